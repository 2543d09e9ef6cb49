"""A wavefront render into a stream under capture is refused before anything is allocated or queued, so that the
capture goes on and its graph holds what the caller put there; a megakernel launch may be captured."""
import ctypes as C

import pytest

from cortexraytracercuda_b200 import _lib, configs
from cortexraytracercuda_b200.renderer import Context, DeviceScene, RtcError
from cortexraytracercuda_b200.scene import ENGINE_MEGAKERNEL, FLAG_SAMPLE_GROUPS, MODE_CLEAN, RenderParams

pytestmark = pytest.mark.gpu


def _capture(refused):
    """Captures an addition before and after `refused(stream)`, then replays the graph twice."""
    import torch
    x = torch.zeros(4, device="cuda")
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        x.add_(1.0)
        refused(s.cuda_stream)
        x.add_(10.0)
    g.replay()
    g.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [22.0] * 4


@pytest.mark.parametrize("first_use", [True, False])
@pytest.mark.parametrize("w,h,kw", [(16, 8, {}), (400, 300, {}), (64, 48, dict(mode=MODE_CLEAN, flags=FLAG_SAMPLE_GROUPS))])
def test_render_device(first_use, w, h, kw):
    import torch
    with Context(0) as c:   # on its first use it has no scratch memory yet
        ds = DeviceScene(c, configs.SCENES["textured"][0]())
        p = RenderParams(width=w, height=h, spp=4, max_depth=5, **kw)
        out = torch.zeros(h, w, 4, device="cuda")
        if not first_use:
            ds.render_device(p, out.data_ptr())

        def refused(stream):
            with pytest.raises(RtcError):
                ds.render_device(p, out.data_ptr(), stream=stream)

        _capture(refused)
        out.zero_()
        ds.render_device(p, out.data_ptr())
        torch.cuda.synchronize()
        assert out[..., :3].sum() > 0
        ds.close()


def test_render_noalloc(ctx):
    import torch
    lib = _lib.load()
    ds = DeviceScene(ctx, configs.SCENES["textured"][0]())
    p = RenderParams(width=64, height=48, spp=4, max_depth=5).to_c()
    out = torch.zeros(48, 64, 4, device="cuda")

    def render(stream):
        return lib.rtc_render_noalloc(ds.handle, C.byref(p), C.c_void_p(out.data_ptr()), stream)

    assert render(None) == 0   # the array's address is looked up outside a capture
    torch.cuda.synchronize()
    want = out.clone()
    out.zero_()

    def refused(stream):
        assert render(C.c_void_p(stream)) == 3   # RTC_ERR_CUDA

    _capture(refused)
    assert out.abs().sum() == 0   # the graph holds nothing of the refused call
    assert render(None) == 0
    torch.cuda.synchronize()
    assert torch.equal(out, want)


def test_megakernel_is_captured(ctx):
    import torch
    ds = DeviceScene(ctx, configs.SCENES["textured"][0]())
    p = RenderParams(width=64, height=48, spp=4, max_depth=5, engine=ENGINE_MEGAKERNEL)
    out = torch.zeros(48, 64, 4, device="cuda")
    ds.render_device(p, out.data_ptr())
    torch.cuda.synchronize()
    want = out.clone()
    out.zero_()
    _capture(lambda stream: ds.render_device(p, out.data_ptr(), stream=stream))
    assert torch.equal(out, want)
