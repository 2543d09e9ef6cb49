"""The drain kernels finish exactly the slots they are given, whatever their number: the wavefront engine
against the megakernel, g++ flavour (no FMA contraction: the sums are identical), at sizes around a warp, a
block of the compacting drain and the number of drain threads (75,776), with chains of one bounce to many.
Scenes without transforms run the drain of one-warp blocks, scenes with them the compacting drain."""
import numpy as np
import pytest

from cortexraytracercuda_b200 import configs
from cortexraytracercuda_b200.renderer import DeviceScene, RtcError
from cortexraytracercuda_b200.scene import (DRAW_ORDER_DEVICE, DRAW_ORDER_HOST, ENGINE_MEGAKERNEL, ENGINE_WAVEFRONT,
                                            FLAG_SAMPLE_GROUPS, MODE_CLEAN, MODE_COMPAT, RenderParams)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["textured", "xforms"])
@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 9, 50), (31, 1, 4, 20), (33, 1, 4, 20), (257, 1, 9, 12), (64, 37, 16, 1),
                                           (275, 276, 9, 10)])
def test_drain_equals_megakernel(ctx, name, w, h, spp, depth):
    ds = DeviceScene(ctx, configs.SCENES[name][0]())
    p = RenderParams(width=w, height=h, spp=spp, max_depth=depth, draw_order=DRAW_ORDER_HOST, engine=ENGINE_MEGAKERNEL)
    a, rgb_a = ds.render(p, want_rgb8=True)
    p.engine = ENGINE_WAVEFRONT
    b, rgb_b = ds.render(p, want_rgb8=True)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert np.array_equal(rgb_a, rgb_b)


@pytest.mark.parametrize("name", ["textured", "xforms"])
def test_drain_sample_groups_repeatable(ctx, name):
    """Sample groups through the drains: every group finishes once and is added in group order."""
    ds = DeviceScene(ctx, configs.SCENES[name][0]())
    p = RenderParams(width=97, height=41, spp=13, max_depth=9, mode=MODE_CLEAN, flags=FLAG_SAMPLE_GROUPS)
    a, _ = ds.render(p)
    b, _ = ds.render(p)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)) and np.isfinite(a).all()


@pytest.mark.parametrize("name,mode,order,flags", [
    ("spheres", MODE_COMPAT, DRAW_ORDER_DEVICE, 0), ("lights", MODE_COMPAT, DRAW_ORDER_HOST, 0),
    ("uvmesh", MODE_COMPAT, DRAW_ORDER_DEVICE, 0), ("xforms", MODE_COMPAT, DRAW_ORDER_DEVICE, 0),
    ("spheres", MODE_CLEAN, DRAW_ORDER_DEVICE, 0), ("xforms", MODE_CLEAN, DRAW_ORDER_DEVICE, FLAG_SAMPLE_GROUPS)])
@pytest.mark.parametrize("w,h", [(1, 1), (33, 7), (275, 276), (641, 479)])
def test_bounces_kernel_equals_split_kernels(ctx, monkeypatch, name, mode, order, flags, w, h):
    """The several-iterations kernel (frames and queues of up to 2,048 slots per SM) against the extend and
    shade kernels, every flavour: the same bits.  Sizes from one pixel over the drain threshold (75,776) to
    a frame that starts in the split kernels and goes over."""
    ds = DeviceScene(ctx, configs.SCENES[name][0]())
    p = RenderParams(width=w, height=h, spp=9, max_depth=12, mode=mode, draw_order=order, flags=flags)
    a, rgb_a = ds.render(p, want_rgb8=True)
    monkeypatch.setenv("RTC_WF_BOUNCES", "0")
    b, rgb_b = ds.render(p, want_rgb8=True)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert np.array_equal(rgb_a, rgb_b)


def test_capture_is_refused(ctx):
    """A render into a stream under capture is refused, small frames (which never poll) included."""
    import torch
    ds = DeviceScene(ctx, configs.SCENES["textured"][0]())
    p = RenderParams(width=16, height=8, spp=4, max_depth=5)
    out = torch.zeros(8, 16, 4, device="cuda")
    ds.render_device(p, out.data_ptr())
    torch.cuda.synchronize()
    want = out.clone()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with pytest.raises(RtcError):
        with torch.cuda.graph(g, stream=s):
            ds.render_device(p, out.data_ptr(), stream=s.cuda_stream)
    out.zero_()
    ds.render_device(p, out.data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(out, want)
