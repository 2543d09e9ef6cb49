"""rtc_get_render_stats gives the number of slots that the drain took over also where the frame was queued without
a poll (fewer units than 512 per SM)."""
import pytest

from cortexraytracercuda_b200 import configs
from cortexraytracercuda_b200.renderer import Context, DeviceScene
from cortexraytracercuda_b200.scene import MODE_CLEAN, Camera, RenderParams, Scene

pytestmark = pytest.mark.gpu


def _misses():
    s = Scene(name="misses")
    s.sphere((0, 0, 50), 0.5, s.lambertian((0.5, 0.5, 0.5)))   # behind the camera
    s.dir_light((0, 0, 60), (1, 0, 0), (0, 1, 0), (1, 1, 1))
    s.set_background_sky()
    s.camera = Camera(look_from=(0, 0, 10), look_at=(0, 0, 0), up=(0, 1, 0), vfov=40.0, aspect=1.0, aperture=0.0, focus=10.0)
    return s


def _stats(c, ds, **kw):
    import torch
    p = RenderParams(mode=MODE_CLEAN, **kw)
    out = torch.empty(p.height, p.width, 4, device="cuda")
    ds.render_device(p, out.data_ptr())
    return c.last_stats()


def test_drained_slots_of_queued_frames():
    with Context(0) as c:
        ds = DeviceScene(c, _misses())
        # one iteration a sample: after the first batch of 8 iterations a pixel of 8 samples is done, one of 9 is not
        assert _stats(c, ds, width=64, height=48, spp=8, max_depth=4)["drained_slots"] == 0
        assert _stats(c, ds, width=64, height=48, spp=9, max_depth=4)["drained_slots"] == 64 * 48
        st = c.last_stats()   # asked again: the same
        assert st["drained_slots"] == 64 * 48 and st["iterations"] == 16
        d2 = DeviceScene(c, configs.textured())
        some = _stats(c, d2, width=101, height=53, spp=4, max_depth=6)["drained_slots"]
        assert 0 < some < 101 * 53
        big = _stats(c, d2, width=640, height=360, spp=4, max_depth=6)["drained_slots"]   # polled
        assert 0 <= big < 640 * 360
        d2.close()
        ds.close()
