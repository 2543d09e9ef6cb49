"""Clean mode's instrumented frames (device counters): the dielectric's dot product has its rounding written out.
These pixels see glass; their sums are those of the kernels before the path state was rearranged.  (The
uninstrumented kernels round it their own way: the images agree to the last bits, not in them.)"""
import numpy as np
import pytest

from cortexraytracercuda_b200 import configs
from cortexraytracercuda_b200.renderer import DeviceScene
from cortexraytracercuda_b200.scene import ENGINE_WAVEFRONT, MODE_CLEAN, RenderParams

pytestmark = pytest.mark.gpu

W, H = 1920, 1080
PIXELS = {(0, 349): (0x41380eb3, 0x41a009a0, 0x4100af9b), (405, 666): (0x411159b8, 0x41646791, 0x40ed350a),
          (510, 895): (0x40eff4d9, 0x40b7e9ee, 0x408eed3d), (552, 853): (0x4225d21c, 0x423de4a7, 0x426aa4c7),
          (656, 698): (0x42312fc5, 0x4246c311, 0x42669d27), (740, 757): (0x419e30f1, 0x41c37c88, 0x41ecc999)}


def test_counted_glass_pixels(ctx):
    import torch
    s = configs.meshes(5, seed=1, env_size=(256, 128))
    s.camera = configs.orbit_camera(s.camera, 0.1, (0, 0.95, 0))
    s.camera.aspect = W / H
    ds = DeviceScene(ctx, s)
    p = RenderParams(width=W, height=H, spp=64, max_depth=6, mode=MODE_CLEAN, seed=82, engine=ENGINE_WAVEFRONT)
    out = torch.empty(H, W, 4, device="cuda")
    cnt = torch.zeros(8, dtype=torch.int64, device="cuda")
    ds.render_device(p, out.data_ptr(), None, cnt.data_ptr())
    torch.cuda.synchronize()
    assert int(cnt[1]) == W * H * 64
    words = out.cpu().numpy().view(np.uint32)
    for at, want in PIXELS.items():
        assert tuple(int(w) for w in words[at][:3]) == want


def test_counted_glass_decision_pixel(ctx):
    """A refraction whose choice against reflection hangs on the incidence cosine's last bit."""
    import torch
    s = configs.SCENES["xforms"][0]()
    s.camera.aspect = W / H
    ds = DeviceScene(ctx, s)
    p = RenderParams(width=W, height=H, spp=64, max_depth=10, mode=MODE_CLEAN, seed=82, engine=ENGINE_WAVEFRONT)
    out = torch.empty(H, W, 4, device="cuda")
    cnt = torch.zeros(8, dtype=torch.int64, device="cuda")
    ds.render_device(p, out.data_ptr(), None, cnt.data_ptr())
    torch.cuda.synchronize()
    words = out.cpu().numpy().view(np.uint32)
    assert tuple(int(w) for w in words[569, 1336][:3]) == (0x41691b6c, 0x3f84cf46, 0x3f816c83)
