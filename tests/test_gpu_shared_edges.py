"""Rays through an edge that two triangles share: which of the two is hit is decided by one rounding (u + v of
the last edge's test, fused with u's product or not), and one pixel in millions shows it.  These pixels hold such
a ray.  Their sums are those of the kernels before their walk was rewritten; they must not move with the code
that the compiler happens to see around the test."""
import numpy as np
import pytest

from cortexraytracercuda_b200 import configs
from cortexraytracercuda_b200.renderer import DeviceScene, Job
from cortexraytracercuda_b200.scene import ENGINE_WAVEFRONT, FLAG_WIDE_BVH, MODE_CLEAN, MODE_COMPAT, RenderParams

pytestmark = pytest.mark.gpu

W, H = 1920, 1080


def _scene(name):
    s = configs.meshes(5, seed=1, env_size=(256, 128))
    s.camera = configs.orbit_camera(s.camera, 0.1, (0, 0.95, 0))
    s.camera.aspect = W / H
    if name == "box":          # triangles beside one transformed box
        s.box((0, 0, 0), (0.2, 0.2, 0.2), s.lambertian((0.7, 0.7, 0.7)),
              transform=configs.placed(s, (-2, 0.2, 2.2), rotate=(0, 20.0, 0)))
    if name == "transformed":  # the meshes themselves transformed
        t = configs.placed(s, (0, 0, 0), rotate=(3, 6, 7), scale=(1.1, 0.9, 1.0))
        for m in s.meshes:
            m["transform"] = t
    return s


@pytest.mark.parametrize("scene,mode,flags,batch,pixels", [
    ("plain", MODE_CLEAN, 0, False, {(556, 777): (0x42a3e9e8, 0x42af2988, 0x42bde965)}),
    ("plain", MODE_CLEAN, FLAG_WIDE_BVH, False, {(556, 777): (0x42206d0d, 0x423e7f3a, 0x426b81da),
                                                 (618, 1011): (0x420d276a, 0x41858453, 0x4148093f)}),
    ("box", MODE_CLEAN, 0, False, {(556, 777): (0x42a3e9e8, 0x42af2988, 0x42bde965),
                                   (618, 1011): (0x420d691a, 0x4185a1e1, 0x41482abe)}),
    ("box", MODE_COMPAT, 0, True, {(430, 485): (0x4213826f, 0x423a2b54, 0x42703013)}),
    ("box", MODE_COMPAT, FLAG_WIDE_BVH, False, {(430, 485): (0x4213968b, 0x423a3826, 0x42703013)}),
    ("transformed", MODE_CLEAN, 0, False, {(437, 1153): (0x41becf25, 0x41467d68, 0x411b2a2e),
                                           (582, 1204): (0x41d5c7fe, 0x41614cc5, 0x4130b0a3)}),
])
def test_shared_edge_pixels(ctx, scene, mode, flags, batch, pixels):
    import torch
    ds = DeviceScene(ctx, _scene(scene))
    p = RenderParams(width=W, height=H, spp=64, max_depth=6, mode=mode, flags=flags, seed=82, engine=ENGINE_WAVEFRONT)
    out = torch.empty(H, W, 4, device="cuda")
    if batch:
        ctx.render_batch([Job(ds, p, out.data_ptr(), None)])
    else:
        ds.render_device(p, out.data_ptr())
    torch.cuda.synchronize()
    words = out.cpu().numpy().view(np.uint32)
    for at, want in pixels.items():
        assert tuple(int(w) for w in words[at][:3]) == want
