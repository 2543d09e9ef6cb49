"""Which scenes take the kernels built without the code that plain scenes never reach: the flag, and that each
feature which clears it, alone in a scene, is rendered - against the megakernel, which has the full code, in the
g++ flavour (no FMA contraction: identical sums)."""
import ctypes as C

import numpy as np
import pytest

from cortexraytracercuda_b200 import configs
from cortexraytracercuda_b200.renderer import DeviceScene
from cortexraytracercuda_b200.scene import DRAW_ORDER_HOST, ENGINE_MEGAKERNEL, ENGINE_WAVEFRONT, Camera, RenderParams, Scene

pytestmark = pytest.mark.gpu


def _plain(ds):
    fn = ds.ctx.lib.rtc_scene_plain
    fn.restype, fn.argtypes = C.c_int, [C.c_void_p]
    return fn(ds.handle)


def _scene(feature, transformed):
    s = Scene(name=feature)
    m = s.lambertian((0.7, 0.5, 0.3))
    t = configs.placed(s, (0.2, 0.1, 0.0), rotate=(0, 20, 0)) if transformed else 0
    s.sphere((0, 0, 0), 1.0, m, transform=t)
    v, f = configs.icosphere(1)
    s.mesh(0.8 * v + np.array([2.0, 0, 0]), f, m, normals=v if feature == "smooth" else None, smooth=feature == "smooth",
           uvs=configs.sphere_uvs(v) if feature == "uvs" else None)
    s.quad((-5, -1, -5), (10, 0, 0), (0, 0, 10), s.lambertian(s.checker_colors(1.0, (0.2, 0.3, 0.1), (0.9, 0.9, 0.9))))
    s.dir_light((0, 5, 0), (2, 0, 0), (0, 0, 2), (4, 4, 4))
    s.set_background_sky()
    if feature == "image":
        s.sphere((-2, 0, 0), 1.0, s.lambertian(s.image(configs.procedural_image(16, 8))))
    if feature == "omni":
        s.omni_light((1, 3, 1), 0.4, (5, 5, 5), invisible=False)
    if feature == "spot":
        s.spot_light((1, 3, 1), (-0.2, -1, -0.2), 40.0, 2.0, (5, 5, 5), radius=0.3)
    if feature == "env":
        s.set_background_env(configs.sky_sun_envmap(32, 16))
    s.camera = Camera(look_from=(0, 2, 8), look_at=(0, 0, 0), up=(0, 1, 0), vfov=45.0, aspect=1.5, aperture=0.0, focus=8.0)
    return s


@pytest.mark.parametrize("transformed", [False, True])
@pytest.mark.parametrize("feature,plain", [("none", 1), ("image", 0), ("smooth", 0), ("uvs", 0), ("omni", 0), ("spot", 0),
                                           ("env", 0)])
def test_one_feature(ctx, feature, plain, transformed):
    ds = DeviceScene(ctx, _scene(feature, transformed))
    assert _plain(ds) == plain
    p = RenderParams(width=96, height=64, spp=9, max_depth=6, draw_order=DRAW_ORDER_HOST, engine=ENGINE_MEGAKERNEL)
    a, rgb_a = ds.render(p, want_rgb8=True)
    p.engine = ENGINE_WAVEFRONT
    b, rgb_b = ds.render(p, want_rgb8=True)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)) and np.array_equal(rgb_a, rgb_b)


@pytest.mark.parametrize("name", ["cornell", "spheres", "icosphere", "xforms"])
def test_scenes_compared_with_the_full_kernels_are_plain(ctx, name):
    """test_gpu_plain.py renders these with and without an image that nothing uses."""
    s = configs.SCENES[name][0]()
    assert _plain(DeviceScene(ctx, s)) == 1
    s.images.append(np.zeros((1, 1, 3), np.uint8))
    assert _plain(DeviceScene(ctx, s)) == 0
