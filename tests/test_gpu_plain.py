"""The one-image kernels built without the code that plain scenes never reach (image textures, environment map,
smooth normals, omni and spot lights) against the full ones: the same bits.  A scene with an image that nothing
uses takes the full kernels and is otherwise the same scene."""
import numpy as np
import pytest

from cortexraytracercuda_b200 import configs
from cortexraytracercuda_b200.renderer import DeviceScene
from cortexraytracercuda_b200.scene import (DRAW_ORDER_DEVICE, DRAW_ORDER_HOST, FLAG_SAMPLE_GROUPS, FLAG_WIDE_BVH,
                                            MODE_CLEAN, MODE_COMPAT, RenderParams)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["cornell", "spheres", "icosphere", "xforms"])
@pytest.mark.parametrize("mode,order,flags", [
    (MODE_COMPAT, DRAW_ORDER_DEVICE, 0), (MODE_COMPAT, DRAW_ORDER_HOST, 0), (MODE_COMPAT, DRAW_ORDER_DEVICE, FLAG_WIDE_BVH),
    (MODE_CLEAN, DRAW_ORDER_DEVICE, 0), (MODE_CLEAN, DRAW_ORDER_DEVICE, FLAG_SAMPLE_GROUPS)])
@pytest.mark.parametrize("w,h", [(1, 1), (275, 276), (641, 479)])
def test_plain_kernels_equal_full_kernels(ctx, name, mode, order, flags, w, h):
    s = configs.SCENES[name][0]()
    p = RenderParams(width=w, height=h, spp=9, max_depth=12, mode=mode, draw_order=order, flags=flags)
    a, rgb_a = DeviceScene(ctx, s).render(p, want_rgb8=True)
    s.images.append(np.zeros((1, 1, 3), np.uint8))
    b, rgb_b = DeviceScene(ctx, s).render(p, want_rgb8=True)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert np.array_equal(rgb_a, rgb_b)
