"""Scenes of 2^20 primitives or more, whose extend kernel (and, in clean mode, whose shade kernel) takes queue
chunks from a counter: a plain scene renders to the same bits as the same scene with an image that nothing uses,
and in the g++ flavour (no FMA contraction) every engine gives the same sums."""
import numpy as np
import pytest

from cortexraytracercuda_b200 import configs
from cortexraytracercuda_b200.renderer import DeviceScene
from cortexraytracercuda_b200.scene import (DRAW_ORDER_DEVICE, DRAW_ORDER_HOST, ENGINE_MEGAKERNEL, ENGINE_WAVEFRONT,
                                            FLAG_SAMPLE_GROUPS, FLAG_WIDE_BVH, MODE_CLEAN, MODE_COMPAT, RenderParams)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scenes(ctx):
    s = configs.icosphere_scene(7)   # 983,042 primitives and 80 K more: over 2^20, no image, no environment map
    v, f = configs.displaced_icosphere(6, 0.1)
    s.mesh(0.3 * v + np.array([0.0, 3.0, 0.0]), f, s.dielectric(1.5))
    plain = DeviceScene(ctx, s)
    assert s.num_primitives >= 1 << 20
    s.images.append(np.zeros((1, 1, 3), np.uint8))
    return plain, DeviceScene(ctx, s)


@pytest.mark.parametrize("mode,order,flags", [
    (MODE_COMPAT, DRAW_ORDER_DEVICE, 0), (MODE_COMPAT, DRAW_ORDER_HOST, 0), (MODE_COMPAT, DRAW_ORDER_DEVICE, FLAG_WIDE_BVH),
    (MODE_CLEAN, DRAW_ORDER_DEVICE, 0), (MODE_CLEAN, DRAW_ORDER_DEVICE, FLAG_SAMPLE_GROUPS),
    (MODE_CLEAN, DRAW_ORDER_DEVICE, FLAG_WIDE_BVH)])
@pytest.mark.parametrize("w,h", [(257, 131), (1280, 720)])
def test_plain_equals_full_above_2_20(scenes, mode, order, flags, w, h):
    p = RenderParams(width=w, height=h, spp=9, max_depth=12, mode=mode, draw_order=order, flags=flags,
                     engine=ENGINE_WAVEFRONT)
    (a, rgb_a), (b, rgb_b) = (s.render(p, want_rgb8=True) for s in scenes)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert np.array_equal(rgb_a, rgb_b)
    if order == DRAW_ORDER_HOST:
        p.engine = ENGINE_MEGAKERNEL
        c, _ = scenes[0].render(p)
        assert np.array_equal(a.view(np.uint32), c.view(np.uint32))
