"""The compacting drain, which RTC_WF_DRAIN_EVERY turns on (read once per process, so a process of its own),
finishes exactly the slots it is given: against the megakernel, g++ flavour, at sizes around a warp, its
256-thread block and the number of drain threads (75,776)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import numpy as np
from cortexraytracercuda_b200 import configs
from cortexraytracercuda_b200.renderer import Context, DeviceScene
from cortexraytracercuda_b200.scene import DRAW_ORDER_HOST, ENGINE_MEGAKERNEL, ENGINE_WAVEFRONT, RenderParams
ctx = Context(0)
for name in ("textured", "xforms"):
    ds = DeviceScene(ctx, configs.SCENES[name][0]())
    for w, h, spp, depth in ((1, 1, 9, 50), (33, 1, 4, 20), (257, 1, 9, 12), (64, 37, 16, 1), (275, 276, 9, 10)):
        p = RenderParams(width=w, height=h, spp=spp, max_depth=depth, draw_order=DRAW_ORDER_HOST, engine=ENGINE_MEGAKERNEL)
        a, _ = ds.render(p)
        p.engine = ENGINE_WAVEFRONT
        b, _ = ds.render(p)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (name, w, h)
print("ok")
"""


@pytest.mark.parametrize("every", ["1", "2"])
def test_packed_drain_equals_megakernel(every):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, env=dict(os.environ, RTC_WF_DRAIN_EVERY=every),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
