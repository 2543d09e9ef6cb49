"""Renders of one context on several streams and threads: they share the context's scratch memory, so each waits
on the device for the one before, and every image is the one that the frame gives alone.  Small frames are queued
without a poll, so nothing on the host keeps them apart."""
import threading

import numpy as np
import pytest

from cortexraytracercuda_b200 import configs
from cortexraytracercuda_b200.renderer import DeviceScene
from cortexraytracercuda_b200.scene import DRAW_ORDER_HOST, FLAG_SAMPLE_GROUPS, MODE_CLEAN, RenderParams

pytestmark = pytest.mark.gpu

FRAMES = [  # (scene, params): queued whole; with sample groups; polled
    ("textured", dict(width=64, height=48, spp=4, max_depth=10, draw_order=DRAW_ORDER_HOST)),
    ("cornell", dict(width=200, height=150, spp=16, max_depth=12, draw_order=DRAW_ORDER_HOST)),
    ("xforms", dict(width=97, height=61, spp=9, max_depth=8, mode=MODE_CLEAN, flags=FLAG_SAMPLE_GROUPS)),
    ("spheres", dict(width=640, height=360, spp=4, max_depth=20, draw_order=DRAW_ORDER_HOST)),
]


@pytest.fixture(scope="module")
def frames(ctx):
    import torch
    out = []
    for name, kw in FRAMES:
        ds, p = DeviceScene(ctx, configs.SCENES[name][0]()), RenderParams(**kw)
        want = torch.empty(p.height, p.width, 4, device="cuda")
        ds.render_device(p, want.data_ptr())
        torch.cuda.synchronize()
        out.append((ds, p, want))
    return out


def _same(got, want):
    return np.array_equal(got.cpu().numpy().view(np.uint32), want.cpu().numpy().view(np.uint32))


@pytest.mark.parametrize("streams", [2, 3])
def test_alternating_streams(frames, streams):
    import torch
    st = [torch.cuda.Stream() for _ in range(streams)]
    got = []
    for k in range(24):
        ds, p, want = frames[(k * 5) % len(frames)]
        out = torch.zeros_like(want)
        torch.cuda.current_stream().synchronize()
        ds.render_device(p, out.data_ptr(), stream=st[k % streams].cuda_stream)
        got.append((out, want))
    torch.cuda.synchronize()
    assert all(_same(o, w) for o, w in got)


def test_host_render_and_rays_behind_a_queued_frame(frames):
    """rtc_render and ray queries run on the context's own stream, right behind a frame on another one."""
    import torch
    s = torch.cuda.Stream()
    rays = np.array([[0, 1, 4, 1e-4, 0.02 * k, -0.1, -1, 1e30] for k in range(-40, 40)], np.float32)
    prim, t = frames[0][0].trace_closest(rays, 0, 8)
    for k in range(12):
        ds, p, want = frames[k % len(frames)]
        out = torch.zeros_like(want)
        torch.cuda.current_stream().synchronize()
        ds.render_device(p, out.data_ptr(), stream=s.cuda_stream)
        if k % 2:
            a, b = frames[0][0].trace_closest(rays, 0, 8)
            assert np.array_equal(a, prim) and np.array_equal(b, t)
        else:
            ds2, p2, want2 = frames[(k + 1) % len(frames)]
            rad, _ = ds2.render(p2)
            assert np.array_equal(rad.view(np.uint32), want2.cpu().numpy().reshape(rad.shape).view(np.uint32))
        torch.cuda.synchronize()
        assert _same(out, want)


def test_threads_with_their_own_streams(frames):
    import torch
    results = []

    def work(first):
        s = torch.cuda.Stream()
        for k in range(first, first + 8):
            ds, p, want = frames[k % len(frames)]
            out = torch.zeros_like(want)
            torch.cuda.current_stream().synchronize()
            ds.render_device(p, out.data_ptr(), stream=s.cuda_stream)
            s.synchronize()
            results.append(_same(out, want))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert len(results) == 32 and all(results)
