"""Closest hits through leaf ranges: the hit leaves of one node are tested as one range of items, found by
their first item's word where the range is consecutive words of one kind and through the item list
otherwise, and transformed primitives reuse the object-space ray of the transform before.

Scenes of 1 to 67 primitives of every kind (single leaves, one node, mixed and uniform leaves, siblings of
different kinds; transforms in runs, interleaved and absent; boxes), against the C restatement's search:
primitive ids and distances are identical, since every test is the same arithmetic (no FMA contraction) and
the primitives are in general position (no two at one distance)."""
import numpy as np
import pytest

from cortexraytracercuda_b200.renderer import DeviceScene
from cortexraytracercuda_b200.scene import BVH_DEVICE, BVH_DEVICE_LBVH, BVH_SAH, FLAG_WIDE_BVH, Scene

import oracles

pytestmark = pytest.mark.gpu


def _scene(kinds, n, seed, transforms=0):
    rng = np.random.default_rng([seed, n])
    s = Scene(name="ranges")
    m = s.lambertian((0.5, 0.5, 0.5))
    refs = [s.transform(translate=tuple(rng.uniform(-1, 1, 3)), rotate=(0.0, float(rng.uniform(-40, 40)), 0.0),
                        scale=tuple(rng.uniform(0.6, 1.4, 3))) for _ in range(transforms)]
    tri = []
    for k in range(n):
        kind = kinds[k % len(kinds)]
        at = rng.uniform(-3, 3, 3)
        ref = int(refs[rng.integers(len(refs))]) if refs and rng.random() < 0.8 else 0
        if kind == "sphere":
            s.sphere(tuple(at), float(rng.uniform(0.2, 0.9)), m, transform=ref)
        elif kind == "quad":
            s.quad(tuple(at), tuple(rng.uniform(-1, 1, 3)), tuple(rng.uniform(-1, 1, 3)), m, transform=ref)
        elif kind == "light":
            s.dir_light(tuple(at), tuple(rng.uniform(-1, 1, 3)), tuple(rng.uniform(-1, 1, 3)), (1, 1, 1), invisible=bool(k & 1))
        elif kind == "box":
            s.box(tuple(at), tuple(rng.uniform(0.3, 1.0, 3)), m, transform=ref)
        elif transforms:
            s.mesh(at + rng.uniform(-1, 1, (6, 3)), [[0, 1, 2], [3, 4, 5]], m, transform=ref)
        else:
            tri.append(at + rng.uniform(-1, 1, (3, 3)))
    if tri:
        s.mesh(np.concatenate(tri), np.arange(3 * len(tri)).reshape(-1, 3), m)
    return s


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-6, 6, (n, 3))
    d = rng.uniform(-3, 3, (n, 3)) - o
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3], r[:, 3], r[:, 4:7], r[:, 7] = o, 1e-4, d, 3e38
    return r


def _check(ds, want, rays, flags=0):
    for (depth, max_depth), (prim, t) in want.items():
        p, tt = ds.trace_closest(rays, depth, max_depth, flags=flags)
        assert np.array_equal(p, prim)
        assert np.array_equal(tt[prim >= 0], t[prim >= 0])


@pytest.mark.parametrize("kinds", [("sphere",), ("tri",), ("quad",), ("light",), ("sphere", "tri"),
                                   ("quad", "sphere", "light", "tri")])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 17, 67])
def test_leaf_ranges(ctx, kinds, n):
    scene = _scene(kinds, n, 31)
    rays = _rays(4000, n)
    o = oracles.port().scene(scene)
    want = {dm: o.trace_closest(rays, *dm) for dm in ((1, 1), (0, 8))}
    for builder in (BVH_SAH, BVH_DEVICE, BVH_DEVICE_LBVH):
        _check(DeviceScene(ctx, scene, builder), want, rays)
    _check(DeviceScene(ctx, scene), want, rays, FLAG_WIDE_BVH)


@pytest.mark.parametrize("transforms", [1, 3])
@pytest.mark.parametrize("n", [1, 2, 9, 41])
def test_transformed_runs(ctx, n, transforms):
    scene = _scene(("box", "sphere", "tri", "quad"), n, 7, transforms)
    rays = _rays(4000, n)
    o = oracles.port().scene(scene)
    want = {dm: o.trace_closest(rays, *dm) for dm in ((1, 1), (0, 8))}
    ds = DeviceScene(ctx, scene)
    _check(ds, want, rays)
    _check(ds, want, rays, FLAG_WIDE_BVH)


def test_trace_block_sizes(ctx):
    """Ray queries of growing and shrinking size share the context's kept block; the last is past what is
    kept (1,677,721 rays) and uses its own.  Every call gives each ray the hit that it has in a call alone."""
    scene = _scene(("sphere", "tri", "quad"), 40, 5)
    ds = DeviceScene(ctx, scene)
    rays = _rays(1000, 3)
    prim, t = ds.trace_closest(rays, 0, 8)
    oracle_prim, oracle_t = oracles.port().scene(scene).trace_closest(rays, 0, 8)
    assert np.array_equal(prim, oracle_prim) and np.array_equal(t[prim >= 0], oracle_t[prim >= 0])
    for n in (1, 33, 5000, 127, 200_003, 1_677_722, 64):
        reps = -(-n // 1000)
        p, tt = ds.trace_closest(np.tile(rays, (reps, 1))[:n], 0, 8)
        assert np.array_equal(p, np.tile(prim, reps)[:n]) and np.array_equal(tt, np.tile(t, reps)[:n])
