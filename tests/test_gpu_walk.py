"""The walk over the compact nodes of large trees against the canonical walk.

aqua_trace without counting walks a large tree through its 64-byte walk
nodes; with AQUA_TRACE_COUNT it walks the full-precision nodes in canonical
order. Closest hits must agree bit for bit and occlusion exactly, on the rays
where conservative boxes could slip: origins on surfaces, axis-aligned and
nearly axis-aligned directions, segments that end or start at a hit,
far-away and unnormalised rays, and directions with a zero or a non-finite
component."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[3, 5], ids=["interior", "spheres"])
def scene(request, gpu_ctx):
    s = gpu_ctx.procedural(request.param, seed=0, width=64, height=36)
    lo, hi = ((-9.9, 0.0, -6.9), (9.9, 4.0, 6.9)) if request.param == 3 else ((-40, 0, -40), (40, 4, 40))
    yield s, np.array(lo, np.float32), np.array(hi, np.float32)
    s.free()


def both(ctx, scene, rays, any_hit):
    a = ctx.trace(scene, rays, any_hit=any_hit)
    b = ctx.trace(scene, rays, any_hit=any_hit, count=True)
    assert np.array_equal(a[3], b[3]), f"{int((a[3] != b[3]).sum())} of {len(rays)} differ"
    for x, y in zip(a[:3], b[:3]):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    return a


def make_rays(kind, lo, hi, n, seed):
    r = np.random.default_rng(seed)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = lo + (hi - lo) * r.random((n, 3))
    d = r.normal(size=(n, 3))
    if kind == "axis":
        d = np.zeros((n, 3))
        d[np.arange(n), r.integers(0, 3, n)] = r.choice([-1.0, 1.0], n)
        rays[:, 0:3] = np.round(rays[:, 0:3])  # on the planes of flat, axis-aligned surfaces
    elif kind == "grazing":
        d[np.arange(n), r.integers(0, 3, n)] *= 10.0 ** r.uniform(-12, -3, n)
    elif kind == "far":
        rays[:, 0:3] = (lo + hi) / 2 - d / np.linalg.norm(d, axis=1, keepdims=True) * 10.0 ** r.uniform(1, 3, (n, 1))
        d += r.normal(size=(n, 3)) * 1e-5
    elif kind == "scaled":
        d *= 10.0 ** r.uniform(-6, 6, (n, 1))
    elif kind == "odd":
        d[r.random((n, 3)) < 0.3] = 0.0
        if hi[0] < 20.0:  # such a ray may walk the whole tree: one of each, on the smaller scene
            d[7, 0], d[11, 1], rays[13, 2] = np.nan, np.inf, np.inf
    rays[:, 4:7] = d
    rays[:, 7] = np.inf
    return rays


@pytest.mark.parametrize("kind", ["random", "axis", "grazing", "far", "scaled", "odd"])
def test_walk_matches_the_canonical_walk(gpu_ctx, scene, kind):
    s, lo, hi = scene
    rays = make_rays(kind, lo, hi, 30_001, seed=len(kind))
    t, u, v, prim = both(gpu_ctx, s, rays, False)[:4]
    both(gpu_ctx, s, rays, True)
    if kind == "odd":
        return
    hit = prim >= 0
    assert hit.any()
    # From the hit points on: origins on surfaces, into every direction, and
    # segments whose ends are the hits themselves.
    o = (rays[hit, 0:3] + t[hit, None] * rays[hit, 4:7]).astype(np.float32)
    again = make_rays("random" if kind == "random" else kind, lo, hi, o.shape[0], seed=7)
    if kind != "far":
        again[:, 0:3] = o
    both(gpu_ctx, s, again, False)
    both(gpu_ctx, s, again, True)
    ends = rays[hit].copy()
    ends[:, 7] = t[hit]
    both(gpu_ctx, s, ends, True)
    ends[:, 7] = np.nextafter(t[hit], np.float32(np.inf))
    both(gpu_ctx, s, ends, False)
    ends[:, 3], ends[:, 7] = t[hit], np.inf
    both(gpu_ctx, s, ends, False)
