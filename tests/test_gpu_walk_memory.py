"""A large scene that leaves no room for its walk nodes loads without them and is
walked through its full-precision nodes, with the same hits."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu


def test_a_scene_without_room_for_walk_nodes_loads(gpu_ctx):
    import aqua

    rays = random_rays(5003, -6.0, 6.0, seed=3)
    rays[:, 1] = np.abs(rays[:, 1]) * 0.5 + 0.1
    # This context's second allocation, the walk nodes, fails; the scene is traced by another.
    with aqua.Context(device=0, fail_alloc_after=2) as small:
        scene = small.procedural(3, seed=0, width=64, height=36)
        info = scene.info()
        assert info.device_bytes == info.upload_bytes
        for any_hit in (False, True):
            a = gpu_ctx.trace(scene, rays, any_hit=any_hit)
            b = gpu_ctx.trace(scene, rays, any_hit=any_hit, count=True)
            for x, y in zip(a[:4], b[:4]):
                assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
        full = gpu_ctx.procedural(3, seed=0, width=64, height=36)
        assert full.info().device_bytes == info.device_bytes + 64 * info.num_bvh_nodes
        assert np.array_equal(gpu_ctx.trace(full, rays)[3], gpu_ctx.trace(scene, rays)[3])
        full.free()
        scene.free()
