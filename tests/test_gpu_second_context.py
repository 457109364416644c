"""Scenes are not tied to the context that loaded them.

A load, and a change of the node format, ends with everything the device
derives from the scene in place, so a context with a stream of its own can
trace the scene at once. The hits are those of the canonical walk."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu


def agree(ctx, scene, rays):
    a, b = ctx.trace(scene, rays), ctx.trace(scene, rays, count=True)
    for x, y in zip(a[:4], b[:4]):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    return a[3]


@pytest.mark.parametrize("config", [3, 5], ids=["interior", "spheres"])
def test_trace_right_after_a_load_through_another_context(config):
    import aqua

    rays = random_rays(5003, -6.0, 6.0, seed=config)
    rays[:, 1] = np.abs(rays[:, 1]) * 0.5 + 0.1
    with aqua.Context(device=0) as owner, aqua.Context(device=0) as other:
        assert (other.trace(owner.procedural(1, seed=0), rays)[3] >= 0).any()  # its kernels are loaded
        scene = owner.procedural(config, seed=0, width=64, height=36)
        first = agree(other, scene, rays)
        assert (first >= 0).any()
        info = scene.info()
        for fmt in (aqua.BVH_QUANTIZED, aqua.BVH_FULL, aqua.BVH_AUTO):
            scene.set_bvh_format(fmt)
            assert np.array_equal(agree(other, scene, rays), first)
        assert scene.info().device_bytes == info.device_bytes
        scene.free()
