"""A scene whose device image could not be rebuilt is refused by every call that
would read it, and works again once a rebuild succeeds."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu


def test_a_scene_without_an_image_is_refused(gpu_ctx):
    torch = pytest.importorskip("torch")
    import aqua

    rays = random_rays(100, -0.5, 0.5, seed=1)
    film = torch.zeros((8, 8, 3), device="cuda")
    torch.cuda.synchronize()
    # This context's second allocation, the rebuilt image, fails; another one makes the calls.
    with aqua.Context(device=0, fail_alloc_after=2) as small:
        scene = small.procedural(2, seed=0, width=8, height=8)
        before = gpu_ctx.trace(scene, rays)
        with pytest.raises(aqua.AquaError) as e:
            scene.set_bvh_format(aqua.BVH_QUANTIZED)
        assert e.value.status == aqua.ERR_OOM
        cfg = gpu_ctx.integrator(spp=1)
        nrc = aqua.Nrc(gpu_ctx)
        ncfg = gpu_ctx.integrator(type=aqua.INTEGRATOR_NRC, spp=1)
        calls = [
            lambda: gpu_ctx.trace(scene, rays),
            lambda: gpu_ctx.render(scene, cfg),
            lambda: gpu_ctx.render(scene, cfg, tuning=gpu_ctx.tuning(kernel=aqua.KERNEL_PERSISTENT)),
            lambda: gpu_ctx.autotune(scene, cfg),
            lambda: gpu_ctx.render_batch([(scene, 8, 8, 1, 3, 0, film.data_ptr())]),
            lambda: gpu_ctx.render_nrc(scene, ncfg, nrc, dev_ptr=film.data_ptr()),
            lambda: gpu_ctx._check(gpu_ctx.lib.aqua_render_noalloc(gpu_ctx.handle, scene.handle, ctypes.byref(cfg),
                                                                   ctypes.c_void_p(film.data_ptr()), None)),
        ]
        for call in calls:
            with pytest.raises(aqua.AquaError) as e:
                call()
            assert e.value.status == aqua.ERR_INVALID_ARG and "no device image" in e.value.message
        # A rebuild through a context with memory.
        gpu_ctx._check(gpu_ctx.lib.aqua_scene_set_bvh_format(gpu_ctx.handle, scene.handle, aqua.BVH_AUTO))
        for x, y in zip(before[:4], gpu_ctx.trace(scene, rays)[:4]):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
        nrc.free()
        scene.free()
