"""A batch job's image depends on the job alone: the same bits by itself, with
jobs that make the batch keep its pixels whole, in a graph or not, and at any launch shape."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (config, width, height, spp, depth, seed): odd sizes, one sample, runs of several
# samples.
JOBS = [(2, 61, 43, 11, 8, 1), (1, 16, 9, 1, 5, 2), (2, 8, 5, 333, 8, 3), (1, 40, 30, 64, 4, 4),
        (1, 300, 200, 37, 3, 5)]
# about 9, 31, 126 and 503 million paths beside them: more than 1, 4, 17 and 68
# samples are split
COMPANY = [(1, 320, 240, 120, 2, 9), (1, 640, 480, 100, 2, 9), (1, 1024, 1024, 120, 2, 9), (1, 2048, 2048, 120, 1, 9)]


def test_a_job_has_the_same_bits_in_any_company(gpu_ctx):
    torch = pytest.importorskip("torch")
    scenes = {c: gpu_ctx.procedural(c, seed=0) for c in (1, 2)}

    def render(specs, **kw):
        films = [torch.full((h, w, 3), -1.0, device="cuda") for (_, w, h, _, _, _) in specs]
        torch.cuda.synchronize()
        jobs = [(scenes[c], w, h, spp, depth, seed, f.data_ptr())
                for (c, w, h, spp, depth, seed), f in zip(specs, films)]
        st, _ = gpu_ctx.render_batch(jobs, gpu_ctx.tuning(**kw) if kw else None)
        assert st.paths == sum(w * h * spp for (_, w, h, spp, _, _) in specs)
        return [f.cpu().numpy() for f in films]

    alone = [render([j])[0] for j in JOBS]
    for kw in ({}, dict(use_graph=0, block_trace=256), dict(use_graph=1, block_trace=64, blocks_per_sm=1)):
        for a, b in zip(alone, render(JOBS, **kw)):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for other in COMPANY:
        for a, b in zip(alone, render(JOBS + [other])):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    # Jobs that share a film (the same view twice) leave the view's image in it.
    film = torch.full((200, 300, 3), -1.0, device="cuda")
    rest = torch.zeros((2048, 2048, 3), device="cuda")
    torch.cuda.synchronize()
    twice = [(scenes[c], w, h, spp, depth, seed, film.data_ptr()) for (c, w, h, spp, depth, seed) in [JOBS[-1]] * 2]
    for company in ([], [(scenes[1], 2048, 2048, 120, 1, 9, rest.data_ptr())]):
        film.fill_(-1.0)
        torch.cuda.synchronize()
        gpu_ctx.render_batch(twice + company)
        assert np.array_equal(film.cpu().numpy().view(np.uint32), alone[-1].view(np.uint32))
    for (c, w, h, spp, depth, seed), img in zip(JOBS, alone):
        s = scenes[c]
        s.set_resolution(w, h)
        cfg = gpu_ctx.integrator(spp=spp, max_depth=depth, rr_depth=3, seed=seed)
        ref, _ = gpu_ctx.render(s, cfg)
        np.testing.assert_allclose(img, ref, rtol=1e-5, atol=1e-6)
    for s in scenes.values():
        s.free()
