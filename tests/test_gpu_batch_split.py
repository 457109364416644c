"""Batches whose pixels are split into runs of samples.

The runs' sums are added in order by the lane that finishes the pixel's last
run, so a job's image is the single render's up to FP32 summation order, the
same bits on every launch shape, replay and order of completion; a job with
fewer samples than a run keeps whole pixels."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (config, width, height, spp, depth, seed): about 16M paths, so runs of two
# samples: even and odd sample counts, one run, a pixel, a last run of one.
MIXED = [(1, 512, 512, 60, 4, 1), (2, 33, 29, 7, 8, 2), (2, 16, 16, 2, 8, 3), (1, 8, 8, 1, 3, 4), (2, 1, 1, 9, 8, 5)]
# few paths: every sample is a run of its own
SMALL = [(1, 40, 30, 5, 5, 1), (2, 17, 13, 33, 8, 2), (2, 5, 3, 1, 8, 3)]


@pytest.mark.parametrize("specs", [MIXED, SMALL], ids=["runs", "samples"])
def test_split_batches_match_single_renders(gpu_ctx, specs):
    torch = pytest.importorskip("torch")
    scenes = {c: gpu_ctx.procedural(c, seed=0) for c in {s[0] for s in specs}}
    films = [torch.full((h, w, 3), -1.0, device="cuda") for (_, w, h, _, _, _) in specs]
    jobs = [(scenes[c], w, h, spp, depth, seed, f.data_ptr())
            for (c, w, h, spp, depth, seed), f in zip(specs, films)]
    torch.cuda.synchronize()
    first = None
    for kw in ({}, dict(use_graph=1), dict(use_graph=1), dict(use_graph=0, block_trace=64, blocks_per_sm=2),
               dict(use_graph=1, block_trace=256)):
        st, job_ms = gpu_ctx.render_batch(jobs, gpu_ctx.tuning(**kw) if kw else None)
        assert st.paths == sum(w * h * spp for (_, w, h, spp, _, _) in specs)
        assert np.all(job_ms > 0) and np.all(job_ms <= st.device_ms * 1.05 + 0.05)
        got = [f.cpu().numpy().copy() for f in films]
        if first is not None:
            assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(first, got))
        first = got
        for f in films:
            f.fill_(-1.0)
        torch.cuda.synchronize()
    for (c, w, h, spp, depth, seed), img in zip(specs, first):
        s = scenes[c]
        info = s.info()
        s.set_resolution(w, h)
        ref, _ = gpu_ctx.render(s, gpu_ctx.integrator(spp=spp, max_depth=depth, rr_depth=3, seed=seed),
                                tuning=gpu_ctx.tuning(replicas=1))
        s.set_resolution(info.width, info.height)
        np.testing.assert_allclose(img, ref, rtol=1e-5, atol=1e-6)
    for s in scenes.values():
        s.free()
