"""How many wavefront iterations a render launches.

A slot runs its work items one after another, each at most max_depth + 1
iterations long, so that product bounds the launches; below it the queue's
length ends the render. Every path must be complete whatever the bound, the
chunking and the split of the samples over slots, and the image must not
depend on the chunking."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp,depth,shape", [
    (1, 1, 1, 0, {}),                      # one ray
    (33, 17, 3, 0, {}),                    # camera rays only
    (64, 64, 4, 5, {}),                    # a sample per slot: exactly depth + 1 iterations
    (40, 30, 7, 6, dict(replicas=3)),      # samples that do not divide over the replicas
    (40, 30, 7, 6, dict(replicas=1)),
    (41, 29, 5, 8, dict(slots=37)),        # several pixels per slot, ragged
    (40, 30, 9, 4, dict(sort_by_material=1)),
    (24, 20, 64, 8, dict(replicas=2)),     # long enough for the shrinking chunks
])
def test_every_path_ends_and_chunking_does_not_matter(gpu_ctx, w, h, spp, depth, shape):
    s = gpu_ctx.procedural(2, seed=3, width=w, height=h)
    cfg = gpu_ctx.integrator(spp=spp, max_depth=depth, rr_depth=3, seed=11)
    images = []
    for chunk in (0, 1, 3, 64):
        img, st = gpu_ctx.render(s, cfg, tuning=gpu_ctx.tuning(iters_per_graph=chunk, **shape))
        assert st.paths == w * h * spp
        slots = shape.get("slots", w * h)
        if "slots" in shape or shape.get("replicas") == 1:
            items = -(-(w * h) // slots) * spp
        else:
            items = -(-spp // shape.get("replicas", spp))
        assert 1 <= st.iterations <= items * (depth + 1)
        images.append(img)
    for img in images[1:]:
        assert np.array_equal(img.view(np.uint32), images[0].view(np.uint32))
    s.free()


@pytest.mark.parametrize("spp,depth,records", [(1, 6, 500), (3, 4, 200), (2, 0, 0)])
def test_cached_frames_end_within_the_bound(gpu_ctx, spp, depth, records):
    import aqua

    s = gpu_ctx.procedural(2, seed=0, width=61, height=43)
    net = aqua.Nrc(gpu_ctx, seed=1)
    cfg = gpu_ctx.integrator(type=aqua.INTEGRATOR_NRC, spp=spp, max_depth=depth, rr_depth=3, seed=2,
                             nrc_train_samples=records, batch_size=128)
    for tune in (None, gpu_ctx.tuning(replicas=1), gpu_ctx.tuning(iters_per_graph=2, sort_by_material=1)):
        _, st = gpu_ctx.render_nrc(s, cfg, net, tuning=tune)
        assert st.paths == 61 * 43 * spp
    net.free()
    s.free()
