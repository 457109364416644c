"""Shading that loads each thread's next queue entry ahead, against the form
without: a render's image does not depend on the number of path slots, and
slots up to the grid's threads use the one form, more the other."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("config", [2, 3])
def test_images_agree_across_the_switch(gpu_ctx, config):
    import torch

    import aqua

    side = 640
    s = gpu_ctx.procedural(config, seed=0, width=side, height=side)
    try:
        cfg = gpu_ctx.integrator(spp=2, max_depth=4, rr_depth=3, seed=5)
        lanes = torch.cuda.get_device_properties(0).multi_processor_count * 128  # one block per SM
        want = None
        for slots in (lanes // 2, lanes, lanes + 1, 2 * lanes, 2 * lanes + 1, 3 * lanes + 77, side * side):
            tuning = aqua.Tuning(slots=slots, blocks_per_sm=1)
            img, _ = gpu_ctx.render(s, cfg, tuning=tuning)
            if want is None:
                want = img.copy()
            assert np.array_equal(img, want), slots
    finally:
        s.free()
