"""The tensor-core training step at the edges of its tiles and grid.

One kernel runs forward, backward and weight gradients over 128-row tiles, two
per CTA and round, and accumulates the gradients over a CTA's tiles; so row
counts around one tile, one tile per CTA, two and more rounds. Gradients and
loss against the mma.sync step, which rounds at the same points and differs in
the order of FP32 sums only; a repeated step must be bit-identical."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAYERS = [slice(4096 * k, min(4096 * (k + 1), 20672)) for k in range(6)]


def batch(n, seed):
    r = np.random.default_rng(seed)
    x = r.uniform(-1, 1, (n, 64)).astype(np.float32)
    x[:, 63] = 1.0
    b = x.view(np.uint32)
    bits = ((b + 0x7FFF + ((b >> 16) & 1)) >> 16).astype(np.uint16)  # round to nearest even bf16
    return bits, np.exp(r.normal(-0.5, 1.0, (n, 3))).astype(np.float32)


@pytest.mark.parametrize("rows", [1, 31, 127, 128, 129, 152 * 128, 152 * 128 + 1, 2 * 152 * 128 - 1,
                                  2 * 152 * 128 + 129, 100_003])
def test_step_matches_mma_sync(gpu_ctx, rows):
    import aqua

    x, t = batch(rows, rows)
    out = []
    for kernel in (aqua.NRC_KERNEL_TCGEN05, aqua.NRC_KERNEL_MMA_SYNC, aqua.NRC_KERNEL_TCGEN05):
        net = aqua.Nrc(gpu_ctx, seed=3, forward_kernel=kernel)
        loss = net.train_step(x, t)
        out.append((loss, net.gradients(), net.weights()))
        net.free()
    (l0, g0, w0), (l1, g1, _), (l2, g2, w2) = out
    assert abs(l0 - l1) <= 1e-4 * abs(l1)
    for sl in LAYERS:
        scale = np.abs(g1[sl]).max()
        assert np.linalg.norm(g0[sl] - g1[sl]) <= 1e-3 * np.linalg.norm(g1[sl])
        assert np.abs(g0[sl] - g1[sl]).max() <= 1e-2 * scale
    assert np.array_equal(g0.view(np.uint32), g2.view(np.uint32)) and np.array_equal(w0, w2)


@pytest.mark.parametrize("ema", [0.0, 0.9])
def test_steps_of_changing_size(gpu_ctx, ema):
    """Consecutive steps share the scratch and the weight images: larger, smaller
    and larger batches in turn, with and without averaged inference weights, must
    leave the network where the mma.sync steps leave it."""
    import aqua

    nets = [aqua.Nrc(gpu_ctx, seed=5, ema_decay=ema, learning_rate=1e-4, forward_kernel=k)
            for k in (aqua.NRC_KERNEL_TCGEN05, aqua.NRC_KERNEL_MMA_SYNC)]
    for i, rows in enumerate((500, 20_000, 129, 40_000, 1)):
        x, t = batch(rows, 100 + i)
        a, b = (net.train_step(x, t) for net in nets)
        assert abs(a - b) <= 2e-3 * abs(b)
    x, _ = batch(1000, 7)
    y0, y1 = (net.forward(x) for net in nets)
    scale = np.abs(y1).max()
    assert np.abs(y0 - y1).max() <= 2e-2 * scale and np.abs(y0 - y1).mean() <= 2e-3 * scale
    for net in nets:
        net.free()
