"""The encoder's two forms: 32- and 16-byte words on aligned buffers, 4-byte
words on others. Same arithmetic, so the same bits, at the edges of the
128-row blocks, and nothing written past the rows."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 127, 128, 129, 1000])
@pytest.mark.parametrize("raw_off,x_off", [(0, 0), (8, 8), (0, 2), (4, 0), (1, 0), (3, 6)])
def test_encode_forms_agree(gpu_ctx, rows, raw_off, x_off):
    import torch

    import aqua

    net = aqua.Nrc(gpu_ctx, seed=3, bbox_min=[-1, -1, -1], bbox_max=[1, 1, 1])
    try:
        raw = np.random.default_rng(rows).uniform(-1, 1, (rows, 16)).astype(np.float32)
        raw[:, 3:6] /= np.linalg.norm(raw[:, 3:6], axis=1, keepdims=True)
        raw[:, 6:9] /= np.linalg.norm(raw[:, 6:9], axis=1, keepdims=True)
        want = net.encode(raw)
        src = torch.zeros(rows * 16 + 16, dtype=torch.float32, device="cuda")
        src[raw_off:raw_off + rows * 16] = torch.from_numpy(raw).cuda().reshape(-1)
        dst = torch.full((rows * 64 + 64,), 0x5A5A, dtype=torch.int16, device="cuda")
        torch.cuda.synchronize()
        net.encode_device(src.data_ptr() + 4 * raw_off, rows, dst.data_ptr() + 2 * x_off)
        got = dst.cpu().numpy().view(np.uint16)
        assert np.array_equal(got[x_off:x_off + rows * 64].reshape(rows, 64), want)
        assert np.all(got[:x_off] == 0x5A5A) and np.all(got[x_off + rows * 64:] == 0x5A5A)
    finally:
        net.free()
