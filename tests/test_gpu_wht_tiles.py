"""Batched FP32 Walsh-Hadamard transform of rows at the edges of its tiles:
8192 elements (1, 2 or 4 rows) per tile, last tiles that are not full, one
tile, one more and one fewer than the tiles in flight, and 16-byte aligned
rows that do not start a 128-byte line.  Tolerance: 2e-6 * max|ref| against
the FP64 transform (FP32 arithmetic over at most 13 add/sub stages)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def reference(x):
    y, n, h = x.astype(np.float64), x.shape[1], 1
    while h < n:
        y = y.reshape(-1, n // (2 * h), 2, h)
        y = np.stack([y[:, :, 0] + y[:, :, 1], y[:, :, 0] - y[:, :, 1]], axis=2).reshape(-1, n)
        h *= 2
    return y


@pytest.mark.parametrize("method", ["tensor", "cuda"])
@pytest.mark.parametrize("rows,log2n", [(1, 11), (3, 11), (5, 11), (1, 12), (3, 12), (1, 13), (2, 13), (147, 13),
                                        (149, 13), (741, 13), (1187, 11)])
@pytest.mark.parametrize("offset", [0, 4])
def test_tile_remainders(gpu, method, rows, log2n, offset):
    import torch

    from compmatmul_b200 import device
    n = 1 << log2n
    x = np.random.default_rng(rows + log2n).standard_normal((rows, n)).astype(np.float32)
    buf = torch.full((rows * n + 64,), 7.0, device="cuda")
    xd = buf[offset:offset + rows * n].view(rows, n)
    xd.copy_(torch.from_numpy(x))
    out = torch.full((rows * n + 64,), -3.0, device="cuda")
    y = device.wht_rows(xd, method, out=out[offset:offset + rows * n].view(rows, n)).cpu().numpy()
    ref = reference(x)
    assert np.abs(y - ref).max() <= 2e-6 * np.abs(ref).max()
    # nothing written before or after the rows
    assert (out[:offset] == -3.0).all() and (out[offset + rows * n:] == -3.0).all()
