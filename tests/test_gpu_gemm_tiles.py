"""Exact FP64 product on the device at the edges of its 64 x 64 tiles and
16-deep slabs, with aligned rows (16-byte copies) and odd ones (8-byte
copies), and from a base that is only 8-byte aligned.  Tolerance: k * 2^-52 *
(|A|^T |B|) per entry (k roundings of a sum whose terms it bounds)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_a,k,n_b", [(1, 1, 1), (64, 16, 64), (65, 17, 63), (128, 15, 66), (63, 160, 130), (2, 33, 200),
                                       (200, 1000, 2), (129, 64, 65)])
@pytest.mark.parametrize("offset", [0, 1])
def test_gemm_tiles(gpu, n_a, k, n_b, offset):
    import torch

    from compmatmul_b200 import device
    rng = np.random.default_rng(n_a * 7 + n_b)
    A, B = rng.standard_normal((k, n_a)), rng.standard_normal((k, n_b))

    def on_device(M):
        buf = torch.full((M.size + 2,), 1e300, dtype=torch.float64, device="cuda")
        v = buf[offset:offset + M.size].view(*M.shape)
        v.copy_(torch.from_numpy(M))
        return v

    C = device.gemm(on_device(A), on_device(B)).cpu().numpy()
    bound = k * 2.0 ** -52 * (np.abs(A).T @ np.abs(B))
    assert (np.abs(C - A.T @ B) <= bound).all()
