"""Additions of the product sketch where their forms change hands: integer
inputs, so that every order of additions gives the same bits as the definition."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n_a, n_inner, n_b, b, d)
SHAPES = [
    (70, 40, 1385, 8192, 3),     # 87 entries a window on average: more than three batches at times
    (65, 33, 750, 512, 2),       # buckets of many entries (six and more of one bucket)
    (65, 33, 767, 512, 2),       # the last columns of the staged form, the first of the lane form
    (65, 33, 768, 512, 2),
    (40, 16, 3071, 2048, 2),
    (40, 16, 3072, 2048, 2),
    (33, 20, 4096, 4096, 1),     # as many columns as buckets
    (31, 20, 4097, 65536, 2),    # a second block of one column
    (1100, 8, 600, 16384, 1),    # several row groups
    (33, 16, 13000, 1 << 17, 1), # gathered, more than three batches at times
]


@pytest.mark.parametrize("n_a,k,n_b,b,d", SHAPES)
@pytest.mark.parametrize("variant", ["fft", "fwht"])
def test_integer_sketches_are_exact(gpu, variant, n_a, k, n_b, b, d, monkeypatch):
    import torch

    from compmatmul_b200 import capi, device, lib
    monkeypatch.setenv("CMM_SKETCH_KERNELS", "product")
    rng = np.random.default_rng(n_a + n_b)
    A, B = rng.integers(-99, 100, (k, n_a)).astype(float), rng.integers(-99, 100, (k, n_b)).astype(float)
    got = device.compressed_product(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), d, b, 3, variant=variant)
    assert lib().cmm_last_sketch_kernel().decode() == "product"
    mas = "multiply add shift"
    cA, cB = capi.hash_codes(mas, d, b, 3, 0, n_a), capi.hash_codes(mas, d, b, 3, 1, n_b)
    C = A.T @ B
    want = np.zeros((d, b))
    for t in range(d):
        hA, hB = (cA[t] & 0x7fffffff)[:, None], (cB[t] & 0x7fffffff)[None, :]
        idx = (hA + hB) % b if variant == "fft" else hA ^ hB
        minus = ((cA[t] >> 31)[:, None] ^ (cB[t] >> 31)[None, :]).astype(bool)
        np.add.at(want[t], idx, np.where(minus, -C, C))
    # (the sign of a code is +1 where its bit is set: two equal bits give +)
    assert np.array_equal(got.cpu().numpy().reshape(d, b), want)
