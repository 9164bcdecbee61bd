"""Dense estimates and top-K on the device at the edges of their kernels.

The estimate's median is compared bit for bit with the exchange network of
minima and maxima over the d values (which passes a NaN by), for every d with a
kernel of its own, with zeros of both signs, infinities and NaNs among the
values, at sizes around the rows and columns of a CTA.  Top-K is compared with
a stable sort, around one CTA's and one thread's share of the entries.  The
inverse transforms are compared with the definition."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def network(v):
    """Entry d / 2 after odd-even transposition with minima and maxima that
    take the other value for a NaN, and -0 below +0."""
    def less(a, b):
        return (a < b) | ((a == b) & np.signbit(a) & ~np.signbit(b))

    v = [x.copy() for x in v]
    d = len(v)
    for k in range(d):
        for i in range(k & 1, d - 1, 2):
            a, b = v[i], v[i + 1]
            na, nb = np.isnan(a), np.isnan(b)
            lo = np.where(na, b, np.where(nb, a, np.where(less(b, a), b, a)))
            hi = np.where(na, b, np.where(nb, a, np.where(less(b, a), a, b)))
            v[i], v[i + 1] = lo, hi
    return v[d // 2]


@pytest.mark.parametrize("variant", ["fft", "fwht"])
@pytest.mark.parametrize("d", list(range(1, 17)))
@pytest.mark.parametrize("n_a,n_b", [(1, 1), (17, 257), (70, 300)])
@pytest.mark.parametrize("values", ["normal", "zeros", "special"])
def test_dense_estimate_is_the_networks(gpu, variant, d, n_a, n_b, values):
    import torch

    from compmatmul_b200 import capi, device
    b, seed = 256, 11 + d
    rng = np.random.default_rng(100 * d + n_a)
    p = rng.standard_normal((d, b))
    if values == "zeros":
        p = np.where(rng.random((d, b)) < 0.7, np.where(rng.random((d, b)) < 0.5, -0.0, 0.0), p)
    elif values == "special":
        u = rng.random((d, b))
        p = np.where(u < 0.2, np.inf, np.where(u < 0.4, -np.inf, np.where(u < 0.5, np.nan, p)))
    C = device.decompress_dense(torch.from_numpy(p).cuda(), n_a, n_b, d, b, seed, variant=variant).cpu().numpy()
    mas = "multiply add shift"
    cA, cB = capi.hash_codes(mas, d, b, seed, 0, n_a), capi.hash_codes(mas, d, b, seed, 1, n_b)
    vals = []
    for t in range(d):
        hA, hB = (cA[t] & 0x7fffffff)[:, None], (cB[t] & 0x7fffffff)[None, :]
        idx = (hA + hB) % b if variant == "fft" else hA ^ hB
        minus = ((cA[t] >> 31)[:, None] ^ (cB[t] >> 31)[None, :]).astype(bool)
        v = p[t][idx]
        vals.append(np.where(minus, -v, v))
    want = network(vals)
    same = (C.view(np.int64) == want.view(np.int64)) | (np.isnan(C) & np.isnan(want))
    assert same.all()


@pytest.mark.parametrize("n_a,n_b", [(1, 1), (1, 33), (255, 257), (700, 1001), (1300, 1000)])
@pytest.mark.parametrize("K", [1, 64, 65, 1000, 4096])
@pytest.mark.parametrize("values", ["normal", "few"])
def test_topk_against_a_stable_sort(gpu, n_a, n_b, K, values):
    import torch

    from compmatmul_b200 import device
    n = n_a * n_b
    K = min(K, n)
    rng = np.random.default_rng(n + K)
    C = rng.standard_normal(n)
    if values == "few":  # ties, more than fit the sort at the larger sizes
        C = np.round(2 * C)
        C[C == 0] = 0.0
    order = np.argsort(-C, kind="stable")[:K]
    i, j, v = device.topk(torch.from_numpy(C.reshape(n_a, n_b)).cuda(), K)
    assert (i * n_b + j == order).all() and (v == C[order]).all()


@pytest.mark.parametrize("variant", ["fft", "fwht"])
@pytest.mark.parametrize("log2b", [1, 2, 6, 10, 12, 13, 14])
@pytest.mark.parametrize("d", [1, 5])
def test_small_sketches_against_the_definition(gpu, variant, log2b, d):
    import torch

    from compmatmul_b200 import capi, device
    n_a, k, n_b, b, seed = 13, 9, 11, 1 << log2b, 5 + d
    rng = np.random.default_rng(log2b)
    A, B = rng.standard_normal((k, n_a)), rng.standard_normal((k, n_b))
    got = device.compressed_product(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), d, b, seed, variant=variant)
    mas = "multiply add shift"
    cA, cB = capi.hash_codes(mas, d, b, seed, 0, n_a), capi.hash_codes(mas, d, b, seed, 1, n_b)
    C = A.T @ B
    want = np.zeros((d, b))
    for t in range(d):
        hA, hB = (cA[t] & 0x7fffffff)[:, None], (cB[t] & 0x7fffffff)[None, :]
        idx = (hA + hB) % b if variant == "fft" else hA ^ hB
        minus = ((cA[t] >> 31)[:, None] ^ (cB[t] >> 31)[None, :]).astype(bool)
        np.add.at(want[t], idx, np.where(minus, -C, C))
    # every stage of the transforms rounds values of at most the 1-norms' products
    bound = (4 * log2b + 8 + n_a * n_b) * 2.0 ** -52 * (np.abs(A).sum(1) * np.abs(B).sum(1)).sum()
    assert np.abs(got.cpu().numpy().reshape(d, b) - want).max() <= bound
