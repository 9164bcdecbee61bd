"""Product sketch (residue planes, int8 tensor-core product, reconstruction,
addition into the sketches) against the oracle.

The shapes sit at the edges of its tiles (128 / 256 columns, 128 inner
indices), of its column windows and of both addition kernels, and are large
enough that the dispatch takes it (checked through cmm_last_sketch_kernel).
Tolerances: FP64 1e-11 * max|p| as for the other kernels.  FP32 inputs: an
entry of the integer product is off by at most 2^-32 (sqrt(k) + sqrt(k)) |a_i||b_j|
(each column's entries are rounded to 2^-32 of its norm bound), and a bucket
sums n_a n_b / b of them, far below 1e-6 * max|p| for these sizes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def capi():
    from compmatmul_b200 import capi as c
    return c


def kernel():
    from compmatmul_b200 import lib
    return lib().cmm_last_sketch_kernel().decode()


def check(oracle, variant, AT, B, d, b, seed=5, h=None, f32=False):
    if f32:
        AT, B = AT.astype(np.float32), B.astype(np.float32)
        p, _ = capi().compressed_product_f32(variant, h, AT, B, d, b, seed)
    else:
        p, _ = capi().compressed_product(variant, h, AT, B, d, b, seed)
    assert kernel() == "product", kernel()
    ref = oracle.compressed_product(variant, h, AT.astype(np.float64), B.astype(np.float64), d, b, seed)
    tol = 1e-6 if f32 else 1e-11
    np.testing.assert_allclose(p, ref, rtol=0, atol=tol * max(float(np.abs(ref).max()), 1e-300))
    return p, ref


# (n_a, n_inner, n_b, b, d)
SHAPES = [(512, 128, 512, 8192, 3), (513, 129, 257, 8192, 2), (255, 127, 1025, 8192, 1), (700, 300, 90, 16384, 5),
          (90, 300, 700, 16384, 5), (1, 2000, 1000, 4096, 3), (1000, 2000, 1, 4096, 3), (640, 33, 900, 8192, 2),
          (300, 700, 300, 1 << 15, 2), (520, 64, 600, 1 << 17, 1), (400, 3000, 1500, 512, 4), (300, 2000, 4200, 2048, 2)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("variant,f32", [("fft", False), ("fwht", False), ("fft", True), ("fwht", True)])
def test_product_sketch_vs_oracle(gpu, oracle, variant, f32, shape):
    n_a, k, n_b, b, d = shape
    rng = np.random.default_rng(n_a + k + b)
    AT = rng.standard_normal((k, n_a))
    B = rng.standard_normal((k, n_b)) * 1e-3
    AT[rng.integers(k), rng.integers(n_a)] += 1e3
    check(oracle, variant, AT, B, d, b, h=["multiply shift", "tabulation8", None][n_a % 3], f32=f32)


@pytest.mark.parametrize("variant", ["fft", "fwht"])
def test_scales_zero_rows_and_columns(gpu, oracle, variant):
    """Row pairs of very different scales, zero rows and columns, tiny and huge values."""
    rng = np.random.default_rng(3)
    AT = rng.standard_normal((300, 300)) * np.logspace(-60, 60, 300)[:, None]
    B = rng.standard_normal((300, 310)) * np.logspace(60, -60, 300)[:, None]
    AT[[0, 7, 299]] = 0.0
    B[[5, 298]] = 0.0
    AT[:, 11] = 0.0
    B[:, 309] = 0.0
    check(oracle, variant, AT, B, 3, 8192)
    check(oracle, variant, AT * 1e-140, B * 1e100, 3, 8192)


@pytest.mark.parametrize("f32", [False, True])
def test_integer_inputs_are_exact(gpu, oracle, f32):
    rng = np.random.default_rng(4)
    p, ref = check(oracle, "fwht", rng.integers(-99, 100, (400, 333)).astype(float),
                   rng.integers(-99, 100, (400, 280)).astype(float), 4, 8192, f32=f32)
    assert np.array_equal(p, ref)


@pytest.mark.parametrize("variant", ["fft", "fwht"])
def test_chunks_of_the_inner_index(gpu, oracle, variant, monkeypatch):
    """A small budget splits the inner index: later chunks add to the product."""
    rng = np.random.default_rng(6)
    AT, B = rng.standard_normal((700, 260)), rng.standard_normal((700, 250))
    whole, _ = check(oracle, variant, AT, B, 3, 8192)
    monkeypatch.setenv("CMM_MATERIALIZE_BYTES", str(1 << 20))
    parts, _ = check(oracle, variant, AT, B, 3, 8192)
    np.testing.assert_allclose(parts, whole, rtol=0, atol=1e-13 * np.abs(whole).max())


@pytest.mark.parametrize("variant", ["fft", "fwht"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_inputs_give_nan(gpu, variant, bad):
    """As through the transforms: one non-finite entry makes every bucket NaN.
    The FFT form skips a row pair whose other row is zero."""
    rng = np.random.default_rng(7)
    AT, B = rng.standard_normal((300, 300)), rng.standard_normal((300, 300))
    AT[17, 3] = bad
    p, _ = capi().compressed_product(variant, None, AT, B, 2, 8192, 1)
    assert kernel() == "product" and np.isnan(p).all()
    B[17] = 0.0
    p, _ = capi().compressed_product(variant, None, AT, B, 2, 8192, 1)
    assert np.isnan(p).all() == (variant == "fwht")


def test_device_entry_and_dense_estimate(gpu, oracle):
    """cmm_dev_matmul forms the product in the dense output first; odd sizes."""
    import torch

    from compmatmul_b200 import device
    rng = np.random.default_rng(8)
    AT, B = rng.standard_normal((301, 303)), rng.standard_normal((301, 299))
    C = device.matmul(torch.from_numpy(AT).cuda(), torch.from_numpy(B).cuda(), 5, 4096, 9, "fft").cpu().numpy()
    assert kernel() == "product"
    p = oracle.compressed_product("fft", None, AT, B, 5, 4096, 9)
    ref = oracle.decompress("fft", None, p, 5, 4096, 9, 303, 299)
    np.testing.assert_allclose(C, ref, rtol=0, atol=1e-11 * np.abs(p).max())
