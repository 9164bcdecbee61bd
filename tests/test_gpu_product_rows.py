"""Row balance of the product sketch: rows of subnormals, of zeros, of NaNs next
to zeros, longer and shorter than a CTA's share, FP32 and FP64.  As in the
transform kernels, the FFT form skips a row pair in which a row has no number
but zero, whatever NaNs it has; the FWHT form and every other non-finite value
make the sketch NaN.  Sketches against the oracle's product of the finite
rows: 1e-11 * max|p| (FP64), 1e-6 (FP32), as for this kernel's other tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sketch(variant, A, B, f32, d=2, b=8192):
    from compmatmul_b200 import capi, lib
    fn = capi.compressed_product_f32 if f32 else capi.compressed_product
    p, _ = fn(variant, None, A, B, d, b, 4)
    assert lib().cmm_last_sketch_kernel().decode() == "product"
    return p


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("variant", ["fft", "fwht"])
@pytest.mark.parametrize("n_a,n_b", [(300, 513), (127, 2000), (1100, 300)])
def test_subnormal_and_zero_rows(gpu, oracle, variant, f32, n_a, n_b):
    dt = np.float32 if f32 else np.float64
    rng = np.random.default_rng(n_a)
    A, B = rng.standard_normal((300, n_a)).astype(dt), rng.standard_normal((300, n_b)).astype(dt)
    A[3] *= np.finfo(dt).tiny / 16
    B[5] = 0.0
    A[7, :] = -0.0
    p = sketch(variant, A, B, f32)
    ref = oracle.compressed_product(variant, None, A.astype(float), B.astype(float), 2, 8192, 4)
    assert np.abs(p - ref).max() <= (1e-6 if f32 else 1e-11) * np.abs(ref).max()


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("variant", ["fft", "fwht"])
@pytest.mark.parametrize("at", [0, 299])
def test_rows_without_a_number(gpu, oracle, variant, f32, at):
    dt = np.float32 if f32 else np.float64
    rng = np.random.default_rng(at)
    A, B = rng.standard_normal((300, 300)).astype(dt), rng.standard_normal((300, 310)).astype(dt)
    A[17] = 0.0
    A[17, at] = np.nan
    p = sketch(variant, A, B, f32)
    if variant == "fwht":
        assert np.isnan(p).all()
    else:
        A[17] = 0.0
        ref = oracle.compressed_product(variant, None, A.astype(float), B.astype(float), 2, 8192, 4)
        assert np.abs(p - ref).max() <= (1e-6 if f32 else 1e-11) * np.abs(ref).max()
    A[17] = 0.0
    A[17, at] = -np.inf
    assert np.isnan(sketch(variant, A, B, f32)).all()
