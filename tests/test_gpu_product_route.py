"""Which kernels a single product runs on where C is sparse in the buckets (few
columns, many buckets), where it is padded to whole tiles, and where it is dense:
the route that was measured to be faster on B200, by 1.2 to 10 times.  Sketches
against the definition on integer inputs: the product route gives the same bits
in every order of additions, the transforms come within 1e-11 * max|p| (2e-5 from
FP32 inputs, their tolerance elsewhere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (variant, f32, d, b, n_a, n_inner, n_b), the faster route
SHAPES = [
    (("fft", False, 7, 1 << 22, 16892, 1, 729), "transforms"),
    (("fwht", False, 5, 1 << 21, 8953, 32, 6096), "transforms"),
    (("fwht", False, 1, 1 << 17, 11076, 79, 1033), "transforms"),
    (("fft", False, 9, 1 << 16, 4099, 25, 1418), "transforms"),
    (("fft", True, 1, 1 << 21, 3695, 40, 123), "transforms"),
    (("fwht", False, 5, 4096, 7340, 77, 88), "transforms"),
    (("fwht", False, 1, 2048, 7183, 4240, 286), "transforms"),
    (("fft", False, 3, 1 << 21, 750, 1350, 58), "product"),
    (("fft", False, 12, 1 << 18, 729, 1000, 122), "product"),
    (("fft", False, 7, 1 << 13, 3000, 500, 3000), "product"),
    (("fwht", True, 9, 1 << 17, 2000, 700, 2100), "product"),
]


@pytest.mark.parametrize("shape,route", SHAPES)
def test_route(gpu, shape, route):
    import torch

    from compmatmul_b200 import capi, device, lib
    variant, f32, d, b, n_a, k, n_b = shape
    dt = torch.float32 if f32 else torch.float64
    g = torch.Generator(device="cuda").manual_seed(1)
    A = torch.randint(-99, 100, (k, n_a), device="cuda", generator=g).to(dt)
    B = torch.randint(-99, 100, (k, n_b), device="cuda", generator=g).to(dt)
    p = device.compressed_product(A, B, d, b, 3, variant=variant)
    assert (lib().cmm_last_sketch_kernel().decode() == "product") == (route == "product")
    mas = "multiply add shift"
    cA, cB = (torch.as_tensor(capi.hash_codes(mas, d, b, 3, side, n).astype(np.int64), device="cuda")
              for side, n in ((0, n_a), (1, n_b)))
    C = A.double().t() @ B.double()
    for t in (0, d - 1):
        hA, hB = (cA[t] & 0x7fffffff)[:, None], (cB[t] & 0x7fffffff)[None, :]
        at = (hA + hB) % b if variant == "fft" else hA ^ hB
        sign = (((cA[t] >> 31)[:, None] ^ (cB[t] >> 31)[None, :]) * -2 + 1).double()
        want = torch.zeros(b, dtype=torch.float64, device="cuda").index_add_(0, at.flatten(), (C * sign).flatten())
        if route == "product":
            assert torch.equal(p[t], want)
        else:
            tol = 2e-5 if f32 else 1e-11
            assert (p[t] - want).abs().max() <= tol * want.abs().max()
