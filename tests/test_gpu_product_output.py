"""The dense output as room for the product C: it may share memory with the
inputs, with another product's output, start 8 bytes off a 16-byte boundary, or
have an odd number of columns.  Against the same call with an output of its own:
the same bits, since the sketch and the estimate do not depend on where C is."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D, BUCKETS, SEED = 5, 8192, 11


def kernel():
    from compmatmul_b200 import lib
    return lib().cmm_last_sketch_kernel().decode()


def inputs(k, n_a, n_b, f32, seed=0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float32 if f32 else torch.float64
    return (torch.randn((k, n_a), device="cuda", generator=g, dtype=dt),
            torch.randn((k, n_b), device="cuda", generator=g, dtype=dt))


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("where", ["AT", "B", "end of AT", "end of B"])
def test_output_over_an_input(gpu, monkeypatch, f32, where):
    """Several chunks of the inner index: the later ones are read after C's
    first entries are there."""
    import torch

    from compmatmul_b200 import device
    monkeypatch.setenv("CMM_MATERIALIZE_BYTES", str(1 << 20))
    n = 512
    AT, B = inputs(n, n, n, f32)
    want = device.matmul(AT, B, D, BUCKETS, SEED)
    assert kernel() == "product"
    # one buffer: room, an input, room, all in units of its type
    size = AT.numel()
    buf = torch.zeros(5 * size, device="cuda", dtype=AT.dtype)
    x = AT if "AT" in where else B
    at = 2 * size
    src = buf[at:at + size].view(n, n)
    src.copy_(x)
    begin = at + (size - 64 if "end" in where else 0)
    out = buf[begin:begin + size * (2 if f32 else 1)].view(torch.float64).view(n, n)
    got = device.matmul(*((src, B) if "AT" in where else (AT, src)), D, BUCKETS, SEED, out=out)
    assert kernel() == "product"
    assert torch.equal(got, want)


@pytest.mark.parametrize("n_b", [300, 301])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("chunks", [False, True])
def test_output_alignment_and_odd_columns(gpu, oracle, monkeypatch, n_b, offset, chunks):
    import torch

    from compmatmul_b200 import device
    if chunks:
        monkeypatch.setenv("CMM_MATERIALIZE_BYTES", str(1 << 20))
    AT, B = inputs(400, 303, n_b, False)
    buf = torch.full((303 * n_b + 3,), 5.0, device="cuda", dtype=torch.float64)
    out = buf[offset:offset + 303 * n_b].view(303, n_b)
    C = device.matmul(AT, B, D, BUCKETS, SEED, "fwht", out=out).cpu().numpy()
    assert kernel() == "product"
    p = oracle.compressed_product("fwht", None, AT.cpu().numpy(), B.cpu().numpy(), D, BUCKETS, SEED)
    ref = oracle.decompress("fwht", None, p, D, BUCKETS, SEED, 303, n_b)
    np.testing.assert_allclose(C, ref, rtol=0, atol=1e-11 * np.abs(p).max())
    assert (buf[:offset] == 5.0).all() and (buf[offset + 303 * n_b:] == 5.0).all()


def run_batch(prods, f32=False):
    """prods: (AT, B, p, C) tensors; one run."""
    import torch

    from compmatmul_b200 import check, lib
    from compmatmul_b200.batch import _Prod
    arr = (_Prod * len(prods))()
    for i, (AT, B, p, C) in enumerate(prods):
        arr[i] = _Prod(0, 1, D, BUCKETS, AT.shape[1], AT.shape[0], B.shape[1], SEED + i, AT.data_ptr(), B.data_ptr(),
                       p.data_ptr(), C.data_ptr())
    h = ctypes.c_void_p()
    check(lib().cmm_batch_create(ctypes.cast(arr, ctypes.c_void_p), len(prods), int(f32), 0, ctypes.byref(h)))
    check(lib().cmm_batch_run(h, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    check(lib().cmm_batch_destroy(h))


def test_batch_products_with_one_output(gpu):
    """Both sketches are those of the products alone; the output is the last's."""
    import torch
    one, two = inputs(300, 400, 300, False, 1), inputs(500, 400, 300, False, 2)
    p = torch.empty((4, D, BUCKETS), device="cuda", dtype=torch.float64)
    C = torch.empty((3, 400, 300), device="cuda", dtype=torch.float64)
    run_batch([(*one, p[0], C[0]), (*two, p[1], C[1])])
    run_batch([(*one, p[2], C[2]), (*two, p[3], C[2])])
    assert torch.equal(p[0], p[2]) and torch.equal(p[1], p[3]) and torch.equal(C[1], C[2])


def test_batch_output_over_another_products_input(gpu):
    """Every input is read before any output is written."""
    import torch
    one, two = inputs(300, 256, 256, False, 1), inputs(256, 256, 400, False, 2)
    p = torch.empty((4, D, BUCKETS), device="cuda", dtype=torch.float64)
    C, E = torch.empty((256, 256), device="cuda", dtype=torch.float64), torch.empty((2, 256, 400), device="cuda",
                                                                                   dtype=torch.float64)
    run_batch([(*one, p[0], C), (*two, p[1], E[0])])
    run_batch([(*one, p[2], two[0]), (*two, p[3], E[1])])
    for a, b in ((p[0], p[2]), (p[1], p[3]), (E[0], E[1]), (C, two[0])):
        # (the transforms, whose order of additions is another one)
        assert (a - b).abs().max() <= 1e-11 * p[:2].abs().max()
