"""Device memory of the product sketch: where it does not fit, or would take far
more than the transforms, calls, plans and requests that the transforms can do
are still done.  What fills or measures the device's memory runs in processes of
their own."""
import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GB = 1 << 30


def child(name, **env):
    r = subprocess.run([sys.executable, __file__, name], env=dict(os.environ, **env), cwd=pathlib.Path(__file__).parents[1],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr


def kernel():
    from compmatmul_b200 import lib
    return lib().cmm_last_sketch_kernel().decode()


def integers(k, n_a, n_b):
    import torch
    g = torch.Generator(device="cuda").manual_seed(1)
    return [torch.randint(-99, 100, (k, n), device="cuda", generator=g).double() for n in (n_a, n_b)]


def repetition(A, B, d, b, t, seed):
    """p_t of the FFT variant, from its definition."""
    import torch

    from compmatmul_b200 import capi
    cA, cB = (torch.as_tensor(capi.hash_codes("multiply add shift", d, b, seed, side, x.shape[1])[t].astype(np.int64),
                              device="cuda") for side, x in ((0, A), (1, B)))
    want = torch.zeros(b, dtype=torch.float64, device="cuda")
    for i in range(0, A.shape[1], 2048):
        C = A[:, i:i + 2048].t() @ B
        at = ((cA[i:i + 2048] & 0x7fffffff)[:, None] + (cB & 0x7fffffff)[None, :]) % b
        sign = ((cA[i:i + 2048] >> 31)[:, None] ^ (cB >> 31)[None, :]) * -2.0 + 1.0
        want.index_add_(0, at.flatten(), (C * sign).flatten())
    return want


def test_a_call_that_the_free_memory_does_not_hold(gpu):
    child("full")


def full():
    """8192 x 2000 x 8192: the product needs 1.9 GB at least, the transforms a chunk of theirs."""
    import torch

    from compmatmul_b200 import device
    A, B = integers(2000, 8192, 8192)
    small = device.compressed_product(A[:, :512].contiguous(), B[:, :512].contiguous(), 3, 1 << 16, 5)
    assert kernel() == "product"
    p = device.compressed_product(A, B, 3, 1 << 16, 5)
    assert kernel() == "product"
    torch.cuda.synchronize()
    import ctypes
    # what the pool of stream-ordered memory keeps goes back to the device, and all but 1.2 GB is taken
    cudart = torch.cuda.cudart()
    assert cudart is not None
    rt = ctypes.CDLL("libcudart.so.12")
    pool = ctypes.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolTrimTo(pool, ctypes.c_size_t(0)) == 0
    fill = torch.empty(torch.cuda.mem_get_info()[0] - 6 * GB // 5, dtype=torch.uint8, device="cuda")
    q = device.compressed_product(A, B, 3, 1 << 16, 5)
    torch.cuda.synchronize()
    assert kernel() != "product", kernel()
    assert (q - p).abs().max() <= 1e-11 * p.abs().max()
    again = device.compressed_product(A[:, :512].contiguous(), B[:, :512].contiguous(), 3, 1 << 16, 5)
    assert kernel() == "product" and torch.equal(again, small)
    del fill


def test_partial_sketches_of_many_buckets(gpu):
    child("buckets", CMM_SKETCH_KERNELS="product")


def buckets():
    """16384 rows and columns, b = 2^24, d = 5: a partial sketch is 0.67 GB, and
    64 row groups would have one each."""
    import torch

    from compmatmul_b200 import device
    A, B = integers(3, 16384, 16384)
    p = torch.empty((5, 1 << 24), dtype=torch.float64, device="cuda")
    before = torch.cuda.mem_get_info()[0]
    device.compressed_product(A, B, 5, 1 << 24, 5, out=p)
    torch.cuda.synchronize()
    assert kernel() == "product"
    used = before - torch.cuda.mem_get_info()[0]
    assert used < 16 * GB, used  # C 2, residues 2, partial sketches 8, planes, lists
    for t in (0, 4):
        assert torch.equal(p[t], repetition(A, B, 5, 1 << 24, t, 5))


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("variant", ["fft", "fwht"])
def test_panels_and_chunks(gpu, monkeypatch, variant, f32):
    """A small scratch limit: the rows of C in panels of 256, the last one short, the
    inner indices in chunks of 128; the planes' rounding differs by chunk."""
    import torch

    from compmatmul_b200 import device
    g = torch.Generator(device="cuda").manual_seed(3)
    dt = torch.float32 if f32 else torch.float64
    A, B = (torch.randn((700, n), device="cuda", generator=g, dtype=dt) for n in (1100, 515))
    whole = device.compressed_product(A, B, 3, 8192, 5, variant)
    assert kernel() == "product"
    monkeypatch.setenv("CMM_MATERIALIZE_BYTES", str(1 << 20))
    parts = device.compressed_product(A, B, 3, 8192, 5, variant)
    assert kernel() == "product"
    assert (parts - whole).abs().max() <= (1e-7 if f32 else 1e-13) * whole.abs().max()


def random(k, n_a, n_b, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn((k, n), device="cuda", generator=g) for n in (n_a, n_b)]


def test_request_between_the_needs_of_both_routes(gpu):
    """1024-square FP32 requests, b = 8192, d = 5: the product sketch holds 35 MB, the
    transforms 12.  Under a cap of 20 MB they are served by the transforms."""
    from compmatmul_b200 import device
    from compmatmul_b200.serve import Server
    AT, B = random(1024, 1024, 1024, 5)
    ref = device.compressed_product(AT.double(), B.double(), 5, 8192, 9).cpu().numpy()
    got = []
    for cap in (20 << 20, 1 << 30):
        srv = Server(mem_cap_bytes=cap, f32=True, streams=2, max_wave=4)
        ids = [srv.submit(AT, B, 5, 8192, 9) for _ in range(3)]
        got.append([srv.result(i, timeout=60) for i in ids])
        st = srv.stats()
        srv.close()
        assert (st["max_mem_in_use"] > 20 << 20) == (cap > 20 << 20), st
    for p in got[0] + got[1]:
        assert np.abs(p - ref).max() <= 2e-5 * np.abs(ref).max()
        assert np.array_equal(p, got[0][0]) or np.array_equal(p, got[1][0])


def test_plan_with_products_above_the_scratch_limit(gpu, monkeypatch):
    """A limit that the small product's work space fits and the large one's does
    not: the large one takes the transforms."""
    import torch

    from compmatmul_b200.batch import BatchPlan
    prods = [dict(AT=m[0], B=m[1], d=5, b=8192, seed=3 + i) for i, m in
             enumerate([random(600, 300, 310, 1), random(1500, 1024, 1024, 2), random(600, 310, 300, 3)])]

    def run(limit):
        if limit:
            monkeypatch.setenv("CMM_MATERIALIZE_BYTES", str(limit))
        plan = BatchPlan(prods, f32=True, tune=False)
        plan.run()
        torch.cuda.synchronize()
        out = [(q["p"].clone(), q["C"].clone()) for q in plan.products]
        plan.close()
        return out

    whole, some, none = run(0), run(16 << 20), run(1 << 20)  # (the small ones need 7 MB each, the large one 60)
    for k in range(3):
        same = torch.equal(whole[k][0], some[k][0])
        assert same == (k != 1)  # the same route gives the same bits
        assert not torch.equal(whole[k][0], none[k][0])
        for a, b, c in zip(whole[k], some[k], none[k]):
            for x in (b, c):
                assert (a - x).abs().max() <= 2e-5 * whole[k][0].abs().max()


if __name__ == "__main__":
    sys.path.insert(0, os.getcwd())
    {"full": full, "buckets": buckets}[sys.argv[1]]()
