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


if __name__ == "__main__":
    sys.path.insert(0, os.getcwd())
    {"full": full, "buckets": buckets}[sys.argv[1]]()
