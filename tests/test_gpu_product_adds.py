"""Additions of the product sketch where their forms change hands: integer
inputs, so that every order of additions gives the same bits as the definition.
The dispatch would give some of these sizes to other kernels, and reads its
override once a process, so the sketches are formed in a process of their own."""
import os
import pathlib
import subprocess
import sys

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


@pytest.mark.parametrize("variant", ["fft", "fwht"])
def test_integer_sketches_are_exact(gpu, variant):
    env = dict(os.environ, CMM_SKETCH_KERNELS="product")
    r = subprocess.run([sys.executable, __file__, variant], env=env, cwd=pathlib.Path(__file__).parents[1],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr


def exact(variant, n_a, k, n_b, b, d):
    import torch

    from compmatmul_b200 import capi, device, lib
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
    return np.array_equal(got.cpu().numpy().reshape(d, b), want)


if __name__ == "__main__":
    sys.path.insert(0, os.getcwd())
    wrong = [s for s in SHAPES if not exact(sys.argv[1], *s)]
    print("differ:", wrong)
    sys.exit(1 if wrong else 0)
