"""Copies of pageable host arrays around the sizes where they change hands (one
thread, the caller with helpers that stay awake, the pool), alone and from
several host threads at once, after pauses in which the helpers fall asleep:
every call gives the device path's estimate, to the rounding of another grouping
of the inner index: 1e-13 of the largest bucket, here 1e-12 of the largest entry
(a bucket is a sum of the same variance as an entry's estimate; a part that was
not copied in time is off by far more)."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n_a, n_inner, n_b): inputs and outputs of 0.1 to 20 MB
SHAPES = [(120, 120, 120), (181, 181, 181), (182, 181, 400), (700, 200, 720), (1250, 130, 1260), (1240, 64, 1280),
          (90, 3000, 700), (1600, 300, 1500)]


def call(A, B, seed=5):
    from compmatmul_b200 import load_dropin
    from compmatmul_b200.planted import aligned_empty
    C = aligned_empty((A.shape[1], B.shape[1]))
    load_dropin().matmul_fft(C, A, B, 3, 4096, seed)
    return C


def inputs(shape, seed):
    from compmatmul_b200.planted import aligned_empty
    n_a, k, n_b = shape
    rng = np.random.default_rng(seed)
    A, B = aligned_empty((k, n_a)), aligned_empty((k, n_b))
    A[...] = rng.standard_normal((k, n_a))
    B[...] = rng.standard_normal((k, n_b))
    return A, B


@pytest.mark.parametrize("shape", SHAPES)
def test_repeated_calls(gpu, shape):
    import torch

    from compmatmul_b200 import device
    A, B = inputs(shape, 1)
    ref = device.matmul(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), 3, 4096, 5).cpu().numpy()
    for i in range(12):
        if i % 4 == 0:
            time.sleep(0.002)
        assert np.abs(call(A, B) - ref).max() <= 1e-12 * np.abs(ref).max()


def test_several_threads(gpu):
    cases = [inputs(s, 10 + i) for i, s in enumerate(SHAPES[1:])]
    want = [call(A, B) for A, B in cases]
    wrong = []

    def work(i):
        for rep in range(8):
            for j in range(len(cases)):
                k = (i + j) % len(cases)
                C = call(*cases[k])
                if np.abs(C - want[k]).max() > 1e-12 * np.abs(want[k]).max():
                    wrong.append((i, rep, k))
            time.sleep(0.001 * (i % 3))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    assert not any(t.is_alive() for t in threads) and not wrong, wrong[:5]
