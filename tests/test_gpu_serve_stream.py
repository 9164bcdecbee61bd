"""A steady stream of requests that take the product sketch, several waves in
flight on as many streams: every request ends, and gives the same bits each time.

The product kernel's CTAs work in pairs; when other streams' kernels shared
their SMs, a pair whose CTAs came and went on their own could stay for good (in
a stream of 2000 requests a second, after a second or two).  In a process of
its own, which ends whether or not a request does."""
import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REQUESTS, POOL, AHEAD = 8000, 24, 24


def test_every_request_ends(gpu):
    r = subprocess.run([sys.executable, __file__], cwd=pathlib.Path(__file__).parents[1], capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr


def main():
    from collections import deque

    from compmatmul_b200.planted import batch_shapes, planted_problem_device
    from compmatmul_b200.serve import Server
    pool = []
    for s in batch_shapes(count=POOL, seed=77, lo=256, hi=2048):
        AT, B, _ = planted_problem_device(s["m"], s["n"], s["p"], s["K"], s["gen_seed"], "float32")
        pool.append((AT, B, s["d"], s["b"], s["seed"], s["variant"]))
    srv = Server(mem_cap_bytes=8 << 30, f32=True, streams=4, max_wave=1, cache_bytes=1 << 30)
    first, live, wrong = {}, deque(), 0
    for i in range(REQUESTS + AHEAD):
        if i < REQUESTS:
            live.append((i % POOL, srv.submit(*pool[i % POOL])))
        if i >= AHEAD:
            k, rid = live.popleft()
            p = srv.result(rid, timeout=30.0)
            wrong += not np.array_equal(first.setdefault(k, p), p)
    st = srv.stats()
    print("differ:", wrong, st)
    return 0 if wrong == 0 and st["completed"] == REQUESTS and st["max_waves_in_flight"] >= 3 else 1


if __name__ == "__main__":
    sys.path.insert(0, os.getcwd())
    code = 2
    try:
        code = main()
    except Exception as e:  # a request that does not end: nothing here may wait for it
        print(f"{type(e).__name__}: {e}")
    sys.stdout.flush()
    os._exit(code)
