"""Batch plans and serving with every product on one route: the batch transform
kernel (one and several slabs, the reductions of small and of large b) and the
product sketch, against the oracle.  The dispatch would give most of these sizes
to the product sketch, and reads its override once a process, so each route runs
in a process of its own.  Tolerances as in these parts' other tests: 1e-11 *
max|p| from FP64 inputs, 2e-5 from FP32."""
import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (variant, n_a, n_inner, n_b, b, d)
SHAPES = [("fft", 300, 90, 260, 1024, 3), ("fwht", 310, 80, 250, 4096, 2), ("fft", 257, 130, 255, 8192, 2),
          ("fwht", 260, 100, 300, 16384, 1), ("fft", 300, 70, 310, 1 << 15, 2), ("fwht", 280, 60, 270, 1 << 16, 2),
          ("fft", 200, 40, 210, 1 << 17, 1), ("fwht", 90, 200, 70, 1 << 17, 1)]


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("route", ["slab", "product"])
def test_route(gpu, route, f32):
    r = subprocess.run([sys.executable, __file__, route, str(int(f32))], env=dict(os.environ, CMM_SKETCH_KERNELS=route),
                       cwd=pathlib.Path(__file__).parents[1], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr


def main(route, f32):
    import torch

    from compmatmul_b200.batch import BatchPlan
    from compmatmul_b200.serve import Server
    from oracle.oracle import Oracle
    orc, rng = Oracle(), np.random.default_rng(12)
    dt, tol = (np.float32, 2e-5) if f32 else (np.float64, 1e-11)
    prods, refs = [], []
    for i, (variant, n_a, k, n_b, b, d) in enumerate(SHAPES):
        AT, B = rng.standard_normal((k, n_a)).astype(dt), rng.standard_normal((k, n_b)).astype(dt)
        prods.append(dict(AT=torch.from_numpy(AT).cuda(), B=torch.from_numpy(B).cuda(), d=d, b=b, seed=40 + i, variant=variant))
        p = orc.compressed_product(variant, None, AT.astype(float), B.astype(float), d, b, 40 + i)
        refs.append((p, orc.decompress(variant, None, p, d, b, 40 + i, n_a, n_b)))
    # which route: the product sketch's work items are tiles of 256 x 256 per modulus
    for q in prods:
        plan = BatchPlan([q], f32=f32, tune=False)
        tiles = -(-q["AT"].shape[1] // 256) * -(-q["B"].shape[1] // 256) * (8 if f32 else 15)
        assert (plan.info()["items"] == tiles) == (route == "product"), (q["b"], plan.info(), tiles)
        plan.close()
    plan = BatchPlan(prods, f32=f32, tune=True)
    for _ in range(2):
        plan.run()
    srv = Server(mem_cap_bytes=2 << 30, f32=f32, streams=2, max_wave=3)
    ids = [srv.submit(q["AT"], q["B"], q["d"], q["b"], q["seed"], q["variant"]) for q in prods]
    served = [srv.result(i, timeout=60) for i in ids]
    srv.close()
    torch.cuda.synchronize()
    for q, s, (p, C) in zip(plan.products, served, refs):
        for name, x, ref in (("plan", q["p"].cpu().numpy(), p), ("served", s, p), ("estimate", q["C"].cpu().numpy(), C)):
            err = float(np.abs(x - ref).max()) / float(np.abs(p).max())
            assert err <= tol, (name, q["variant"], q["b"], err)
        if route == "product":  # the same jobs in both
            assert np.array_equal(q["p"].cpu().numpy(), s)
    plan.close()


if __name__ == "__main__":
    sys.path.insert(0, os.getcwd())
    main(sys.argv[1], sys.argv[2] == "1")
