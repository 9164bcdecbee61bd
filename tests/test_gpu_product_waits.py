"""Waits of the product sketch's kernels that run out.  The test hook lets their
barriers wait for an arrival that nobody makes, for a millisecond instead of two
seconds: the kernels end, the sketch is NaN, and the caller whose sketch it is
gets an error: not another thread's call, plan, server or request.  What comes
next is unaffected."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n_a, n_inner, n_b, b, d): staged additions in one and two row blocks, lane additions
SHAPES = [(300, 200, 300, 8192, 2), (40, 300, 4200, 8192, 3), (300, 2000, 4200, 2048, 2)]


def kernel():
    from compmatmul_b200 import lib
    return lib().cmm_last_sketch_kernel().decode()


def matrices(shape, seed=0):
    n_a, k, n_b, _, _ = shape
    rng = np.random.default_rng(seed)
    return rng.standard_normal((k, n_a)), rng.standard_normal((k, n_b))


@pytest.mark.parametrize("variant", ["fft", "fwht"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("where", ["product", "add"])
def test_the_call_reports_it(gpu, oracle, monkeypatch, variant, shape, where):
    from compmatmul_b200 import capi
    d, b = shape[4], shape[3]
    AT, B = matrices(shape)
    monkeypatch.setenv("CMM_TEST_PRODUCT_WAIT", where)
    with pytest.raises(RuntimeError, match="a wait ran out"):
        capi.compressed_product(variant, None, AT, B, d, b, 7)
    monkeypatch.delenv("CMM_TEST_PRODUCT_WAIT")
    p, _ = capi.compressed_product(variant, None, AT, B, d, b, 7)
    assert kernel() == "product"
    ref = oracle.compressed_product(variant, None, AT, B, d, b, 7)
    np.testing.assert_allclose(p, ref, rtol=0, atol=1e-11 * np.abs(ref).max())


def test_only_the_callers_thread_reports_it(gpu, monkeypatch):
    """A device call returns before its kernels run: its sketch is NaN and the
    thread's next call says so.  Calls of another thread in between are good."""
    import torch

    from compmatmul_b200 import capi, device
    AT, B = matrices(SHAPES[0])
    dAT, dB = torch.from_numpy(AT).cuda(), torch.from_numpy(B).cuda()
    good, _ = capi.compressed_product("fft", None, AT, B, 2, 8192, 7)
    seen, go, done = {}, threading.Event(), threading.Event()

    def other():
        monkeypatch.setenv("CMM_TEST_PRODUCT_WAIT", "product")
        p = device.compressed_product(dAT, dB, 2, 8192, 7)
        torch.cuda.synchronize()
        seen["nan"] = bool(torch.isnan(p).all())
        monkeypatch.delenv("CMM_TEST_PRODUCT_WAIT")
        done.set()
        go.wait(60)
        try:
            device.compressed_product(dAT, dB, 2, 8192, 7)
        except RuntimeError as e:
            seen["error"] = str(e)
        seen["after"] = device.compressed_product(dAT, dB, 2, 8192, 7).cpu().numpy()

    t = threading.Thread(target=other)
    t.start()
    assert done.wait(60)
    p, _ = capi.compressed_product("fft", None, AT, B, 2, 8192, 7)
    np.testing.assert_array_equal(p, good)
    go.set()
    t.join(60)
    assert seen["nan"] and "a wait ran out" in seen["error"]
    assert np.abs(seen["after"] - good).max() <= 1e-13 * np.abs(good).max()


def problems(count, f32, lo=400, hi=1200):
    import torch

    from compmatmul_b200.planted import batch_shapes, planted_problem_device
    out = []
    for s in batch_shapes(count=count, seed=61, lo=lo, hi=hi):
        AT, B, _ = planted_problem_device(s["m"], s["n"], s["p"], s["K"], s["gen_seed"], "float32" if f32 else "float64")
        out.append(dict(AT=AT, B=B, d=s["d"], b=s["b"], seed=s["seed"], variant=s["variant"]))
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("where", ["product", "add"])
@pytest.mark.parametrize("own_stream", [False, True])
def test_only_the_plan_reports_it(gpu, monkeypatch, where, own_stream):
    """On the plan's stream a run returns when it has ended and reports it;
    on a caller's stream the plan's next run does."""
    import torch

    from compmatmul_b200.batch import BatchPlan
    probs = problems(12, True)
    good, bad = BatchPlan(probs, f32=True, tune=False), BatchPlan(probs, f32=True, tune=False)
    stream = None if own_stream else torch.cuda.Stream()
    monkeypatch.setenv("CMM_TEST_PRODUCT_WAIT", where)  # (captured with the kernels of the first run)
    if own_stream:
        with pytest.raises(RuntimeError, match="a wait ran out"):
            bad.run()
    else:
        bad.run(stream)
    torch.cuda.synchronize()
    monkeypatch.delenv("CMM_TEST_PRODUCT_WAIT")
    for _ in range(2):
        good.run(stream)
    torch.cuda.synchronize()
    assert all(torch.isnan(q["p"]).all() for q in bad.products)
    assert not any(torch.isnan(q["p"]).any() for q in good.products)
    with pytest.raises(RuntimeError, match="a wait ran out"):
        bad.run(stream)
    bad.close()
    good.close()


@pytest.mark.parametrize("where", ["product", "add"])
def test_only_the_request_reports_it(gpu, monkeypatch, where):
    from compmatmul_b200.serve import Server
    probs = problems(3, True)

    def submit(srv, q):
        return srv.submit(q["AT"], q["B"], q["d"], q["b"], q["seed"], q["variant"])

    srv, other = (Server(mem_cap_bytes=2 << 30, f32=True, streams=2, max_wave=2) for _ in range(2))
    want = [srv.result(submit(srv, q), timeout=60) for q in probs]
    monkeypatch.setenv("CMM_TEST_PRODUCT_WAIT", where)
    rid = submit(srv, probs[0])
    with pytest.raises(RuntimeError, match="a wait ran out"):
        srv.result(rid, timeout=60)
    monkeypatch.delenv("CMM_TEST_PRODUCT_WAIT")
    for s in (other, srv):
        for q, p in zip(probs, want):
            np.testing.assert_array_equal(s.result(submit(s, q), timeout=60), p)
        assert s.stats()["in_flight"] == 0 and s.stats()["mem_in_use"] == 0
        s.close()
