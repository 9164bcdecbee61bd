"""Timed workloads of the compressed product: what users of this framework run,
through its public entry points.

A case is a plain dict; ``op`` names the entry point:

* ``matmul``   device.matmul: sketch + dense median estimate on CUDA tensors;
* ``dropin``   compmatmul.matmul_fft / matmul_fwht on host numpy arrays;
* ``recover``  Sketch.compute + topk: the largest entries without the dense estimate;
* ``sketch``   device.compressed_product: the d x b sketch alone;
* ``batch``    BatchPlan.run: many uneven float32 products with dense estimates;
* ``serve``    Server: a burst of float32 requests from host memory;
* ``gemm``     device.gemm: the exact FP64 product;
* ``wht``      device.wht_rows: the Walsh-Hadamard transform of float32 rows.

Inputs are planted-entry problems: noise N(0, 0.01^2) plus K planted pairs of
+10, as in the benchmark configurations.  Programs with float32 inputs (the
mixed-precision path) keep float32 results.
"""
import math

import numpy as np
import torch

import compmatmul_b200
from compmatmul_b200 import device
from compmatmul_b200.batch import BatchPlan
from compmatmul_b200.planted import aligned_empty, batch_shapes
from compmatmul_b200.serve import Server
from compmatmul_b200.sketch import Sketch

SIGMA, BIG = 0.01, 10.0


def _product(name, op, n_a, n_inner, n_b, b, d, variant, hash="multiply add shift", dtype="float64", K=0):
    return {"name": name, "op": op, "n_a": n_a, "n_inner": n_inner, "n_b": n_b, "b": b, "d": d, "variant": variant,
            "hash": hash, "dtype": dtype, "K": K or max(1, min(256, n_a // 16, n_inner // 16, n_b // 16))}


def listed():
    return [
        # the smallest call, as in the smoke run and unit tests: launches and latency
        _product("matmul_tiny", "matmul", 96, 96, 96, 1024, 5, "fft"),
        # the 512-square configuration, called as the reference's Python module is
        _product("dropin_512", "dropin", 512, 512, 512, 4096, 5, "fft", K=32),
        # a rectangular product of odd sizes, XOR variant, table hashing
        _product("matmul_ragged_fwht", "matmul", 1000, 777, 1303, 8192, 7, "fwht", "tabulation8"),
        # the 4096-square FP64 configuration: sketch, then its 256 largest entries
        _product("recover_fft_4096", "recover", 4096, 4096, 4096, 1 << 16, 9, "fft", K=256),
        # the sketch of a large rectangular product, kept for later queries
        _product("sketch_fwht_ragged", "sketch", 5000, 3001, 7000, 1 << 16, 9, "fwht", "multiply shift"),
        # the headline configuration: 16384-square FP64 with the dense estimate
        _product("matmul_fft_16384", "matmul", 16384, 16384, 16384, 1 << 16, 9, "fft", K=256),
        # the mixed-precision configuration: float32 inputs, b = 2^18
        _product("mixed_fft_16384", "matmul", 16384, 16384, 16384, 1 << 18, 9, "fft", dtype="float32", K=1024),
        # mixed precision, rectangular, XOR variant, sketch only
        _product("mixed_fwht_ragged", "sketch", 6001, 3000, 4500, 1 << 17, 7, "fwht", "tabulation8", "float32"),
        # many uneven products per iteration of a job (the batched configuration's shapes)
        {"name": "batch_64", "op": "batch", "count": 64, "lo": 256, "hi": 4096, "shapes": 4004, "dtype": "float32"},
        # a burst of requests to the serving engine (the serving configuration's shapes)
        {"name": "serve_48", "op": "serve", "count": 48, "lo": 256, "hi": 4096, "shapes": 5005, "dtype": "float32"},
        # the exact comparator of the reference's module
        {"name": "gemm_fp64", "op": "gemm", "n_a": 3000, "n_inner": 2048, "n_b": 2500, "dtype": "float64"},
        # the transform alone on many rows, with the entry point's default method
        {"name": "wht_rows_8192", "op": "wht", "rows": 16384, "n": 8192, "method": "tensor", "dtype": "float32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


HASHES = ["multiply shift", "multiply add shift", "tabulation8"]


def draw(rng):
    """One more case of the listed ranges: sizes log-uniform (odd ones among
    them), every variant, hash family and data type that is listed."""
    op = rng.choice(["matmul", "matmul", "dropin", "recover", "sketch", "sketch", "batch", "serve", "gemm", "wht"])
    if op in ("batch", "serve"):
        return {"op": op, "count": rng.randint(8, 56), "lo": 256, "hi": 4096, "shapes": rng.randint(1, 1 << 20),
                "dtype": "float32"}
    if op == "gemm":
        return {"op": op, "n_a": _log_int(rng, 64, 6000), "n_inner": _log_int(rng, 64, 6000),
                "n_b": _log_int(rng, 64, 6000), "dtype": "float64"}
    if op == "wht":
        return {"op": op, "rows": _log_int(rng, 64, 16384), "n": 1 << rng.randint(11, 13),
                "method": rng.choice(["tensor", "cuda"]), "dtype": "float32"}
    hi = 4096 if op == "dropin" else 12000
    while True:
        dtype = "float64" if op in ("dropin", "recover") else rng.choice(["float64", "float32"])
        c = _product("", op, _log_int(rng, 96, hi), _log_int(rng, 96, hi), _log_int(rng, 96, hi),
                     1 << rng.randint(10, 18), rng.choice([5, 7, 9]), rng.choice(["fft", "fwht"]), rng.choice(HASHES),
                     dtype)
        if _transform_flops(c) <= 0.5 * _transform_flops(listed()[5]):
            del c["name"]
            return c


# ------------------------------------------------------------------ inputs
def _planted(n_a, n_inner, n_b, K, dtype, seed):
    """AT (n_inner x n_a), B (n_inner x n_b): noise plus K planted pairs."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dt = torch.float32 if dtype == "float32" else torch.float64
    AT = torch.randn((n_inner, n_a), generator=g, device="cuda", dtype=dt) * SIGMA
    B = torch.randn((n_inner, n_b), generator=g, device="cuda", dtype=dt) * SIGMA
    r = np.random.default_rng(int(seed))
    K = min(K, n_a, n_inner, n_b)
    k, i, j = (torch.as_tensor(r.choice(n, size=K, replace=False), device="cuda") for n in (n_inner, n_a, n_b))
    AT[k, i] += BIG
    B[k, j] += BIG
    return AT, B


def _seeds(case, seed):
    """Input seed and hash seed of a state."""
    return int(seed) * 7919 + 1, int(seed) * 104729 + 9001


def _job_list(case, seed):
    """Products of a batch or a burst: the shapes are the case's, the contents
    and hash seeds the state's."""
    s_in, s_hash = _seeds(case, seed)
    out = []
    for i, s in enumerate(batch_shapes(count=case["count"], seed=case["shapes"], lo=case["lo"], hi=case["hi"])):
        AT, B = _planted(s["m"], s["n"], s["p"], s["K"], case["dtype"], s_in + 1009 * i)
        out.append({"AT": AT, "B": B, "d": s["d"], "b": s["b"], "seed": s_hash + 17 * i, "variant": s["variant"]})
    return out


def _inputs(case, seed):
    s_in, s_hash = _seeds(case, seed)
    if case["op"] == "wht":
        g = torch.Generator(device="cuda").manual_seed(s_in)
        return {"x": torch.randn((case["rows"], case["n"]), generator=g, device="cuda", dtype=torch.float32)}
    K = case.get("K", 0)
    AT, B = _planted(case["n_a"], case["n_inner"], case["n_b"], K, case["dtype"], s_in)
    return {"AT": AT, "B": B, "seed": s_hash}


def prepare(case, seed):
    st = {"case": case}
    if case["op"] == "batch":
        st["plan"] = BatchPlan(_job_list(case, seed), f32=True, tune=True, dense=True)
    elif case["op"] == "serve":
        st["jobs"] = [dict(q, AT=q["AT"].cpu().pin_memory(), B=q["B"].cpu().pin_memory())
                      for q in _job_list(case, seed)]
        st["server"] = Server(mem_cap_bytes=4 << 30, f32=True, streams=4, max_wave=32)
    else:
        st.update(_inputs(case, seed))
    if case["op"] == "dropin":
        for k in ("AT", "B"):
            h = aligned_empty(tuple(st[k].shape))
            h[...] = st[k].cpu().numpy()
            st[k] = h
        st["C"] = aligned_empty((case["n_a"], case["n_b"]))
        st["module"] = compmatmul_b200.load_dropin()
    elif case["op"] in ("matmul", "gemm"):
        st["C"] = torch.empty((case["n_a"], case["n_b"]), dtype=torch.float64, device="cuda")
    elif case["op"] == "wht":
        st["y"] = torch.empty_like(st["x"])
    return st


# -------------------------------------------------------------------- runs
def run(state):
    c = state["case"]
    op = c["op"]
    if op == "batch":
        state["plan"].run()
        return {"p": torch.cat([q["p"].flatten().float() for q in state["plan"].products]),
                "C": torch.cat([q["C"].flatten().float() for q in state["plan"].products])}
    if op == "serve":
        srv = state["server"]
        ids = [srv.submit(q["AT"], q["B"], q["d"], q["b"], q["seed"], q["variant"]) for q in state["jobs"]]
        return [srv.result(i).astype(np.float32) for i in ids]
    if op == "gemm":
        return device.gemm(state["AT"], state["B"], out=state["C"])
    if op == "wht":
        return device.wht_rows(state["x"], c["method"], out=state["y"])
    args = (c["d"], c["b"], state["seed"])
    if op == "dropin":
        f = state["module"].matmul_fft if c["variant"] == "fft" else state["module"].matmul_fwht
        f(state["C"], state["AT"], state["B"], *args, c["hash"])
        return state["C"]
    if op == "recover":
        s = Sketch.compute(state["AT"], state["B"], *args, variant=c["variant"], hash=c["hash"])
        return {"p": s.p, "top": s.topk(c["K"])}
    if op == "sketch":
        out = device.compressed_product(state["AT"], state["B"], *args, variant=c["variant"], hash=c["hash"])
    else:
        out = device.matmul(state["AT"], state["B"], *args, variant=c["variant"], hash=c["hash"], out=state["C"])
    return out.float() if c["dtype"] == "float32" else out


# -------------------------------------------------------------------- work
def _transform_flops(c):
    """d transform pairs per inner index (2.5 b log b flops per real FFT, b log b
    per WHT), pointwise products and scatter."""
    lg = math.log2(c["b"])
    per = 5 * c["b"] * lg + 4 * c["b"] if c["variant"] == "fft" else 2 * c["b"] * lg + 2 * c["b"]
    return c["d"] * c["n_inner"] * (per + c["n_a"] + c["n_b"])


def _sketch_work(c, dense, esz):
    """Inputs read once, the sketch (and the estimate) written once; the
    cheaper of d transforms per inner index, or the product once and d signed
    additions per entry."""
    nn = c["n_a"] * c["n_b"]
    by = esz * c["n_inner"] * (c["n_a"] + c["n_b"]) + 8 * c["d"] * c["b"] + (8 * nn if dense else 0)
    fl = min(_transform_flops(c), 2.0 * c["n_inner"] * nn + c["d"] * nn)
    return by, fl + (c["d"] * nn if dense else 0)


def work(case):
    op = case["op"]
    if op in ("batch", "serve"):
        by = fl = 0.0
        for s in batch_shapes(count=case["count"], seed=case["shapes"], lo=case["lo"], hi=case["hi"]):
            q = {"n_a": s["m"], "n_inner": s["n"], "n_b": s["p"], "b": s["b"], "d": s["d"], "variant": s["variant"]}
            x, y = _sketch_work(q, op == "batch", 4)
            by, fl = by + x, fl + y
        return {"bytes": by, "flops": fl}
    if op == "gemm":
        a, k, b = case["n_a"], case["n_inner"], case["n_b"]
        return {"bytes": 8.0 * (k * (a + b) + a * b), "flops": 2.0 * a * k * b}
    if op == "wht":
        n = case["rows"] * case["n"]
        return {"bytes": 8.0 * n, "flops": n * math.log2(case["n"])}
    by, fl = _sketch_work(case, op in ("matmul", "dropin"), 4 if case["dtype"] == "float32" else 8)
    if op == "recover":  # the estimates are formed and compared, not stored
        fl += (case["d"] + 1) * case["n_a"] * case["n_b"]
    return {"bytes": by, "flops": fl}


# ------------------------------------------------- the same in 64 bits, plainly
_M64 = (1 << 64) - 1


def _stream(seed):
    """xoshiro256** seeded by splitmix64: the reference's random stream."""
    s, x = [], seed & _M64
    for _ in range(4):
        x = (x + 0x9E3779B97F4A7C15) & _M64
        z = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & _M64
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _M64
        s.append(z ^ (z >> 31))
    while True:
        r = (s[1] * 5) & _M64
        yield (((r << 7) | (r >> 57)) * 9) & _M64
        t = (s[1] << 17) & _M64
        s[2] ^= s[0]
        s[3] ^= s[1]
        s[1] ^= s[2]
        s[0] ^= s[3]
        s[2] ^= t
        s[3] = ((s[3] << 45) | (s[3] >> 19)) & _M64


def _hash_words(kind, d, seed, n):
    """d x n hash words (top bits are the bucket or the sign) of keys 0..n-1."""
    r, key, out = _stream(seed), np.arange(n, dtype=np.uint64), []
    for _ in range(d):
        if kind == "multiply shift":
            a = next(r)
            while a & 1 == 0:
                a = next(r)
            out.append(np.uint64(a) * key)
        elif kind == "multiply add shift":
            a, b = next(r), next(r)
            out.append(np.uint64(a) * key + np.uint64(b))
        else:  # tabulation8: four byte tables
            T = np.array([next(r) & 0xFFFFFFFF for _ in range(1024)], dtype=np.uint64).reshape(4, 256)
            k = key.astype(np.int64)
            h = T[0][k & 255] ^ T[1][(k >> 8) & 255] ^ T[2][(k >> 16) & 255] ^ T[3][(k >> 24) & 255]
            out.append(h << np.uint64(32))
    return np.stack(out)


def _buckets_signs(kind, d, b, seed, side, n):
    h = _hash_words(kind, d, seed + side, n) >> np.uint64(64 - (b.bit_length() - 1))
    s = _hash_words(kind, d, seed + 2 + side, n) >> np.uint64(63)
    return (torch.as_tensor(h.astype(np.int64), device="cuda"),
            torch.as_tensor(s.astype(np.float64) * 2 - 1, device="cuda"))


def _exact(AT, B, d, b, seed, variant, kind, dense):
    """p_t[idx] = sum over (i, j) of s1 s2 (A B)[i][j], and the median estimates."""
    AT, B = AT.double(), B.double()
    n_a, n_b = AT.shape[1], B.shape[1]
    h1, s1 = _buckets_signs(kind, d, b, seed, 0, n_a)
    h2, s2 = _buckets_signs(kind, d, b, seed, 1, n_b)
    p = torch.zeros((d, b), dtype=torch.float64, device="cuda")
    rows = max(1, (1 << 25) // n_b)

    def where(t, i0, i1):
        x, y = h1[t, i0:i1, None], h2[t, None, :]
        return ((x + y) & (b - 1)) if variant == "fft" else (x ^ y)

    for i0 in range(0, n_a, rows):
        i1 = min(n_a, i0 + rows)
        C = AT[:, i0:i1].t() @ B
        for t in range(d):
            v = C * s1[t, i0:i1, None] * s2[t, None, :]
            p[t].index_add_(0, where(t, i0, i1).flatten(), v.flatten())
    if not dense:
        return p, None
    E = torch.empty((n_a, n_b), dtype=torch.float64, device="cuda")
    rows = max(1, rows // 8)
    for i0 in range(0, n_a, rows):
        i1 = min(n_a, i0 + rows)
        v = torch.stack([p[t][where(t, i0, i1)] * s1[t, i0:i1, None] * s2[t, None, :] for t in range(d)])
        E[i0:i1] = v.sort(dim=0).values[d // 2]
    return p, E


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        both = [_exact(q["AT"], q["B"], q["d"], q["b"], q["seed"], q["variant"], "multiply add shift", True)
                for q in _job_list(case, seed)]
        return {"p": torch.cat([p.flatten() for p, _ in both]), "C": torch.cat([e.flatten() for _, e in both])}
    if op == "serve":
        return [_exact(q["AT"], q["B"], q["d"], q["b"], q["seed"], q["variant"], "multiply add shift", False)[0].cpu()
                for q in _job_list(case, seed)]
    st = _inputs(case, seed)
    if op == "gemm":
        return st["AT"].t() @ st["B"]
    if op == "wht":
        y, n = st["x"].double(), case["n"]
        h = 1
        while h < n:
            y = y.view(-1, n // (2 * h), 2, h)
            y = torch.cat([y[:, :, :1] + y[:, :, 1:], y[:, :, :1] - y[:, :, 1:]], dim=2).view(-1, n)
            h *= 2
        return y
    p, E = _exact(st["AT"], st["B"], case["d"], case["b"], st["seed"], case["variant"], case["hash"],
                  op in ("matmul", "dropin"))
    if op == "recover":
        return {"p": p, "top": None}
    if op == "sketch":
        return p
    return E.cpu() if op == "dropin" else E
