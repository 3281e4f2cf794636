"""Performance cases of the library: what its users run, through the public entry points, over the range they run it in.

Each kind of case below says which use it stands for. All device work goes through one context, as in a program that
serves one GPU; weights, codes and models are made from the seed and stay on the device (or, for the entries that take
host pointers, in host memory) between calls, the way a user's program keeps them.
"""
import ctypes as C
import math
import weakref

import numpy as np
import torch

from libinferbit_b200 import Backend, LinearT, PqT
from libinferbit_b200 import _ffi

_shared = {}


def _backend():
    if "be" not in _shared:
        _shared["be"] = Backend(0)
    return _shared["be"]


def _host():
    if "host" not in _shared:
        host = _ffi.load_host()
        if host.ib_b200_init(0) != 0:
            raise RuntimeError(host.ib_b200_last_error().decode())
        _shared["host"] = host
    return _shared["host"]


def _check(rc):
    if rc != 0:
        _backend()._check(rc)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _bytes(g, *shape):
    return torch.randint(0, 256, shape, generator=g, device="cuda", dtype=torch.uint8)


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)


def _half(g, lo, hi, *shape):
    return (torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo).to(torch.float16)


def _out(*shape, dtype=torch.float32):
    return torch.zeros(shape, device="cuda", dtype=dtype)


def listed():
    return [
        # one call of the reference-shaped kernel table, host vectors in and out: the TinyLlama up projection
        {"name": "table int4 5632x2048", "kind": "table", "bits": 4, "M": 5632, "N": 2048, "B": 1},
        # INT8 attention projections of Mistral-7B shape over sixteen layers: one token, and sixteen at once
        {"name": "attention int8 b1", "kind": "attention", "bits": 8, "hidden": 4096, "kv": 1024, "layers": 16, "B": 1},
        {"name": "attention int8 b16", "kind": "attention", "bits": 8, "hidden": 4096, "kv": 1024, "layers": 16, "B": 16},
        # INT4 weights times INT8-quantised activations (the reference's default for INT4 tensors): the MLP of a 7B layer
        {"name": "mlp w4a8 b1", "kind": "mlp_w4a8", "hidden": 4096, "inter": 14336, "layers": 8, "B": 1},
        # product-quantised down projection of every layer: one token, and eight at once
        {"name": "pq down b1", "kind": "pq", "M": 4096, "N": 14336, "G": 16, "K": 256, "K2": 0, "outliers": 0, "tensors": 24, "B": 1},
        {"name": "pq down b8", "kind": "pq", "M": 4096, "N": 14336, "G": 16, "K": 256, "K2": 0, "outliers": 0, "tensors": 24, "B": 8},
        # candidates for the next token from a two-level product-quantised LM head
        {"name": "pq lm head top 64", "kind": "pq_topk", "M": 32000, "N": 4096, "G": 16, "K": 256, "K2": 16, "top": 64},
        # one token through group-scaled INT4 matrices
        {"name": "int4 groups 14336x4096", "kind": "int4g", "M": 14336, "N": 4096, "G": 128, "tensors": 8},
        # codebook training: resident points with chunks of eight values, and a converter's call with host arrays
        {"name": "kmeans 4M x 8", "kind": "kmeans", "points": 1 << 22, "D": 8, "K": 256, "iters": 10},
        {"name": "kmeans host 262147 x 4", "kind": "kmeans_host", "points": 262147, "D": 4, "K": 256, "iters": 10},
        # Mistral-7B shape: the next token after 512, and a prompt of 64 tokens into an empty cache
        {"name": "decode 7b", "kind": "model", "hidden": 4096, "inter": 14336, "layers": 32, "heads": 32, "kv_heads": 8, "vocab": 32000,
         "attn_bits": 8, "mlp_bits": 4, "head_bits": 8, "pos": 512, "tokens": 1},
        {"name": "prompt 7b", "kind": "model", "hidden": 4096, "inter": 14336, "layers": 32, "heads": 32, "kv_heads": 8, "vocab": 32000,
         "attn_bits": 8, "mlp_bits": 4, "head_bits": 8, "pos": 0, "tokens": 64},
    ]


def _between(rng, lo, hi, step=1):
    """a multiple of step, spread over the logarithm of [lo, hi]"""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["table", "attention", "mlp_w4a8", "pq", "pq_topk", "int4g", "kmeans", "kmeans_host", "model", "model"])
    if kind == "table":
        bits = rng.choice([4, 8])
        return {"kind": kind, "bits": bits, "M": _between(rng, 256, 14336), "N": _between(rng, 1024, 8192, 32),
                "B": 1 if bits == 4 else rng.choice([1, 1, _between(rng, 2, 8)])}
    if kind == "attention":
        hidden = _between(rng, 1024, 5120, 128)
        return {"kind": kind, "bits": rng.choice([8, 8, 4]), "hidden": hidden, "kv": max(128, hidden // rng.choice([1, 4, 8]) // 64 * 64),
                "layers": rng.randint(8, 16), "B": _between(rng, 1, 32)}
    if kind == "mlp_w4a8":
        hidden = _between(rng, 1024, 5120, 128)
        return {"kind": kind, "hidden": hidden, "inter": _between(rng, 2 * hidden, 4 * hidden, 128), "layers": rng.randint(4, 8), "B": _between(rng, 1, 8)}
    if kind == "pq":
        G = rng.choice([16, 16, 8, 32])
        n_out = rng.choice([0, 0, 0, 32])
        K2 = rng.choice([0, 0, 0, 16, 256])
        return {"kind": kind, "M": _between(rng, 1024, 14336), "N": _between(rng, 1024, 14336 if G > 8 else 8192, G) + n_out, "G": G,
                "K": rng.choice([256, 256, 128]), "K2": K2, "outliers": n_out, "tensors": rng.randint(8, 16), "B": _between(rng, 1, 16)}
    if kind == "pq_topk":
        return {"kind": kind, "M": _between(rng, 8000, 64000), "N": _between(rng, 1024, 4096, 16), "G": 16, "K": 256,
                "K2": rng.choice([0, 16, 256]), "top": _between(rng, 8, 256)}
    if kind == "int4g":
        G = rng.choice([128, 128, 64, 32])
        return {"kind": kind, "M": _between(rng, 1024, 14336), "N": _between(rng, 1024, 14336, 128), "G": G, "tensors": rng.randint(4, 12)}
    if kind == "kmeans":
        D, K = rng.choice([8, 8, 4, 16]), rng.choice([256, 256, 128, 200, 64])
        most = (1 << 22) * 8 * 256 // (D * K)
        return {"kind": kind, "points": _between(rng, 50000, min(most, 1 << 22) // (2 if D == 16 else 1)), "D": D, "K": K, "iters": rng.randint(4, 10)}
    if kind == "kmeans_host":
        return {"kind": kind, "points": _between(rng, 20000, 600000), "D": rng.choice([4, 8, 8, 16]), "K": rng.choice([256, 256, 128, 16]),
                "iters": rng.randint(4, 10)}
    heads = rng.choice([8, 16, 20, 24, 32])
    hidden = 128 * heads
    return {"kind": "model", "hidden": hidden, "inter": _between(rng, 2 * hidden, int(3.5 * hidden), 128), "layers": rng.randint(4, 24), "heads": heads,
            "kv_heads": heads // rng.choice([1, 4]), "vocab": _between(rng, 8000, 32000), "attn_bits": rng.choice([8, 8, 4]),
            "mlp_bits": rng.choice([4, 4, 8]), "head_bits": 8, "pos": _between(rng, 1, 1024) - 1,
            "tokens": rng.choice([1, 1, _between(rng, 2, 64)])}


# ── calls of the kernel table: host vectors, weights registered once like the mapping of a model file ──
def _table_prepare(case, seed):
    host, rng = _host(), np.random.default_rng(seed)
    M, N, B, bits = case["M"], case["N"], case["B"], case["bits"]
    w = np.frombuffer(rng.bytes(M * N * bits // 8), np.uint8)
    scales = rng.uniform(0.002, 0.02, M).astype(np.float32) if bits == 4 else rng.uniform(0.001, 0.01, M).astype(np.float32)
    x = rng.standard_normal((B, N)).astype(np.float32)
    out = np.zeros((B, M), np.float32)
    if host.ib_b200_register(w.ctypes.data, w.nbytes) != 0:
        raise RuntimeError(host.ib_b200_last_error().decode())
    p = (out.ctypes.data, w.ctypes.data, scales.ctypes.data, x.ctypes.data, M, N)
    if bits == 4:
        call, args = host.ib_b200_matmul_int4, p
    elif B == 1:
        call, args = host.ib_b200_matmul_int8, p
    else:
        call, args = host.ib_b200_matmul_int8_batch, p + (B, M)
    state = _State(call=call, args=args, out=out, keep=(w, scales, x))
    weakref.finalize(state, lambda a=w: host.ib_b200_unregister(a.ctypes.data))
    return state


def _table_run(s):
    s.call(*s.args)
    if _shared["host"].ib_b200_status() != 0:
        raise RuntimeError(_shared["host"].ib_b200_last_error().decode())
    return s.out


class _State:
    def __init__(self, **kw):
        self.__dict__.update(kw)


def _calls_run(s):
    for fn, args in s.calls:
        rc = fn(*args)
        if rc != 0:
            _check(rc)
    return s.out


# ── attention projections: q, k, v share an activation and a launch, o follows ──
def _attention_prepare(case, seed):
    be, g = _backend(), _gen(seed)
    H, kv, L, B, bits = case["hidden"], case["kv"], case["layers"], case["B"], case["bits"]
    lo = 0.001 if bits == 8 else 0.002
    x, att = _normal(g, L, B, H), _normal(g, L, B, H)
    out = {"q": _out(L, B, H), "k": _out(L, B, kv), "v": _out(L, B, kv), "o": _out(L, B, H)}
    rows = {"q": H, "k": kv, "v": kv, "o": H}
    w = {n: _bytes(g, L, r, H * bits // 8) for n, r in rows.items()}
    sc = {n: _half(g, lo, 10 * lo, L, r) for n, r in rows.items()}
    calls = []
    for i in range(L):
        t = {n: LinearT(w[n][i].data_ptr(), sc[n][i].data_ptr(), out[n][i].data_ptr(), r, r, 0, 0) for n, r in rows.items()}
        calls.append((be.lib.ibcu_linear, (be.ctx, (LinearT * 3)(t["q"], t["k"], t["v"]), 3, x[i].data_ptr(), H, B, bits)))
        calls.append((be.lib.ibcu_linear, (be.ctx, (LinearT * 1)(t["o"]), 1, att[i].data_ptr(), H, B, bits)))
    return _State(calls=calls, out=out, keep=(x, att, w, sc))


# ── the MLP of a layer on the INT4 x INT8 route: gate and up, silu(gate) * up, down ──
def _mlp_prepare(case, seed):
    be, g = _backend(), _gen(seed)
    H, I, L, B = case["hidden"], case["inter"], case["layers"], case["B"]
    rows, cols = {"gate": I, "up": I, "down": H}, {"gate": H, "up": H, "down": I}
    w = {n: _bytes(g, L, rows[n], cols[n] // 2) for n in rows}
    sc = {n: _half(g, 0.0002, 0.002, L, rows[n]) for n in rows}
    x = _normal(g, L, B, H)
    out = {"gate": _out(L, B, I), "up": _out(L, B, I), "hidden": _out(L, B, I), "down": _out(L, B, H)}
    calls = []
    for i in range(L):
        for n in ("gate", "up", "down"):
            t = (LinearT * 1)(LinearT(w[n][i].data_ptr(), sc[n][i].data_ptr(), out[n][i].data_ptr(), rows[n], rows[n], 0, 0))
            src = out["hidden"][i] if n == "down" else x[i]
            if n == "down":
                calls.append((be.lib.ibcu_silu_mul, (be.ctx, out["hidden"][i].data_ptr(), out["gate"][i].data_ptr(), out["up"][i].data_ptr(), B * I)))
            calls.append((be.lib.ibcu_linear_w4a8_fp32, (be.ctx, t, src.data_ptr(), cols[n], B)))
    return _State(calls=calls, out=out, keep=(x, w, sc))


# ── product-quantised tensors, prepared once ──
def _pq_tensor(be, g, case, cb, cb2):
    M, N, G, K, K2, n_out = case["M"], case["N"], case["G"], case["K"], case["K2"], case.get("outliers", 0)
    Cn = (N - n_out) // G
    t, keep = PqT(), []

    def put(v):
        keep.append(v)
        return v.data_ptr()
    t.M, t.N, t.G, t.K, t.K_l2, t.n_outlier, t.cb_chunk_stride = M, N, G, K, K2, n_out, 0
    t.codebook_l, t.codebook_r = put(cb[0]), put(cb[1])
    t.idx_l, t.idx_r = (put(torch.randint(0, K, (M, Cn), generator=g, device="cuda", dtype=torch.uint8)) for _ in range(2))
    t.row_scale = put(_half(g, 0.5, 2.0, M))
    if K2:
        t.codebook2_l, t.codebook2_r = put(cb2[0]), put(cb2[1])
        t.idx2_l, t.idx2_r = (put(_bytes(g, M, (Cn + 1) // 2) if K2 == 16 else torch.randint(0, K2, (M, Cn), generator=g, device="cuda", dtype=torch.uint8))
                              for _ in range(2))
    if n_out:
        t.outlier_cols = put(torch.randperm(N, generator=g, device="cuda")[:n_out].sort().values.to(torch.int32))
        t.outlier_sidecar = put(torch.randint(-127, 128, (M, n_out), generator=g, device="cuda", dtype=torch.int8))
        t.outlier_scale = put(_half(g, 0.001, 0.01, n_out))
    place = put(torch.empty(int(be.lib.ibcu_pq_prepared_bytes(C.byref(t))), device="cuda", dtype=torch.uint8))
    torch.cuda.synchronize()
    _check(be.lib.ibcu_pq_prepare(be.ctx, C.byref(t), place))
    return t, keep


def _codebooks(g, case):
    half = case["G"] // 2
    cb = [(_normal(g, case["K"], half) * 0.02).to(torch.float16) for _ in range(2)]
    cb2 = [(_normal(g, max(1, case["K2"]), half) * 0.004).to(torch.float16) for _ in range(2)]
    return cb, cb2


def _pq_prepare(case, seed):
    be, g = _backend(), _gen(seed)
    L, B = case["tensors"], case["B"]
    cb, cb2 = _codebooks(g, case)
    x, out = _normal(g, L, B, case["N"]), _out(L, B, case["M"])
    calls, keep = [], [x, cb, cb2]
    for i in range(L):
        t, k = _pq_tensor(be, g, case, cb, cb2)
        keep.append((t, k))
        calls.append((be.lib.ibcu_pq_matmul_fp32, (be.ctx, C.byref(t), x[i].data_ptr(), out[i].data_ptr(), B)))
    return _State(calls=calls, out=out, keep=keep)


def _topk_prepare(case, seed):
    be, g = _backend(), _gen(seed)
    cb, cb2 = _codebooks(g, case)
    x, out = _normal(g, case["N"]), {"logits": _out(case["top"]), "ids": _out(case["top"], dtype=torch.int32)}
    t, keep = _pq_tensor(be, g, case, cb, cb2)
    calls = [(be.lib.ibcu_pq_lm_head_topk, (be.ctx, C.byref(t), x.data_ptr(), case["top"], out["logits"].data_ptr(), out["ids"].data_ptr()))]
    return _State(calls=calls, out=out, keep=(x, t, keep, cb, cb2))


# ── INT4 rows with one scale per group of columns ──
def _int4g_prepare(case, seed):
    be, g = _backend(), _gen(seed)
    M, N, G, L = case["M"], case["N"], case["G"], case["tensors"]
    w, sc = _bytes(g, L, M, N // 2), _half(g, 0.002, 0.02, L, M, N // G)
    x, out = _normal(g, L, N), _out(L, M)
    calls = []
    for i in range(L):
        t = _ffi.Int4gT()
        t.M, t.N, t.G, t.K_out, t.q, t.s = M, N, G, 0, w[i].data_ptr(), sc[i].data_ptr()
        calls.append((be.lib.ibcu_int4g_matmul_fp32, (be.ctx, C.pointer(t), x[i].data_ptr(), out[i].data_ptr(), 0.0)))
    return _State(calls=calls, out=out, keep=(w, sc, x))


# ── k-means: Lloyd iterations from the first K points ──
def _kmeans_prepare(case, seed):
    be, g = _backend(), _gen(seed)
    n, D, K = case["points"], case["D"], case["K"]
    X = _normal(g, n, D) * 0.02
    first = X[:K].clone()
    out = {"centers": _out(K, D), "codes": _out(n, dtype=torch.int32), "dist": _out(n), "inertia": _out(1, dtype=torch.float64)}
    room = {"sums": _out(K, D), "counts": _out(K, dtype=torch.int32)}         # working tables of an iteration
    a = {k: v.data_ptr() for k, v in {**out, **room}.items()}
    calls = [(be.lib.ibcu_memcpy_d2d, (be.ctx, a["centers"], first.data_ptr(), K * D * 4))]
    calls += [(be.lib.ibcu_kmeans_lloyd_iter, (be.ctx, X.data_ptr(), n, D, a["centers"], K, a["codes"], a["dist"], a["sums"], a["counts"], a["inertia"]))] * case["iters"]
    return _State(calls=calls, out=out, keep=(X, first, room))


def _kmeans_host_prepare(case, seed):
    host = _host()
    n, D, K = case["points"], case["D"], case["K"]
    X = (np.random.default_rng(seed).standard_normal((n, D), dtype=np.float32) * np.float32(0.02))
    out = {"centers": np.zeros((K, D), np.float32), "codes": np.zeros(n, np.int32), "inertia": np.zeros(1, np.float64)}
    args = (X.ctypes.data, n, D, K, case["iters"], -1.0, out["centers"].ctypes.data, out["codes"].ctypes.data, out["inertia"].ctypes.data)
    return _State(X=X, out=out, args=args, K=K, iters=case["iters"])


def _kmeans_host_run(s):
    s.out["centers"][:] = s.X[:s.K]
    if _shared["host"].ib_b200_kmeans_lloyd(*s.args) != s.iters:
        raise RuntimeError(_shared["host"].ib_b200_last_error().decode())
    return s.out


# ── a model step: tokens in host memory, logits of the last one in host memory; longer prompts go through in groups of 32 positions ──
MAX_CTX, GROUP = 1152, 32


def _model_prepare(case, seed):
    be, host, rng = _backend(), _host(), np.random.default_rng(seed)
    cfg = _ffi.ModelCfg(case["hidden"], case["inter"], case["layers"], case["heads"], case["kv_heads"], case["hidden"] // case["heads"], case["vocab"],
                        MAX_CTX, 1e-5, 10000.0, case["attn_bits"], case["mlp_bits"], case["head_bits"])
    m = host.ib_b200_model_create(be.ctx, C.byref(cfg))
    if not m:
        raise RuntimeError("model allocation failed")
    tokens = rng.integers(0, case["vocab"], case["tokens"]).astype(np.int32)
    logits = np.zeros(case["vocab"], np.float32)
    state = _State(calls=[], out=logits, keep=tokens)
    weakref.finalize(state, host.ib_b200_model_free, m)
    _check(host.ib_b200_model_fill_random(m, seed + 1, case["pos"]))
    for done in range(0, case["tokens"], GROUP):
        n = min(GROUP, case["tokens"] - done)
        last = done + n == case["tokens"]
        state.calls.append((host.ib_b200_forward_step_last, (m, tokens.ctypes.data + 4 * done, case["pos"] + done, n, logits.ctypes.data if last else None)))
    return state


_PREPARE = {"table": _table_prepare, "attention": _attention_prepare, "mlp_w4a8": _mlp_prepare, "pq": _pq_prepare, "pq_topk": _topk_prepare,
            "int4g": _int4g_prepare, "kmeans": _kmeans_prepare, "kmeans_host": _kmeans_host_prepare, "model": _model_prepare}
_RUN = {"table": _table_run, "kmeans_host": _kmeans_host_run}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state.run = _RUN.get(case["kind"], _calls_run)
    torch.cuda.synchronize()                      # the library's stream does not wait for torch's
    return state


def run(state):
    return state.run(state)


def work(case):
    """bytes: weights, scales or codes and activations read once, results written once; flops: multiplications and additions of the products"""
    kind = case["kind"]
    if kind == "table":
        M, N, B = case["M"], case["N"], case["B"]
        return {"bytes": M * N * case["bits"] // 8 + 4 * M + 4 * B * (N + M), "flops": 2 * M * N * B}
    if kind == "attention":
        H, kv, L, B = case["hidden"], case["kv"], case["layers"], case["B"]
        rows = 2 * H + 2 * kv
        return {"bytes": L * (rows * H * case["bits"] // 8 + 2 * rows + 4 * B * (2 * H + rows)), "flops": 2 * L * rows * H * B}
    if kind == "mlp_w4a8":
        H, I, L, B = case["hidden"], case["inter"], case["layers"], case["B"]
        return {"bytes": L * (3 * H * I // 2 + 2 * (2 * I + H) + 4 * B * (2 * H + 3 * I)), "flops": 6 * L * H * I * B}
    if kind in ("pq", "pq_topk"):
        M, N, G, K2, n_out = case["M"], case["N"], case["G"], case["K2"], case.get("outliers", 0)
        L, B, Cn = case.get("tensors", 1), case.get("B", 1), (N - n_out) // G
        second = 0 if not K2 else (Cn + 1) // 2 * 2 if K2 == 16 else 2 * Cn      # bytes per row
        books = 2 * G * (case["K"] + K2)
        if kind == "pq_topk":                     # first level of every row, every level of the chosen rows
            return {"bytes": M * (2 * Cn + 2) + case["top"] * (2 * Cn + second + 8) + books + 4 * N, "flops": 2 * G * Cn * (case["K"] + K2) + 2 * Cn * M}
        levels = 2 if K2 else 1
        return {"bytes": L * (M * (2 * Cn + second + 2 + n_out) + 4 * B * (N + M)) + books,
                "flops": L * B * (2 * G * Cn * (case["K"] + K2) + 2 * Cn * M * levels + 2 * n_out * M)}
    if kind == "int4g":
        M, N, L = case["M"], case["N"], case["tensors"]
        return {"bytes": L * (M * N // 2 + 2 * M * N // case["G"] + 4 * (N + M)), "flops": 2 * L * M * N}
    if kind in ("kmeans", "kmeans_host"):
        n, D, K, it = case["points"], case["D"], case["K"], case["iters"]
        return {"bytes": it * n * D * 4 + n * (8 if kind == "kmeans" else 4) + 2 * K * D * 4, "flops": it * n * (2 * K * D + D)}
    H, I, L, n, kv = case["hidden"], case["inter"], case["layers"], case["tokens"], case["hidden"] // case["heads"] * case["kv_heads"]
    attn, mlp, head = 2 * H * (H + kv), 3 * H * I, case["vocab"] * H
    cache = 2 * L * 4 * kv * (case["pos"] + 2 * n)           # earlier positions read, new ones written and read
    return {"bytes": L * (attn * case["attn_bits"] + mlp * case["mlp_bits"]) // 8 + head * case["head_bits"] // 8 + cache + 4 * case["vocab"] + n * H,
            "flops": 2 * n * L * (attn + mlp) + 2 * head + 4 * n * L * H * (case["pos"] + n // 2 + 1)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("table", "attention", "pq", "int4g"):
        return {"rel": 1e-5}                      # sums of 32-bit products
    if kind == "pq_topk":
        return {"rel": 1e-5, "differ": 0.01}      # nearly equal logits may change places
    if kind == "mlp_w4a8":
        return {"rel": 1e-4}                      # integer sums, but a last-bit difference of silu can move an 8-bit rounding of one activation
    if kind in ("kmeans", "kmeans_host"):
        # sums in another order move the centroids by their last bits, over the iterations a few points in a million between two
        # clusters with them, and each of those moves the mean of a cluster of n points by about 1 / n of its width
        return {"rel": 1e-3, "max": 0.1, "differ": 1e-3}
    return {"rel": 1e-4}                          # last-bit differences of every layer's sums, carried through all layers
