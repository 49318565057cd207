"""The measured work of the engine: what its users have it do, through its public entry points.

Every case is one call pattern of README / INTEGRATION over the sizes the engine serves:

  mertens   one exact M(X) (Engine.mertens): table build, planning, S1/S2 sums, result
            read back -- from X = 10^6, where launches and the host path are the time, to
            X = 10^17, under each parameter policy a caller can choose (the reference's
            default, its dense and its streamed-table parameters, the B200 policy)
  stream    the same for a table above the context's resident limit (built in bands)
  batch     many uneven M(X) in one call (Engine.mertens_batch), with the default
            parameters or with one shared table as the batch autotuner writes them
  read      a Mertens / Mobius table for the caller: Engine.table_build + table_read
  noalloc   the table build into the caller's own device buffers (dr_table_build_noalloc)
  train     full-batch training of the learned parameter tuner's network (MLP.train)

Seeds move the inputs (X, table limits, weights, examples) within a case's size.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deleglise-rivat_b200"))
import dr_b200  # noqa: E402

POLICIES = {
    "reference": dr_b200.POLICY_REFERENCE,
    "dense": dr_b200.POLICY_DENSE,
    "compressed": dr_b200.POLICY_COMPRESSED,
    "b200": dr_b200.POLICY_GPU,
}


def listed():
    return [
        # compute_mertens(X) as a drop-in caller makes it, answered from a table of X values: latency
        {"name": "m1e6_default", "kind": "mertens", "X": 10**6, "policy": "reference"},
        # a small X with outer terms: every kernel of the path, hardly any work in each
        {"name": "m1e9_default", "kind": "mertens", "X": 10**9, "policy": "reference"},
        # the plain dense engine (MERTENS_USE_CHMT=0 parameters) at 10^12: int16 prefix only
        {"name": "m1e12_dense", "kind": "mertens", "X": 10**12, "policy": "dense"},
        # the streamed-table parameters of the reference at 10^15: dense prefix + bit planes
        {"name": "m1e15_compressed", "kind": "mertens", "X": 10**15, "policy": "compressed"},
        # the headline query, with the policy a B200 user picks
        {"name": "m1e16_b200", "kind": "mertens", "X": 10**16, "policy": "b200"},
        # the largest single query
        {"name": "m1e17_b200", "kind": "mertens", "X": 10**17, "policy": "b200"},
        # a table above the resident limit, streamed in bands (6e9 of 2.27e10 values resident)
        {"name": "m1e16_streamed", "kind": "stream", "X": 10**16, "resident": 6 * 10**9, "band": 5 * 10**9},
        # a few small queries in one call, default parameters
        {"name": "batch32_default", "kind": "batch", "count": 32, "lo": 9.0, "hi": 12.0, "u": 0, "cx": 0.0},
        # 256 uneven queries on one shared table, as the batch autotuner sets it up
        {"name": "batch256_tuned", "kind": "batch", "count": 256, "lo": 9.0, "hi": 14.0, "u": 8600000000, "cx": 1.4},
        # a caller that wants M(n) and mu(n) themselves
        {"name": "read_3e6", "kind": "read", "u": 3000000, "dense": 1000000},
        # a table in the caller's own device memory
        {"name": "noalloc_2e9", "kind": "noalloc", "u": 2000000000, "dense": 128000000},
        # the tuner's training set: 305 (features -> parameters) examples
        {"name": "train_305", "kind": "train", "examples": 305, "steps": 100},
    ]


def _log(rng, lo, hi):
    return int(round(10 ** rng.uniform(math.log10(lo), math.log10(hi))))


def draw(rng):
    kind = rng.choice(["mertens"] * 6 + ["stream", "batch", "batch", "read", "noalloc", "train"])
    if kind == "mertens":
        policy = rng.choice(["reference", "reference", "dense", "compressed", "b200", "b200"])
        hi = {"reference": 10**16, "dense": 10**14, "compressed": 10**16, "b200": 8 * 10**16}[policy]
        lo = {"reference": 10**6, "dense": 10**8, "compressed": 10**10, "b200": 10**10}[policy]
        return {"kind": kind, "X": _log(rng, lo, hi), "policy": policy}
    if kind == "stream":
        X = _log(rng, 10**14, 2 * 10**16)
        u = dr_b200.default_params(X, dr_b200.POLICY_GPU).u_total
        return {"kind": kind, "X": X, "resident": int(u * rng.uniform(0.25, 0.7)), "band": int(u * rng.uniform(0.1, 0.4))}
    if kind == "batch":
        tuned = rng.random() < 0.5
        lo = rng.uniform(8.0, 10.0)
        hi = lo + rng.uniform(1.0, 4.0)
        u = int(dr_b200.default_params(int(10**hi), dr_b200.POLICY_GPU).u_total * rng.uniform(1.0, 4.0)) if tuned else 0
        return {"kind": kind, "count": _log(rng, 4, 400), "lo": lo, "hi": hi, "u": u,
                "cx": rng.choice([1.2, 1.4, 1.7]) if tuned else 0.0}
    if kind == "read":
        u = _log(rng, 10**5, 10**7)
        return {"kind": kind, "u": u, "dense": int(u * rng.choice([0.25, 0.5, 1.0]))}
    if kind == "noalloc":
        u = _log(rng, 10**7, 5 * 10**9)
        return {"kind": kind, "u": u, "dense": int(u * rng.uniform(0.02, 0.3))}
    return {"kind": kind, "examples": _log(rng, 32, 1000), "steps": _log(rng, 20, 300)}


def _query(case, seed):
    """The X and parameters of a single-query case: X within 1% below the case's."""
    rng = np.random.default_rng([seed, 1])
    X = case["X"] - int(rng.integers(1, max(2, case["X"] // 100)))
    policy = POLICIES["b200" if case["kind"] == "stream" else case["policy"]]
    return X, dr_b200.default_params(X, policy)


def _batch(case, seed):
    rng = np.random.default_rng([seed, 2])
    xs = [int(round(10**v)) for v in rng.uniform(case["lo"], case["hi"], size=case["count"])]
    if not case["u"]:
        return xs, None
    # one table for all queries, every endpoint inside it (the shape dr_autotune_batch writes)
    u = (max(case["u"], 10**6) + 255) // 256 * 256
    top = max(xs)
    a_max = int(case["cx"] * math.sqrt(top)) + 1000
    n_max = top // u + 1000
    dense = min(u, max((a_max + 255) // 256 * 256, min(128000000, (u // 4 + 255) // 256 * 256)))
    p = dr_b200.Params(u_total=u, u_dense=dense, cx=case["cx"], mu_limit=min(u, max(a_max, n_max)),
                       segment_log2=18, block_threads=1024, chunk_log2=0)
    return xs, [p] * len(xs)


def _limits(case, seed):
    """Table limits: the case's, less a seeded part of a thousand values."""
    rng = np.random.default_rng([seed, 3])
    cut = int(rng.integers(1, 1000))
    u = case["u"] - cut
    dense = min(u, max(0, case["dense"] - cut - int(rng.integers(0, 64))))
    return u, dense


def _examples(case, seed):
    """Features as the tuner sees them (X, budget) and smooth targets near its outputs."""
    rng = np.random.default_rng([seed, 4])
    n = case["examples"]
    x = np.stack([dr_b200.tuner_features(int(10 ** rng.uniform(10, 16)), int(2 ** rng.uniform(33, 37.3)))
                  for _ in range(n)]).astype(np.float32)
    t = np.stack([0.3 * x[:, 0] + 0.1, -0.4 * x[:, 1] * x[:, 0], 0.5 * x[:, 1] - 0.2,
                  np.tanh(2 * x[:, 0])], 1) + 0.02 * rng.standard_normal((n, 4))
    a = [math.sqrt(6 / 4), math.sqrt(6 / 64), 0.1 * math.sqrt(6 / 64)]
    z = np.zeros
    w = np.concatenate([a[0] * rng.uniform(-1, 1, 256), z(64), a[1] * rng.uniform(-1, 1, 4096), z(64),
                        a[2] * rng.uniform(-1, 1, 256), z(4)])
    return x, t.astype(np.float32), w.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("mertens", "stream"):
        s["engine"] = dr_b200.Engine(0)
        s["X"], s["params"] = _query(case, seed)
        if kind == "stream":
            s["engine"].set_resident_limit(case["resident"], case["band"])
    elif kind == "batch":
        s["engine"] = dr_b200.Engine(0)
        s["xs"], s["params"] = _batch(case, seed)
    elif kind == "read":
        s["engine"] = dr_b200.Engine(0)
        s["u"], s["dense"] = _limits(case, seed)
        s["count"] = case["u"] - 1000
        s["first"] = s["u"] - s["count"] + 1
    elif kind == "noalloc":
        s["u"], s["dense"] = u, dense = _limits(case, seed)
        s["mu"] = min(u, 10 * math.isqrt(u))
        # buffers with room for every seed's limits, as a pool hands them out
        words = (case["u"] - max(0, case["dense"] - 1064) + 63) // 64 + 1
        s["dM"] = torch.zeros(case["dense"] + 8, dtype=torch.int16, device="cuda")
        s["planes"] = torch.zeros(2 * words, dtype=torch.int64, device="cuda")
        s["ckpt"] = torch.zeros(words, dtype=torch.int32, device="cuda")
        s["wheel"] = torch.zeros(4 * (10 * math.isqrt(case["u"]) // 192 + 3), dtype=torch.int32, device="cuda")
    else:
        s["engine"] = dr_b200.Engine(0)
        s["mlp"] = dr_b200.MLP(s["engine"], seed=1)
        s["x"], s["t"], s["w"] = _examples(case, seed)
        s["steps"] = case["steps"]
    return s


def _i64(v):
    """An unsigned 64-bit checksum as the int64 of the same bits."""
    return v - 2**64 if v >= 2**63 else v


def run(s):
    kind = s["kind"]
    if kind in ("mertens", "stream"):
        r = s["engine"].mertens(s["X"], s["params"])
        return [r.M, _i64(r.stats.C), _i64(r.stats.S1), _i64(r.stats.S2)]
    if kind == "batch":
        out, _ = s["engine"].mertens_batch(s["xs"], s["params"])
        return np.array(out, dtype=np.int64)
    if kind == "read":
        s["engine"].table_build(s["u"], s["dense"], s["u"])
        M, mu = s["engine"].table_read(s["first"], s["count"])
        return {"M": M, "mu": mu}
    if kind == "noalloc":
        p = ctypes.c_void_p
        rc = dr_b200.lib().dr_table_build_noalloc(
            0, p(torch.cuda.current_stream().cuda_stream), s["u"], s["dense"], s["mu"], p(s["dM"].data_ptr()),
            p(s["planes"].data_ptr()), p(s["ckpt"].data_ptr()), p(s["wheel"].data_ptr()))
        if rc:
            raise dr_b200.DRError(rc, dr_b200.lib().dr_last_error().decode())
        return {"dM": s["dM"], "planes": s["planes"], "ckpt": s["ckpt"], "wheel": s["wheel"]}
    s["mlp"].set_weights(s["w"])
    loss = s["mlp"].train(s["x"], s["t"], s["steps"])
    return {"loss": loss, "weights": s["mlp"].get_weights()}


def _table_bytes(u, dense, mu):
    return 2.0 * dense + 0.3125 * (u - dense) + mu / 4.0


def _sums(X, u, cx):
    """Quotients of the S1 and S2 sums (lookups plus summands), from the lengths of their ranges:
    sum over squarefree k <= N = X/u coprime to 6 of sqrt(X/k)/cx divisors and cx sqrt(X/k) wheel values."""
    if X <= u:
        return 0.0, 0.0
    r = math.sqrt(float(X) * max(1.0, X / u))
    return 0.57 * r / cx, 0.27 * r * cx


def work(case):
    """Bytes: the table written once, and read once by the sums.  Operations: two (multiply and
    add) per quotient of the sums; for a table alone its values times the average number of
    prime factors, for the network the products of its passes."""
    kind = case["kind"]
    if kind in ("mertens", "stream"):
        p = dr_b200.default_params(case["X"], POLICIES["b200" if kind == "stream" else case["policy"]])
        s1, s2 = _sums(case["X"], p.u_total, p.cx)
        return {"bytes": 2.0 * _table_bytes(p.u_total, p.u_dense, p.mu_limit), "flops": 2.0 * (s1 + s2)}
    if kind == "batch":
        xs, ps = _batch(case, 0)
        ps = ps or [dr_b200.default_params(x) for x in xs]
        sums = sum(sum(_sums(x, p.u_total, p.cx)) for x, p in zip(xs, ps))
        u, d, m = (max(getattr(p, k) for p in ps) for k in ("u_total", "u_dense", "mu_limit"))
        return {"bytes": 2.0 * _table_bytes(u, d, m), "flops": 2.0 * sums}
    if kind == "read":
        return {"bytes": 2.0 * _table_bytes(case["u"], case["dense"], case["u"]) + 5.0 * case["u"],
                "flops": 3.0 * case["u"]}
    if kind == "noalloc":
        return {"bytes": _table_bytes(case["u"], case["dense"], 10 * math.isqrt(case["u"])), "flops": 3.0 * case["u"]}
    per = 2.0 * (4 * 64 + 64 * 64 + 64 * 4)
    return {"bytes": 8.0 * 4740 + 32.0 * case["examples"], "flops": 3.0 * per * case["examples"] * case["steps"]}


# --- the same results from plain numpy -------------------------------------------------


def _mobius(n):
    """mu(0..n) as int8: sign flips at the primes, zeros at their squares."""
    mu = np.ones(n + 1, dtype=np.int8)
    mu[0] = 0
    flag = np.ones(n + 1, dtype=bool)
    flag[:2] = False
    for p in range(2, n + 1):
        if p > n // p:
            break
        if flag[p]:
            flag[p * p::p] = False
    left = np.arange(n + 1, dtype=np.int64)  # what the primes up to sqrt(n) leave of n
    for p in np.flatnonzero(flag[: math.isqrt(n) + 1]):
        p = int(p)
        mu[p::p] *= -1
        mu[p * p::p * p] = 0
        q = p
        while q <= n:
            left[q::q] //= p
            q *= p
    mu[left > 1] *= -1
    return mu


def _mertens(X):
    """M(X) by the hyperbola recursion over the values floor(X/i)."""
    small = max(2, int(round(X ** (2.0 / 3.0))))
    M = np.cumsum(_mobius(small).astype(np.int64))
    if X <= small:
        return int(M[X])
    top = X // (small + 1)
    big = np.zeros(top + 1, dtype=np.int64)  # M(X // i)
    for i in range(top, 0, -1):
        y = X // i
        r = math.isqrt(y)
        d = np.arange(2, y // (r + 1) + 1, dtype=np.int64)
        near = d[d * i <= top]
        total = int(big[near * i].sum()) + int(M[y // d[len(near):]].sum())
        q = np.arange(1, r + 1, dtype=np.int64)
        total += int((M[q] * (y // q - y // (q + 1))).sum())
        big[i] = 1 - total
    return int(big[1])


def _train(case, seed):
    x, t, w = (v.astype(np.float64) for v in _examples(case, seed))
    cut = np.cumsum([256, 64, 4096, 64, 256])
    m, v = np.zeros_like(w), np.zeros_like(w)
    loss = 0.0
    b1, b2, eps, lr = (float(np.float32(k)) for k in (0.9, 0.999, 1e-8, 3e-3))
    c1, c2 = (float(np.float32(1) - np.float32(k)) for k in (0.9, 0.999))
    for step in range(1, case["steps"] + 1):
        W1, c_1, W2, c_2, W3, c_3 = np.split(w, cut)
        W1, W2, W3 = W1.reshape(64, 4), W2.reshape(64, 64), W3.reshape(4, 64)
        h1 = np.maximum(x @ W1.T + c_1, 0.0)
        h2 = np.maximum(h1 @ W2.T + c_2, 0.0)
        e = h2 @ W3.T + c_3 - t
        loss = float(np.mean(e * e))
        dy = 2.0 * e / e.size
        d2 = (dy @ W3) * (h2 > 0)
        d1 = (d2 @ W2) * (h1 > 0)
        g = np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), (dy.T @ h2).ravel(),
                            dy.sum(0)])
        m = b1 * m + c1 * g
        v = b2 * v + c2 * g * g
        w = w - lr * (m / (1 - b1**step)) / (np.sqrt(v / (1 - b2**step)) + eps)
    return {"loss": loss, "weights": w}


def exact(case, seed):
    kind = case["kind"]
    if kind == "mertens":
        X, _ = _query(case, seed)
        return [_mertens(X), None, None, None] if X <= 10**10 else None
    if kind == "read":
        u, _ = _limits(case, seed)
        count = case["u"] - 1000
        mu = _mobius(u)
        M = np.cumsum(mu.astype(np.int64)).astype(np.int32)
        return {"M": M[u - count + 1:], "mu": mu[u - count + 1:]}
    if kind == "train":
        return _train(case, seed)
    return None
