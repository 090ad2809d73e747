"""The batched calls whose speed this library is kept to, as a program makes them.

Fixed-size batches go through the torch-facing functions of ``magma_b200.api`` (the caller
has tensors); variable-size batches go through the C ABI with pointer and size arrays that
the caller keeps, as a C program does. Routines that work in place are given a fresh copy of
the caller's matrices on every pass. ``listed`` has the library's own workloads with one
member at each end of the range; ``draw`` gives others of the same ranges, odd orders,
transposed and upper forms among them. Entries are seeded; sizes depend on the case alone.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from magma_b200 import api

DEV = "cuda"
LOWER, UPPER = 122, 121
LEFT, RIGHT = 141, 142


def listed():
    return [
        # a few small systems: the latency of one call (a quadrature point, a small block Jacobi)
        dict(name="gesv_64x8", op="gesv", n=8, batch=64, nrhs=1),
        # many small systems, one right-hand side (element-local problems)
        dict(name="gesv_10000x32", op="gesv", n=32, batch=10000, nrhs=1),
        # blocked orders in plain FP64, and the same systems in mixed precision
        dict(name="gesv_2048x256", op="gesv", n=256, batch=2048, nrhs=4),
        dict(name="dsgesv_2048x256", op="dsgesv", n=256, batch=2048, nrhs=4),
        # a request loop's micro-batch: orders log-uniform up to the largest it admits, up to 16 right-hand sides
        dict(name="gesv_v256", op="gesv_v", lo=8, hi=1024, batch=256, nrhs=16),
        # small products of mixed sizes (fronts of a sparse solver), both precisions
        dict(name="gemm_v20000_f64", op="gemm_v", dtype="f64", lo=8, hi=128, batch=20000, ta=False, tb=False),
        dict(name="gemm_v20000_f32", op="gemm_v", dtype="f32", lo=8, hi=128, batch=20000, ta=False, tb=False),
        # SPD systems, many small and few large orders, FP64; and FP32 factors with FP64 refinement
        dict(name="posv_v50000", op="posv_v", lo=4, hi=512, batch=50000, nrhs=8, upper=False),
        dict(name="dsposv_v10000", op="dsposv_v", lo=4, hi=512, batch=10000, nrhs=8),
        # triangular solves of mixed sizes
        dict(name="trsm_v20000", op="trsm_v", lo=8, hi=128, batch=20000, left=True, lower=True, trans=False),
        # QR of small square matrices
        dict(name="geqrf_10000x64", op="geqrf", m=64, n=64, batch=10000),
        # factor and invert (block preconditioners that keep inverses)
        dict(name="getri_10000x32", op="getri", n=32, batch=10000),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["gesv", "gesv", "dsgesv", "gesv_v", "gemm_v", "gemm_v", "posv_v", "dsposv_v", "trsm_v", "geqrf", "getri"])
    if op == "gesv":
        n = _log(rng, 8, 256)
        return dict(op=op, n=n, batch=_log(rng, 64, max(64, min(10000, int(2.0e10 / n ** 3)))), nrhs=rng.randint(1, 4))
    if op == "dsgesv":
        n = _log(rng, 96, 256)
        return dict(op=op, n=n, batch=_log(rng, 256, 2048), nrhs=rng.randint(1, 4))
    if op == "gesv_v":
        return dict(op=op, lo=8, hi=_log(rng, 128, 1024), batch=_log(rng, 64, 256), nrhs=rng.randint(1, 16))
    if op == "gemm_v":
        return dict(op=op, dtype=rng.choice(["f64", "f32"]), lo=8, hi=rng.randint(32, 128), batch=_log(rng, 2000, 20000),
                    ta=rng.random() < 0.25, tb=rng.random() < 0.25)
    if op == "posv_v":
        return dict(op=op, lo=4, hi=_log(rng, 64, 512), batch=_log(rng, 2000, 50000), nrhs=rng.randint(1, 8), upper=rng.random() < 0.25)
    if op == "dsposv_v":
        return dict(op=op, lo=4, hi=_log(rng, 64, 512), batch=_log(rng, 2000, 10000), nrhs=rng.randint(1, 8))
    if op == "trsm_v":
        return dict(op=op, lo=8, hi=rng.randint(32, 128), batch=_log(rng, 2000, 20000), left=rng.random() < 0.75,
                    lower=rng.random() < 0.75, trans=rng.random() < 0.25)
    if op == "geqrf":
        n = _log(rng, 16, 128)
        return dict(op=op, m=n + rng.choice([0, 0, rng.randint(0, n)]), n=n, batch=_log(rng, 1000, min(10000, int(2.6e9 / n ** 3))))
    n = _log(rng, 8, 64)
    return dict(op=op, n=n, batch=_log(rng, 64, min(10000, int(2.0e9 / n ** 3))))


# ------------------------------------------------------------------ sizes (of the case alone)
def _sizes(case):
    """Per-instance sizes of a variable-size case: {"m", "n", "k", "r"} as needed."""
    op, lo, hi, b = case["op"], case["lo"], case["hi"], case["batch"]
    g = np.random.default_rng([lo, hi, b, len(op)])
    if op in ("gemm_v", "trsm_v"):
        m, n, k = (g.integers(lo, hi + 1, b) for _ in range(3))
        return dict(m=m, n=n, k=k)
    u = g.random(b)
    if op == "gesv_v":
        n = np.exp(math.log(lo) + u * (math.log(hi) - math.log(lo)))
    else:   # density ~ n^-1.5 on [lo, hi]
        a, c = lo ** -0.5, hi ** -0.5
        n = (a - u * (a - c)) ** -2.0
    return dict(n=np.rint(n).astype(np.int64).clip(lo, hi), r=g.integers(1, case["nrhs"] + 1, b))


def _r8(v):
    return (v + 7) // 8 * 8


def _offsets(sizes):
    """Offsets of instances packed at multiples of four entries, and the total."""
    pad = (sizes + 3) // 4 * 4
    return np.concatenate([[0], np.cumsum(pad)[:-1]]).astype(np.int64), int(pad.sum())


def work(case):
    op = case["op"]
    if op in ("gesv", "dsgesv", "getri"):
        n, r, b = float(case["n"]), float(case.get("nrhs", 0)), case["batch"]
        if op == "gesv":
            return dict(bytes=b * (16 * n * n + 16 * n * r + 4 * n + 4), flops=b * (2 / 3 * n ** 3 + 2 * n * n * r))
        if op == "dsgesv":
            return dict(bytes=b * (8 * n * n + 16 * n * r + 4 * n + 8), flops=b * (2 / 3 * n ** 3 + 4 * n * n * r))
        return dict(bytes=b * (24 * n * n + 4 * n + 8), flops=b * 2 * n ** 3)
    if op == "geqrf":
        m, n, b = float(case["m"]), float(case["n"]), case["batch"]
        return dict(bytes=b * 8 * (2 * m * n + n), flops=b * (2 * m * n * n - 2 / 3 * n ** 3))
    s = {k: v.astype(np.float64) for k, v in _sizes(case).items()}
    if op == "gemm_v":
        e = 8 if case["dtype"] == "f64" else 4
        m, n, k = s["m"], s["n"], s["k"]
        return dict(bytes=float(e * (m * k + k * n + 2 * m * n).sum()), flops=float((2 * m * n * k).sum()))
    if op == "trsm_v":
        m, n = s["m"], s["n"]
        t = m if case["left"] else n
        return dict(bytes=float(8 * (t * (t + 1) / 2 + 2 * m * n).sum()), flops=float((t * m * n).sum()))
    n, r = s["n"], s["r"]
    if op == "gesv_v":
        return dict(bytes=float((16 * n * n + 16 * n * r + 4 * n + 4).sum()), flops=float((2 / 3 * n ** 3 + 2 * n * n * r).sum()))
    if op == "posv_v":
        return dict(bytes=float((8 * n * (n + 1) + 16 * n * r + 4).sum()), flops=float((n ** 3 / 3 + 2 * n * n * r).sum()))
    return dict(bytes=float((4 * n * (n + 1) + 16 * n * r + 8).sum()), flops=float((n ** 3 / 3 + 4 * n * n * r).sum()))


def tolerance(case):
    # four times and a little more of what the results differ from 64-bit ones in another order of operations
    # ("exact" below). Solutions of a few ill-conditioned systems carry most of an LU batch's difference.
    op = case["op"]
    if op == "gemm_v":
        return dict(rel=1e-15) if case["dtype"] == "f64" else dict(rel=2.5e-6)
    if op == "posv_v":
        return dict(rel=1e-15, max=1e-12)
    if op == "dsposv_v":
        return dict(rel=1e-14, max=1e-12, differ=0.01)
    if op in ("trsm_v", "geqrf"):
        return dict(rel=5e-15, max=1e-11)
    if op == "dsgesv":
        return dict(rel=5e-10, max=1e-6, differ=0.01)
    return dict(rel=1e-10, max=1e-6)


# ------------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, dtype=torch.float64, device=DEV, generator=g) * 2 - 1


def _haar(g, b, n):
    G = torch.randn(b, n, n, dtype=torch.float64, device=DEV, generator=g)
    for _ in range(2):   # G R^-1 with R the Cholesky factor of G^T G, twice: Q with R's diagonal positive
        L = torch.linalg.cholesky(G.transpose(1, 2) @ G)
        G = torch.linalg.solve_triangular(L.transpose(1, 2), G, upper=True, left=False)
    return G


def _graded(g, b, n):
    """U diag(s) V^T, U and V Haar, s log-uniform, condition numbers log-uniform on [1e2, 1e6]."""
    kappa = torch.exp(math.log(1e2) + torch.rand(b, 1, dtype=torch.float64, device=DEV, generator=g) * math.log(1e4))
    s = torch.exp(-torch.rand(b, n, dtype=torch.float64, device=DEV, generator=g) * torch.log(kappa))
    return ((_haar(g, b, n) * s[:, None, :]) @ _haar(g, b, n).transpose(1, 2)).contiguous()


def _ints(v):
    """Device size array of batch + 1 entries, as the variable-size entry points take it."""
    return torch.from_numpy(np.concatenate([v, [0]]).astype(np.int32)).to(DEV)


def _ptrs(buf, off):
    return buf.data_ptr() + torch.from_numpy(off * buf.element_size()).to(DEV)


def _groups(n):
    """(order, instances of that order) of a variable-size batch."""
    order = np.argsort(n, kind="stable")
    edge = np.flatnonzero(np.diff(n[order])) + 1
    return [(int(n[ids[0]]), ids) for ids in np.split(order, edge)]


def _index(off, ids, count):
    return torch.from_numpy(off[ids]).to(DEV)[:, None] + torch.arange(count, device=DEV)[None, :]


def _inputs(case, seed):
    """The caller's matrices: dense tensors, or flat buffers with offsets."""
    g, op = _gen(seed), case["op"]
    if op in ("gesv", "dsgesv", "getri"):
        n, b = case["n"], case["batch"]
        graded = op == "dsgesv" or n >= 96
        d = dict(A0=_graded(g, b, n) if graded else _uniform(g, b, n, n))
        if op != "getri":
            d["B0"] = torch.randn(b, case["nrhs"], n, dtype=torch.float64, device=DEV, generator=g) if graded else _uniform(g, b, case["nrhs"], n)
        return d
    if op == "geqrf":
        return dict(A0=_uniform(g, case["batch"], case["n"], case["m"]))
    s = _sizes(case)
    if op == "gemm_v":
        dt = torch.float64 if case["dtype"] == "f64" else torch.float32
        ra, ca = (s["k"], s["m"]) if case["ta"] else (s["m"], s["k"])
        rb, cb = (s["n"], s["k"]) if case["tb"] else (s["k"], s["n"])
        d = dict(s, lda=_r8(ra), ldb=_r8(rb), ldc=_r8(s["m"]))
        for key, ld, cols in (("A0", d["lda"], ca), ("B0", d["ldb"], cb), ("C0", d["ldc"], s["n"])):
            d["off" + key[0]], total = _offsets(ld * cols)
            d[key] = torch.randn(total, dtype=dt, device=DEV, generator=g)
        return d
    if op == "trsm_v":
        t = s["m"] if case["left"] else s["n"]
        d = dict(s, t=t, lda=_r8(t), ldb=_r8(s["m"]))
        d["offA"], ta = _offsets(d["lda"] * t)
        d["offB"], tb = _offsets(d["ldb"] * s["n"])
        d["A0"] = torch.randn(ta, dtype=torch.float64, device=DEV, generator=g)
        d["B0"] = torch.randn(tb, dtype=torch.float64, device=DEV, generator=g)
        for nv, ids in _groups(t):   # N(0,1)/sqrt(n) + 2 I
            ld = int(_r8(nv))
            i = _index(d["offA"], ids, ld * nv)
            M = d["A0"][i].reshape(len(ids), nv, ld) / math.sqrt(nv)
            M[:, range(nv), range(nv)] += 2
            d["A0"][i] = M.reshape(len(ids), -1)
        return d
    n, r = s["n"], s["r"]
    d = dict(s)
    d["offA"], ta = _offsets(n * n)
    d["offB"], tb = _offsets(n * r)
    d["B0"] = torch.randn(tb, dtype=torch.float64, device=DEV, generator=g)
    if op == "gesv_v":
        d["A0"] = _uniform(g, ta)
        return d
    d["A0"] = torch.zeros(ta, dtype=torch.float64, device=DEV)
    for nv, ids in _groups(n):       # G G^T + n I
        G = torch.randn(len(ids), nv, nv, dtype=torch.float64, device=DEV, generator=g)
        S = torch.baddbmm(nv * torch.eye(nv, dtype=torch.float64, device=DEV).expand_as(G), G, G.transpose(1, 2))
        d["A0"][_index(d["offA"], ids, nv * nv)] = S.reshape(len(ids), -1)
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    op = case["op"]
    d["case"], d["q"] = case, api.default_queue()
    if op == "dsgesv":
        d["A"] = d["A0"]             # only an instance that falls back to FP64 is overwritten
    elif op not in ("gemm_v", "trsm_v", "dsposv_v"):
        d["A"] = torch.empty_like(d["A0"])
    if op == "gesv":
        d["B"] = torch.empty_like(d["B0"])
    if not op.endswith("_v"):
        return d
    for key in ("m", "n", "k", "r", "lda", "ldb", "ldc"):
        if key in d:
            d["d" + key] = _ints(d[key])
    A = d.get("A", d["A0"])
    d["pA"] = _ptrs(A, d["offA"])
    if op == "gemm_v":
        d["C"] = torch.empty_like(d["C0"])
        d["pB"], d["pC"] = _ptrs(d["B0"], d["offB"]), _ptrs(d["C"], d["offC"])
        return d
    if op == "dsposv_v":
        words = d["n"] * (d["n"] + d["r"])
        off, total = _offsets(words)
        d["X"] = torch.zeros_like(d["B0"])
        d["W"] = torch.empty(total, dtype=torch.float32, device=DEV)
        d["pB"], d["pX"], d["pW"] = _ptrs(d["B0"], d["offB"]), _ptrs(d["X"], d["offB"]), _ptrs(d["W"], off)
        d["it"] = torch.zeros(len(words) + 1, dtype=torch.int32, device=DEV)
    else:
        d["B"] = torch.empty_like(d["B0"])
        d["pB"] = _ptrs(d["B"], d["offB"])
    if op == "gesv_v":
        off, total = _offsets(d["n"])
        d["ipiv"] = torch.zeros(total, dtype=torch.int32, device=DEV)
        d["pP"] = _ptrs(d["ipiv"], off)
    d["info"] = torch.zeros(case["batch"] + 1, dtype=torch.int32, device=DEV)
    return d


# ---------------------------------------------------------------------------------- calls
def _p(t):
    return C.c_void_p(t.data_ptr())


def _ok(rc):
    if rc:
        raise RuntimeError(f"the call returned {rc}")


def run(d):
    case, q = d["case"], d["q"]
    op, L, b, hi = case["op"], q.lib, case["batch"], case.get("hi")
    if op == "dsgesv":
        X, ipiv, it, info = api.dsgesv_batched(d["A"], d["B0"], queue=q)
        return dict(X=X, ipiv=ipiv, iter=it, info=info)
    if op == "dsposv_v":
        _ok(L.magma_dsposv_vbatched_max_nocheck(LOWER, _p(d["dn"]), _p(d["dr"]), _p(d["pA"]), _p(d["dn"]), _p(d["pB"]), _p(d["dn"]),
                                                _p(d["pX"]), _p(d["dn"]), _p(d["pW"]), _p(d["it"]), _p(d["info"]), b, hi,
                                                case["nrhs"], q.handle))
        return dict(X=d["X"], iter=d["it"][:b], info=d["info"][:b])
    if op == "gemm_v":
        d["C"].copy_(d["C0"])
        fn = L.magmablas_dgemm_vbatched_max_nocheck if case["dtype"] == "f64" else L.magmablas_sgemm_vbatched_max_nocheck
        fn(112 if case["ta"] else 111, 112 if case["tb"] else 111, _p(d["dm"]), _p(d["dn"]), _p(d["dk"]), 1.0, _p(d["pA"]),
           _p(d["dlda"]), _p(d["pB"]), _p(d["dldb"]), 0.5, _p(d["pC"]), _p(d["dldc"]), b, hi, hi, hi, q.handle)
        return dict(C=d["C"])
    if op == "trsm_v":
        d["B"].copy_(d["B0"])
        L.magmablas_dtrsm_vbatched_max_nocheck(LEFT if case["left"] else RIGHT, LOWER if case["lower"] else UPPER,
                                               112 if case["trans"] else 111, 131, _p(d["dm"]), _p(d["dn"]), 1.0, _p(d["pA"]),
                                               _p(d["dlda"]), _p(d["pB"]), _p(d["dldb"]), b, hi, hi, q.handle)
        return dict(B=d["B"])
    d["A"].copy_(d["A0"])
    if op == "getri":
        ipiv, info = api.dgetrf_batched(d["A"], queue=q)
        inv, info2 = api.dgetri_outofplace_batched(d["A"], ipiv, queue=q)
        return dict(A=d["A"], ipiv=ipiv, info=info, inv=inv, info2=info2)
    if op == "geqrf":
        tau = api.dgeqrf_batched(d["A"], case["m"], queue=q)
        return dict(A=d["A"], tau=tau)
    d["B"].copy_(d["B0"])
    if op == "gesv":
        ipiv, info = api.dgesv_batched(d["A"], d["B"], queue=q)
        return dict(A=d["A"], B=d["B"], ipiv=ipiv, info=info)
    if op == "gesv_v":
        _ok(L.magma_dgesv_vbatched_max_nocheck(_p(d["dn"]), _p(d["dr"]), _p(d["pA"]), _p(d["dn"]), _p(d["pP"]), _p(d["pB"]), _p(d["dn"]),
                                               _p(d["info"]), b, hi, case["nrhs"], q.handle))
        return dict(A=d["A"], B=d["B"], ipiv=d["ipiv"], info=d["info"][:b])
    _ok(L.magma_dposv_vbatched_max_nocheck(UPPER if case["upper"] else LOWER, _p(d["dn"]), _p(d["dr"]), _p(d["pA"]), _p(d["dn"]), _p(d["pB"]),
                                           _p(d["dn"]), _p(d["info"]), b, hi, case["nrhs"], q.handle))
    return dict(A=d["A"], B=d["B"], info=d["info"][:b])


# ------------------------------------------------------------------------ 64-bit results
def _cm(flat, off, ids, ld, cols):
    """Instances of one shape from a flat buffer, as (count, ld, cols) matrices."""
    return flat[_index(off, ids, ld * cols)].reshape(len(ids), cols, ld).transpose(1, 2)


def _put(flat, off, ids, M):
    flat[_index(off, ids, M.shape[1] * M.shape[2])] = M.transpose(1, 2).reshape(len(ids), -1)


def _by_shape(*sizes):
    """(shape, instances) for each combination of sizes."""
    u, inv = np.unique(np.stack(sizes, 1), axis=0, return_inverse=True)
    order = np.argsort(inv.reshape(-1), kind="stable")
    edge = np.flatnonzero(np.diff(inv.reshape(-1)[order])) + 1
    return [(tuple(int(x) for x in u[inv.reshape(-1)[ids[0]]]), ids) for ids in np.split(order, edge)]


def exact(case, seed):
    op, b = case["op"], case["batch"]
    d = _inputs(case, seed)
    info = torch.zeros(b, dtype=torch.int32)
    if op in ("gesv", "dsgesv", "getri"):
        LU, piv = torch.linalg.lu_factor(d["A0"].transpose(1, 2))
        if op == "getri":
            inv = torch.linalg.lu_solve(LU, piv, torch.eye(case["n"], dtype=torch.float64, device=DEV).expand_as(LU))
            return dict(A=LU.transpose(1, 2), ipiv=piv, info=info, inv=inv.transpose(1, 2), info2=info)
        X = torch.linalg.lu_solve(LU, piv, d["B0"].transpose(1, 2)).transpose(1, 2)
        if op == "dsgesv":
            return dict(X=X, ipiv=None, iter=None, info=info)
        return dict(A=LU.transpose(1, 2), B=X, ipiv=piv, info=info)
    if op == "geqrf":
        a, tau = torch.geqrf(d["A0"].transpose(1, 2).cpu())
        return dict(A=a.transpose(1, 2), tau=tau)
    if op == "gemm_v":
        A0, B0, out = d["A0"].double(), d["B0"].double(), d["C0"].double()
        for (m, n, k), ids in _by_shape(d["m"], d["n"], d["k"]):
            A = _cm(A0, d["offA"], ids, int(_r8(k if case["ta"] else m)), m if case["ta"] else k)
            B = _cm(B0, d["offB"], ids, int(_r8(n if case["tb"] else k)), k if case["tb"] else n)
            A = A[:, :k, :].transpose(1, 2) if case["ta"] else A[:, :m, :]
            B = B[:, :n, :].transpose(1, 2) if case["tb"] else B[:, :k, :]
            M = _cm(out, d["offC"], ids, int(_r8(m)), n).clone()
            M[:, :m, :] = A @ B + 0.5 * M[:, :m, :]
            _put(out, d["offC"], ids, M)
        return dict(C=out)
    if op == "trsm_v":
        out = d["B0"].clone()
        for (m, n), ids in _by_shape(d["m"], d["n"]):
            t = m if case["left"] else n
            A = _cm(d["A0"], d["offA"], ids, int(_r8(t)), t)[:, :t, :]
            M = _cm(out, d["offB"], ids, int(_r8(m)), n).clone()
            T = torch.tril(A) if case["lower"] else torch.triu(A)
            up = not case["lower"]
            if case["trans"]:
                T, up = T.transpose(1, 2), not up
            M[:, :m, :] = torch.linalg.solve_triangular(T, M[:, :m, :].contiguous(), upper=up, left=case["left"])
            _put(out, d["offB"], ids, M)
        return dict(B=out)
    A, B = d["A0"].clone(), torch.zeros_like(d["B0"]) if op == "dsposv_v" else d["B0"].clone()
    ipiv = None
    if op == "gesv_v":
        poff, total = _offsets(d["n"])
        ipiv = torch.zeros(total, dtype=torch.int32, device=DEV)
    for (n, r), ids in _by_shape(d["n"], d["r"]):
        M, R = _cm(d["A0"], d["offA"], ids, n, n), _cm(d["B0"], d["offB"], ids, n, r)
        if op == "gesv_v":
            F, piv = torch.linalg.lu_factor(M)
            X = torch.linalg.lu_solve(F, piv, R)
            ipiv[_index(poff, ids, n)] = piv
        else:
            F = torch.linalg.cholesky(M)
            X = torch.cholesky_solve(R, F)
            F = F.transpose(1, 2).triu() + M.tril(-1) if case.get("upper") else F.tril() + M.triu(1)
        _put(A, d["offA"], ids, F)
        _put(B, d["offB"], ids, X)
    if op == "gesv_v":
        return dict(A=A, B=B, ipiv=ipiv, info=info)
    if op == "dsposv_v":
        return dict(X=B, iter=None, info=info)
    return dict(A=A, B=B, info=info)
