"""GPU tests of the variable-size mixed-precision Cholesky solve (magma_dsposv_vbatched).

Criterion (as magma_dsposv_gpu, src/zcposv_gpu.cpp:134-330): every solution has
normwise backward error <= 1e-14 against the FP64 data; refined instances leave
A untouched; instances that fall back to FP64 hold the FP64 Cholesky factor,
bit-identical to the oracle, and their info is LAPACK's."""
import numpy as np
import pytest

import oracle
from magma_b200 import testing as T

pytestmark = pytest.mark.gpu


def _mixed_batch(count, seed, n_hi=512):
    rng = np.random.default_rng(seed)
    ns = np.concatenate([[1, 31, 32, 33, 64, 65, 200, n_hi], rng.integers(2, n_hi + 1, count - 8)])
    nrhs = rng.integers(1, 9, count)
    As = [np.ascontiguousarray(T.spd_gram(int(n), seed, i)) for i, n in enumerate(ns)]
    Bs = [rng.standard_normal((int(r), int(n))) for n, r in zip(ns, nrhs)]
    return ns, nrhs, As, Bs


def _bwd(A, X, B):
    """max over RHS of ||b - A x||_inf / (||A||_inf ||x||_inf + ||b||_inf); arrays (cols, n)."""
    R = B.T - A @ X.T
    an = np.abs(A).sum(axis=1).max()
    return float((np.abs(R).max(axis=0) / (an * np.abs(X.T).max(axis=0) + np.abs(B.T).max(axis=0))).max())


@pytest.mark.parametrize("checked", [True, False])
def test_dsposv_vbatched_backward_error(cuda, checked):
    import magma_b200 as mb
    from magma_b200.api import VarBatch
    ns, nrhs, As, Bs = _mixed_batch(60, 21)
    gA, gB = VarBatch(As, cuda), VarBatch(Bs, cuda)
    ms = (int(ns.max()), int(nrhs.max())) if not checked else None
    X, it, info = mb.dsposv_vbatched(gA, gB, ns, nrhs, max_sizes=ms)
    it, info = it.cpu().numpy(), info.cpu().numpy()
    Xs = X.unpack()
    assert np.all(info == 0)
    assert np.all(it >= 0), it                      # SPD and well conditioned: all refine in FP32
    for i in range(len(ns)):
        assert _bwd(As[i], Xs[i], Bs[i]) <= 1e-14, (i, ns[i])
    Aout = gA.unpack()
    for i in range(len(ns)):
        assert np.array_equal(Aout[i], As[i])       # A untouched
    for i in range(len(Bs)):
        assert np.array_equal(gB.unpack()[i], Bs[i])


def test_dsposv_vbatched_fallbacks(cuda):
    import magma_b200 as mb
    from magma_b200.api import VarBatch
    ns = np.array([40, 70, 90, 20])
    nrhs = np.array([2, 1, 3, 4])
    As = [np.ascontiguousarray(T.spd_gram(int(n), 5, i)) for i, n in enumerate(ns)]
    As[1][3, 3] = 1e39                              # overflows single precision -> iter -2, FP64 succeeds
    As[2][10, 10] = -5.0                            # not positive definite -> iter -3, info 11 in FP64
    rng = np.random.default_rng(3)
    Bs = [rng.standard_normal((int(r), int(n))) for n, r in zip(ns, nrhs)]
    gA, gB = VarBatch(As, cuda), VarBatch(Bs, cuda)
    X, it, info = mb.dsposv_vbatched(gA, gB, ns, nrhs)
    it, info = it.cpu().numpy(), info.cpu().numpy()
    assert it[0] >= 0 and it[3] >= 0
    assert it[1] == -2 and it[2] == -3
    O = [As[1].copy(), As[2].copy()]
    Ob = [np.zeros((1, 70)), np.zeros((1, 90))]
    oinfo = oracle.dposv_vbatched(O, Ob, [70, 90], [1, 1], [70, 90], [70, 90], solve=False, upper=False)
    assert list(info[[1, 2]]) == list(oinfo)
    assert oinfo[1] == 11
    Aout = gA.unpack()
    assert np.array_equal(np.tril(Aout[1]), np.tril(O[0]))   # FP64 factor, bit-identical to the oracle
    Xs = X.unpack()
    for i in (0, 1, 3):
        assert _bwd(As[i], Xs[i], Bs[i]) <= 1e-14, i


def test_dsposv_vbatched_independent_of_the_batch(cuda):
    """An instance's solution and iteration count follow from the instance alone: not from the
    caller's maximum of right-hand sides, nor from another instance with more of them."""
    import magma_b200 as mb
    from magma_b200.api import VarBatch
    ns = np.repeat([20, 32, 33, 40, 64, 65, 128, 129, 256], 12)
    rng = np.random.default_rng(8)
    nrhs = rng.integers(1, 5, len(ns))
    As = [np.ascontiguousarray(T.spd_gram(int(n), 44, i)) for i, n in enumerate(ns)]
    Bs = [rng.standard_normal((int(r), int(n))) for n, r in zip(ns, nrhs)]
    extra = (np.ascontiguousarray(T.spd_gram(50, 45, 0)), rng.standard_normal((8, 50)))
    results = []
    for most, more in ((4, False), (8, False), (8, True)):
        a, b, n, r = (As + [extra[0]], Bs + [extra[1]], np.append(ns, 50), np.append(nrhs, 8)) if more else (As, Bs, ns, nrhs)
        X, it, info = mb.dsposv_vbatched(VarBatch(a, cuda), VarBatch(b, cuda), n, r, max_sizes=(256, most))
        assert not info.cpu().numpy().any()
        results.append((X.unpack()[:len(ns)], it.cpu().numpy()[:len(ns)]))
    for X, it in results[1:]:
        assert np.array_equal(it, results[0][1])
        for i in range(len(ns)):
            assert np.array_equal(X[i], results[0][0][i]), (i, ns[i])


def test_single_precision_factor(cuda):
    """The FP32 factor that the refinement solves with, left in the caller's workspace: the oracle's
    bits at the edges of the 32-column panels and of the team sizes, at odd leading dimensions of A. A
    wrong entry would otherwise cost passes only."""
    import ctypes as C

    import torch

    from magma_b200.api import VarBatch, default_queue
    ns = np.array([20, 33, 64, 65, 96, 97, 128, 129, 160, 255, 256, 257, 300, 480, 511, 512], np.int32)
    batch, rng = len(ns), np.random.default_rng(12)
    lda = ns + ns % 3
    As = []
    for i, n in enumerate(ns):
        a = np.zeros((n, lda[i]))
        a[:, :n] = T.spd_gram(int(n), 71, i)
        As.append(a)
    Bs = [rng.standard_normal((2, int(n))) for n in ns]
    gA, gB, gX = VarBatch(As, cuda), VarBatch(Bs, cuda), VarBatch([np.zeros_like(b) for b in Bs], cuda)
    gW = VarBatch([np.zeros((int(n) + 2, int(n))) for n in ns], cuda, torch.float32)
    it, info = gA.ints(np.zeros(batch)), gA.ints(np.zeros(batch))
    dn, dr, dla = gA.ints(ns), gA.ints(np.full(batch, 2)), gA.ints(lda)
    q = default_queue()
    p = lambda t: C.c_void_p(t.data_ptr())
    rc = q.lib.magma_dsposv_vbatched_max_nocheck(122, p(dn), p(dr), p(gA.ptrs), p(dla), p(gB.ptrs), p(dn), p(gX.ptrs), p(dn),
                                                 p(gW.ptrs), p(it), p(info), batch, 512, 2, q.handle)
    q.sync()
    assert rc == 0 and (it.cpu().numpy()[:batch] >= 0).all()
    for i, (n, W) in enumerate(zip(ns, gW.unpack())):
        ref = np.ascontiguousarray(As[i][:, :n]).astype(np.float32)
        assert oracle.spotrf(ref) == 0
        lower = np.triu(np.ones((n, n), bool))         # [column, row]
        assert np.array_equal(W[:n][lower], ref[lower]), n


def test_dsposv_vbatched_argument_errors(cuda):
    import magma_b200 as mb
    from magma_b200.api import VarBatch
    gA = VarBatch([np.eye(4), np.eye(3)], cuda)
    gB = VarBatch([np.ones((1, 4)), np.ones((1, 3))], cuda)
    with pytest.raises(ValueError, match="-2"):
        mb.dsposv_vbatched(gA, gB, [4, -3], [1, 1])
    with pytest.raises(ValueError, match="-5"):
        mb.dsposv_vbatched(gA, gB, [4, 3], [1, 1], lda=[4, 2])
