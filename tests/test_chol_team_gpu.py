"""FP64 Cholesky and solve by a team of warps (orders 33..512, and solves up to 1024): factors,
solutions and info equal the oracle's bit for bit at the edges of the 32-column panels and of the
team sizes, for one, several and more than eight right-hand sides, in both triangles; the triangle
that is not named stays as it was."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("upper", [False, True])
@pytest.mark.parametrize("n,nrhs", [(33, 1), (64, 9), (65, 2), (96, 8), (97, 17), (128, 1), (129, 40), (256, 9), (257, 3),
                                    (511, 16), (512, 8), (600, 11)])
def test_posv_bit_identical(cuda, n, nrhs, upper):
    import torch

    import magma_b200 as mb
    import oracle
    from magma_b200 import testing as T
    lda, batch = n + n % 3, 3
    A = np.random.default_rng(n).uniform(-1, 1, (batch, n, lda))
    for i in range(batch):
        A[i, :, :n] = T.spd_gram(n, 40, i)
    bad = n // 2 + 3
    A[2, bad, bad] = -1.0                        # leading minor bad + 1 is not positive
    B = np.random.default_rng(n + 1).standard_normal((batch, nrhs, n + 1))
    dA, dB = torch.from_numpy(A).to(cuda), torch.from_numpy(B).to(cuda)
    info = mb.dposv_batched(dA, dB, upper=upper).cpu().numpy()
    gA, gB = dA.cpu().numpy(), dB.cpu().numpy()
    OA, OB = [A[i].copy() for i in range(batch)], [B[i].copy() for i in range(batch)]
    full = np.full(batch, n, np.int32)
    oinf = oracle.dposv_vbatched(OA, OB, full, np.full(batch, nrhs, np.int32), np.full(batch, lda, np.int32),
                                 np.full(batch, n + 1, np.int32), upper=upper)
    assert np.array_equal(info, oinf)
    tri = np.tril(np.ones((n, n), bool)) if not upper else np.triu(np.ones((n, n), bool))   # [row, column]
    for i in range(batch):
        got, ref, was = gA[i, :, :n].T, OA[i][:, :n].T, A[i, :, :n].T
        assert np.array_equal(got[~tri], was[~tri])
        if i < 2:
            assert np.array_equal(got[tri], ref[tri])
            assert np.array_equal(gB[i], OB[i])
        elif not upper:                          # the finished columns of the failed factorisation
            assert np.array_equal(np.tril(got)[:, :bad], np.tril(ref)[:, :bad])
        else:
            assert np.array_equal(np.triu(got)[:bad], np.triu(ref)[:bad])
