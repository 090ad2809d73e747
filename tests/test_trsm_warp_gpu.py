"""FP64 trsm on the warp kernel (triangles up to 176 rows; from the left with a transposed triangle
and at most 32 columns up to 224): every side / uplo / trans / diag form equals the oracle bit for
bit at the edges of its 8-row pieces, 8-column groups and 32-column blocks, at its largest sizes and
just past them (the panel kernel), with odd leading dimensions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = [(left, lower, trans, unit) for left in (True, False) for lower in (True, False) for trans in (False, True)
         for unit in (False, True)]
SIZES = [(1, 1), (7, 9), (8, 8), (33, 31), (65, 1), (100, 40), (176, 17), (17, 176), (256, 17), (17, 256), (257, 9), (9, 257)]
NARROW = [(224, 32), (32, 224), (200, 5), (5, 200)]


@pytest.mark.parametrize("left,lower,trans,unit", FORMS)
def test_trsm_warp_bit_identical(cuda, left, lower, trans, unit):
    import oracle
    from magma_b200.api import VarBatch, tri_vbatched
    narrow = [s for s in NARROW if s[0 if left else 1] > 32]
    # up to the warp kernel's sizes, past them, and with one panel of columns on both sides of 224
    for limit in (SIZES[:8], SIZES[:10], SIZES, narrow, narrow + [(225, 8) if left else (8, 225)]):
        rng = np.random.default_rng(5)
        M, N = [m for m, _ in limit], [n for _, n in limit]
        R = [m if left else n for m, n in limit]
        lda, ldb = [r + r % 3 for r in R], [m + 1 for m in M]
        As = [rng.uniform(-1, 1, (r, la)) / r for r, la in zip(R, lda)]
        for a, r in zip(As, R):
            a[range(r), range(r)] += 1.5
        Bs = [rng.uniform(-1, 1, (n, lb)) for n, lb in zip(N, ldb)]
        gA, gB = VarBatch(As, cuda), VarBatch(Bs, cuda)
        tri_vbatched("trsm", gA, gB, M, N, lda, ldb, alpha=0.75, left=left, lower=lower, trans=trans, unit=unit,
                     max_sizes=(max(M), max(N)))
        for i, out in enumerate(gB.unpack()):
            ref = Bs[i].copy()
            oracle.dtri(True, left, lower, trans, unit, M[i], N[i], 0.75, As[i], ref)
            assert np.array_equal(out, ref), (M[i], N[i])
