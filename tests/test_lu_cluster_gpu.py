"""The FP64 LU of one matrix per thread-block cluster (orders above 64): factors, pivots and
info equal the oracle's bit for bit at the edges of its launch shapes (128, 256, 512 and 1024
rows; one, two and four blocks a matrix), for panels cut short, wide and tall matrices, odd
leading dimensions, singular instances and tiny pivots, with and without pivoting."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(m, n, lda):
    rng = np.random.default_rng(1000 * m + n)
    A = rng.uniform(-1, 1, (4, n, lda))
    A[1, min(n - 1, 40), :] = 0.0                 # a zero column: info set, the factorisation goes on
    A[2, :, :m] *= 2.0 ** -1040                   # every pivot below the smallest normal number
    A[3, :, m // 2] = A[3, :, m // 3]             # two equal rows: ties go to the lower position
    return A


SHAPES = [(65, 65), (128, 128), (129, 97), (255, 256), (256, 255), (257, 257), (300, 90), (512, 511), (513, 513),
          (1024, 70), (1000, 1024), (70, 300), (270, 1500)]


@pytest.mark.parametrize("m,n", SHAPES)
def test_getrf_cluster_bit_identical(cuda, m, n):
    import torch

    import magma_b200 as mb
    import oracle
    lda = m + (m + n) % 3
    A = _inputs(m, n, lda)
    O = A.copy()
    oip, oinf = oracle.dgetrf_batched(O, m)
    D = torch.from_numpy(A).to(cuda)
    ipiv, info = mb.dgetrf_batched(D, m=m)
    k = min(m, n)
    assert np.array_equal(ipiv.cpu().numpy()[:, :k], oip[:, :k])
    assert np.array_equal(info.cpu().numpy(), oinf)
    assert np.array_equal(D.cpu().numpy(), O)


@pytest.mark.parametrize("m", [65, 130, 257, 513])
def test_getrf_nopiv_cluster_bit_identical(cuda, m):
    import torch

    import magma_b200 as mb
    import oracle
    rng = np.random.default_rng(m)
    A = rng.uniform(-1, 1, (3, m, m))
    A[:, range(m), range(m)] += m
    A[1, 0, 0] = 0.0
    O = A.copy()
    _, oinf = oracle.dgetrf_nopiv_batched(O, m)
    D = torch.from_numpy(A).to(cuda)
    info = mb.dgetrf_nopiv_batched(D)
    assert np.array_equal(info.cpu().numpy(), oinf)
    assert np.array_equal(D.cpu().numpy(), O)


def _random_bit_identical(cuda, m, n, batch):
    import torch

    import magma_b200 as mb
    import oracle
    A = np.random.default_rng(m + n).uniform(-1, 1, (batch, n, m))
    O = A.copy()
    oip, oinf = oracle.dgetrf_batched(O, m)
    D = torch.from_numpy(A).to(cuda)
    ipiv, info = mb.dgetrf_batched(D, m=m)
    k = min(m, n)
    assert np.array_equal(ipiv.cpu().numpy()[:, :k], oip[:, :k])
    assert np.array_equal(info.cpu().numpy(), oinf)
    assert np.array_equal(D.cpu().numpy(), O)


@pytest.mark.parametrize("m,n,batch", [(700, 17, 74), (1024, 20, 60), (600, 129, 300), (260, 161, 400)])
def test_many_clusters(cuda, m, n, batch):
    """Short factorisations in as many clusters as the machine holds at once, and more: a cluster's
    first exchange comes right after it starts, while its blocks replace other clusters'."""
    _random_bit_identical(cuda, m, n, batch)


@pytest.mark.parametrize("m,few,many", [(257, 96, 160), (512, 96, 160), (513, 16, 128), (1024, 16, 128)])
@pytest.mark.parametrize("past", [0, 1])
def test_tall_rule(cuda, m, few, many, past):
    """Matrices on both sides of the lines between the block and the cluster kernel, for few and for
    many matrices; and the fewest columns."""
    _random_bit_identical(cuda, m, few + past, 5)
    _random_bit_identical(cuda, m, many + past, 80)
    _random_bit_identical(cuda, m, 1 + past, 80)


@pytest.mark.parametrize("cols", [40, 300])
def test_tall_vbatched(cuda, cols):
    """Variable sizes with tall instances, under a maximum of few and of many columns."""
    import magma_b200 as mb
    import oracle
    from magma_b200.api import VarBatch
    rng = np.random.default_rng(cols)
    m = np.array([300, 512, 257, 513, 1024, 700, 40, 256, 128, 1000] * 9)
    n = np.minimum(rng.integers(1, cols + 1, len(m)), np.where(m > 256, cols, 64))
    n[3] = cols
    As = [rng.uniform(-1, 1, (c, r)) for r, c in zip(m, n)]
    gA = VarBatch(As, cuda)
    ipiv, info = mb.dgesv_vbatched(gA, None, n, m=m, solve=False, max_sizes=(1024, cols))
    ip = ipiv.cpu().numpy()
    assert not info.cpu().numpy().any()
    for i, out in enumerate(gA.unpack()):
        O = As[i].copy()[None]
        oip, _ = oracle.dgetrf_batched(O, int(m[i]))
        assert np.array_equal(out, O[0]) and np.array_equal(ip[i, :oip.shape[1]], oip[0]), (m[i], n[i])
