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


@pytest.mark.parametrize("m,n", [(257, 1), (400, 2), (513, 1), (1024, 3)])
def test_short_factorisations(cuda, m, n):
    """A panel of one to three steps in more clusters than the machine holds at once: each cluster's
    first exchange comes right after it starts, while its blocks replace other clusters'."""
    import torch

    import magma_b200 as mb
    import oracle
    A = np.random.default_rng(m).uniform(-1, 1, (1500, n, m))
    O = A.copy()
    oip, oinf = oracle.dgetrf_batched(O, m)
    D = torch.from_numpy(A).to(cuda)
    ipiv, info = mb.dgetrf_batched(D, m=m)
    assert np.array_equal(ipiv.cpu().numpy()[:, :n], oip[:, :n])
    assert np.array_equal(info.cpu().numpy(), oinf)
    assert np.array_equal(D.cpu().numpy(), O)
