"""FP64 solves with LU factors of orders above 64 (tensor-core sweeps, eight right-hand sides at
a time): solutions equal the oracle's bit for bit at the edges of the launch shapes and of the
32-row blocks, for partial and several groups of right-hand sides, zero right-hand sides, tiny
and huge diagonals (the division's slow path) and singular factors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(65, 1), (96, 8), (127, 9), (128, 3), (129, 17), (255, 2), (256, 4), (257, 16), (512, 1), (513, 40), (1024, 9)]


def _problem(n, nrhs):
    rng = np.random.default_rng(n * 100 + nrhs)
    A = rng.uniform(-1, 1, (4, n, n + n % 2))
    B = rng.uniform(-1, 1, (4, nrhs, n + 1))
    B[0, :, : n // 2] = 0.0
    B[0, 0, 3] = -0.0
    A[1, :, :n] *= (2.0 ** rng.integers(-480, 480, n))[:, None]     # columns scaled: extreme diagonals of U
    A[2, 40, :] = 0.0                                               # singular: divisions by zero
    return A, B


@pytest.mark.parametrize("n,nrhs", CASES)
def test_getrs_bit_identical(cuda, n, nrhs):
    import torch

    import magma_b200 as mb
    import oracle
    A, B = _problem(n, nrhs)
    ipiv, _ = oracle.dgetrf_batched(A, n)
    X = B.copy()
    oracle.dgetrs_batched(A, ipiv, X)
    dA, dB, dP = (torch.from_numpy(v).to(cuda) for v in (A, B, ipiv))
    mb.dgetrs_batched(dA, dP, dB)
    assert np.array_equal(dB.cpu().numpy(), X, equal_nan=True)


@pytest.mark.parametrize("n,nrhs", CASES[::2])
def test_getrs_trans(cuda, n, nrhs):
    import torch

    import magma_b200 as mb
    import oracle
    A, B = _problem(n, nrhs)
    A, B = A[3:], B[3:]
    ipiv, _ = oracle.dgetrf_batched(A, n)
    X = B.copy()
    oracle.dgetrs_batched(A, ipiv, X, trans=True)
    dA, dB, dP = (torch.from_numpy(v).to(cuda) for v in (A, B, ipiv))
    mb.dgetrs_batched(dA, dP, dB, trans=True)
    got = dB.cpu().numpy()
    # each solution carries the backward error of two n-term substitutions, amplified by cond(A);
    # the oracle sums in another order: 64 n eps of the largest entry, as for the smaller orders
    assert np.abs(got - X).max() <= 64 * n * np.finfo(float).eps * np.abs(X).max()


@pytest.mark.parametrize("n", [65, 128])
@pytest.mark.parametrize("past", [0, 1])
def test_one_rhs_many(cuda, n, past):
    """One right-hand side on both sides of the line of five matrices an SM: the oracle's solutions,
    and with trans the bits of the same solve beside a second right-hand side (always the sweeps)."""
    import torch

    import magma_b200 as mb
    import oracle
    batch = 5 * torch.cuda.get_device_properties(0).multi_processor_count + past
    rng = np.random.default_rng(n + past)
    A, B = rng.uniform(-1, 1, (batch, n, n)), rng.uniform(-1, 1, (batch, 2, n))
    ipiv, _ = oracle.dgetrf_batched(A, n)
    X = B[:, :1].copy()
    oracle.dgetrs_batched(A, ipiv, X)
    dA, dP = torch.from_numpy(A).to(cuda), torch.from_numpy(ipiv).to(cuda)
    for trans in (False, True):
        one, two = torch.from_numpy(B[:, :1].copy()).to(cuda), torch.from_numpy(B).to(cuda)
        mb.dgetrs_batched(dA, dP, one, trans=trans)
        mb.dgetrs_batched(dA, dP, two, trans=trans)
        assert torch.equal(one, two[:, :1])
        if not trans:
            assert np.array_equal(one.cpu().numpy(), X)
