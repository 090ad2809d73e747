"""The FP64 tensor-core GEMM tile fed by asynchronous copies (no-transpose form, max(M, N) > 32):
bit-identical to the CUDA-core tiles at the edges of its 64x64 tiles, 8x8 sub-tiles and 16-wide K
chunks, with even and odd leading dimensions and with operands that start on 8 but not 16 bytes."""
import numpy as np
import pytest

from magma_b200 import _lib

pytestmark = pytest.mark.gpu

SHAPES = [(33, 1, 3), (64, 64, 16), (65, 40, 17), (72, 97, 31), (128, 128, 128), (127, 57, 33), (8, 100, 15), (130, 66, 2)]


@pytest.mark.parametrize("shift", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_gemm_dmma_edges(cuda, m, n, k, pad, shift):
    import ctypes as C

    import torch

    import magma_b200 as mb
    lib = _lib.load()
    count = lib.magma_b200_tuning_get(None, 0)
    vals = (C.c_int * count)()
    lib.magma_b200_tuning_get(vals, count)
    rng = np.random.default_rng(m * 131 + n * 7 + k)
    batch, lda, ldb, ldc = 3, m + pad, k + pad, m + 1

    def dev(cols, ld, off):
        buf = torch.from_numpy(rng.standard_normal(batch * cols * ld + 2)).to(cuda)
        return buf[off:off + batch * cols * ld].view(batch, cols, ld)
    A, B, C0 = dev(k, lda, shift[0]), dev(n, ldb, shift[1]), dev(n, ldc, 0)
    out = {}
    try:
        for variant in (0, 3):
            new = (C.c_int * count)(*([variant] * 4 + list(vals)[4:]))
            assert lib.magma_b200_tuning_set(new, count) == 0
            for beta in (0.0, 0.5):
                D = C0.clone()
                mb.gemm_batched(A, B, D, m, n, k, alpha=1.25, beta=beta)
                out[variant, beta] = D.cpu().numpy()
    finally:
        lib.magma_b200_tuning_set(vals, count)
    for beta in (0.0, 0.5):
        assert np.array_equal(out[0, beta], out[3, beta])
    assert np.array_equal(out[3, 0.5][:, :, m:], C0.cpu().numpy()[:, :, m:])
