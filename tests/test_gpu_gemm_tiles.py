"""The FP64 GEMM engine at the edges of its CTA tiles (64 x 64, 64 x 32, 32 x 32,
128 x 16, 128 x 8) and of its k tile of 16, for every operand layout, with and
without 16-byte copies, split and unsplit, against numpy (float64).  Tolerance: as
tests/test_gpu_gemm.py, 1e-13 relative to sum |a||b| (contractions of at most 700
terms: 700 x 2^-53 = 8e-14 bounds the rounding of any summation order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [
    # (m, n): one row or column, just below / at / above a tile edge, thin, wide
    (1, 1), (31, 33), (32, 32), (65, 63), (64, 31), (127, 8), (128, 1), (129, 9), (257, 16),
    (300, 17), (33, 515), (7, 2050), (2100, 1030), (4133, 12),
]


def _operands(rng, m, n, k, nbr, a_k, b_n, pad):
    lda, ldb = (k if a_k else m) + pad, (n if b_n else k) + pad
    A = rng.standard_normal((nbr, m if a_k else k, lda))  # C order: columns of lda
    B = rng.standard_normal((nbr, k if b_n else n, ldb))
    Am = [x[:, :k] if a_k else x[:, :m].T for x in A]
    Bm = [x[:, :n] if b_n else x[:, :k].T for x in B]
    return A, B, np.concatenate(Am, axis=1), np.concatenate(Bm, axis=0), lda, ldb


@pytest.mark.parametrize("a_k,b_n", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("k,nbr,split", [(1, 1, 0), (16, 1, 0), (35, 3, 0), (700, 1, 5),
                                         (15, 40, 64)])
def test_tile_edges(uw12lib, cuda_device, a_k, b_n, pad, k, nbr, split):
    import torch
    for m, n in SIZES:
        rng = np.random.default_rng(m * 7 + n * 3 + k)
        A, B, Am, Bm, lda, ldb = _operands(rng, m, n, k, nbr, a_k, b_n, pad)
        C = rng.standard_normal((n, m))
        dA, dB, dC = (torch.from_numpy(x).cuda() for x in (A, B, C.copy()))
        uw12lib.dgemm(m, n, k, 2.0, dA.data_ptr(), lda, a_k, dB.data_ptr(), ldb, b_n, 0.5,
                      dC.data_ptr(), m, nbr1=nbr, sr=(A[0].size, 0, B[0].size, 0), split=split)
        torch.cuda.synchronize()
        ref = 2.0 * Am @ Bm + 0.5 * C.T
        scale = 2.0 * np.abs(Am) @ np.abs(Bm) + 0.5 * np.abs(C.T)
        assert np.all(np.abs(dC.cpu().numpy().T - ref) <= 1e-13 * scale), (m, n)
