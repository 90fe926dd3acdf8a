"""Split-precision products at the edges of their output tiles: one CTA (128 columns)
and CTA pair (256), every tile height (128 to 256 rows in steps of 32), one and several
K chunks, batches with and without a shared operand.  Small-integer operands, whose
products are exact in FP64 and in the residue arithmetic, so the results are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 128, 129, 256, 257, 300, 513])
@pytest.mark.parametrize("m,k", [(1, 1), (31, 130), (160, 128), (161, 129), (224, 40), (300, 257),
                                 (385, 64), (700, 33)])
def test_exact_products(uw12lib, cuda_device, m, n, k):
    import torch
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    for nb, shared in ((1, False), (3, False), (3, True)):
        A = rng.integers(-9, 10, (1 if shared else nb, k, m)).astype(np.float64)
        B = rng.integers(-9, 10, (nb, n, k)).astype(np.float64)
        C = rng.integers(-9, 10, (nb, n, m)).astype(np.float64)
        dA, dB, dC = (torch.from_numpy(x).cuda() for x in (A, B, C.copy()))
        uw12lib.dgemm_split(m, n, k, 1.0, dA.data_ptr(), m, False, dB.data_ptr(), k, False, 2.0,
                            dC.data_ptr(), m, nbo1=nb,
                            so=(0 if shared else m * k, 0, n * k, 0, m * n, 0))
        torch.cuda.synchronize()
        ref = np.stack([B[b] @ A[0 if shared else b] for b in range(nb)]) + 2.0 * C
        assert np.array_equal(dC.cpu().numpy(), ref)


def test_long_contraction(uw12lib, cuda_device):
    """More K than one accumulator chunk holds (65536), for both kinds of tile."""
    import torch
    k = 70000
    rng = np.random.default_rng(3)
    for m, n in ((160, 300), (96, 256)):
        A = rng.integers(-3, 4, (k, m)).astype(np.float64)
        B = rng.integers(-3, 4, (n, k)).astype(np.float64)
        dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
        dC = torch.empty((n, m), dtype=torch.float64, device="cuda")
        uw12lib.dgemm_split(m, n, k, 1.0, dA.data_ptr(), m, False, dB.data_ptr(), k, False, 0.0,
                            dC.data_ptr(), m)
        torch.cuda.synchronize()
        assert np.array_equal(dC.cpu().numpy(), B @ A)


@pytest.mark.parametrize("a_k", [False, True])
@pytest.mark.parametrize("b_n", [False, True])
@pytest.mark.parametrize("m,n,k,nbr,pad,off", [(33, 65, 20, 3, 0, 0), (32, 64, 21, 3, 0, 0),
                                               (34, 66, 20, 3, 1, 0), (34, 66, 20, 3, 0, 1),
                                               (1, 1, 130, 1, 0, 0), (515, 131, 258, 2, 2, 0)])
def test_operand_loads(uw12lib, cuda_device, a_k, b_n, m, n, k, nbr, pad, off):
    """Operands read in pairs and singly: odd and even extents, leading dimensions and
    base addresses, both orders, several reduction batches."""
    import torch
    rng = np.random.default_rng(m + n + k)
    lda, ldb = (k if a_k else m) + pad, (n if b_n else k) + pad
    A = rng.integers(-9, 10, off + nbr * (m if a_k else k) * lda).astype(np.float64)
    B = rng.integers(-9, 10, off + nbr * (k if b_n else n) * ldb).astype(np.float64)
    Av = A[off:].reshape(nbr, m if a_k else k, lda)
    Bv = B[off:].reshape(nbr, k if b_n else n, ldb)
    ref = sum((x[:, :k] if a_k else x[:, :m].T) @ (y[:, :n] if b_n else y[:, :k].T)
              for x, y in zip(Av, Bv))
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    for moduli in (7, 14, 16):
        dC = torch.full((n, m), float("nan"), dtype=torch.float64, device="cuda")
        uw12lib.dgemm_split(m, n, k, 1.0, dA.data_ptr() + 8 * off, lda, a_k,
                            dB.data_ptr() + 8 * off, ldb, b_n, 0.0, dC.data_ptr(), m, nbr1=nbr,
                            sr=(Av[0].size, 0, Bv[0].size, 0), n_moduli=moduli)
        torch.cuda.synchronize()
        assert np.array_equal(dC.cpu().numpy().T, ref)
