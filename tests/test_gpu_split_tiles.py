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
