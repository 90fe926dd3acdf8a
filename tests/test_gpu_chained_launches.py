"""Products and streaming kernels whose blocks may start before the previous kernel of
their stream has finished: every step reads what the step before wrote and overwrites
what that step read.  Signed permutation matrices and integer data, so every product is
exact and the result has to be equal to numpy's (tolerance zero), on the legacy, a side
and a captured stream, and behind an event of another stream."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (rows, columns, split): one tile, split-K with its reduction, several waves of tiles
SIZES = [(5, 3, 0), (64, 64, 0), (96, 40, 6), (700, 33, 16), (1500, 1500, 0), (513, 4097, 0)]
STEPS = 24


def _problem(m, n):
    rng = np.random.default_rng(m + 31 * n)
    perm = [rng.permutation(m) for _ in range(3)]
    sign = [rng.choice([-1.0, 1.0], m) for _ in range(3)]
    A = np.zeros((3, m, m))  # column-major m x m: A[q][col, row]
    for q in range(3):
        A[q][perm[q], np.arange(m)] = sign[q]
    X = rng.integers(-9, 10, (n, m)).astype(np.float64)
    want = X
    for s in range(STEPS):
        q = s % 3
        want = sign[q] * want[:, perm[q]]
    return A, X, want


def _chain(lib, m, n, split, dA, dX, dY):
    # X -> Y -> X -> ...: each product overwrites what the previous one read
    src, dst = dX, dY
    for s in range(STEPS):
        lib.dgemm(m, n, m, 1.0, dA[s % 3].data_ptr(), m, False, src.data_ptr(), m, False, 0.0,
                  dst.data_ptr(), m, split=split)
        src, dst = dst, src
    return src


@pytest.mark.parametrize("where", ["default", "side", "event", "captured"])
@pytest.mark.parametrize("m,n,split", SIZES)
def test_dependent_products(uw12lib, cuda_device, m, n, split, where):
    import torch
    A, X, want = _problem(m, n)
    dA, x = torch.from_numpy(A).cuda(), torch.from_numpy(X).cuda()
    dX, dY = x.clone(), torch.full_like(x, float("nan"))
    torch.cuda.synchronize()
    if where == "default":
        out = _chain(uw12lib, m, n, split, dA, dX, dY)
    else:
        stream, other = torch.cuda.Stream(), torch.cuda.Stream()
        uw12lib.set_stream(stream.cuda_stream)
        try:
            if where == "side":
                out = _chain(uw12lib, m, n, split, dA, dX, dY)
            elif where == "event":
                # the operand arrives on another stream, behind copies that take a while;
                # the product before the wait is the chained launch's predecessor
                dX.zero_()
                big = torch.ones(1 << 26, device="cuda", dtype=torch.float64)
                torch.cuda.synchronize()
                uw12lib.dgemm(m, n, m, 1.0, dA[0].data_ptr(), m, False, dX.data_ptr(), m, False,
                              0.0, dY.data_ptr(), m, split=split)
                with torch.cuda.stream(other):
                    for _ in range(8):
                        big.mul_(1.0)
                    other.wait_stream(stream)  # the product above reads dX
                    dX.copy_(x)
                stream.wait_stream(other)
                out = _chain(uw12lib, m, n, split, dA, dX, dY)
            else:
                _chain(uw12lib, m, n, split, dA, dX, dY)  # kernels loaded, pools filled
                stream.synchronize()
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=stream):
                    out = _chain(uw12lib, m, n, split, dA, dX, dY)
                for _ in range(2):
                    dX.copy_(x)
                    torch.cuda.synchronize()
                    graph.replay()
                    torch.cuda.synchronize()
        finally:
            stream.synchronize()
            uw12lib.set_stream(0)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
