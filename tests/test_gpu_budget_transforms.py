"""The transforms of stored W and V keep to an explicit chunk budget: the unpacked blocks
of both (83 MB at this size) are formed whole under a large budget, in chunks under a
small one, with the same energy (1e-12 relative: the sums run in another order).  The
device memory that the library takes is read from the free memory around the call on a
trimmed pool: one 32 MiB block of small buffers, and nothing of the size of the blocks."""
import pytest

from tests.parity_cases import Case, make_case

pytestmark = pytest.mark.gpu

CASE = Case("thin", 120, 360, 60, (1,), (1,), "baseline", 5, 8.0)


def test_small_budget_chunks_the_transforms(uw12lib, cuda_device):
    import torch
    L = uw12lib
    d = make_case(CASE)
    W = L.setup_base_integrals(d.W3, d.W2, d.W3_ri)
    V = L.setup_base_integrals(d.V3, d.V2, d.V3_ri)
    WV = L.setup_base_integrals(d.WV3, d.WV2)
    A = L.setup_abs_projectors(d.S, CASE.n_ao, CASE.n_ri)

    def energy(budget):
        L.set_memory_budget(budget)
        try:
            L.trim_memory()
            torch.cuda.synchronize()
            free0, _ = torch.cuda.mem_get_info()
            n0 = L.launch_count()
            e, _, _ = L.form_fock(W, V, WV, A, d.orbitals, d.occ, CASE.n_active, False, False,
                                  1.0, 0.0)
            torch.cuda.synchronize()
            free1, _ = torch.cuda.mem_get_info()
            return e, L.launch_count() - n0, free0 - free1
        finally:
            L.set_memory_budget(0)

    energy(1 << 30)  # loads the kernels
    whole, n_whole, _ = energy(1 << 30)
    # 8 MiB: the whole transforms (2.2 MB) fit, the unpacked blocks do not; at most half
    # of it (36 of 360 aux functions) is unpacked at a time
    chunked, n_chunked, taken = energy(8 << 20)
    assert abs(chunked - whole) <= 1e-12 * abs(whole)
    assert n_chunked >= n_whole + 2 * 2 * 9  # an unpack and a product per chunk, W and V
    assert taken <= 96 << 20
