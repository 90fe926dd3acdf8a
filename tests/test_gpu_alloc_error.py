"""A call that fails for device memory leaves no error behind: the host thread's next CUDA
check (the caller's) and next evaluation succeed, with the results of an empty device."""
import pytest

from tests.parity_cases import Case, make_case

pytestmark = pytest.mark.gpu


def test_failed_allocation_leaves_no_error(uw12lib, cuda_device):
    import torch
    L = uw12lib
    c = Case("full", 96, 288, 384, (20,), (19,), "baseline", 5, 8.0)
    d = make_case(c)
    W = L.setup_base_integrals(d.W3, d.W2, d.W3_ri)
    V = L.setup_base_integrals(d.V3, d.V2, d.V3_ri)
    WV = L.setup_base_integrals(d.WV3, d.WV2)
    A = L.setup_abs_projectors(d.S, c.n_ao, c.n_ri)

    def evaluate():
        return L.form_fock(W, V, WV, A, d.orbitals, d.occ, c.n_active, True, True, 1.0, 0.5)

    whole = evaluate()
    torch.cuda.synchronize()
    L.trim_memory()
    torch.cuda.empty_cache()
    left = 24 << 20  # less than any evaluation of this size takes
    fill = []
    try:
        free, _ = torch.cuda.mem_get_info()
        while free > left + (16 << 20):
            fill.append(torch.empty(min(free - left, 8 << 30), dtype=torch.uint8, device="cuda"))
            free, _ = torch.cuda.mem_get_info()
        with pytest.raises(L.UW12Error, match="status 4"):
            evaluate()
    finally:
        fill.clear()
        torch.cuda.empty_cache()
    x = torch.zeros(4, device="cuda") + 1.0  # the caller's own kernel and check
    assert float(x.sum()) == 4.0
    again = evaluate()
    assert again[0] == whole[0]
