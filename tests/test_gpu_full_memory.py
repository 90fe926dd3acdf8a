"""An evaluation whose whole chunks an almost empty device would hold, on a device
with little memory left: its first attempt runs out of memory, the second chunks
within what is there, and the results are those of the same call on the empty
device (1e-12 relative: the chunked terms are summed in another order)."""
import numpy as np
import pytest

from tests.parity_cases import Case, make_case

pytestmark = pytest.mark.gpu


def test_evaluation_with_little_memory_left(uw12lib, cuda_device):
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

    n0 = L.launch_count()
    whole = evaluate()
    n_whole = L.launch_count() - n0
    torch.cuda.synchronize()
    L.trim_memory()
    torch.cuda.empty_cache()
    left = 400 << 20  # the unchunked evaluation takes about 700 MiB
    fill = []
    try:
        free, _ = torch.cuda.mem_get_info()
        while free > left + (16 << 20):
            fill.append(torch.empty(min(free - left, 8 << 30), dtype=torch.uint8, device="cuda"))
            free, _ = torch.cuda.mem_get_info()
        n0 = L.launch_count()
        tight = evaluate()
        n_tight = L.launch_count() - n0
    finally:
        fill.clear()
        torch.cuda.empty_cache()
    assert n_tight > n_whole  # repeated, in chunks
    assert abs(tight[0] - whole[0]) <= 1e-12 * abs(whole[0])
    assert np.max(np.abs(tight[1][0] - whole[1][0])) <= 1e-12 * np.max(np.abs(whole[1][0]))
