"""An evaluation that runs out of memory is repeated in chunks: on a device with 300 MiB left
it launches more than twice the kernels of the unchunked evaluation, so the repeat alone
(all but the failed attempt's, fewer than one evaluation's) launches more than one that runs
whole, and so does the same call under an explicit budget of that size."""
import numpy as np
import pytest

from tests.parity_cases import Case, make_case

pytestmark = pytest.mark.gpu


def test_repeat_is_chunked(uw12lib, cuda_device):
    import torch
    L = uw12lib
    c = Case("full", 96, 288, 384, (20,), (19,), "baseline", 5, 8.0)
    d = make_case(c)
    W = L.setup_base_integrals(d.W3, d.W2, d.W3_ri)
    V = L.setup_base_integrals(d.V3, d.V2, d.V3_ri)
    WV = L.setup_base_integrals(d.WV3, d.WV2)
    A = L.setup_abs_projectors(d.S, c.n_ao, c.n_ri)

    def evaluate(budget=0):
        L.set_memory_budget(budget)
        try:
            n0 = L.launch_count()
            e, f, _ = L.form_fock(W, V, WV, A, d.orbitals, d.occ, c.n_active, True, True, 1.0, 0.5)
            return e, f[0], L.launch_count() - n0
        finally:
            L.set_memory_budget(0)

    whole = evaluate()
    budgeted = evaluate(60 << 20)
    assert budgeted[2] > whole[2]
    torch.cuda.synchronize()
    L.trim_memory()
    torch.cuda.empty_cache()
    left = 300 << 20
    fill = []
    try:
        free, _ = torch.cuda.mem_get_info()
        while free > left + (16 << 20):
            fill.append(torch.empty(min(free - left, 8 << 30), dtype=torch.uint8, device="cuda"))
            free, _ = torch.cuda.mem_get_info()
        tight = evaluate()
    finally:
        fill.clear()
        torch.cuda.empty_cache()
    print("launches", whole[2], budgeted[2], tight[2])
    assert tight[2] - whole[2] > whole[2]
    for x in (tight, budgeted):
        assert abs(x[0] - whole[0]) <= 1e-12 * abs(whole[0])
        assert np.max(np.abs(x[1] - whole[1])) <= 1e-12 * np.max(np.abs(whole[1]))
