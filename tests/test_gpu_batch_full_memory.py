"""A batch of small molecules on a device that holds one of them at a time in chunks, but
not eight: no molecule fails, and each result is that of a single call on the empty device
(1e-12 relative: the chunked terms are summed in another order)."""
import numpy as np
import pytest

from tests.parity_cases import Case, make_case

pytestmark = pytest.mark.gpu


def test_batch_with_little_memory_left(uw12lib, cuda_device):
    import torch
    L = uw12lib
    c = Case("full", 96, 288, 384, (18,), (17,), "baseline", 5, 8.0)
    d = make_case(c)
    W = L.setup_base_integrals(d.W3, d.W2, d.W3_ri)
    V = L.setup_base_integrals(d.V3, d.V2, d.V3_ri)
    WV = L.setup_base_integrals(d.WV3, d.WV2)
    A = L.setup_abs_projectors(d.S, c.n_ao, c.n_ri)
    e1, f1, _ = L.form_fock(W, V, WV, A, d.orbitals, d.occ, c.n_active, True, True, 1.0, 0.5)
    mol = {"W": W, "V": V, "WV": WV, "abs": A, "orbitals": d.orbitals, "occ": d.occ,
           "n_active": list(c.n_active)}
    torch.cuda.synchronize()
    L.trim_memory()
    torch.cuda.empty_cache()
    left = 400 << 20  # a single evaluation takes about 600 MiB unchunked
    fill = []
    try:
        free, _ = torch.cuda.mem_get_info()
        while free > left + (16 << 20):
            fill.append(torch.empty(min(free - left, 8 << 30), dtype=torch.uint8, device="cuda"))
            free, _ = torch.cuda.mem_get_info()
        res = L.fock_batched([mol] * 12, True, True, 1.0, 0.5, n_streams=8)
    finally:
        fill.clear()
        torch.cuda.empty_cache()
    for e, f, _ in res:
        assert abs(e - e1) <= 1e-12 * abs(e1)
        assert np.max(np.abs(f[0] - f1[0])) <= 1e-12 * np.max(np.abs(f1[0]))
