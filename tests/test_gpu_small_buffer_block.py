"""An evaluation on a device with just the memory for its large buffers: the block that
serves its small buffers (32 MiB, of which this one uses 5) does not get in their way.
Frozen core, so that nothing but the AO transforms is large: four buffers of 41 to 48 MiB
at a time under the given budget."""
import pytest

from tests.parity_cases import Case, make_case

pytestmark = pytest.mark.gpu


def test_large_buffers_come_before_the_block(uw12lib, cuda_device):
    import torch
    L = uw12lib
    c = Case("core", 300, 300, 100, (60,), (1,), "baseline", 5, 8.0)
    d = make_case(c)
    W = L.setup_base_integrals(d.W3, d.W2, d.W3_ri)
    V = L.setup_base_integrals(d.V3, d.V2, d.V3_ri)
    WV = L.setup_base_integrals(d.WV3, d.WV2)
    A = L.setup_abs_projectors(d.S, c.n_ao, c.n_ri)

    def energy():
        return L.form_fock(W, V, WV, A, d.orbitals, d.occ, c.n_active, False, False, 1.0, 0.0)[0]

    L.set_memory_budget(96 << 20)
    fill = []
    try:
        whole = energy()
        torch.cuda.synchronize()
        L.trim_memory()
        torch.cuda.empty_cache()
        left = 212 << 20
        free, _ = torch.cuda.mem_get_info()
        while free > left + (4 << 20):
            fill.append(torch.empty(min(free - left, 8 << 30), dtype=torch.uint8, device="cuda"))
            free, _ = torch.cuda.mem_get_info()
        tight = energy()
    finally:
        L.set_memory_budget(0)
        fill.clear()
        torch.cuda.empty_cache()
    assert abs(tight - whole) <= 1e-12 * abs(whole)
