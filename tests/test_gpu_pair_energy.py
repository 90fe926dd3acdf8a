"""Same-spin three-electron energy and gradients over symmetric orbital pairs: energies
against the oracle and gradients against the CPU reverse sweep, whole and in chunks of
occupied orbitals of several sizes, with and without frozen core, odd and even sizes.
Tolerances: those of tests/test_gpu_parity.py (well-conditioned inputs) and
tests/test_gpu_adjoint_same_spin.py."""
import numpy as np
import pytest

from oracle import uw12_oracle as O
from tests import adjoint_ref as AR
from tests.parity_cases import Case, make_case, oracle_form_fock

pytestmark = pytest.mark.gpu

CASES = [Case("closed", 11, 30, 16, (6,), (6,), "unit", 1),
         Case("core", 12, 31, 17, (7, 6), (5, 3), "unit", 2),
         Case("one_active", 9, 22, 10, (4, 3), (1, 1), "unit", 3)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
@pytest.mark.parametrize("budget_kib", [0, 64, 128, 256])
def test_energy_and_gradients(uw12lib, cuda_device, case, budget_kib):
    L = uw12lib
    d = make_case(case)
    W = L.setup_base_integrals(d.W3, d.W2, d.W3_ri)
    V = L.setup_base_integrals(d.V3, d.V2, d.V3_ri)
    WV = L.setup_base_integrals(d.WV3, d.WV2)
    A = L.setup_abs_projectors(d.S, case.n_ao, case.n_ri)
    act = list(case.n_active)
    try:
        L.set_memory_budget(budget_kib << 10)
        energy = L.uw12_energy(W, V, WV, A, d.orbitals, d.occ, act, 1.0, 0.5)
        _, _, _, g = L.fock_backward(W, V, WV, A, d.orbitals, d.occ, act, 1.0, 0.5,
                                     indirect_term=True)
    finally:
        L.set_memory_budget(0)
    e_ref, _, _ = oracle_form_fock(d, True, False, 1.0, 0.5)
    assert abs(energy - e_ref) <= 1e-8 * max(1.0, abs(e_ref))
    Wo = O.BaseIntegrals(d.W3, d.W2, d.W3_ri)
    Vo = O.BaseIntegrals(d.V3, d.V2, d.V3_ri)
    WVo = O.BaseIntegrals(d.WV3, d.WV2)
    absp = O.calculate_abs_projectors(d.S, case.n_ao, case.n_ri)
    gd = AR.direct_adjoint(Wo, Vo, WVo, absp, d.orbitals, d.occ, act, 1.0, 0.5)
    gi = AR.indirect_adjoint(Wo, Vo, WVo, absp, d.orbitals, d.occ, act)
    for key in gd:
        r = gd[key] + 0.5 * gi[key]
        scale = max(np.max(np.abs(r)), np.max(np.abs(gd[key])), 0.5 * np.max(np.abs(gi[key])))
        assert np.max(np.abs(g[key] - r)) <= 1e-9 * scale, key
