"""Fock terms over symmetric orbital pairs against the oracle: whole, and in chunks of
every size that a range of budgets gives (mirror images inside a chunk, behind it, and
none), frozen core, matrices of odd and even size, over pairs and over aux functions, and
the shards of the pair sums on one device.  Tolerances: tests/test_gpu_parity.py's for
well-conditioned inputs."""
import numpy as np
import pytest

from tests.parity_cases import Case, make_case, oracle_form_fock

pytestmark = pytest.mark.gpu

CASES = [Case("odd", 13, 60, 18, (8,), (8,), "unit", 1),
         Case("odd_core", 13, 60, 18, (8, 7), (6, 4), "unit", 2),
         Case("even_core", 12, 60, 17, (9,), (7,), "unit", 3),
         Case("aux_form", 12, 13, 11, (9, 8), (8, 8), "unit", 4),
         Case("one_active", 11, 40, 9, (4, 3), (1, 1), "unit", 5)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
@pytest.mark.parametrize("s_ss", [0.5, 0.0])
@pytest.mark.parametrize("budget_kib", [0, 64, 160, 320, 640])
def test_pairs_match_oracle(uw12lib, cuda_device, case, s_ss, budget_kib):
    L = uw12lib
    d = make_case(case)
    W = L.setup_base_integrals(d.W3, d.W2, d.W3_ri)
    V = L.setup_base_integrals(d.V3, d.V2, d.V3_ri)
    WV = L.setup_base_integrals(d.WV3, d.WV2)
    A = L.setup_abs_projectors(d.S, case.n_ao, case.n_ri)
    try:
        L.set_memory_budget(budget_kib << 10)
        e, f, _ = L.form_fock(W, V, WV, A, d.orbitals, d.occ, case.n_active, s_ss != 0, True, 1.0,
                              s_ss)
    finally:
        L.set_memory_budget(0)
    e_ref, f_ref, _ = oracle_form_fock(d, s_ss != 0, True, 1.0, s_ss)
    assert abs(e - e_ref) <= 1e-8 * max(1.0, abs(e_ref))
    for x, y in zip(f, f_ref):
        assert np.max(np.abs(x - y)) <= 1e-7 * max(1.0, np.max(np.abs(y)))
