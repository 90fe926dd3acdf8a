"""Packed-symmetric storage at the edges of the streaming kernels' 32 x 32 tiles:
energy and Fock matrix against the oracle, and the packed gradients against the CPU
adjoint, for AO counts around one and two tiles.  Tolerances: as
tests/test_gpu_parity.py (well-conditioned inputs) and tests/test_gpu_adjoint.py."""
import numpy as np
import pytest

from oracle import uw12_oracle as O
from tests import adjoint_ref as AR
from tests.parity_cases import Case, make_case, oracle_form_fock

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ao", [1, 31, 32, 33, 64, 65])
def test_tile_edges(uw12lib, cuda_device, n_ao):
    o = min(3, n_ao)
    case = Case("tiles", n_ao, 9, 7, (o, 1), (o, 1), "unit", n_ao)
    d = make_case(case)
    W = uw12lib.setup_base_integrals(d.W3, d.W2, d.W3_ri)
    V = uw12lib.setup_base_integrals(d.V3, d.V2, d.V3_ri)
    WV = uw12lib.setup_base_integrals(d.WV3, d.WV2)
    A = uw12lib.setup_abs_projectors(d.S, case.n_ao, case.n_ri)
    args = (W, V, WV, A, d.orbitals, d.occ, case.n_active)
    e, f, _ = uw12lib.form_fock(*args, True, True, 1.0, 0.5)
    e_ref, f_ref, _ = oracle_form_fock(d, True, True, 1.0, 0.5)
    assert abs(e - e_ref) <= 1e-8 * max(1.0, abs(e_ref))
    for a, b in zip(f, f_ref):
        assert np.max(np.abs(a - b)) <= 1e-7 * max(1.0, np.max(np.abs(b)))
    _, _, _, g = uw12lib.fock_backward(*args, 1.0, 0.5)
    ref = AR.direct_adjoint(O.BaseIntegrals(d.W3, d.W2, d.W3_ri),
                            O.BaseIntegrals(d.V3, d.V2, d.V3_ri), O.BaseIntegrals(d.WV3, d.WV2),
                            O.calculate_abs_projectors(d.S, case.n_ao, case.n_ri), d.orbitals,
                            d.occ, list(case.n_active), 1.0, 0.5)
    for key in ("W3", "V3", "WV3"):
        assert np.max(np.abs(g[key] - ref[key])) <= 1e-9 * np.max(np.abs(ref[key])), key
