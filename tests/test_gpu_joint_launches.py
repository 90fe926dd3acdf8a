"""Products of W and V in one launch: stored integrals (formed side by side) against the
oracle and against produced ones (one after the other), at odd and even sizes, for energies
and Fock matrices, closed and open shell, frozen core, with and without the same-spin
terms.  Tolerances: tests/test_gpu_parity.py's for well-conditioned inputs."""
import ctypes

import numpy as np
import pytest

from tests.parity_cases import Case, make_case, oracle_form_fock

pytestmark = pytest.mark.gpu

CASES = [Case("odd", 15, 43, 21, (4,), (4,), "unit", 1),
         Case("odd_open", 15, 43, 21, (4, 3), (3, 2), "unit", 2),
         Case("even_open", 16, 48, 20, (5, 4), (5, 4), "unit", 3),
         Case("tiny", 3, 5, 4, (1,), (1,), "unit", 4),
         Case("one_spin", 10, 31, 12, (3, 2), (3, 0), "unit", 5),
         Case("no_active", 10, 31, 12, (2,), (0,), "unit", 6)]


def _produce(x):
    def fn(first, count, out, ld, stream):
        v = np.ctypeslib.as_array(ctypes.cast(out, ctypes.POINTER(ctypes.c_double)),
                                  shape=(count, ld))
        v[:, :x.shape[0]] = x[:, first:first + count].T
    return fn


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
@pytest.mark.parametrize("s_ss", [0.5, 0.0])
@pytest.mark.parametrize("fock", [True, False])
def test_side_by_side(uw12lib, cuda_device, case, s_ss, fock):
    L = uw12lib
    d = make_case(case)
    N, M, R = case.n_ao, case.n_df, case.n_ri
    A = L.setup_abs_projectors(d.S, N, R)
    stored = [L.setup_base_integrals(d.W3, d.W2, d.W3_ri),
              L.setup_base_integrals(d.V3, d.V2, d.V3_ri), L.setup_base_integrals(d.WV3, d.WV2)]
    produced = [L.setup_base_integrals_callback(j2, _produce(j3), _produce(ri), N, M, R, False,
                                                False)
                for j3, j2, ri in ((d.W3, d.W2, d.W3_ri), (d.V3, d.V2, d.V3_ri))] + stored[2:]
    e_ref, f_ref, _ = oracle_form_fock(d, s_ss != 0, fock, 1.0, s_ss)
    for handles in (stored, produced):
        e, f, _ = L.form_fock(*handles, A, d.orbitals, d.occ, case.n_active, s_ss != 0, fock, 1.0,
                              s_ss)
        assert abs(e - e_ref) <= 1e-8 * max(1.0, abs(e_ref))
        if fock:
            for x, y in zip(f, f_ref):
                assert np.max(np.abs(x - y)) <= 1e-7 * max(1.0, np.max(np.abs(y)))
