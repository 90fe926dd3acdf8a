"""Both forms of the t~ dX Fock term (over orbital pairs, over aux functions) against
the oracle: few and many occupied orbitals per aux function, closed and open shell,
frozen core, with and without the same-spin terms, whole and in chunks of one occupied
orbital (64 KiB budget), stored and produced integrals, FP64 and every product split.
Tolerances: tests/test_gpu_parity.py's for well-conditioned inputs."""
import numpy as np
import pytest

from tests.parity_cases import Case, make_case, oracle_form_fock

pytestmark = pytest.mark.gpu

CASES = [Case("few", 13, 40, 17, (3,), (3,), "unit", 1),
         Case("few_core", 13, 40, 17, (4, 3), (2, 1), "unit", 2),
         Case("many", 12, 9, 11, (9,), (8,), "unit", 3),
         Case("many_open", 12, 9, 11, (9, 7), (9, 7), "unit", 4),
         Case("one_spin", 9, 14, 8, (3, 2), (3, 0), "unit", 5)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
@pytest.mark.parametrize("scales", [(1.0, 0.5), (1.0, 0.0), (0.0, 1.0)])
@pytest.mark.parametrize("mode", ["whole", "chunks", "produced", "split"])
def test_fock_matches_oracle(uw12lib, cuda_device, case, scales, mode):
    L = uw12lib
    d = make_case(case)
    N, M, R = case.n_ao, case.n_df, case.n_ri

    def handle(j3, j2, ri):
        if mode != "produced":
            return L.setup_base_integrals(j3, j2, ri)

        def fn(x):
            def produce(first, count, out, ld, stream):
                import ctypes
                v = np.ctypeslib.as_array(ctypes.cast(out, ctypes.POINTER(ctypes.c_double)),
                                          shape=(count, ld))
                v[:, :x.shape[0]] = x[:, first:first + count].T
            return produce

        return L.setup_base_integrals_callback(j2, fn(j3), fn(ri) if ri is not None else None, N,
                                               M, R if ri is not None else 0, False, False)

    W, V, WV = handle(d.W3, d.W2, d.W3_ri), handle(d.V3, d.V2, d.V3_ri), handle(d.WV3, d.WV2, None)
    A = L.setup_abs_projectors(d.S, N, R)
    s_os, s_ss = scales
    try:
        if mode in ("chunks", "produced"):
            L.set_memory_budget(64 << 10)
        if mode == "split":
            L.set_precision(14)
            L.set_split_threshold(0.0)
        e, f, _ = L.form_fock(W, V, WV, A, d.orbitals, d.occ, case.n_active, s_ss != 0, True, s_os,
                              s_ss)
    finally:
        L.set_memory_budget(0)
        L.set_precision(0)
        L.set_split_threshold(2e9)
    e_ref, f_ref, _ = oracle_form_fock(d, s_ss != 0, True, s_os, s_ss)
    assert abs(e - e_ref) <= 1e-8 * max(1.0, abs(e_ref))
    for x, y in zip(f, f_ref):
        assert np.max(np.abs(x - y)) <= 1e-7 * max(1.0, np.max(np.abs(y)))
