"""How often an integral-direct evaluation without same-spin terms runs the producers.

Form over aux functions (60 AO, 100 DF and 60 RI functions, 18 orbitals: 171 pairs against
100 aux functions), closed shell, a 9.6 MB budget for the chunks: V's integrals are produced
once for the transforms and once per chunk of W's aux functions.  The chunk has the budget
but for V's blocks (a quarter for RI, a sixteenth for AO), and holds two R' x N matrices and
a packed column per aux function, so 0.825 M / 16.2 k = 50 of the 100: two chunks.

Two spins whose chunks fit whole, host producers: over aux functions W and V are produced once
for the transforms and once more, over orbital pairs once more for each spin, which costs more
across the host link than the pairs save.  Each tensor is asked for twice, and the block read
ahead of the second request is dropped: at most three passes.

The results are the oracle's (tests/test_gpu_parity.py's tolerances for well-conditioned inputs)."""
import ctypes

import numpy as np
import pytest

from tests.parity_cases import Case, make_case, oracle_form_fock

pytestmark = pytest.mark.gpu


def _check(got, d):
    e_ref, f_ref, _ = oracle_form_fock(d, False, True, 1.0, 0.0)
    assert abs(got[0] - e_ref) <= 1e-8 * max(1.0, abs(e_ref))
    for x, y in zip(got[1], f_ref):
        assert np.max(np.abs(x - y)) <= 1e-7 * max(1.0, np.max(np.abs(y)))


def _handles(L, d, c, columns):
    import torch
    from libuw12_b200.distributed import device_view

    def device(name, x):
        t = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()

        def fn(first, count, out, ld, stream):
            columns[name] = columns.get(name, 0) + count
            with torch.cuda.stream(torch.cuda.ExternalStream(stream) if stream else
                                   torch.cuda.default_stream()):
                device_view(out, ld * count, t.device).view(count, ld)[:, :x.shape[0]] = \
                    t[first:first + count]
        return fn

    # device producers: nothing is read ahead, so the count is what the evaluation asks for
    return [L.setup_base_integrals_callback(j2, device(n, j3), device(n + "_ri", ri), c.n_ao,
                                            c.n_df, c.n_ri, False, False, device=True)
            for n, j3, j2, ri in (("W", d.W3, d.W2, d.W3_ri), ("V", d.V3, d.V2, d.V3_ri))]


def test_aux_form_chunks(uw12lib, cuda_device):
    L = uw12lib
    c = Case("aux", 60, 100, 60, (18,), (18,), "unit", 3)
    d = make_case(c)
    columns = {}
    W, V = _handles(L, d, c, columns)
    WV = L.setup_base_integrals(d.WV3, d.WV2)
    A = L.setup_abs_projectors(d.S, c.n_ao, c.n_ri)
    L.set_memory_budget(8 * 1200000)
    try:
        got = L.form_fock(W, V, WV, A, d.orbitals, d.occ, c.n_active, False, True, 1.0, 0.0)
    finally:
        L.set_memory_budget(0)
    _check(got, d)
    assert columns == {"W": 2 * 100, "W_ri": 2 * 100, "V": 3 * 100, "V_ri": 3 * 100}


def test_host_producers_of_two_spins(uw12lib, cuda_device):
    L = uw12lib
    c = Case("host", 24, 72, 96, (3, 2), (3, 2), "unit", 4)
    d = make_case(c)
    columns = {}

    def produce(name, x):
        def fn(first, count, out, ld, stream):
            columns[name] = columns.get(name, 0) + count
            v = np.ctypeslib.as_array(ctypes.cast(out, ctypes.POINTER(ctypes.c_double)),
                                      shape=(count, ld))
            v[:, :x.shape[0]] = x[:, first:first + count].T
        return fn

    W, V = [L.setup_base_integrals_callback(j2, produce(n, j3), produce(n + "_ri", ri), c.n_ao,
                                            c.n_df, c.n_ri, False, False)
            for n, j3, j2, ri in (("W", d.W3, d.W2, d.W3_ri), ("V", d.V3, d.V2, d.V3_ri))]
    WV = L.setup_base_integrals(d.WV3, d.WV2)
    A = L.setup_abs_projectors(d.S, c.n_ao, c.n_ri)
    got = L.form_fock(W, V, WV, A, d.orbitals, d.occ, c.n_active, False, True, 1.0, 0.0)
    for h in (W, V):  # joins what is being read ahead
        h.close()
    _check(got, d)
    assert max(columns.values()) <= 3 * 72, columns
