"""A producer that takes most of the device's memory for itself at its first call, in an
evaluation that cannot be repeated (its gradients leave through a sink): the later phases
chunk within what is left, with the results of the empty device (1e-12 relative: the
chunked terms are summed in another order)."""
import ctypes

import numpy as np
import pytest

from tests.parity_cases import Case, make_case

pytestmark = pytest.mark.gpu


def test_producer_that_takes_memory(uw12lib, cuda_device):
    import torch
    L = uw12lib
    c = Case("full", 96, 288, 384, (30,), (29,), "baseline", 5, 8.0)
    d = make_case(c)
    fill = []
    left = [0]

    def produce(first, count, out, ld, stream):
        free, _ = torch.cuda.mem_get_info()
        while left[0] and free > left[0] + (16 << 20):
            fill.append(torch.empty(min(free - left[0], 8 << 30), dtype=torch.uint8,
                                    device="cuda"))
            free, _ = torch.cuda.mem_get_info()
        v = np.ctypeslib.as_array(ctypes.cast(out, ctypes.POINTER(ctypes.c_double)),
                                  shape=(count, ld))
        v[:, :d.WV3.shape[0]] = d.WV3[:, first:first + count].T

    W = L.setup_base_integrals(d.W3, d.W2, d.W3_ri)
    V = L.setup_base_integrals(d.V3, d.V2, d.V3_ri)
    WV = L.setup_base_integrals_callback(d.WV2, produce, None, c.n_ao, c.n_df, 0, False, False)
    A = L.setup_abs_projectors(d.S, c.n_ao, c.n_ri)

    def gradients():
        out = np.zeros_like(d.W3)

        def sink(first, count, block):
            out[:, first:first + count] = block
        e, f, _, _ = L.fock_backward_blocks(W, V, WV, A, d.orbitals, d.occ, c.n_active, 1.0, 0.5,
                                            {"W3": sink}, indirect_term=True)
        return e, f, out

    whole = gradients()
    torch.cuda.synchronize()
    L.trim_memory()
    torch.cuda.empty_cache()
    left[0] = 1000 << 20  # the unchunked Fock matrix takes about 2 GB
    try:
        tight = gradients()
    finally:
        fill.clear()
        torch.cuda.empty_cache()
    assert abs(tight[0] - whole[0]) <= 1e-12 * abs(whole[0])
    assert np.max(np.abs(tight[1][0] - whole[1][0])) <= 1e-12 * np.max(np.abs(whole[1][0]))
    assert np.max(np.abs(tight[2] - whole[2])) <= 1e-12 * np.max(np.abs(whole[2]))
