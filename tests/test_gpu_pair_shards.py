"""Shards of the Fock terms over orbital pairs on the GPU.

* With frozen core and ranges that start inside the active orbitals (mirror images behind
  the first block), whole and in chunks, three shards on threads of one device add up to the
  oracle's Fock matrix (tests/test_gpu_parity.py's tolerances for well-conditioned inputs).
* Eight shards of 64 active orbitals have about the same GEMM work.  A range ends within
  half an orbital's pairs (32) of its even place, so its pairs are 260 +- 32 (ratio 1.28),
  and all other work but shard 0's is dealt out evenly: at most 1.3 between shards 1 to 7.
  Even ranges of orbitals give shard 7 five times the pairs of shard 1."""
import numpy as np
import pytest

from tests.parity_cases import Case, make_case, oracle_form_fock
from tests.test_gpu_shards import _sharded

pytestmark = pytest.mark.gpu

CASES = [Case("core", 13, 60, 18, (9,), (7,), "unit", 1),
         Case("open_core", 12, 60, 17, (8, 7), (6, 4), "unit", 2),
         Case("one_active", 11, 40, 9, (4, 3), (1, 1), "unit", 5)]


def _handles(L, d, c):
    return (L.setup_base_integrals(d.W3, d.W2, d.W3_ri),
            L.setup_base_integrals(d.V3, d.V2, d.V3_ri), L.setup_base_integrals(d.WV3, d.WV2),
            L.setup_abs_projectors(d.S, c.n_ao, c.n_ri))


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
@pytest.mark.parametrize("s_ss", [0.5, 0.0])
@pytest.mark.parametrize("budget_kib", [0, 320])
def test_shards_inside_the_active_orbitals(uw12lib, cuda_device, case, s_ss, budget_kib):
    d = make_case(case)
    out = _sharded(uw12lib, _handles(uw12lib, d, case), d, case, 3, (1.0, s_ss), budget_kib << 10)
    e_ref, f_ref, _ = oracle_form_fock(d, s_ss != 0, True, 1.0, s_ss)
    assert abs(sum(o[0] for o in out) - e_ref) <= 1e-8 * max(1.0, abs(e_ref))
    for s, f in enumerate(f_ref):
        f_sum = sum(o[1][s] for o in out)
        assert np.max(np.abs(f_sum - f)) <= 1e-7 * max(1.0, np.max(np.abs(f)))


def test_shards_have_even_work(uw12lib, cuda_device):
    L = uw12lib
    c = Case("even", 64, 48, 40, (64,), (64,), "baseline", 5, 8.0)
    d = make_case(c)
    h = _handles(L, d, c)
    flops = []
    for shard in range(1, 8):
        # the others' parts of the intermediates are left out: the work is the same
        L.set_shard(shard, 8)
        L.set_allreduce(lambda ptr, count, stream: None)
        L.profile_enable(True)
        try:
            L.profile_read()
            L.form_fock(*h, d.orbitals, d.occ, c.n_active, True, True, 1.0, 0.5)
            flops.append(L.profile_read()["flops"])
        finally:
            L.profile_enable(False)
            L.set_allreduce(None)
            L.set_shard(0, 1)
    print(["%.3g" % f for f in flops])
    assert max(flops) <= 1.3 * min(flops)
