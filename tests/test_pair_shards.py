"""Shards of the Fock terms over orbital pairs.  The library's own ranges (csrc/kernels.cuh,
compiled into tests/cpp/pair_check.cpp) cover the orbitals with about equal numbers of pairs;
and with those ranges the pair sums of t~ dX and of the same-spin three-electron Fock, formed
over each range's distinct pairs on two gloo ranks and added up by the collective, equal the
sums over aux functions and over all pairs (1e-12 relative: sums of a few thousand terms)."""
import datetime
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch
import torch.distributed as dist
import torch.multiprocessing as mp

from oracle import uw12_oracle as O
from tests.parity_cases import Case, make_case
from tests.schedule_model import T3, sq_all
from tests.sharded_model import _h1, _h2
from tests.test_distributed_cpu import _free_port

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def pair_check(tmp_path_factory):
    out = tmp_path_factory.mktemp("cpp") / "pair_check"
    cmd = ["g++", "-std=c++17", "-O1", "-x", "c++", f"-I{ROOT / 'libuw12_b200' / 'csrc'}",
           "-I/usr/local/cuda/include", str(ROOT / "tests" / "cpp" / "pair_check.cpp"), "-o",
           str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def _bounds(program, a, c, n):
    r = subprocess.run([str(program), str(a), str(c), str(n)], capture_output=True, text=True)
    assert r.returncode == 0
    return [int(x) for x in r.stdout.split()]


def test_ranges_and_columns(pair_check):
    r = subprocess.run([str(pair_check)], capture_output=True, text=True)
    assert r.returncode == 0, r.returncode


CASES = [Case("closed", 6, 10, 9, (4,), (4,), "baseline", 3, 4.0),
         Case("core", 7, 11, 9, (5,), (3,), "baseline", 5, 4.0),
         Case("one", 6, 10, 9, (2,), (1,), "baseline", 5, 4.0)]


def _parts(case):
    """The pair quantities of a closed-shell case: G and Y of W and V over all (j, k), S^-1."""
    d = make_case(case)
    vals, vecs = O.eigen_decomposition(d.S, 1e-6, 1e-8)
    S = (vecs / vals) @ vecs.T
    Co = O.occupation_weighted_orbitals(d.orbitals, d.occ)[0]
    a, o = case.n_active[0], case.n_occ[0]
    Ca = Co[:, o - a:]
    N, R = case.n_ao, case.n_ri
    Rp = N + R
    G, Y, xh, J = {}, {}, {}, {}
    for nm, X in (("W", O.BaseIntegrals(d.W3, d.W2, d.W3_ri)),
                  ("V", O.BaseIntegrals(d.V3, d.V2, d.V3_ri))):
        M, lam = X.n_df, X.df_vals
        B1 = _h1(X.J3_0, Co, 0, M) @ X.P2
        B2 = T3(B1, Ca)
        st = np.zeros((Rp, a, M))
        st[N:] = (_h2(X.J3_ri_0, Ca, R, 0, M) @ X.P2).reshape((R, a, M), order="F")
        st[:N] = B1.reshape((N, o, M), order="F")[:, o - a:, :]
        xh[nm] = (X.P2 @ (lam[:, None] * B2.T)).reshape((M, a, o), order="F")
        J[nm] = np.concatenate([sq_all(X.J3_0), X.J3_ri_0.reshape((R, N, M), order="F")], axis=0)
        G[nm] = np.einsum("pnA,Ajk->jkpn", J[nm], xh[nm])
        Y[nm] = np.einsum("pjA,A,nkA->jkpn", st, lam, B1.reshape((N, o, M), order="F"))
    return S, G, Y, xh, J, a, o - a, o


def _reference(case):
    S, G, Y, xh, J, a, c, o = _parts(case)
    T2 = np.einsum("Ajk,Bjk->AB", xh["W"], xh["V"])
    D = np.einsum("AB,pmA,pq,qnB->mn", T2, J["W"], S, J["V"])
    ss = (np.einsum("jkpm,pq,jkqn->mn", G["W"], S, Y["V"])
          + np.einsum("jkpm,pq,jkqn->mn", G["V"], S, Y["W"])
          + np.einsum("ijpm,pq,jiqn->mn", Y["W"][:, c:], S, Y["V"][:, c:]))
    return D, ss + ss.T  # the Fock matrix is symmetrised


def _shard(case, lo, hi):
    """The distinct pairs of orbitals [lo, hi): D and the same-spin terms."""
    S, G, Y, _, _, a, c, o = _parts(case)
    N = case.n_ao
    D, F = np.zeros((N, N)), np.zeros((N, N))
    SY = np.einsum("pq,jkqn->jkpn", S, Y["V"])
    for k in range(lo, hi):
        for j in range(a if k < c else k - c + 1):
            i = k - c
            twin = k >= c and j != i
            sgv = (2.0 if twin else 1.0) * S @ G["V"][j, k]
            yw = 0.5 * (Y["W"][j, k] + Y["W"][i, c + j]) if twin else Y["W"][j, k]
            syv = SY[j, k] + SY[i, c + j] if twin else SY[j, k]
            D += G["W"][j, k].T @ sgv
            F += sgv.T @ yw + G["W"][j, k].T @ syv
            if k >= c:
                F += Y["W"][i, c + j].T @ SY[j, k]
                if twin:
                    F += Y["W"][j, k].T @ SY[i, c + j]
    return D, F + F.T


def _rank(rank, world, port, case, bounds, out_q):
    os.environ["MASTER_ADDR"] = "127.0.0.1"
    os.environ["MASTER_PORT"] = str(port)
    dist.init_process_group("gloo", rank=rank, world_size=world,
                            timeout=datetime.timedelta(seconds=60))
    try:
        parts = [torch.from_numpy(np.ascontiguousarray(x))
                 for x in _shard(case, bounds[rank], bounds[rank + 1])]
        for t in parts:
            dist.all_reduce(t, op=dist.ReduceOp.SUM)
        if rank == 0:
            out_q.put([t.numpy() for t in parts])
    finally:
        dist.destroy_process_group()


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
def test_two_ranks_sum_to_whole(pair_check, case):
    a, o = case.n_active[0], case.n_occ[0]
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    port = _free_port()
    bounds = _bounds(pair_check, a, o - a, 2)
    ps = [ctx.Process(target=_rank, args=(r, 2, port, case, bounds, q)) for r in range(2)]
    for p in ps:
        p.start()
    got = q.get(timeout=120)
    for p in ps:
        p.join(timeout=60)
        assert p.exitcode == 0
    for x, ref in zip(got, _reference(case)):
        assert np.max(np.abs(x - ref)) <= 1e-12 * np.max(np.abs(ref))
