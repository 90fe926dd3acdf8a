"""The pair form of the t~ dX Fock term and the same-spin three-electron Fock (numpy):
with T2 = sum_s c_s x^_W[s] x^_V[s]^T the sum over aux functions equals the sum over
orbital pairs, and the pair sums of the three same-spin terms equal the direct
contraction, whole and over chunks of occupied orbitals in the engine's pair order
(k - k0) + nk j.  Products of random matrices of a few dozen terms: 1e-12 relative."""
import numpy as np
import pytest


def _setup(N, M, R, o, a, seed):
    g = np.random.default_rng(seed)
    P = N + R
    G = {x: g.standard_normal((M, P, N)) for x in "WV"}       # aux, AO + RI, AO
    B1 = {x: g.standard_normal((M, o, N)) for x in "WV"}      # aux (eigenbasis), occupied, AO
    st = {x: g.standard_normal((M, a, P)) for x in "WV"}      # stacked transforms
    lam = {x: g.uniform(0.5, 2.0, M) for x in "WV"}
    xh = {x: g.standard_normal((M, a, o)) for x in "WV"}
    S = g.standard_normal((P, P))
    return G, B1, st, lam, xh, S + S.T


@pytest.mark.parametrize("N,M,R,o,a,kc", [(4, 7, 5, 3, 3, 3), (4, 7, 5, 4, 2, 4), (3, 5, 6, 5, 4, 2),
                                          (2, 3, 3, 1, 1, 1)])
def test_pair_sums(N, M, R, o, a, kc):
    G, B1, st, lam, xh, S = _setup(N, M, R, o, a, 7)
    c = o - a
    # over aux functions
    T2 = np.einsum("ajk,bjk->ab", xh["W"], xh["V"])
    D_aux = np.einsum("ab,apm,pq,bqn->mn", T2, G["W"], S, G["V"])
    Gx = {x: np.einsum("ajk,apm->jkpm", xh[x], G[x]) for x in "WV"}
    Y = {x: np.einsum("ajp,a,akn->jkpn", st[x], lam[x], B1[x]) for x in "WV"}
    ss = (np.einsum("jkpm,pq,jkqn->mn", Gx["W"], S, Y["V"])
          + np.einsum("jkpm,pq,jkqn->mn", Gx["V"], S, Y["W"])
          + np.einsum("ijpm,pq,jiqn->mn", Y["W"][:, c:], S, Y["V"][:, c:]))
    # over chunks of pairs
    D, F = np.zeros((N, N)), np.zeros((N, N))
    P = N + R
    for k0 in range(0, o, kc):
        nk = min(kc, o - k0)

        def pairs(t):  # (k - k0) + nk j
            return t[:, k0:k0 + nk].reshape(a * nk, P, N)

        SG = np.einsum("pq,xqn->xpn", S, pairs(Gx["V"]))
        Z = np.einsum("pq,xqn->xpn", S, pairs(Y["V"]))
        F += np.einsum("xpm,xpn->mn", SG, pairs(Y["W"]))
        F += np.einsum("xpm,xpn->mn", pairs(Gx["W"]), Z)
        D += np.einsum("xpm,xpn->mn", pairs(Gx["W"]), SG)
        for i in range(max(k0, c) - c, max(k0 + nk, c) - c):
            for j in range(a):
                # whole chunk: Y_W of pair (i, c + j) from the chunk itself
                yw = pairs(Y["W"])[(c + j - k0) + nk * i] if nk == o else Y["W"][i, c + j]
                F += yw.T @ Z[(c + i - k0) + nk * j]
    assert np.max(np.abs(D - D_aux)) <= 1e-12 * np.max(np.abs(D_aux))
    # term 1 is transposed where S^-1 moves to the other factor; the Fock matrix is symmetrised
    sym = lambda x: x + x.T  # noqa: E731
    assert np.max(np.abs(sym(F) - sym(ss))) <= 1e-12 * np.max(np.abs(ss))
