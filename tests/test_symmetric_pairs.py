"""Sums over orbital pairs restricted to j <= i for the active ones (numpy): with x^
symmetric in the active pair, the Fock terms over all pairs equal those over chunks of
occupied orbitals in the engine's pair order, with the mirror images taken from the
chunk's own block of Y or from the block behind it.  Products of random matrices of a few
dozen terms: 1e-12 relative."""
import numpy as np
import pytest


def _count(a, c, k):
    i = max(k - c, 0)
    return a * min(k, c) + i * (i + 1) // 2


@pytest.mark.parametrize("o,a,kc", [(3, 3, 3), (5, 3, 5), (5, 3, 2), (6, 5, 2), (7, 4, 3), (4, 4, 1),
                                    (1, 1, 1)])
def test_symmetric_pair_sums(o, a, kc):
    g = np.random.default_rng(3)
    c, P, N = o - a, 6, 4
    G = {x: g.standard_normal((a, o, P, N)) for x in "WV"}
    for x in "WV":  # G[j, c + i] = G[i, c + j]
        G[x][:, c:] = 0.5 * (G[x][:, c:] + G[x][:, c:].swapaxes(0, 1))
    Y = g.standard_normal((a, o, P, N))                    # Y_W
    Z = g.standard_normal((a, o, P, N))                    # S^-1 Y_V
    S = g.standard_normal((P, P))
    S = S + S.T
    SG = np.einsum("pq,jkqn->jkpn", S, G["V"])
    ref = {"D": np.einsum("jkpm,jkpn->mn", G["W"], SG),
           "V": np.einsum("jkpm,jkpn->mn", SG, Y),
           "W": np.einsum("jkpm,jkpn->mn", G["W"], Z),
           "k": np.einsum("ijpm,jipn->mn", Y[:, c:], Z[:, c:])}
    got = {q: np.zeros((N, N)) for q in ref}
    k0 = 0
    while k0 < o:
        nk = min(kc, o - k0)
        if nk < o and k0 < c:
            nk = min(nk, c - k0)
        i0, i1 = max(k0, c) - c, max(k0 + nk, c) - c
        nj = a if k0 < c else i1
        pairs = ([(p % a, k0 + p // a) for p in range(a * max(0, min(k0 + nk, c) - k0))]
                 + [(j, c + i) for i in range(i0, i1) for j in range(i + 1)])
        assert len(pairs) == _count(a, c, k0 + nk) - _count(a, c, k0)

        def blocks(t):
            first = [t[j, k0 + q] for j in range(nj) for q in range(nk)]
            return first + [t[i, c + j] for i in range(i0, i1) for j in range(i0)]

        def mirror(j, k):
            i = k - c
            if i < 0 or j == i:
                return None
            return nk * nj + j + i0 * (i - i0) if j < i0 else (c + j - k0) + nk * i

        y, z = blocks(Y), blocks(Z)
        for j, k in pairs:
            m = mirror(j, k)
            w = 2.0 if m is not None else 1.0

            def both(t, h):
                own = t[(k - k0) + nk * j]
                return own if m is None else h * (own + t[m])

            sg = w * SG[j, k]
            got["D"] += G["W"][j, k].T @ sg
            got["V"] += sg.T @ both(y, 0.5)
            got["W"] += G["W"][j, k].T @ both(z, 1.0)
        first, back = c + i0 - k0, nk * nj
        for i in range(i1 - i0):
            for j in range(i1 - i0):
                blk = first + nk * i0
                got["k"] += y[blk + nk * i + j].T @ z[blk + i + nk * j]
            for j in range(i0):
                got["k"] += y[back + i0 * i + j].T @ z[first + i + nk * j]
                got["k"] += y[first + i + nk * j].T @ z[back + i0 * i + j]
        k0 += nk
    for q in ref:
        assert np.max(np.abs(got[q] - ref[q])) <= 1e-12 * np.max(np.abs(ref[q])), q
