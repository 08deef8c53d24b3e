"""The folded FP64 DFT against the direct sum, at the sizes where its tiles end:
odd and even sizes (the unpaired row and column), one slot, a partial and a
second tile of column slots, more tiles than warps, and rows beyond one
shared-memory table of phases (128).

The bound: a value is a sum of D1 D2 terms; each term carries a few roundings
of the folded operands, the phases and the running sum, at most ~D1 + D2 + 32
of them, so the error is below (D1 + D2 + 32) 2^-53 sum|P| per point.
"""
import numpy as np
import pytest

from tests.conftest import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D1,D2", [(2, 2), (3, 2), (2, 3), (7, 15), (16, 16), (17, 18), (32, 65), (66, 34), (258, 6),
                                   (300, 67)])
def test_fold_matches_direct_sum(lib, ctx, D1, D2):
    rng = np.random.default_rng(D1 * 1000 + D2)
    P = rng.standard_normal((D1, D2, 1)) + 0.5
    # ratio 1, one projection: a grid point's value is its one DFT value (the
    # average of a single contribution)
    p = params(lib, D1, D2, 1, oversamplingRatio=1.0, interpolationCutoffDistance=0.2)
    ang = np.array([[17.0, 23.0, 41.0]])
    M, _, nk = ctx.grid_dft(p, P, ang, want_rec=False)
    ind, dist, u, v = ctx.select(p, *ang[0])
    assert nk[0] == len(ind) > 0
    n1, n2 = lib.grid_size(p)
    l1, l2 = n1 // 2 + 1, 2 * (n2 // 2) + 1
    k1, k2, k3 = ind % l1, (ind // l1) % l2, ind // (l1 * l2)  # offsets of k from its lowest value
    inside = (k2 < n2) & (k3 < n1)
    a = np.arange(D1) - D1 // 2
    b = np.arange(D2) - D2 // 2
    Eu = np.exp(-2j * np.pi * np.outer(u.astype(np.float64), a) / n1)
    Ev = np.exp(-2j * np.pi * np.outer(v.astype(np.float64), b) / n2)
    F = np.einsum("ja,ab,jb->j", Eu, P[:, :, 0], Ev)
    got = M[k1[inside], k2[inside], k3[inside]]
    # the average (F / D) / (1 / D) adds at most 4 roundings of F
    bar = 2 * (D1 + D2 + 32) * 2.0 ** -53 * np.abs(P).sum()
    assert np.abs(got - F[inside]).max() < bar
