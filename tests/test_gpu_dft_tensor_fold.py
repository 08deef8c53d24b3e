"""The folded tensor-core DFT at the edges of its blocks: odd and even sizes (the
row without a partner), one and several K chunks, a second row block (from 258
rows), a second column block (from 129 columns), padded columns, grids that
are a power of two or not, against the direct sum.

Bars (relative 2-norm over the points): the split keeps 16 (BF16) or 22 (FP16)
significant bits of each operand and drops one product of low parts, 3 2^-17
and 3 2^-23 with random signs; the phases are products of up to ten rotations
of 2^-24 each.
"""
import numpy as np
import pytest

from tests.conftest import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bar", [("mixed", 3 * 2.0 ** -17 + 20 * 2.0 ** -24), ("fp16", 3 * 2.0 ** -23 + 20 * 2.0 ** -24)])
@pytest.mark.parametrize("D1,D2", [(2, 2), (3, 5), (31, 17), (64, 64), (65, 33), (127, 129), (128, 16), (130, 144),
                                   (256, 130), (258, 9), (300, 15), (514, 4)])
def test_points_against_the_direct_sum(lib, ctx, D1, D2, precision, bar):
    rng = np.random.default_rng(D1 * 1000 + D2)
    P = rng.random((D1, D2, 2)) * np.array([1.0, 3e3])
    p = params(lib, D1, D2, 2, oversamplingRatio=1.0, interpolationCutoffDistance=0.1, precision=precision)
    angles = np.array([[17.0, 23.0, 41.0], [120.0, -35.0, 10.0]])
    n1, n2 = lib.grid_size(p)
    l1, l2 = n1 // 2 + 1, 2 * (n2 // 2) + 1
    M, _, _ = ctx.grid_dft(p, P, angles, want_rec=False)
    a, b = np.arange(D1) - D1 // 2, np.arange(D2) - D2 // 2
    num = np.zeros((l1, l2, 2 * (n1 // 2) + 1), complex)
    ws = np.zeros(num.shape)
    hit = np.zeros(num.shape, bool)
    val = np.zeros(num.shape, complex)
    for q in range(2):
        ind, dist, u, v = ctx.select(p, *angles[q])
        k = (ind % l1, (ind // l1) % l2, ind // (l1 * l2))
        Eu = np.exp(-2j * np.pi * np.outer(u.astype(np.float64), a) / n1)
        Ev = np.exp(-2j * np.pi * np.outer(v.astype(np.float64), b) / n2)
        F = ((Eu @ P[:, :, q]) * Ev).sum(1)
        exact = dist.astype(np.float64) < 1e-7
        w = np.where(exact, 0.0, 1.0 / np.maximum(dist.astype(np.float64), 1e-30))
        num[k] += F * w
        ws[k] += w
        e = tuple(x[exact] for x in k)
        hit[e] = True
        val[e] = F[exact]
    want = np.where(hit, val, num / np.maximum(ws, 1e-300))[:, :n2, :n1]
    got = M[:l1]
    filled = (hit | (ws > 0))[:, :n2, :n1]
    assert filled.sum() > 0 and (got[~filled] == 0).all()
    assert np.linalg.norm((got - want)[filled]) < bar * np.linalg.norm(want[filled])
