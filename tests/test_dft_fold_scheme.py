"""CPU restatement of the folded tensor-core DFT: the folded blocks' index map
(every row pair and column once, nothing outside the projection), the fold as
an identity, its split-BF16 error against the unfolded products', and the
stage protocol of the two producer groups."""
import random

import numpy as np
import pytest

from tests.test_split_and_mixed_radix import bf16

KN, KR, KC = 128, 128, 32


@pytest.mark.parametrize("D1,D2", [(2, 2), (3, 5), (64, 64), (65, 130), (255, 16), (256, 256), (258, 129), (600, 3)])
def test_block_indices(D1, D2):
    m = D1 // 2
    Kp, D2p = (m + KC - 1) // KC * KC, (D2 + 15) // 16 * 16
    nnc, nkr = (D2p + KN - 1) // KN, (Kp + KR - 1) // KR
    rows = np.zeros(D1, int)
    cols = np.zeros(D2, int)
    for kr in range(nkr):
        nkc = min(KR // KC, Kp // KC - KR // KC * kr)
        assert 1 <= nkc <= 4
        for kc in range(4):
            a = 1 + kr * KR + kc * KC + np.arange(KC)
            used = a <= m
            assert kc < nkc or not used.any()  # chunks that are not multiplied hold nothing
            lo = m - a[used]
            assert (lo >= 0).all()
            np.add.at(rows, lo, 1)
            hi = (m + a[used])[m + a[used] < D1]
            np.add.at(rows, hi, 1)
    rows[m] += 1  # a = 0: the epilogue's row
    assert (rows == 1).all()
    for nc in range(nnc):
        Nc = min(KN, D2p - KN * nc)
        assert Nc % 16 == 0 and 16 <= Nc <= KN
        b = nc * KN + np.arange(Nc)
        np.add.at(cols, b[b < D2], 1)
    assert (cols == 1).all()


def _split(x):
    hi = bf16(x.astype(np.float32))
    return hi.astype(np.float64), bf16((x.astype(np.float32) - hi).astype(np.float32)).astype(np.float64)


def _product(A, B):
    (Ah, Al), (Bh, Bl) = _split(A), _split(B)
    return Ah @ Bh + Ah @ Bl + Al @ Bh


@pytest.mark.parametrize("D1", [17, 64, 150, 256])
def test_fold_and_its_error(D1):
    rng = np.random.default_rng(D1)
    D2, n, m = 40, 2 * D1, D1 // 2
    P = rng.random((D1, D2))
    u = rng.uniform(-D1, D1, 200)
    a = np.arange(D1) - m
    E = np.exp(-2j * np.pi * np.outer(u, a) / n)
    Q = E @ P
    Pe, Po = np.zeros((m, D2)), np.zeros((m, D2))
    for k in range(1, m + 1):
        hi = P[m + k] if m + k < D1 else 0.0
        Pe[k - 1], Po[k - 1] = hi + P[m - k], hi - P[m - k]
    Ek = np.exp(-2j * np.pi * np.outer(u, np.arange(1, m + 1)) / n)
    assert np.allclose(P[m] + Ek.real @ Pe + 1j * (Ek.imag @ Po), Q)
    err = np.linalg.norm(P[m] + _product(Ek.real, Pe) + 1j * _product(Ek.imag, Po) - Q)
    old = np.linalg.norm(_product(E.real, P) + 1j * _product(E.imag, P) - Q)
    assert err < 1.15 * old


@pytest.mark.parametrize("seed", range(40))
def test_two_producer_groups_share_the_stages(seed):
    """Random interleavings of the two groups and the consumer: with parity waits
    (a wait for phase n passes exactly when the completed count is n modulo 2) the
    hand-off between the groups keeps every fill of a stage after the consumption
    of its last content, and nothing waits for ever."""
    rng = random.Random(seed)
    units = [rng.randint(1, 4) for _ in range(rng.randint(1, 12))]
    base = [sum(units[:i]) for i in range(len(units))]
    S = 3
    empty, full, hand = [0] * S, [0] * S, [0, 0]  # completed phases
    filled = []

    def passes(completed, want):  # wait with parity (want - 1) & 1
        return (completed & 1) != ((want - 1) & 1)

    def producer(pg):
        for i in range(pg, len(units), 2):
            for kc in range(units[i]):
                g = base[i] + kc
                if kc == 0 and i > 0:
                    n = (i - 1) // 2 + 1
                    while not passes(hand[1 - pg], n):
                        yield
                if g >= S:
                    while not passes(empty[g % S], g // S):
                        yield
                    assert empty[g % S] == g // S  # the stage's last content is consumed
                yield
                filled.append(g)
                full[g % S] += 1
            hand[pg] += 1
            yield

    def consumer():
        for g in range(sum(units)):
            while not passes(full[g % S], g // S + 1):
                yield
            assert full[g % S] == g // S + 1
            yield
            empty[g % S] += 1

    live = [producer(0), producer(1), consumer()]
    for _ in range(200000):
        if not live:
            break
        x = rng.choice(live)
        try:
            next(x)
        except StopIteration:
            live.remove(x)
    assert not live and filled == list(range(sum(units)))
