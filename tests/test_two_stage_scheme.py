"""CPU restatement of the two-stage passes' index arithmetic (fft_two.cuh): for
every length that splits, each thread of the launched CTA -- the ones beyond a
stage's count included -- stays inside its buffers, the loads and stores of the
active threads cover every element once, and the scheme computes the DFT."""
import numpy as np
import pytest

RADICES = {2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 18, 20, 21, 24, 25, 27, 28, 30, 32}


def split(n):
    for r in range(2, 33):
        if n % r == 0 and 2 <= n // r <= r and r in RADICES and n // r in RADICES:
            return n // r, r
    return None


LENGTHS = [n for n in range(4, 1025) if split(n)]


@pytest.mark.parametrize("W", [2, 4, 8])
def test_column_pass_indices(W):
    for n in LENGTHS:
        R1, R2 = split(n)
        row = R2 | 1
        nt = (W * R2 + 31) // 32 * 32
        t = np.arange(nt) // W
        on_a, on_b = t < R2, t < R1
        ta, tb = np.minimum(t, R2 - 1), np.minimum(t, R1 - 1)
        tile = R1 * row  # elements per column
        assert tile >= n
        k = np.arange(R1)
        assert (k[None, :] * row + t[on_a][:, None]).max() < tile
        assert (tb[:, None] * row + np.arange(R2)[None, :]).max() < tile
        assert (ta[:, None] + R2 * k[None, :]).max() < n
        assert (ta[:, None] * k[None, :]).max() < n  # twiddle index
        for centre in {0, n // 4, n // 2, n - 1}:
            for cnt in {n, n // 2, 1}:
                for inverse in (False, True):
                    # loads: e wraps at most once per step
                    e = ta + centre
                    e = np.where(e >= n, e - n, e)
                    for m in range(R1):
                        assert ((e >= 0) & (e < n)).all()
                        assert (e == (ta + R2 * m + centre) % n).all()
                        e = e + R2
                        e = np.where(e >= n, e - n, e)
                    # stores
                    e = (np.where(tb > 0, n - tb, 0) if inverse else tb) + centre
                    e = np.where(e >= n, e - n, e)
                    limit = np.where(on_b, cnt, 0)
                    seen = np.zeros(n, int)
                    for m in range(R2):
                        go = e < limit
                        assert (e[go] >= 0).all() and (e[go] < cnt).all()
                        x = tb + R1 * m
                        assert (e == ((-x if inverse else x) + centre) % n).all()
                        np.add.at(seen, e[go], 1)
                        e = e + (-R1 if inverse else R1)
                        e = np.where(e >= n, e - n, e)
                        e = np.where(e < 0, e + n, e)
                    assert (seen[:cnt] == W).all() and (seen[cnt:] == 0).all()


@pytest.mark.parametrize("W", [2, 4, 8])
def test_row_pass_indices(W):
    for n in LENGTHS:
        R1, R2 = split(n)
        nt = (W * R2 + 31) // 32 * 32
        cp = (R1 * (R2 | 1)) | 1
        room = cp * ((nt + R2 - 1) // R2)
        c, t = np.arange(nt) // R2, np.arange(nt) % R2
        assert (c * cp + (R1 - 1) * (R2 | 1) + t).max() < room
        assert (c * cp + np.minimum(t, R1 - 1) * (R2 | 1) + R2 - 1).max() < room
        assert cp >= n
        assert room * 8 <= 48 * 1024 or W != 8 or n > 512
        if (W == 8 and n <= 512) or (W == 4 and n > 512):
            assert room * 8 <= 48 * 1024   # complex64: no opt-in of shared memory
        if (W == 4 and n <= 512) or (W == 2 and n > 512):
            assert room * 16 <= 48 * 1024  # complex128


@pytest.mark.parametrize("n", [6, 35, 63, 100, 225, 300, 450, 567, 784, 960])
def test_scheme_is_the_dft(n):
    R1, R2 = split(n)
    rng = np.random.default_rng(n)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    # stage 1: rows t of x[t + R2 m], twiddled; stage 2: columns k1
    Y = np.fft.fft(x.reshape(R1, R2), axis=0)  # [k1, t]
    Y = Y * np.exp(-2j * np.pi * np.outer(np.arange(R1), np.arange(R2)) / n)
    X = np.fft.fft(Y, axis=1)  # [k1, k2]
    out = np.empty(n, complex)
    k = np.arange(R1)[:, None] + R1 * np.arange(R2)[None, :]
    out[k] = X
    assert np.allclose(out, np.fft.fft(x))
    inv = np.empty(n, complex)
    inv[(n - k) % n] = X  # the inverse transform, unnormalised
    assert np.allclose(inv, np.fft.ifft(x) * n)
