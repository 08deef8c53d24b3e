"""recIFFT of a DFT gridding: the Hermitian part of the centred grid is formed
by one warp per row (odd and even lengths, rows shorter and longer than a warp,
fewer rows than a CTA holds), against the oracle on the same grid.

Bars: three transforms of at most 2^10 points and one average, a few roundings
per butterfly level: relative 2-norm 2e-6 in complex64 and 1e-13 in complex128.
"""
import numpy as np
import pytest

from tests.conftest import params, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D1,D2,os_,prec", [
    (6, 5, 1.0, "mixed"), (7, 9, 1.0, "mixed"), (9, 4, 7.0, "mixed"), (64, 6, 2.0, "mixed"), (256, 5, 2.0, "mixed"),
    (128, 3, 4.0, "mixed"), (512, 4, 2.0, "mixed"), (7, 4, 3.0, "fp64"), (63, 5, 1.0, "fp64")])
def test_rec_ifft(lib, ctx, oracle, D1, D2, os_, prec):
    rng = np.random.default_rng(D1 + D2)
    P = 3
    projs = np.asfortranarray(rng.random((D1, D2, P)))
    angles = np.asfortranarray(np.stack([rng.uniform(0, 360, P), rng.uniform(-70, 70, P), rng.uniform(0, 360, P)], 1))
    p = params(lib, D1, D2, P, oversamplingRatio=os_, interpolationCutoffDistance=0.4, precision=prec)
    M, rec, _ = ctx.grid_dft(p, projs, angles)
    want = oracle.rec_ifft(M.astype(np.complex128), D1, D2)
    assert rel(rec, want) < (2e-6 if prec == "mixed" else 1e-13)
