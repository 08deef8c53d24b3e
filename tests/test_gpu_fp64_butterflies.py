"""complex128 register passes (butterflies in fused multiply-adds): every stage
split of the power-of-two lengths, the box being the centred half of the grid
(whose first stage leaves out the zero inputs) or less of it, against numpy and
against the generic engine's iterations.

Bars: a transform of n points adds a few roundings at each of log2(n) levels, so
its relative 2-norm error is below 4 log2(n) units in the last place; an
iteration is four transforms of n1 and two of n2 points, each engine off by
that much, and errors of 6 iterations add up.
"""
import numpy as np
import pytest

from tests.conftest import params, rel
from tests.test_gpu_recon import _measured, _support

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("n", [64, 128, 256, 512, 1024])
def test_transforms(lib, ctx, n):
    rng = np.random.default_rng(n)
    for shape in [(n, 3, 1), (9, 1, n)]:  # columns n apart; 9 adjacent columns: a full and a partial tile
        a = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        bar = 4 * (np.log2(n) + np.log2(9)) * EPS
        assert rel(ctx.fftn(a, precision=lib.PREC_FP64), np.fft.fftn(a)) < bar
        assert rel(ctx.fftn(a, inverse=True, precision=lib.PREC_FP64), np.fft.ifftn(a)) < bar + EPS


@pytest.mark.parametrize("D1,D2,os_", [(32, 32, 2.0), (16, 9, 4.0), (64, 5, 2.0), (32, 6, 4.0), (128, 3, 2.0), (40, 5, 3.2),
                                       (256, 2, 2.0), (128, 2, 4.0), (512, 2, 2.0)])
def test_iterations_against_the_generic_engine(lib, ctx, D1, D2, os_, monkeypatch):
    support = _support(D1, D2, shrink=0)
    M, _ = _measured(D1 + D2, D1, D2, os_, keep=0.3, support=support)
    monkeypatch.setenv("GENFIRE_AUTOTUNE", "0")
    p = params(lib, D1, D2, 1, oversamplingRatio=os_, numIterations=6, constraintEnforcementMode=3, precision="fp64")
    out = []
    for variant in ("1", "0"):
        monkeypatch.setenv("GENFIRE_COL_VARIANT", variant)
        out.append(ctx.reconstruct(p, M, support=support))
    bar = 2 * 6 * 6 * 4 * np.log2(D1 * os_) * EPS
    assert rel(out[0][0], out[1][0]) < bar
    assert np.abs(out[0][1] - out[1][1]).max() < bar
