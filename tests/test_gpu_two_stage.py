"""The two-stage passes (lengths R1 * R2 with both factors up to 32): the
splits with kernels of their own (complex64 from 72 points) and the run-time
ones, equal and unequal factors, every radix, few columns and partial tiles,
against numpy and, for whole iterations, the oracle.

Bars for the transforms: each of the log2(n) butterfly levels adds a relative
error of a few roundings, so the relative 2-norm error of a transform along
one axis is below 4 log2(n) units in the last place.
"""
import numpy as np
import pytest

from tests.conftest import params, rel
from tests.test_gpu_recon import _measured, _support

pytestmark = pytest.mark.gpu

# every radix of the engine appears as a factor: 2..10, 12, 14, 15, 16, 18, 20, 21, 24, 25, 27, 28, 30, 32
LENGTHS = [6, 15, 18, 27, 35, 36, 49, 63, 70, 72, 75, 81, 96, 100, 125, 147, 150, 162, 175, 196, 200, 225, 243, 250,
           294, 300, 315, 375, 378, 405, 441, 450, 486, 500, 560, 567, 576, 600, 625, 672, 729, 756, 784, 800, 840,
           900, 960]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_transform_along_each_axis(lib, ctx, n, precision):
    prec = lib.PREC_FP64 if precision == "fp64" else lib.PREC_MIXED
    eps = 2.0 ** -53 if precision == "fp64" else 2.0 ** -24
    bar = 4 * np.log2(n) * eps
    rng = np.random.default_rng(n)
    for shape in [(n, 3, 1), (9, 1, n)]:  # columns n apart; 9 adjacent columns: a full and a partial tile
        a = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        a = a.astype(np.complex128 if precision == "fp64" else np.complex64).astype(np.complex128)
        axes = tuple(i for i, s in enumerate(shape) if s > 1)
        extra = 4 * np.log2(9) * eps
        assert rel(ctx.fftn(a, precision=prec), np.fft.fftn(a, axes=axes)) < bar + extra
        assert rel(ctx.fftn(a, inverse=True, precision=prec), np.fft.ifftn(a, axes=axes)) < bar + extra + eps


@pytest.mark.parametrize("D1,D2,os_,prec", [
    (24, 7, 3.0, "mixed"), (36, 5, 2.0, "mixed"), (75, 5, 3.0, "mixed"), (150, 4, 2.0, "mixed"), (125, 3, 5.0, "mixed"),
    (240, 3, 3.0, "mixed"), (225, 4, 2.0, "mixed"), (450, 3, 2.0, "mixed"), (75, 5, 3.0, "fp64"), (150, 4, 2.0, "fp64"),
    (225, 4, 2.0, "fp64"), (288, 3, 2.0, "fp64")])
def test_reconstruct_against_the_oracle(lib, ctx, oracle, D1, D2, os_, prec):
    support = _support(D1, D2, shrink=1)
    M, _ = _measured(D1 + D2, D1, D2, os_, keep=0.3, support=support)
    kw = dict(oversamplingRatio=os_, numIterations=3, constraintEnforcementMode=3)
    Mg = M.astype(np.complex64) if prec == "mixed" else M
    rec, errK, _, _, _ = ctx.reconstruct(params(lib, D1, D2, 1, precision=prec, **kw), Mg, support=support)
    reco, errKo, _, _, _ = oracle.reconstruct(oracle.make_params(D1, D2, 1, **kw), M, support=support)
    assert rel(rec, reco) < (1e-10 if prec == "fp64" else 1e-4)
    assert np.abs(errK - errKo).max() < (1e-10 if prec == "fp64" else 1e-5)
