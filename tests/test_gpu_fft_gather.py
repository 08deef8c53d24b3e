"""FFT gridding's gather at its edges, against the oracle: groups of one, a few
and more than 32 projections per warp, odd and even cubes (rows and samples
without a mirror), slices along the axes and diagonals (whole rows within reach,
ties in the rounding), cutoffs below and above the shift range, one voxel per
sample only.

Bars: equal pair counts and filled sets; the sums are FP64 in another order
(1e-12 relative for values of a few hundred terms), complex64 holds a voxel to
a few of its roundings and those of the FP32 transforms (1e-5).
"""
import numpy as np
import pytest

from tests.conftest import params, rel

pytestmark = pytest.mark.gpu

AXES = [(0, 0, 0), (0, 90, 0), (90, 90, 0), (45, 90, 45), (90, 45, 0), (0, 45, 90), (180, 0, 0), (30, 180, 60)]


@pytest.mark.parametrize("D,os_,P,cut,am", [
    (4, 2.0, 1, 0.7, 1), (5, 2.0, 3, 0.7, 1), (7, 1.0, 8, 0.49, 1), (8, 2.0, 8, 0.5, 1), (8, 2.0, 33, 0.7, 1),
    (9, 1.0, 140, 0.7, 1), (8, 1.0, 129, 1.2, 0), (8, 2.0, 6, 2.5, 1), (9, 1.75, 6, 2.5, 0), (10, 2.0, 5, 0.05, 1)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_gather(lib, ctx, oracle, D, os_, P, cut, am, precision):
    rng = np.random.default_rng(D * 100 + P)
    projs = np.asfortranarray(rng.standard_normal((D, D, P)) + 0.2)
    angles = np.stack([rng.uniform(0, 360, P), rng.uniform(-180, 180, P), rng.uniform(0, 360, P)], 1)
    for i, a in enumerate(AXES[:P]):
        angles[i] = a
    kw = dict(oversamplingRatio=os_, interpolationCutoffDistance=cut)
    M, _, n = ctx.grid_fft(params(lib, D, D, P, precision=precision, allowMultipleGridMatches=am, **kw), projs,
                           np.asfortranarray(angles), want_rec=False)
    Mo, _, no = oracle.grid_fft(oracle.make_params(D, D, P, **kw), projs, np.asfortranarray(angles), allow_multiple=am)
    assert n == no
    if precision == "fp64":
        assert np.array_equal(M != 0, Mo != 0)
    assert rel(M, Mo) < (1e-12 if precision == "fp64" else 1e-5)
