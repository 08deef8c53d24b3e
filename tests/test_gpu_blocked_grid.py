"""Iterations on grids whose dim-2 and dim-3 passes have tiles of different
widths (the half-transformed grid is stored in blocks of the wider one), with
whole and partial last blocks, against the oracle.  Bars as for every reconstruction: FP64
1e-10, MIXED 1e-4 on the volume."""
import numpy as np
import pytest

from tests.conftest import params, rel
from tests.test_gpu_recon import _measured, _support

pytestmark = pytest.mark.gpu


# grid lengths: complex64 tiles are 8 columns wide up to 512 points, 4 up to 1024 and 2 up to 2048;
# complex128 ones half as wide from half the length
@pytest.mark.parametrize("D1,D2", [(8, 300), (300, 4), (9, 640), (640, 2), (256, 3), (12, 256), (512, 2), (35, 384)])
@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_tile_widths_that_differ(lib, ctx, oracle, D1, D2, prec):
    support = _support(D1, D2, shrink=0)
    M, _ = _measured(D1 + D2, D1, D2, 2.0, keep=0.2, support=support)
    kw = dict(oversamplingRatio=2.0, numIterations=3, constraintEnforcementMode=3)
    Mg = M.astype(np.complex64) if prec == "mixed" else M
    rec, errK, _, _, _ = ctx.reconstruct(params(lib, D1, D2, 1, precision=prec, **kw), Mg, support=support)
    reco, errKo, _, _, _ = oracle.reconstruct(oracle.make_params(D1, D2, 1, **kw), M, support=support)
    assert rel(rec, reco) < (1e-10 if prec == "fp64" else 1e-4)
    assert np.abs(errK - errKo).max() < (1e-10 if prec == "fp64" else 1e-5)
