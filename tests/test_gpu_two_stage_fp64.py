"""complex128 lengths with an unbalanced split of the two-stage engine (a second
factor above 16 and 1.5 times the first, no factor of 7, up to 256) run on the
generic engine, which is faster there; their neighbours keep the two-stage one.
Both agree with the oracle to 1e-10, the bar of the other FP64 iteration tests."""
import numpy as np
import pytest

from tests.conftest import params, rel
from tests.test_gpu_recon import _measured, _support

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D1,D2,os_,variant", [
    (25, 4, 5.0, 0), (27, 3, 6.0, 0), (50, 4, 4.0, 0), (36, 3, 6.0, 0), (27, 3, 9.0, 0), (50, 3, 5.0, 0),
    (36, 3, 5.0, 6), (63, 3, 3.0, 6), (45, 3, 5.0, 6), (45, 4, 6.0, 6), (84, 3, 3.0, 6), (75, 4, 3.0, 6)])
def test_engine(lib, ctx, oracle, D1, D2, os_, variant):
    support = _support(D1, D2, shrink=1)
    M, _ = _measured(D1 + D2, D1, D2, os_, keep=0.2, support=support)
    kw = dict(oversamplingRatio=os_, numIterations=3, constraintEnforcementMode=3)
    r = ctx.recon(params(lib, D1, D2, 1, **kw), M, support=support)
    assert r.tuning()[1] in ((0, -1) if variant == 0 else (variant,))
    r.iterate(3)
    rec, errK = r.result()[:2]
    r.close()
    reco, errKo = oracle.reconstruct(oracle.make_params(D1, D2, 1, **kw), M, support=support)[:2]
    assert rel(rec, reco) < 1e-10
    assert np.abs(errK - errKo).max() < 1e-10
