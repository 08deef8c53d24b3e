"""The two-stage column passes are never a choice by time: at lengths with another
engine they run by a fixed rule (the fused complex64 pass at five times a power of
two) or when asked for (GENFIRE_COL_VARIANT=6), so that two processes get the same
bits there; and asked for, they agree with the oracle."""
import numpy as np
import pytest

from tests.conftest import params, rel
from tests.test_gpu_recon import _measured, _support

pytestmark = pytest.mark.gpu

SIZES = [(32, 32, 2.0), (64, 64, 2.0), (64, 64, 3.0), (128, 32, 2.0), (160, 32, 2.0), (96, 96, 2.0), (128, 32, 3.0),
         (256, 32, 2.0), (320, 32, 2.0), (160, 64, 2.0), (192, 192, 2.0), (128, 128, 3.0)]


def _recon(lib, ctx, D1, D2, os_, prec, n):
    support = _support(D1, D2, shrink=1)
    M, _ = _measured(D1 + D2, D1, D2, os_, keep=0.3, support=support)
    kw = dict(oversamplingRatio=os_, numIterations=n, constraintEnforcementMode=3)
    Mg = M.astype(np.complex64) if prec == "mixed" else M
    return ctx.recon(params(lib, D1, D2, 1, precision=prec, **kw), Mg, support=support), M, support, kw


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_never_chosen_by_time(lib, ctx, prec):
    rng = np.random.default_rng(0)
    for size in SIZES:
        n1, n2 = int(size[0] * size[2]), int(size[1] * size[2])
        M = np.zeros((n1, n2, n1), dtype=np.complex64 if prec == "mixed" else np.complex128, order="F")
        M[:, :, ::3] = rng.random((n1, n2, 1))
        r = ctx.recon(params(lib, size[0], size[1], 1, precision=prec, oversamplingRatio=size[2], numIterations=1), M)
        chosen = r.tuning()
        r.close()
        five = prec == "mixed" and n1 in (320, 640)
        two_only = [n2 not in (64, 128, 192, 256, 320, 384, 640) or (prec == "fp64" and n2 == 320)] * 3
        two_only[1] = five or (prec == "fp64" and n1 in (320, 640))
        for v, two in zip(chosen, two_only):
            assert (v == 6) == two, (size, chosen)


@pytest.mark.parametrize("D1,D2,os_", [(64, 4, 2.0), (64, 4, 3.0), (128, 4, 2.0), (160, 3, 2.0), (128, 4, 3.0), (320, 3, 2.0)])
@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_forced_two_stage(lib, ctx, oracle, monkeypatch, D1, D2, os_, prec):
    monkeypatch.setenv("GENFIRE_COL_VARIANT", "6")
    r, M, support, kw = _recon(lib, ctx, D1, D2, os_, prec, 3)
    r.iterate(3)
    assert r.tuning()[1] == 6
    rec, errK = r.result()[:2]
    r.close()
    reco, errKo = oracle.reconstruct(oracle.make_params(D1, D2, 1, **kw), M, support=support)[:2]
    assert rel(rec, reco) < (1e-10 if prec == "fp64" else 1e-4)
    assert np.abs(errK - errKo).max() < (1e-10 if prec == "fp64" else 1e-5)
