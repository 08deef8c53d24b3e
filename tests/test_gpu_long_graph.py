"""Calls that run several iterations per graph launch (96 and more at once)
against the same iterations one call each: the same launches in the same order,
so the same bits; with the R-factor monitor's stops between, after calls of
other lengths, and with the Rfree monitor's extra launch."""
import numpy as np
import pytest

from tests.conftest import params
from tests.test_gpu_recon import _measured, _support

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,os_,prec", [(16, 2.0, "mixed"), (32, 2.0, "fp64"), (24, 3.0, "mixed"), (48, 2.0, "mixed")])
@pytest.mark.parametrize("monitor", [0, 7])
def test_long_calls_equal_single_iterations(lib, ctx, D, os_, prec, monitor, monkeypatch):
    monkeypatch.setenv("GENFIRE_AUTOTUNE", "0")  # the same engines on both sides
    N = 131
    support = _support(D, D, shrink=2)
    M, _ = _measured(D, D, D, os_, keep=0.2, support=support)
    rng = np.random.default_rng(D)
    projs = np.asfortranarray(rng.random((D, D, 3)))
    angles = np.asfortranarray(rng.uniform(0, 90, (3, 3)))
    p = params(lib, D, D, 3, oversamplingRatio=os_, numIterations=N, constraintEnforcementMode=1, precision=prec,
               monitor_R=1 if monitor else 0, monitorR_loopLength=monitor or 10)
    Mg = M.astype(np.complex64) if prec == "mixed" else M
    kw = dict(support=support, projections=projs if monitor else None, angles=angles if monitor else None)
    shells = [np.flatnonzero((M != 0).ravel(order="F"))[:5].astype(np.int64)] if not monitor else None
    out = []
    for chunks in ([N], [1] * 20 + [N - 20], [1] * N):
        r = ctx.recon(p, Mg, **kw)
        if shells:
            r.set_rfree(shells)
        for c in chunks:
            r.iterate(c)
        out.append(r.result() + ((r.rfree(),) if shells else ()))
        r.close()
    for got in out[:2]:
        for x, y in zip(got, out[2]):
            assert np.array_equal(x, y)
