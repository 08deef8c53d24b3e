"""Calls that run several iterations per graph launch against the same iterations
one call each, on the engines that test_gpu_long_graph's small grids do not reach:
the radix-32 passes (512 points, with the centred half of a box), the two-stage
passes with kernels of their own (300 points) and the fused one at five times a
power of two (320).  The same launches in the same order: the same bits."""
import numpy as np
import pytest

from tests.conftest import params
from tests.test_gpu_recon import _measured, _support

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D1,D2,os_", [(256, 3, 2.0), (100, 6, 3.0), (160, 4, 2.0)])
def test_long_calls_equal_single_iterations(lib, ctx, monkeypatch, D1, D2, os_):
    monkeypatch.setenv("GENFIRE_AUTOTUNE", "0")  # the same engines on both sides
    N = 103
    support = _support(D1, D2, shrink=1)
    M, _ = _measured(D1, D1, D2, os_, keep=0.1, support=support)
    p = params(lib, D1, D2, 1, oversamplingRatio=os_, numIterations=N, constraintEnforcementMode=1, precision="mixed")
    out = []
    for chunks in ([N], [1] * N):
        r = ctx.recon(p, M.astype(np.complex64), support=support)
        for c in chunks:
            r.iterate(c)
        out.append(r.result())
        r.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)
