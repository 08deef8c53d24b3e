"""The tensor-core gridding kernel with wait limits from one cycle to a fraction of
its run time: a wait may expire in any role and at any unit, also while the other
roles' barriers complete.  The call either reports the timeout or is right, and
the context grids normally after it.  (Limits are polled with the non-blocking
test; the drain of what is in flight keeps the full limit.)"""
import numpy as np
import pytest

from tests.conftest import params, rel

pytestmark = pytest.mark.gpu

ENV = "GENFIRE_DEBUG_DFT_WAIT_CYCLES"


@pytest.mark.parametrize("D,P,precision", [(32, 4, "mixed"), (160, 6, "mixed"), (64, 40, "fp16")])
def test_expiry_at_any_point(lib, ctx, monkeypatch, D, P, precision):
    rng = np.random.default_rng(D)
    projs = np.asfortranarray(rng.random((D, D, P)))
    angles = np.asfortranarray(np.stack([rng.uniform(0, 360, P), rng.uniform(-70, 70, P), rng.uniform(0, 360, P)], 1))
    p = params(lib, D, D, P, precision=precision, oversamplingRatio=2.0, interpolationCutoffDistance=0.3)
    good = ctx.grid_dft(p, projs, angles, want_rec=False)[0]
    expired = 0
    for cycles in (1, 100, 300, 1000, 2000, 3000, 5000, 10000, 30000):
        monkeypatch.setenv(ENV, str(cycles))
        try:
            M = ctx.grid_dft(p, projs, angles, want_rec=False)[0]
            assert np.array_equal(M, good)
        except lib.GenfireError as e:
            assert e.status == 4, str(e)  # GENFIRE_ERR_TIMEOUT
            expired += 1
        monkeypatch.delenv(ENV)
        assert np.array_equal(ctx.grid_dft(p, projs, angles, want_rec=False)[0], good)
    assert expired
