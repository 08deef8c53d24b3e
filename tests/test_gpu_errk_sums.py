"""errK's sums at complex64 lengths of the two-stage passes keep 64-bit accuracy.

From an empty object the spectrum is exactly zero, so the first iteration's
errK = sum |0 - |M|| / sum |M| is 1 but for the rounding of the two sums.  A sum of
at most 2^10 rounded additions in a row (per thread, warp, block and over the
partial sums) with 2^-47 each or better is within 1e-11 of it; single precision
partial sums are 1e-9 and more away."""
import numpy as np
import pytest

from tests.conftest import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D1,D2,os_", [(24, 7, 3.0), (36, 5, 2.0), (75, 5, 3.0), (125, 3, 5.0), (225, 4, 2.0), (150, 105, 3.0)])
def test_first_errk_of_an_empty_object(lib, ctx, D1, D2, os_):
    n1, n2 = int(round(D1 * os_)), int(round(D2 * os_))
    rng = np.random.default_rng(D1)
    M = np.asfortranarray((rng.random((n1, n2, n1)) * (rng.random((n1, n2, n1)) < 0.4)).astype(np.complex64))
    p = params(lib, D1, D2, 1, precision="mixed", oversamplingRatio=os_, numIterations=1, constraintEnforcementMode=3)
    errK = ctx.reconstruct(p, M)[1]
    assert abs(errK[0] - 1.0) < 1e-11


def test_infinite_terms_stay_infinite(lib, ctx):
    """A measured value whose square overflows has an infinite magnitude in single
    precision, and so has errK."""
    D1, D2, os_ = 24, 7, 3.0
    M = np.zeros((72, 21, 72), dtype=np.complex64, order="F")
    M[::5, ::2, ::3] = 1
    M[10, 3, 11] = 1e30
    p = params(lib, D1, D2, 1, precision="mixed", oversamplingRatio=os_, numIterations=1, constraintEnforcementMode=3)
    _, errK, _, _, _ = ctx.reconstruct(p, M)
    assert not np.isfinite(errK[0])
