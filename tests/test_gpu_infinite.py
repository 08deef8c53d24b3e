"""An inverse transform that overflows single precision gives infinities, not NaN:
the last pass's factor has two parts, and neither may turn an infinite sum into
NaN.  Four frequencies of 1.5e38 (zero and the Nyquist frequency of dims 1 and 2)
sum to 6e38 at the even points, in the row pass's last additions at these
lengths, and to zero elsewhere."""
import numpy as np
import pytest

from tests.conftest import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [8, 12])
def test_recifft_overflow(lib, ctx, D):
    P = np.zeros((D, D, 1), order="F")
    P[::2, ::2] = 4 * 1.5e38 / D ** 2
    p = params(lib, D, D, 1, precision="mixed", oversamplingRatio=1.0, interpolationCutoffDistance=0.3)
    rec = ctx.grid_dft(p, P, np.zeros((1, 3)))[1]
    assert np.isposinf(rec[::2, ::2]).all()
    assert not np.isnan(rec).any()
