"""The texture projector's clipped lines where a line is nearly parallel to a face
of the volume: a coordinate that stays within half a unit in the last place of
the last plane rounds onto it, and its samples count as the load kernel counts
them (single-projection calls, below 2^22 samples).  Bars of
test_gpu_project_texture."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILTS = [1e-4, -1e-4, 6e-5, -6e-5, 3e-4, 1e-3, -2e-3, 0.01]


@pytest.mark.parametrize("shape", [(300, 9, 300), (9, 300, 300), (513, 5, 300), (600, 4, 600)])
@pytest.mark.parametrize("phi", [0.0, 90.0, 180.0, 270.0])
@pytest.mark.parametrize("theta", [0.0, 90.0])
def test_lines_along_the_faces(lib, ctx, shape, phi, theta):
    rng = np.random.default_rng(sum(shape))
    vol = np.asfortranarray((rng.random(shape) + 1).astype(np.float32))
    angles = np.asfortranarray([(phi, theta + t, 0.0) for t in TILTS])
    assert np.prod(shape) * len(TILTS) >= 1 << 22 > np.prod(shape)
    got = ctx.project(vol, angles, precision=lib.PREC_MIXED)
    for q in range(len(TILTS)):
        one = ctx.project(vol, angles[q:q + 1], precision=lib.PREC_MIXED)
        assert np.abs(got[:, :, q] - one[:, :, 0]).max() <= 1e-6 * np.abs(one).max(), TILTS[q]
