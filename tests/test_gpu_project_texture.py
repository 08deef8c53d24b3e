"""The float projector through texture gathers (calls of 2^22 samples and more)
against the load kernel (the same projections one call each, which are below
that), for volume sizes with partial pixel tiles, one to several slices across
the texture, and views inside a larger volume; and its R-factor sums.

Both kernels form the same coordinates and the same products; the compiler may
contract a multiply and an add in one of them only, so a sample differs by a
few units in the last place: 1e-6 relative to the largest pixel.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _angles(rng, P):
    a = np.stack([rng.uniform(0, 360, P), rng.uniform(-180, 180, P), rng.uniform(0, 360, P)], 1)
    a[:4] = [(0, 0, 0), (0, 90, 0), (90, 90, 0), (45, 30, 60)]
    return np.asfortranarray(a)


@pytest.mark.parametrize("shape,P", [((33, 47, 29), 96), ((64, 64, 64), 17), ((16, 300, 130), 8), ((130, 9, 300), 14),
                                     ((300, 21, 70), 12), ((2, 3, 700), 1100)])
def test_texture_equals_loads(lib, ctx, shape, P):
    assert np.prod(shape) * P >= 1 << 22 > np.prod(shape)
    rng = np.random.default_rng(sum(shape))
    vol = np.asfortranarray(rng.standard_normal(shape).astype(np.float32))
    angles = _angles(rng, P)
    got = ctx.project(vol, angles, precision=lib.PREC_MIXED)
    for q in list(range(4)) + list(range(4, P, max(1, P // 8))):
        one = ctx.project(vol, angles[q:q + 1], precision=lib.PREC_MIXED)
        assert np.abs(got[:, :, q] - one[:, :, 0]).max() <= 1e-6 * np.abs(one).max()


def test_rfactor_sums_and_a_second_size(lib, ctx):
    rng = np.random.default_rng(5)
    for shape, P in [((40, 56, 40), 60), ((50, 50, 50), 40), ((40, 56, 40), 60)]:  # back to the first size
        vol = np.asfortranarray(rng.random(shape).astype(np.float32))
        angles = _angles(rng, P)
        measured = ctx.project(vol.astype(np.float64), angles) * (1 + 0.01 * rng.standard_normal(shape[:2] + (P,)))
        r, r1, r2 = ctx.rfactor(vol, angles, measured, precision=lib.PREC_MIXED)
        assert abs(r - r1.mean()) < 1e-12
        for q in range(P):  # one projection a call: the load kernel
            _, s1, s2 = ctx.rfactor(vol, angles[q:q + 1], np.asfortranarray(measured[:, :, q:q + 1]),
                                    precision=lib.PREC_MIXED)
            # differences of 1 % of a pixel, each pixel to a few roundings
            assert abs(r1[q] - s1[0]) < 1e-4 * s1[0] and abs(r2[q] - s2[0]) < 1e-4 * s2[0]
