"""The float projector at volume sizes that no texture holds: more slices than a
grid has z blocks, and dimensions beyond the texture's sides; both take the load
kernel.

(8, 8, 70000) is above 2^22 samples with one projection, so it is compared with
the oracle at rotations about dim 3, where a line stays in one column: sixteen
FP32 terms at a time, summed in FP64, of interpolated values of a few roundings
each, 1e-6 relative to the largest pixel.  The other shapes are compared with
single-projection calls, which are far below 2^22 samples: equal.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_more_slices_than_a_grid_has_blocks(lib, ctx, oracle):
    rng = np.random.default_rng(1)
    vol = np.asfortranarray(rng.random((8, 8, 70000)).astype(np.float32))
    angles = np.asfortranarray(np.array([(0., 0., 0.), (90., 0., 0.), (30., 0., 0.)]))
    got = ctx.project(vol, angles, precision=lib.PREC_MIXED)
    want = np.stack([oracle.project(vol, *a) for a in angles], axis=2)
    assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()


@pytest.mark.parametrize("shape", [(2, 40000, 2), (40000, 2, 2), (2, 33000, 3), (3, 2, 40000)])
def test_sides_beyond_the_texture(lib, ctx, shape):
    rng = np.random.default_rng(2)
    vol = np.asfortranarray(rng.standard_normal(shape).astype(np.float32))
    P = (1 << 22) // int(np.prod(shape)) + 1
    angles = np.asfortranarray(np.stack([rng.uniform(0, 360, P), rng.uniform(-1, 1, P), rng.uniform(0, 360, P)], 1))
    angles[0] = 0
    got = ctx.project(vol, angles, precision=lib.PREC_MIXED)
    for q in range(0, P, 5):
        one = ctx.project(vol, angles[q:q + 1], precision=lib.PREC_MIXED)
        assert np.abs(got[:, :, q] - one[:, :, 0]).max() <= 1e-6 * max(np.abs(one).max(), 1)


def test_thin_volumes_take_no_longer(lib, ctx):
    """The same number of samples in slices of 2 x 4096 and of 2048 x 4 pixels; two
    threads of 256 at work made it ten times the time."""
    import time
    rng = np.random.default_rng(3)
    angles = np.asfortranarray([(30., 40., 50.)])
    best = []
    for shape in ((2, 4096, 2048), (2048, 4, 2048)):
        vol = np.asfortranarray(rng.random(shape).astype(np.float32))
        t = []
        for _ in range(8):
            t0 = time.perf_counter()
            ctx.project(vol, angles, precision=lib.PREC_MIXED)
            t.append(time.perf_counter() - t0)
        best.append(min(t))
    assert best[0] < 4 * best[1], best
