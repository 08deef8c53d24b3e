"""Calls of fewer than five projections do not write the volume into a texture
first (which cost them up to a fifth of their time), unless their lines are too few
to fill the chip; the results are the same on both sides of the rule, by the bar of
test_gpu_project_texture."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_no_texture_for_few_projections(lib):
    torch = pytest.importorskip("torch")

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    vol = np.asfortranarray(np.random.default_rng(5).random((512, 512, 256)).astype(np.float32))  # 256 MiB
    angles = np.asfortranarray([(0., t, 0.) for t in np.linspace(-75, 75, 8)])
    with lib.Context(0) as c:
        c.project(vol.astype(np.float64), angles)  # the allocator's pool grows to its size; no texture
        before = free()
        for P in (1, 3, 4):
            c.project(vol, angles[:P], precision=lib.PREC_MIXED)
        assert before - free() < 64 << 20
        c.project(vol, angles[:5], precision=lib.PREC_MIXED)
        assert before - free() > 192 << 20


@pytest.mark.parametrize("shape", [(180, 190, 200), (181, 182, 128), (64, 63, 1500), (64, 64, 1100)])
def test_both_sides_agree(lib, ctx, shape):
    rng = np.random.default_rng(sum(shape))
    vol = np.asfortranarray((rng.random(shape) + 0.1).astype(np.float32))
    angles = np.asfortranarray(np.stack([rng.uniform(0, 360, 8), rng.uniform(-80, 80, 8), rng.uniform(0, 360, 8)], 1))
    angles[0] = 0
    got = ctx.project(vol, angles, precision=lib.PREC_MIXED)
    for P in (1, 2, 4):
        some = ctx.project(vol, angles[:P], precision=lib.PREC_MIXED)
        assert np.abs(got[:, :, :P] - some).max() <= 1e-6 * np.abs(got).max()
