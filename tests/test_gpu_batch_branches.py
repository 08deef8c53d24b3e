"""Batches whose members are spread over the branches by size: large grids (six
million points and more) on two or three of them, small ones on the rest or all.
Every member's result must be bit-identical to the same problem iterated alone."""
import numpy as np
import pytest

from tests.conftest import params
from tests.test_gpu_recon import _support

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    (96, 96, 16, 12),                    # two large branches, one small
    (96, 96, 96),                        # three large branches
    (16, 96) + (8,) * 10,                # small members on several branches beside one large
    (96,) * 9,                           # more large members than branches
    (24, 12, 16, 8, 9, 10, 15, 18, 20),  # small ones only, more than branches
    (96,), (16,),
])
def test_members_equal_themselves_alone(lib, ctx, sizes, monkeypatch):
    monkeypatch.setenv("GENFIRE_AUTOTUNE", "0")  # the same engines on both sides
    out = []
    for batched in (False, True):
        rs = []
        for i, D in enumerate(sizes):
            rng = np.random.default_rng(100 + i)
            n = 2 * D
            M = (rng.standard_normal((n, n, n)) + 1j * rng.standard_normal((n, n, n))).astype(np.complex64)
            M[rng.random(M.shape) > 0.2] = 0
            p = params(lib, D, D, 1, oversamplingRatio=2.0, numIterations=4, constraintEnforcementMode=3, precision="mixed")
            rs.append(ctx.recon(p, np.asfortranarray(M), support=_support(D, D)))
        if batched:
            b = lib.ReconBatch(ctx, rs)
            b.iterate(4)
            b.close()
        else:
            for r in rs:
                r.iterate(4)
        out.append([r.result()[:2] for r in rs])
        for r in rs:
            r.close()
    for (x, ex), (y, ey) in zip(*out):
        assert np.array_equal(x, y) and np.array_equal(ex, ey)
