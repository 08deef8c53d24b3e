"""FFT gridding where many samples share voxels: repeated angles, tilt series and
wide cutoffs, which made the row gather's sums a chain of retries, and the sizes
on both sides of the rule that sends such calls to the scatter.  Results against
the oracle with the bars of test_gpu_fft_gather; times against a call with the
same number of pairs, or a known multiple of them, that has no such chains (each
bar lies halfway, as a factor, between the times with and without the fault)."""
import time

import numpy as np
import pytest

from tests.conftest import params, rel

pytestmark = pytest.mark.gpu


def _angles(kind, P, rng):
    if kind == "same":
        return np.asfortranarray(np.tile([10., 20., 30.], (P, 1)))
    if kind == "tilt":
        return np.asfortranarray(np.stack([np.zeros(P), np.linspace(-75, 75, P), np.zeros(P)], 1))
    return np.asfortranarray(np.stack([rng.uniform(0, 360, P), rng.uniform(-70, 70, P), rng.uniform(0, 360, P)], 1))


@pytest.mark.parametrize("D,os_,P,cut,am,kind", [
    (8, 2.0, 69, 0.7, 1, "euler"), (8, 2.0, 70, 0.7, 1, "euler"), (8, 2.0, 199, 0.3, 1, "euler"), (8, 2.0, 200, 0.3, 1, "euler"),
    (9, 1.0, 100, 0.9, 0, "euler"), (9, 1.0, 99, 0.9, 0, "euler"), (6, 1.5, 24, 1.0, 1, "euler"), (9, 1.75, 8, 1.5, 1, "tilt"),
    (8, 2.0, 3, 2.4, 1, "euler"), (8, 2.0, 4, 2.4, 1, "same"), (5, 1.0, 40, 1.6, 1, "euler"), (4, 1.0, 40, 1.6, 1, "euler"),
    (36, 2.0, 96, 0.7, 1, "tilt"), (10, 2.0, 100, 0.3, 1, "tilt"), (10, 2.0, 95, 0.3, 1, "tilt"), (10, 2.0, 16, 0.7, 1, "same"), (10, 2.0, 15, 0.7, 1, "same"),
    (10, 2.0, 60, 0.7, 1, "same"), (10, 2.0, 60, 0.7, 1, "tilt"), (24, 2.0, 90, 0.7, 1, "tilt"), (12, 2.0, 4, 9.0, 1, "euler")])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_results(lib, ctx, oracle, D, os_, P, cut, am, kind, precision):
    rng = np.random.default_rng(D * 100 + P)
    projs = np.asfortranarray(rng.standard_normal((D, D, P)) + 0.2)
    angles = _angles(kind, P, rng)
    kw = dict(oversamplingRatio=os_, interpolationCutoffDistance=cut)
    M, _, n = ctx.grid_fft(params(lib, D, D, P, precision=precision, allowMultipleGridMatches=am, **kw), projs, angles, want_rec=False)
    Mo, _, no = oracle.grid_fft(oracle.make_params(D, D, P, **kw), projs, angles, allow_multiple=am)
    assert n == no
    if precision == "fp64":
        assert np.array_equal(M != 0, Mo != 0)
    assert rel(M, Mo) < (1e-12 if precision == "fp64" else 1e-5)


def _time(lib, ctx, torch, D, P, cut, kind):
    rng = np.random.default_rng(D + P)
    projs = torch.from_numpy(rng.random((P, D, D))).cuda()
    M = torch.empty((2 * D) ** 3, dtype=torch.complex64, device="cuda")
    p = params(lib, D, D, P, precision="mixed", oversamplingRatio=2.0, interpolationCutoffDistance=cut)
    angles = _angles(kind, P, rng)
    t = []
    for _ in range(12):
        t0 = time.perf_counter()
        ctx.grid_fft_device(p, projs.data_ptr(), angles, M.data_ptr())
        t.append(time.perf_counter() - t0)
    return min(t)


@pytest.mark.parametrize("slow,base,bar", [
    ((128, 31, 0.7, "same"), (128, 31, 0.7, "euler"), 1.1),  # 355 and 211 us against 260
    ((64, 400, 0.7, "tilt"), (64, 400, 0.7, "euler"), 1.5),  # 716 and 469 against 394
    ((64, 31, 3.0, "euler"), (64, 31, 0.7, "euler"), 10.5),  # 1503 and 789 against 105
    ((32, 400, 0.7, "euler"), (32, 31, 0.7, "euler"), 3.2),  # 295 and 172 against 72
])
def test_no_chains_of_retries(lib, ctx, slow, base, bar):
    torch = pytest.importorskip("torch")
    assert _time(lib, ctx, torch, *slow) < bar * _time(lib, ctx, torch, *base)
