"""Contexts on threads of their own (one context per host thread is the C API's
rule), each gridding cubes of another size: what a call sets on the device must
not depend on its own size.  The FFT gridding kernel's shared memory grows with
the cube, and a launch above the device's limit for the kernel fails, so a small
cube's call may not lower the limit between a larger one's setting and its launch."""
import threading

import numpy as np
import pytest

from tests.conftest import params

pytestmark = pytest.mark.gpu


def test_fft_gridding_of_several_sizes_at_once(lib):
    torch = pytest.importorskip("torch")
    cases = []
    for D in (2, 2, 2, 4, 8, 16):  # cubes of 4 to 32 points
        rng = np.random.default_rng(D)
        M = torch.empty(2 * (2 * D) ** 3, dtype=torch.float32, device="cuda")
        cases.append((params(lib, D, D, 1, precision="mixed", oversamplingRatio=2.0),
                      torch.from_numpy(rng.random((D, D))).cuda(), rng.uniform(0, 90, (1, 3)), M))
    torch.cuda.synchronize()
    errors, counts = [], [set() for _ in cases]
    go = threading.Barrier(len(cases))

    def work(i):
        p, projs, angles, M = cases[i]
        with lib.Context(0) as c:
            go.wait()
            for _ in range(3000):
                try:
                    counts[i].add(c.grid_fft_device(p, projs.data_ptr(), angles, M.data_ptr()))
                except lib.GenfireError as e:
                    errors.append((p.Dim1, str(e)))
                    break

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert all(len(c) == 1 for c in counts)
