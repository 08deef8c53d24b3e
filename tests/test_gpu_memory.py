"""Device memory that a context keeps between calls (the projector's texture) is
given back when an allocation fails, and the context goes on."""
import ctypes as C

import numpy as np
import pytest

from genfire_gb300._lib import load, ptr

pytestmark = pytest.mark.gpu


def _out_of_memory(lib, c):
    """A projector call whose volume (1.3 TB) no device holds: it fails before it
    reads any of its arrays."""
    a = np.zeros(3)
    b = np.zeros(1, dtype=np.float32)
    st = load().genfire_project(c.handle, lib.PREC_MIXED, ptr(b), 33000, 33000, 300, 1, ptr(a, C.c_double), None, ptr(b))
    assert st == 2, st  # GENFIRE_ERR_OOM


def test_failed_allocation_releases_the_projector_texture(lib):
    torch = pytest.importorskip("torch")

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    rng = np.random.default_rng(3)
    vol = np.asfortranarray(rng.random((512, 512, 256)).astype(np.float32))  # a texture of 256 MiB
    angles = np.asfortranarray([(10., 20., 30.)])
    with lib.Context(0) as c, lib.Context(0) as other:
        small = c.project(vol[:32, :32, :32], angles, precision=lib.PREC_MIXED)
        c.project(vol.astype(np.float64), angles)  # the allocator's pool grows to its size; no texture
        _out_of_memory(lib, c)
        before = free()
        for failing in (c, other):
            first = c.project(vol, angles, precision=lib.PREC_MIXED)
            _out_of_memory(lib, failing)
            assert before - free() < 64 << 20
            assert np.array_equal(c.project(vol, angles, precision=lib.PREC_MIXED), first)
        assert np.array_equal(c.project(vol[:32, :32, :32], angles, precision=lib.PREC_MIXED), small)
