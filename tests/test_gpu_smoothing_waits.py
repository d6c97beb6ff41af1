"""The smoothing's waits last while slabs are being done, however many they wait behind.

With half a millisecond's patience a slab far down the chain, or one that waits for the previous
pass, sees nothing arrive for longer than that; the slabs before it are being done all the while.
"""
import ctypes

import numpy as np
import pytest

import quickses_gb300 as q
from quickses_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("passes", [1, 4])
def test_waits_last_while_slabs_are_being_done(passes):
    xyz, rad, _ = q.molecules.ball(50000, 41)
    lib = L.lib()
    with q.Context(0) as c:
        c.set_smoothing_shape(512, 1024)
        want = c.compute(xyz, rad, voxel=0.3, smooth=passes)
        assert lib.qses_debug_smoothing_wait(c.handle, 1_000_000) == L.QSES_OK
        for _ in range(3):
            got = c.compute(xyz, rad, voxel=0.3, smooth=passes)
            assert np.array_equal(got.vertices, want.vertices)


def test_limits_are_checked():
    lib = L.lib()
    with q.Context(0) as c:
        for bad in (-1, 999_999, 4_000_000_001):
            assert lib.qses_debug_smoothing_wait(c.handle, ctypes.c_longlong(bad)) == L.QSES_ERR_INVALID_ARG
        assert lib.qses_debug_smoothing_wait(c.handle, 0) == L.QSES_OK
    assert lib.qses_debug_smoothing_wait(None, 0) == L.QSES_ERR_INVALID_ARG
