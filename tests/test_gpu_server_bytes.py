"""What a server counts for a request is what a context reserves for it.

A lattice of separate atoms has about as many edges as the estimate allows for its grid; a lane's
workspaces for it must not exceed the estimate, or a batch could exceed the lane's share.
"""
import ctypes

import numpy as np
import pytest

import quickses_gb300 as q
from quickses_gb300 import _lib as L

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _lattice(k, step):
    a = np.arange(k, dtype=np.float32) * np.float32(step)
    xyz = np.stack(np.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3)
    return np.ascontiguousarray(xyz), np.full(len(xyz), 1.7, np.float32)


def _bytes(xyz, rad, voxel, passes):
    r = L.Request(xyz.ctypes.data, rad.ctypes.data, len(xyz), voxel, passes, 0)
    need, reserved = ctypes.c_ulonglong(0), ctypes.c_ulonglong(0)
    assert L.lib().qses_debug_request_bytes(ctypes.byref(r), ctypes.byref(need), ctypes.byref(reserved)) == L.QSES_OK
    return need.value, reserved.value


@pytest.mark.parametrize("passes", [0, 1])
def test_a_context_reserves_no_more(passes):
    xyz, rad = _lattice(14, 9.0)
    voxel = 0.4
    need, reserved = _bytes(xyz, rad, voxel, passes)
    G = q.grid_info(xyz, rad, voxel).G
    with q.Context(0) as c:
        c.compute_batch([dict(xyz=xyz[:2], radii=rad[:2], voxel=voxel, smooth=passes)])
        free = torch.cuda.mem_get_info()[0]
        out = c.compute_batch([dict(xyz=xyz, radii=rad, voxel=voxel, smooth=passes)])
        used = free - torch.cuda.mem_get_info()[0]
        assert 0.75 * 12 * G * G < len(out[0].vertices) < 12 * G * G  # edges: a few more
    assert 0.5 * reserved < used <= reserved + (8 << 20)  # and the slab tables, and whole pages
    assert need < reserved < 1.3 * need + (4 << 20)
