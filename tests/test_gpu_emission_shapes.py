"""The emission's time on a surface that lies in a few grid planes.

A warp takes consecutive words of the grid, plane after plane along x, so a sheet normal to x gives a
few warps all the work if each takes many.
"""
import numpy as np
import pytest

import quickses_gb300 as q

pytestmark = pytest.mark.gpu


def _sheet(axis, side):
    k = np.arange(side, dtype=np.float32)
    a, b = np.meshgrid(k, k, indexing="ij")
    xyz = np.zeros((a.size, 3), np.float32)
    xyz[:, (axis + 1) % 3], xyz[:, (axis + 2) % 3] = a.ravel(), b.ravel()
    return xyz, np.full(len(xyz), 1.7, np.float32)


def test_a_sheet_normal_to_x_takes_little_longer_than_one_normal_to_z():
    # 520^3 words: 14 times as long with 512 words to a warp, 4 with 128
    best = {}
    with q.Context(0) as c:
        c.set_profiling(True)
        for axis in (0, 2):
            xyz, rad = _sheet(axis, 200)
            times = []
            for _ in range(6):
                c.compute(xyz, rad, voxel=0.4, smooth=0)
                times.append(dict(c.stage_times())["mc_emit"])
            best[axis] = min(times)
    assert best[0] < 7 * best[2], best
