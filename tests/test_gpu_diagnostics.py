"""Smoothing diagnostics of profiled calls: every documented value is counted, and counting does not
change the mesh.
"""
import numpy as np
import pytest

import quickses_gb300 as q

pytestmark = pytest.mark.gpu

CYCLES = ["update_cycles", "release_cycles", "id_wait_cycles", "position_wait_cycles", "store_fence_cycles"]


@pytest.mark.parametrize("n,voxel,passes", [(300, 0.5, 1), (2000, 0.2, 1), (800, 0.3, 3)])  # 0.2 A: long lists too
def test_profiled_calls_count_the_parts_of_an_update(n, voxel, passes):
    xyz, rad, _ = q.molecules.ball(n, 51)
    with q.Context(0) as c:
        want = c.compute(xyz, rad, voxel=voxel, smooth=passes)
        assert all(c.diagnostics()[k] == 0 for k in CYCLES + ["vertices", "max_polls"])
        for level in (1, 2, True):
            c.set_profiling(level)
            got = c.compute(xyz, rad, voxel=voxel, smooth=passes)
            assert np.array_equal(got.vertices, want.vertices) and np.array_equal(got.triangles, want.triangles)
            d = c.diagnostics()
            assert d["vertices"] == passes * len(want.vertices) and d["unfinished_slabs"] == 0
            if level == 2:
                assert all(d[k] == 0 for k in CYCLES)
                continue
            assert all(d[k] > 0 for k in CYCLES)
            # parts of the update, and a step of one or two vertices takes hundreds of cycles
            assert d["id_wait_cycles"] + d["position_wait_cycles"] + d["store_fence_cycles"] <= d["update_cycles"]
            assert 100 < d["update_cycles"] / d["vertices"] < 100_000
