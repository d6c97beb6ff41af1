"""The degenerate filter at the ends of its tiles of 4 096 triangles.

Molecules whose triangles, many of them with a repeated corner, end just before, at and just behind a
tile's end, and not at one of a thread's eight; filtered in place (no smoothing), beside the smoothing
into an array of their own, and side by side in batches whose molecules start anywhere in a tile.
"""
import numpy as np
import pytest

import quickses_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# triangles before the filter: (atoms, seed, voxel)
MESHES = {4092: (9, 36, 0.35), 4096: (9, 30, 0.35), 4100: (7, 32, 0.35), 4104: (7, 41, 0.35), 8184: (23, 34, 0.35),
          8188: (19, 7, 0.35), 8192: (20, 14, 0.35), 8196: (22, 11, 0.35), 12288: (36, 50, 0.35), 12292: (35, 43, 0.35),
          16380: (33, 20, 0.28), 16388: (12, 39, 0.2)}


def _molecule(nt):
    n, seed, voxel = MESHES[nt]
    xyz, rad, _ = q.molecules.ball(n, seed)
    t = O.compute_ses(xyz, rad, voxel, smooth=0, fp64=False).triangles
    a, b, c = t.T
    kept = t[(a != b) & (b != c) & (a != c)]
    assert len(t) == nt and len(kept) < nt
    return xyz, rad, voxel, t, kept


@pytest.mark.parametrize("passes", [0, 1])
@pytest.mark.parametrize("nt", MESHES)
def test_filter_at_the_end_of_a_tile(nt, passes):
    xyz, rad, voxel, every, kept = _molecule(nt)
    with q.Context(0) as c:
        assert np.array_equal(c.compute(xyz, rad, voxel=voxel, smooth=passes).triangles, kept)
        assert np.array_equal(c.compute(xyz, rad, voxel=voxel, smooth=passes, keep_degenerate=True).triangles, every)
        assert np.array_equal(c.compute(xyz, rad, voxel=voxel, smooth=passes).triangles, kept)


@pytest.mark.parametrize("passes", [0, 1])
@pytest.mark.parametrize("order", [(4096, 4096), (4092, 4100, 4096), (4092, 4104, 4092, 8196, 12292), (8188, 4100, 4096, 4092),
                                   (4104, 8184, 16380, 4092, 16388)])
def test_batches_at_the_ends_of_tiles(order, passes):
    mols = [_molecule(nt) for nt in order]
    for keep in (set(), {0}, {len(order) - 1}, set(range(len(order)))):
        reqs = [dict(xyz=m[0], radii=m[1], voxel=m[2], smooth=passes, keep_degenerate=k in keep) for k, m in enumerate(mols)]
        with q.Context(0) as c:
            for k, got in enumerate(c.compute_batch(reqs)):
                assert np.array_equal(got.triangles, mols[k][3 if k in keep else 4])
