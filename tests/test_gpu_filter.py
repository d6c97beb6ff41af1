"""The degenerate filter where its tiles of 1024 triangles and its molecules end.

Meshes of a dozen triangles and of several tiles, filtered or kept, alone and side by side in one
batch (molecules that start and end inside a tile, next to ones that keep every triangle).
"""
import numpy as np
import pytest

import quickses_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# (atoms, seed, voxel, keep): voxels of 0.2 A collapse the most triangles
CASES = [(2, 2, 2.5, False), (2, 2, 2.5, True), (2, 1, 0.2, False), (2, 5, 1.3, False), (30, 6, 0.2, False),
         (30, 6, 0.2, True), (3, 7, 1.0, True), (400, 8, 0.3, False), (2, 9, 2.0, False)]


@pytest.fixture(scope="module")
def meshes():
    got = []
    for n, seed, voxel, keep in CASES:
        xyz, rad, _ = q.molecules.ball(n, seed)
        t = O.compute_ses(xyz, rad, voxel, smooth=0, fp64=False).triangles
        a, b, c = t.T
        got.append((xyz, rad, t if keep else t[(a != b) & (b != c) & (a != c)]))
    return got


def test_some_triangles_are_dropped(meshes):
    full = [len(O.compute_ses(x, r, CASES[k][2], smooth=0, fp64=False).triangles) for k, (x, r, _) in enumerate(meshes)]
    assert any(len(m[2]) < f for m, f in zip(meshes, full)) and min(full) < 1024 < 20 * 1024 < max(full)


@pytest.mark.parametrize("k", range(len(CASES)))
def test_filter_matches_oracle(meshes, k):
    xyz, rad, want = meshes[k]
    with q.Context(0) as c:
        got = c.compute(xyz, rad, voxel=CASES[k][2], smooth=0, keep_degenerate=CASES[k][3])
    assert np.array_equal(got.triangles, want)


@pytest.mark.parametrize("order", [range(9), (4, 0), (0, 1), (8, 5, 7, 2, 6, 4, 1, 3, 0), (0,) * 40 + (7,) + (1,) * 40])
def test_filter_of_a_batch_matches_oracle(meshes, order):
    reqs = [dict(xyz=meshes[k][0], radii=meshes[k][1], voxel=CASES[k][2], smooth=0, keep_degenerate=CASES[k][3])
            for k in order]
    with q.Context(0) as c:
        for got, k in zip(c.compute_batch(reqs), order):
            assert np.array_equal(got.triangles, meshes[k][2])
