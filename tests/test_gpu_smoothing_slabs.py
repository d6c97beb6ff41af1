"""The smoothing kernel where its slabs, lists and halves end.

Small slabs put most neighbours into other slabs (both ways, several slabs apart), 0.2 A voxels
give lists on both sides of the 16 entries that are packed (up to 56), and a slab of a few vertices
or of a whole molecule is one chain or many at once.  Every result is the sequential pass's, bit
for bit: the sums and divisions are the same operations in the same order, so nothing may differ.
"""
import numpy as np
import pytest

import quickses_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def meshes():
    got = {}
    for n, seed, voxel in ((2, 1, 0.5), (90, 5, 0.2), (700, 6, 0.3)):
        xyz, rad, _ = q.molecules.ball(n, seed)
        got[n] = xyz, rad, voxel, O.compute_ses(xyz, rad, voxel, smooth=0, fp64=False)
    return got


def test_lists_cover_both_forms(meshes):
    lengths = 2 * np.bincount(meshes[90][3].triangles.ravel())
    assert lengths.max() > 32 and (lengths > 16).mean() > 0.05 and (lengths <= 16).any()


@pytest.mark.parametrize("n", [2, 90, 700])
@pytest.mark.parametrize("passes", [1, 3])
@pytest.mark.parametrize("threads,target,wave", [(0, 0, 0), (512, 256, 0), (1024, 257, 0), (512, 300, 1000),
                                                 (512, 5376, 0), (1024, 25000, 0), (512, 777, 4099)])
def test_slabs_match_the_sequential_pass(meshes, n, passes, threads, target, wave):
    xyz, rad, voxel, m = meshes[n]
    want = O.smooth_f32(m.vertices_q.astype(np.float32), m.triangles, passes)
    with q.Context(0) as c:
        if threads:
            c.set_smoothing_shape(threads, target, 0, wave)
        got = c.compute(xyz, rad, voxel=voxel, smooth=passes, keep_degenerate=True)
    assert np.array_equal(got.triangles, m.triangles)
    assert np.array_equal(got.vertices, want)
