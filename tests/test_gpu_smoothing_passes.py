"""Several smoothing passes in one launch where slabs share a word of release counters.

A slab's end sets its vertices' byte counters for the next pass while lower slabs may still count down
the bytes next to them, so slabs and molecules start at every place within a word here, and dozens
are under way together.  Every result is the sequential passes', bit for bit.
"""
import numpy as np
import pytest

import quickses_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MOLECULES = [(40, 1), (300, 2), (2, 3), (150, 4), (900, 5), (3, 6), (60, 7)]


@pytest.fixture(scope="module")
def meshes():
    got = []
    for n, seed in MOLECULES:
        xyz, rad, _ = q.molecules.ball(n, seed)
        got.append((xyz, rad, O.compute_ses(xyz, rad, 0.4, smooth=0, fp64=False)))
    return got


@pytest.mark.parametrize("passes", [2, 5])
@pytest.mark.parametrize("target", [257, 258, 259, 260, 1000])
def test_batches_match_the_sequential_passes(meshes, passes, target):
    starts = np.cumsum([len(m.vertices_q) for _, _, m in meshes])
    assert 2 in starts % 4  # molecules that share words (a closed surface has an even number of vertices)
    with q.Context(0) as c:
        c.set_smoothing_shape(512, target, 0, 0)
        got = c.compute_batch([dict(xyz=x, radii=r, voxel=0.4, smooth=passes, keep_degenerate=True) for x, r, _ in meshes])
    for g, (_, _, m) in zip(got, meshes):
        assert np.array_equal(g.vertices, O.smooth_f32(m.vertices_q.astype(np.float32), m.triangles, passes))
