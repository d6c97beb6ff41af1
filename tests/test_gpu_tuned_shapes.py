"""A tuned smoothing shape applies to calls like the one it was tuned on.

The best slab size depends on the number of passes and, in a batch, on its largest molecule: a shape
found for one pass, or for a batch of small molecules, says nothing about other calls of as many
vertices.  Meshes are the same with any shape.
"""
import numpy as np
import pytest

import quickses_gb300 as q

pytestmark = pytest.mark.gpu


def _slab_sizes(c, xyz, rad):
    out = {}
    for passes in (1, 2, 3):
        m = c.compute(xyz, rad, voxel=0.37, smooth=passes)
        out[passes] = c.diagnostics()["slab_size"], m.vertices
    return out


@pytest.mark.parametrize("tuned,others", [(1, (2, 3)), (3, (1,))])
def test_single_molecules(tuned, others):
    xyz, rad, _ = q.molecules.ball(30 if tuned == 1 else 120, 61)  # two sizes, so two entries of the table
    with q.Context(0) as c:
        before = _slab_sizes(c, xyz, rad)
        c.autotune(xyz, rad, voxel=0.37, smooth=tuned)
        after = _slab_sizes(c, xyz, rad)
    for passes in others:
        assert after[passes][0] == before[passes][0]
    for passes in (1, 2, 3):
        assert np.array_equal(after[passes][1], before[passes][1])


def test_batches_of_other_molecules():
    small = [q.molecules.ball(25, 70 + i)[:2] for i in range(40)]
    mixed = [q.molecules.ball(n, 70)[:2] for n in (2600, 30, 40)]

    def run(c, mols):
        out = c.compute_batch([dict(xyz=x, radii=r, voxel=0.45, smooth=1) for x, r in mols])
        return c.diagnostics()["slab_size"], out

    with q.Context(0) as c:
        size, want = run(c, mixed)
    with q.Context(0) as c:
        vertices = [sum(len(m.vertices) for m in out) for out in (want, run(c, small)[1])]
        assert vertices[0].bit_length() == vertices[1].bit_length()  # as many in all
        c.autotune_batch([dict(xyz=x, radii=r, voxel=0.45, smooth=1) for x, r in small])
    with q.Context(0) as c:
        got = run(c, mixed)
    assert got[0] == size
    assert all(np.array_equal(a.vertices, b.vertices) for a, b in zip(got[1], want))
