"""Atoms that are nowhere: a coordinate that is not a number.

Such an atom bounds nothing and reaches no voxel, in the reference and in the batch form, whose bounds
are taken on the host; the single form takes them on the device and has to agree.  The mesh is the
other atoms'; only the numbers of the atoms in cell order may shift.
"""
import numpy as np
import pytest

import quickses_gb300 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [50, 9000])  # ordered in one launch, and by the sort
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("axes", [(0,), (2,), (0, 1, 2)])
def test_the_mesh_is_the_other_atoms(n, sign, axes):
    xyz, rad, _ = q.molecules.ball(n, 91)
    xyz = xyz * np.float32([1.0, 0.5, 0.5])  # longest along x, which then has no bound of its own
    bad = np.insert(xyz, n // 2, np.float32(1.0), axis=0)
    bad[n // 2, list(axes)] = np.copysign(np.float32(np.nan), np.float32(sign))
    radii = np.insert(rad, n // 2, rad[0])
    with q.Context(0) as c:
        want = c.compute(xyz, rad, voxel=0.5, smooth=1)
        got = c.compute(bad, radii, voxel=0.5, smooth=1)
        batch, = c.compute_batch([dict(xyz=bad, radii=radii, voxel=0.5, smooth=1)])
        for m in (got, batch):
            assert np.array_equal(m.vertices, want.vertices) and np.array_equal(m.triangles, want.triangles)
            assert np.array_equal(m.atom_input - (m.atom_input > n // 2), want.atom_input)
        assert np.array_equal(c.compute(xyz, rad, voxel=0.5, smooth=1).vertices, want.vertices)
