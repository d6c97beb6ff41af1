"""The weld where its planes, bins and widths end.

Grids of a few planes and of hundreds, planes with no edge and with thousands, voxels down to the
smallest supported (many positions fall on one quantum), coordinates of either sign and as far out
as they go (a float there is no finer than the quantum).  Positions, their order and the triangles
are whole numbers: nothing may differ.
"""
import numpy as np
import pytest

import quickses_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _molecule(n, seed, shift):
    if n >= 2000:  # planes of thousands of edges: the x ranges come from a part of them
        xyz, rad, _ = q.molecules.shell(n, seed, r_in=20.0)
    else:
        xyz, rad, _ = q.molecules.ball(n, seed)
    return (xyz + np.float32(shift)).astype(np.float32), rad


CASES = [(2, 1, 0.0, 0.157), (2, 2, 0.0, 2.5), (2, 3, -15900.0, 0.3), (2, 4, 15900.0, 0.5), (40, 5, 0.0, 0.16),
         (40, 6, -7.0, 1.1), (300, 7, 4000.0, 0.4), (1500, 8, 0.0, 0.2),
         (2000, 9, 3.0, 0.3)]


def _want(n, seed, shift, dx):
    xyz, rad = _molecule(n, seed, shift)
    return xyz, rad, O.compute_ses(xyz, rad, dx, smooth=0, fp64=False)


@pytest.mark.parametrize("n,seed,shift,dx", CASES)
def test_weld_matches_oracle(n, seed, shift, dx):
    xyz, rad, m = _want(n, seed, shift, dx)
    with q.Context(0) as c:
        got = c.compute(xyz, rad, voxel=dx, smooth=0, keep_degenerate=True)
    assert np.array_equal(got.vertices, m.vertices_q.astype(np.float32))
    assert np.array_equal(got.triangles, m.triangles)


def test_weld_of_a_batch_matches_oracle():
    order = [8, 7, 0, 3, 1, 6, 2, 5, 4]
    with q.Context(0) as c:
        for idx in (order, order[1:4]):
            wants = [_want(*CASES[k]) for k in idx]
            got = c.compute_batch([dict(xyz=x, radii=r, voxel=CASES[k][3], smooth=0, keep_degenerate=True)
                                   for k, (x, r, _) in zip(idx, wants)])
            for g, (_, _, m) in zip(got, wants):
                assert np.array_equal(g.vertices, m.vertices_q.astype(np.float32))
                assert np.array_equal(g.triangles, m.triangles)
