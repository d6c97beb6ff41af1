"""The SAS classification where a tile's candidates stop fitting, and at its rows' ends.

Crowded atoms (several hundred to several thousand around one tile), coarse voxels, radii far from
an atom's, atoms whose spheres end on a voxel; voxel codes equal the oracle's.
"""
import numpy as np
import pytest

import quickses_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _crowd(n, spread, seed, low=1.2, high=2.0):
    r = np.random.default_rng(seed)
    return r.normal(0, spread, (n, 3)).astype(np.float32), r.uniform(low, high, n).astype(np.float32)


MOLECULES = {
    "crowd-500": (_crowd(500, 2.0, 1), 0.3),
    "crowd-513": (_crowd(513, 0.3, 2), 0.5),
    "crowd-3000": (_crowd(3000, 2.5, 3), 0.5),
    "coarse": (_crowd(4000, 9.0, 4), 2.0),
    "small and large radii": (_crowd(60, 6.0, 5, 0.05, 12.0), 0.4),
    "voxel ends": ((np.float32([[0, 0, 0], [0, 0, 3], [1.5, 0, 0]]), np.float32([1.6, 1.6, 1.1])), 0.5),
    "one word": (_crowd(2, 0.5, 6), 0.157),
}


@pytest.mark.parametrize("name", sorted(MOLECULES))
def test_codes_match_oracle(name):
    (xyz, rad), dx = MOLECULES[name]
    g = O.grid(xyz, rad, dx)[0]
    with q.Context(0) as c:
        c.compute(xyz, rad, voxel=dx, smooth=0)
        codes = c.debug_codes(g.G)
    assert np.array_equal(codes, O.field_codes(xyz, rad, g, fp64=False))


def test_batch_matches_single():
    reqs = [dict(xyz=m[0], radii=m[1], voxel=dx, smooth=0) for m, dx in MOLECULES.values()]
    with q.Context(0) as c:
        for got, r in zip(c.compute_batch(reqs), reqs):
            want = c.compute(r["xyz"], r["radii"], voxel=r["voxel"], smooth=0)
            assert np.array_equal(got.vertices, want.vertices) and np.array_equal(got.triangles, want.triangles)
