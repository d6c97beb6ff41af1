"""The marching-cubes emission where rows, words and a warp's share of them end.

Grids whose cells end on, before and behind a 32-voxel word, from a few words to many shares, alone
and side by side in a batch (each molecule's shares start at its own first word).
"""
import numpy as np
import pytest

import quickses_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ENDS = (0, 1, 2, 30, 31)  # cells per axis modulo 32


def _cases():
    """(atoms, voxel) with cells per axis at each end of a word, small and large."""
    got = {}
    for n in (3, 25, 500):
        xyz, rad, _ = q.molecules.ball(n, 40 + n)
        for dx in np.linspace(0.24, 0.5, 105).astype(np.float32):
            gc = O.grid(xyz, rad, float(dx))[0].Gc
            if gc % 32 in ENDS:
                got.setdefault((n, gc % 32), (n, float(dx)))
    return [got[k] for k in sorted(got)]


CASES = _cases()


def _molecule(n):
    return q.molecules.ball(n, 40 + n)[:2]


def test_cases_cover_the_ends():
    assert len(CASES) == 3 * len(ENDS)


@pytest.mark.parametrize("n,dx", CASES)
def test_emission_matches_oracle(n, dx):
    xyz, rad = _molecule(n)
    m = O.compute_ses(xyz, rad, dx, smooth=0, fp64=False)
    with q.Context(0) as c:
        got = c.compute(xyz, rad, voxel=dx, smooth=0, keep_degenerate=True)
    assert np.array_equal(got.triangles, m.triangles)
    assert np.array_equal(got.vertices, m.vertices_q.astype(np.float32))


def test_emission_of_a_batch_matches_oracle():
    reqs = [dict(xyz=_molecule(n)[0], radii=_molecule(n)[1], voxel=dx, smooth=0, keep_degenerate=True) for n, dx in CASES]
    with q.Context(0) as c:
        for got, (n, dx) in zip(c.compute_batch(reqs), CASES):
            m = O.compute_ses(*_molecule(n), dx, smooth=0, fp64=False)
            assert np.array_equal(got.triangles, m.triangles)
            assert np.array_equal(got.vertices, m.vertices_q.astype(np.float32))
