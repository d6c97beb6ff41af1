"""The closest atom where several are equally close and where there are few or none around.

Lattices give exact ties, of which the first in cell order wins; spread-out atoms leave most of the
27 cells empty; coordinates far out round the most.  Compared with every atom, in the kernel's
arithmetic, by exact sums.
"""
import numpy as np
import pytest

import quickses_gb300 as q

pytestmark = pytest.mark.gpu


def _lattice(n, step, shift):
    k = np.arange(n, dtype=np.float32) * np.float32(step)
    return np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3).astype(np.float32) + np.float32(shift)


MOLECULES = {
    "lattice": (_lattice(4, 1.5, 0.0), 1.7),
    "coarse": (_lattice(3, 4.0, -3.0), 1.5),
    "cells": (_lattice(3, 3.1, 0.25), 1.7),
    "far": (_lattice(3, 2.0, 15900.0), 1.8),
    "apart": (np.float32([[0, 0, 0], [30, 0, 0], [0, 29, 31]]), 1.4),
    "ball": (q.molecules.ball(150, 5)[0], 1.6),
}


def _distances(v, atoms):
    """fma(ez, ez, fma(ey, ey, ex * ex)) in 32 bits, each rounded once from an exact sum."""
    wide = np.longdouble
    e = atoms[None] - v[:, None]
    d = (e[..., 0].astype(wide) ** 2).astype(np.float32)
    for c in (1, 2):
        d = (e[..., c].astype(wide) ** 2 + d.astype(wide)).astype(np.float32)
    return d


@pytest.mark.parametrize("name", sorted(MOLECULES))
@pytest.mark.parametrize("batch", [False, True])
def test_closest_atom(name, batch):
    xyz, radius = MOLECULES[name]
    rad = np.full(len(xyz), radius, np.float32)
    with q.Context(0) as c:
        alone = c.compute(xyz, rad, voxel=0.5, smooth=0)
        order = c.debug_atom_order(len(xyz))[0]
        if batch:
            got = c.compute_batch([dict(xyz=MOLECULES["ball"][0], radii=np.full(150, 1.6, np.float32), voxel=0.7, smooth=0),
                                   dict(xyz=xyz, radii=rad, voxel=0.5, smooth=0)])[1]
        else:
            got = alone
    d = _distances(got.vertices, xyz[order])
    assert d.min(1).max() < 7.8  # within the cells around each vertex, 2.8 A and more wide
    assert np.array_equal(got.atom_sorted, d.argmin(1))  # the first of the least
    assert np.array_equal(got.atom_input, order[d.argmin(1)])
