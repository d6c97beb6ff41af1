"""The order of few atoms, where blocks and the one-launch path end.

The same atoms inside a larger molecule of the same bounds take the radix sort: each atom's cell key
is the same there, and the order is the stable one of the keys.
"""
import numpy as np
import pytest

import quickses_gb300 as q

pytestmark = pytest.mark.gpu


def _box(n, size, seed):
    r = np.random.default_rng(seed)
    xyz = r.uniform(0, size, (n, 3)).astype(np.float32)
    xyz[0], xyz[1] = 0, size  # the bounds
    return xyz, np.full(n, 1.7, np.float32)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 257, 4096, 8191, 8192, 8193])
@pytest.mark.parametrize("size", [6.0, 70.0, 265.0])
def test_few_atoms_are_in_stable_key_order(n, size):
    xyz, rad = _box(12000, size, n)
    dx = 1.5 if size > 100 else 0.7
    with q.Context(0) as c:
        c.compute(xyz, rad, voxel=dx, smooth=0)
        order, keys = c.debug_atom_order(len(xyz))
        want = np.empty(len(xyz), keys.dtype)
        want[order] = keys
        c.compute(xyz[:n], rad[:n], voxel=dx, smooth=0)
        order, keys = c.debug_atom_order(n)
    assert np.array_equal(order, np.argsort(want[:n], kind="stable"))
    assert np.array_equal(keys, want[:n][order])
