"""The weld of meshes that crowd a few grid planes.

A face normal to x has all its edges in one or two x layers; one normal to y and a fibre along z have
a layer's edges at a few y: a layer by itself then takes ever longer, and the weld sorts all edges
instead.  Sheets
and fibres along each axis, alone, beside ordinary molecules and in slices: positions, their order
and the triangles are whole numbers, so nothing may differ.
"""
import numpy as np
import pytest

import quickses_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _sheet(axis, side, step, jitter=0.0, shift=0.0):
    k = np.arange(int(side / step), dtype=np.float32) * np.float32(step)
    a, b = np.meshgrid(k, k, indexing="ij")
    xyz = np.zeros((a.size, 3), np.float32)
    xyz[:, (axis + 1) % 3], xyz[:, (axis + 2) % 3] = a.ravel(), b.ravel()
    xyz += np.random.default_rng(axis).normal(0.0, jitter, xyz.shape).astype(np.float32) + np.float32(shift)
    return xyz, np.full(len(xyz), 1.7, np.float32)


def _fibre(axis, length, step):
    xyz = np.zeros((int(length / step), 3), np.float32)
    xyz[:, axis] = np.arange(len(xyz)) * np.float32(step)
    return xyz, np.full(len(xyz), 6.0, np.float32)


def _ball(n, seed):
    return q.molecules.ball(n, seed)[:2]


# name -> (molecule, voxel, whether a layer is crowded)
SHAPES = {
    "sheet x": (_sheet(0, 60, 1.0), 0.4, True),
    "sheet y": (_sheet(1, 60, 1.0), 0.4, False),
    "sheet z": (_sheet(2, 60, 1.0), 0.4, False),
    "rough sheet x": (_sheet(0, 75, 1.5, 0.3, -40.0), 0.4, True),
    "sheet x at 0.2": (_sheet(0, 40, 0.8, 0.0, 900.0), 0.2, True),
    "fibre x": (_fibre(0, 150, 0.3), 0.25, False),
    "fibre z": (_fibre(2, 150, 0.3), 0.25, True),
    "ball": (_ball(500, 3), 0.4, False),
    "two atoms": (_ball(2, 4), 0.3, False),
}


@pytest.fixture(scope="module")
def meshes():
    return {k: O.compute_ses(*mol, dx, smooth=0, fp64=False) for k, (mol, dx, _) in SHAPES.items()}


def _same(got, want):
    assert np.array_equal(got.vertices, want.vertices_q.astype(np.float32))
    assert np.array_equal(got.triangles, want.triangles)


@pytest.mark.parametrize("name", SHAPES)
def test_weld_of_a_shape_matches_oracle(meshes, name):
    (xyz, rad), dx, crowded = SHAPES[name]
    with q.Context(0) as c:
        c.compute(*SHAPES["ball"][0], voxel=0.4, smooth=0, keep_degenerate=True)
        usual = c.last_launch_count()
        for graphs in (True, False, True):
            c.set_graphs(graphs)
            _same(c.compute(xyz, rad, voxel=dx, smooth=0, keep_degenerate=True), meshes[name])
            assert (c.last_launch_count() > usual + 8) == crowded  # the sort's passes


@pytest.mark.parametrize("names", [("sheet x",), ("ball", "sheet x", "two atoms"),
                                   ("two atoms", "rough sheet x", "ball", "fibre z", "sheet x at 0.2", "fibre x", "ball"),
                                   ("sheet z", "ball")])
def test_weld_of_a_batch_of_shapes_matches_oracle(meshes, names):
    reqs = [dict(xyz=SHAPES[k][0][0], radii=SHAPES[k][0][1], voxel=SHAPES[k][1], smooth=0, keep_degenerate=True)
            for k in names]
    with q.Context(0) as c:
        for _ in range(2):
            for got, k in zip(c.compute_batch(reqs), names):
                _same(got, meshes[k])


@pytest.mark.parametrize("slice_", [130, 400])
def test_slices_of_a_sheet_match_oracle(slice_):
    (xyz, rad), dx, _ = SHAPES["sheet x"]
    want = O.compute_ses_slices(xyz, rad, dx, slice_, smooth=1)
    with q.Context(0) as c:
        got = c.compute(xyz, rad, voxel=dx, smooth=1, keep_degenerate=True, slice=slice_, reference_slices=True)
    assert np.array_equal(got.vertices, want.vertices.astype(np.float32))
    assert np.array_equal(got.triangles, want.triangles)


@pytest.mark.parametrize("passes", [1, 3])
def test_smoothing_behind_a_sorted_weld(meshes, passes):
    (xyz, rad), dx, _ = SHAPES["sheet x"]
    want = O.compute_ses(xyz, rad, dx, smooth=passes, fp64=False)
    with q.Context(0) as c:
        got = c.compute(xyz, rad, voxel=dx, smooth=passes, keep_degenerate=True)
    assert np.array_equal(got.vertices, want.vertices.astype(np.float32))
    assert np.array_equal(got.triangles, want.triangles)


@pytest.mark.parametrize("molecule,dx", [(_sheet(0, 200, 1.0), 0.4), (_sheet(0, 300, 1.5, 0.3), 0.4), (_sheet(1, 600, 1.0), 0.4),
                                         (_fibre(2, 400, 0.3), 0.25)])
def test_the_weld_takes_no_longer_than_the_rest(molecule, dx):
    # 0.05 to 0.3 of it where the sort takes over, 20 to 30 times as long where a layer stayed one CTA's
    with q.Context(0) as c:
        c.set_profiling(True)
        best = np.inf
        for _ in range(5):
            c.compute(*molecule, voxel=dx, smooth=0, keep_degenerate=True)
            times = dict(c.stage_times())
            best = min(best, times["weld"] / (sum(times.values()) - times["weld"]))
    assert best < 1.0
