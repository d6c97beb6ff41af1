"""Host results of smoothed calls: the smoothing kernel itself stores the vertices to the host's block,
while triangles and atom ids come over the side stream, which starts with the smoothing or with its
neighbour lists.

Both are compared with the same call's device mesh and with a profiled call, which has one stream.
"""
import numpy as np
import pytest

import quickses_gb300 as q

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


class _DeviceArray:
    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


def _same(a, b):
    assert np.array_equal(a.vertices, b.vertices) and np.array_equal(a.triangles, b.triangles)
    assert np.array_equal(a.atom_sorted, b.atom_sorted) and np.array_equal(a.atom_input, b.atom_input)


@pytest.mark.parametrize("n,voxel", [(2, 2.0), (200, 0.5), (3000, 0.3)])
@pytest.mark.parametrize("passes", [1, 3])
@pytest.mark.parametrize("wave", [0, 2000])  # several launches a pass, each storing its own vertices
def test_vertices_on_the_host_are_the_device_mesh(n, voxel, passes, wave):
    xyz, rad, _ = q.molecules.ball(n, 81)
    d_xyz, d_rad = torch.from_numpy(xyz).cuda(), torch.from_numpy(rad).cuda()
    torch.cuda.synchronize()
    with q.Context(0) as c:
        c.set_smoothing_shape(512, 512, 0, wave)
        host = c.compute(xyz, rad, voxel=voxel, smooth=passes)
        dm = c.compute_device(d_xyz.data_ptr(), d_rad.data_ptr(), n, voxel=voxel, smooth=passes)
        v = torch.as_tensor(_DeviceArray(dm.d_vertices, (dm.n_vertices, 3), "<f4"), device="cuda").cpu().numpy()
        assert np.array_equal(v, host.vertices)
        c.set_profiling(2)
        _same(c.compute(xyz, rad, voxel=voxel, smooth=passes), host)


# Two CTAs an SM: the side stream waits for the lists unless there are more than two slabs to a CTA.
@pytest.mark.parametrize("target,late", [(256, False), (5376, True)])
@pytest.mark.parametrize("batch", [False, True])
def test_the_side_stream_at_either_place(target, late, batch):
    mols = [q.molecules.ball(n, 82)[:2] for n in ((3000,) if not batch else (2500, 40, 900, 2))]
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def run(c):
        if not batch:
            return [c.compute(*mols[0], voxel=0.3, smooth=1)]
        return c.compute_batch([dict(xyz=x, radii=r, voxel=0.3, smooth=1) for x, r in mols])

    with q.Context(0) as c:
        c.set_smoothing_shape(512, target)
        got = run(c)
        slabs = c.diagnostics()["slabs"]
        assert slabs <= 2 * sms if late else slabs > 4 * sms
        again = run(c)
        c.set_profiling(2)
        for a, b, d in zip(got, again, run(c)):
            _same(a, b)
            _same(a, d)
