"""The work this library is measured on: molecules of the sizes its users mesh, through the entry points they call.

Atom counts, voxel sizes and batch shapes are those of ``quickses_gb300.molecules`` (the benchmark's workloads, the
trajectory, the uneven batch and the range of the served stream), the tests and the command line's defaults.  The
molecules are synthetic: heavy atoms at protein density in a ball, or in a thick shell.
"""
import ctypes
import math

import numpy as np
import torch

import quickses_gb300 as q
from quickses_gb300 import _lib as L


def listed():
    return [
        # a ligand or a peptide through the Python call: nothing but latency, launches and read-backs
        {"name": "peptide", "call": "compute", "atoms": 200, "voxel": 0.5, "passes": 1},
        # the benchmark's 1 000-atom molecule through the drop-in API_* functions of the original library
        {"name": "protein", "call": "reference_api", "atoms": 1000, "voxel": 0.5, "passes": 1},
        # a viewer that redraws one frame of a simulation and keeps the mesh on the device
        {"name": "frame", "call": "device", "atoms": 5000, "voxel": 0.4, "passes": 1},
        # the command line's options: three passes, triangles with a repeated corner kept
        {"name": "three_passes", "call": "device", "atoms": 12001, "voxel": 0.3, "passes": 3, "keep": True},
        # a fine mesh for analysis, held on the device
        {"name": "fine", "call": "device", "atoms": 20000, "voxel": 0.2, "passes": 1},
        # the headline workload, host atoms in and a host mesh out
        {"name": "complex", "call": "host", "atoms": 50000, "voxel": 0.2, "passes": 1},
        # the largest molecule of the served stream
        {"name": "large", "call": "device", "atoms": 200000, "voxel": 0.3, "passes": 1},
        # the benchmark's million-atom capsid-like shell, without smoothing
        {"name": "shell", "call": "device", "shape": "shell", "atoms": 1000000, "voxel": 0.5, "passes": 0},
        # frames of a trajectory in one batch
        {"name": "trajectory", "call": "frames", "atoms": 5000, "voxel": 0.4, "passes": 1, "count": 16},
        # unrelated molecules of uneven size in one batch
        {"name": "uneven_batch", "call": "batch", "atoms": 500, "most": 20000, "voxel": 0.4, "passes": 1, "count": 16},
        # a mesh to be compared with one the original program wrote: its slices, seams and all
        {"name": "slices", "call": "slices", "atoms": 5000, "voxel": 0.3, "passes": 1, "slice": 150},
        # a plugin that may not allocate: the voxel field into its own buffer
        {"name": "plugin_field", "call": "field", "atoms": 1000, "voxel": 0.5, "passes": 0},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["compute", "reference_api", "device", "device", "device", "host", "frames", "batch", "slices", "field"])
    voxel = rng.choice([0.2, 0.25, 0.3, 0.4, 0.5, round(rng.uniform(0.2, 0.6), 3)])
    passes = rng.choice([0, 1, 1, 1, 2, 3])
    case = {"call": call, "atoms": 0, "voxel": voxel, "passes": passes}
    if call in ("compute", "reference_api"):
        case["atoms"] = log_int(150, 3000)
    elif call == "device":
        case["shape"] = rng.choice(["ball", "ball", "shell"])
        most = 200000 if voxel >= 0.3 else 50000
        if case["shape"] == "shell":  # all surface: many vertices to an atom
            most = min(most, int(2e7 * voxel ** 2 / (34.6 * (1 + passes))))
        case["atoms"] = log_int(300, most)
        case["keep"] = rng.random() < 0.3
    elif call == "host":
        case["atoms"] = log_int(2000, 50000)
    elif call == "frames":
        case.update(atoms=log_int(500, 5000), voxel=max(voxel, 0.3), count=rng.randint(2, 16))
    elif call == "batch":
        case.update(atoms=log_int(150, 1000), most=log_int(3000, 20000), voxel=max(voxel, 0.3), count=rng.randint(2, 16))
    elif call == "slices":
        case.update(atoms=log_int(800, 5000), voxel=max(voxel, 0.3), passes=min(passes, 1), slice=rng.randint(100, 300))
    else:
        case.update(atoms=log_int(200, 1500), voxel=max(voxel, 0.45), passes=0)
    return case


def _molecules(case):
    n = case["atoms"]
    if case["call"] == "frames":
        base, rad, _ = q.molecules.ball(n, 77)
        return [(q.molecules.jitter(base, 0.3, 7700 + f), rad) for f in range(case["count"])]
    if case["call"] == "batch":
        sizes = np.exp(np.linspace(math.log(n), math.log(case["most"]), case["count"])).astype(int)
        return [q.molecules.ball(int(k), 2024 + i)[:2] for i, k in enumerate(np.random.default_rng(2024).permutation(sizes))]
    if case.get("shape") == "shell":
        # the benchmark's shell has 1 000 000 atoms between 400 and 430 A; smaller ones keep its density and thickness
        return [q.molecules.shell(n, 1, r_in=max(20.0, 400.0 * math.sqrt(n / 1e6)))[:2]]
    return [q.molecules.ball(n, 1)[:2]]


def _atoms(case, seed):
    """The molecules of a case, [(coordinates, radii)], their atoms in an order of the seed's.  A file lists atoms in any
    order; the ids of the closest atoms go by it, while the mesh keeps its size, so that passes on other inputs can be
    compared."""
    got = []
    if case["call"] == "field":
        # the field has no ids in it: another seed's molecule is another frame, inside the same box
        xyz, rad = _molecules(case)[0]
        moved = np.clip(q.molecules.jitter(xyz, 0.3, int(seed) % (1 << 60)), xyz.min(0), xyz.max(0))
        ends = np.concatenate([xyz.argmin(0), xyz.argmax(0)])
        moved[ends] = xyz[ends]
        return [(moved, rad)]
    for i, (xyz, rad) in enumerate(_molecules(case)):
        order = np.random.default_rng([int(seed) % (1 << 60), i]).permutation(len(rad))
        got.append((np.ascontiguousarray(xyz[order]), np.ascontiguousarray(rad[order])))
    return got


class _DeviceArray:
    """A buffer of the state's context, for torch.as_tensor, which keeps this object and with it the state."""

    def __init__(self, ptr, shape, dtype, state):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": dtype, "data": (int(ptr), False), "version": 3}
        self.state = state


def _tensor(ptr, shape, dtype, state):
    if not ptr or not shape[0]:
        return torch.empty(shape, dtype=torch.float32 if dtype == "<f4" else torch.int32, device="cuda")
    return torch.as_tensor(_DeviceArray(ptr, shape, dtype, state), device="cuda")


def _views(m, state):
    """The arrays of a mesh that the library holds for its caller until it is released; they keep the state."""
    nv, nt = m.n_vertices, m.n_triangles

    def view(p, shape, kind):
        if not shape[0]:
            return np.zeros(shape, kind)
        block = (kind * math.prod(shape)).from_address(ctypes.addressof(p.contents))
        block.state = state
        return np.frombuffer(block, kind).reshape(shape)

    return (view(m.vertices, (nv, 3), ctypes.c_float), view(m.triangles, (nt, 3), ctypes.c_int),
            view(m.atom_sorted, (nv,), ctypes.c_int), view(m.atom_input, (nv,), ctypes.c_int))


class _State:
    """A program's context, its molecules and the meshes it holds."""

    def __init__(self, case, seed):
        self.lib, self.meshes = L.lib(), None
        self.case, self.mols = case, _atoms(case, seed)
        call = case["call"]
        if call == "reference_api":
            self.api = q.ReferenceAPI()
        elif call != "field":
            self.ctx = q.Context(0)
        if call in ("device", "field"):
            self.xyz, self.rad = (torch.from_numpy(a).cuda() for a in self.mols[0])
        if call == "field":
            g = q.grid_info(*self.mols[0], case["voxel"]).G
            self.codes = torch.zeros((g, g, g), dtype=torch.uint8, device="cuda")
        if call in ("host", "frames", "batch"):
            n = len(self.mols)
            self.requests, self.meshes, self.status = (L.Request * n)(), (L.Mesh * n)(), (ctypes.c_int * n)()
            for r, (xyz, rad) in zip(self.requests, self.mols):
                r.atoms, r.radii, r.n = xyz.ctypes.data, rad.ctypes.data, xyz.shape[0]
                r.voxel, r.smooth_passes, r.flags = case["voxel"], case["passes"], 0
            self.params = L.Params(case["voxel"], case["passes"], 300, 0)

    def release(self):
        for m in self.meshes or ():
            self.lib.qses_mesh_release(ctypes.byref(m))

    def __del__(self):
        self.release()


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    case, call = state.case, state.case["call"]
    voxel, passes = case["voxel"], case["passes"]
    if call == "compute":
        m = state.ctx.compute(*state.mols[0], voxel=voxel, smooth=passes)
        return m.vertices, m.triangles, m.atom_sorted, m.atom_input
    if call == "slices":
        m = state.ctx.compute(*state.mols[0], voxel=voxel, smooth=passes, slice=case["slice"], reference_slices=True)
        return m.vertices, m.triangles, m.atom_sorted, m.atom_input
    if call == "reference_api":
        nv, nidx = state.api.computeSES(voxel, *state.mols[0], smooth=passes)
        mesh = state.api.getVertices(nv), state.api.getTriangles(nidx).reshape(-1, 3), state.api.getAtomIdPerVert(nv)
        state.api.freeMesh()
        return mesh
    if call == "device":
        d = state.ctx.compute_device(state.xyz.data_ptr(), state.rad.data_ptr(), state.xyz.shape[0], voxel=voxel,
                                     smooth=passes, keep_degenerate=case.get("keep", False))
        nv, nt = d.n_vertices, d.n_triangles
        return (_tensor(d.d_vertices, (nv, 3), "<f4", state), _tensor(d.d_triangles, (nt, 3), "<i4", state),
                _tensor(d.d_atom_sorted, (nv,), "<i4", state), _tensor(d.d_atom_input, (nv,), "<i4", state))
    if call == "field":
        rc = state.lib.qses_field_codes_noalloc(state.xyz.data_ptr(), state.rad.data_ptr(), state.xyz.shape[0], voxel,
                                                state.codes.data_ptr(), state.codes.numel(), torch.cuda.current_stream().cuda_stream)
        if rc:
            raise q.QSESError(rc, L.status_string(rc))
        return state.codes
    # the C interface, as a C or C++ program uses it: the meshes stay in the library's blocks until they are released
    state.release()
    if call == "host":
        r = state.requests[0]
        rc = state.lib.qses_compute(state.ctx.handle, ctypes.byref(state.params), r.atoms,
                                    ctypes.cast(r.radii, ctypes.POINTER(ctypes.c_float)), r.n, ctypes.byref(state.meshes[0]))
    else:
        rc = state.lib.qses_compute_batch(state.ctx.handle, state.requests, len(state.mols), state.meshes, state.status)
        rc = rc or next((s for s in state.status if s), 0)
    if rc:
        raise q.QSESError(rc, L.status_string(rc))
    return [_views(m, state) for m in state.meshes]


def _mesh_size(n, voxel, shape):
    """Vertices of a molecule's mesh, about: a ball has its outer surface and, in proportion, cavities; a shell is all surface."""
    return (34.6 * n if shape == "shell" else 63.9 * n ** (2 / 3) + 1.1 * n) / voxel ** 2


def work(case):
    """Atoms in; vertices, triangles (two to a vertex) and two atom ids out.  Sums and divisions of the smoothing, one
    distance test of each vertex against the atoms around it, and the interpolation of each vertex."""
    n, voxel, shape = case["atoms"], case["voxel"], case.get("shape", "ball")
    if case["call"] == "batch":
        sizes = np.exp(np.linspace(math.log(n), math.log(case["most"]), case["count"])).tolist()
    else:
        sizes = [n] * case.get("count", 1)
    if case["call"] == "field":
        g = (2 * (3 * n / (4 * math.pi * 0.05)) ** (1 / 3) + 9.2) / voxel
        return {"bytes": 16 * n + g ** 3, "flops": 8 * g ** 3}
    nv = sum(_mesh_size(k, voxel, shape) for k in sizes)
    return {"bytes": 16 * float(sum(sizes)) + nv * (12 + 24 + 8), "flops": nv * (39 * case["passes"] + 8 * 30 + 10)}


# ---------------------------------------------------------------- the path in plain numpy

# Triangles of the 256 marching-cubes cases, as the edges of their corners in hex.
_TABLE = """
- 083 019 183981 12a 08312a 92a029 2832a8a98 3b2 0b28b0 19023b 1b219b98b 3a1ba3 0a108a8ba 3903b9ba9 98aa8b 478
430734 019847 419471731 12a847 34730412a 92a902847 2a9297273794 8473b2 b47b24204 90184723b 47b94b9b2921
3a13ba784 1ba14b1047b4 47890b9bab03 47b4b99ba 954 954083 054150 854835315 12a954 30812a495 52a542402
2a5325354348 95423b 0b208b495 05401523b 21525828b485 a3ba13954 4950818a18ba 54050b5bab03 54858aa8b 978579
930953573 078017157 153357 978957a12 a12950530573 802825857a52 2a5253357 7957893b2 95797292027b 23b018178157
b21b17715 958857a13a3b 5705097b010aba0 ba0b03a50807570 ba57b5 a65 0835a6 9015a6 1831985a6 165261 165126308
965906026 598582526328 23ba65 b08b20a65 01923b5a6 5a61929b298b 63b653513 08b0b50515b6 3b6036065059 65969bb98
5a6478 43047365a 1905a6847 a65197173794 612651478 125526304347 847905065026 739794329596269 3b2784a65
5a647242027b 01947823b5a6 9219b294b7b45a6 8473b53515b6 51b5b610b7b404b 059065036b63847 65969b4797b9 a4964a
4a649a083 a01a60640 83181686461a 149124264 308129249264 024426 832824426 a49a64b23 08228b49a4a6 3b201606461a
64161a48121b8b1 964936913b63 8b1810b61914641 3b6360064 648b68 7a678a89a 0730a709a67a a671a7178180 a67a71173
126168189867 269291679093739 780706602 732672 23ba68a89867 20727b09767a9a7 1801781a767a23b b21b17a61671
896867916b63136 091b67 7807063b0b60 7b6 76b 308b76 019b76 819831b76 a126b7 12a3086b7 2902a96b7 6b72a3a83a98
723627 708760620 276237019 162186198876 a76a17137 a7617a187108 03707a0a96a7 76a7a88a9 684b86 36b306046 86b846901
946963931b36 6846b82a1 12a30b06b046 4b846b0292a9 a93a32943b36463 823842462 042462 190234246438 194142246
8138618466a1 a10a06604 4634386a3039a93 a946a4 49576b 083495b76 50154076b b76834354315 954a1276b 6b712a083495
76b54a42a402 348354325a52b76 723762549 954086062687 362376150540 628687218485158 954a16176137 16a176107870954
40a4a503a6a737a 76a7a854a48a 6956b9b89 36b063056095 0b805b01556b 6b3635531 12a95b9b8b56 0b306b09656912a
b85b56805a52025 6b36352a3a53 589528562382 956960062 158180568382628 156216 13616a386569896 a10a06950560 03856a
a56 b5a75b b5ab75830 5b75ab190 a75ab7981831 b12b71751 08312717572b 9759279022b7 75272b592328982 25a235375
820852875a25 9015a35373a2 982921872a25752 135375 087071175 903935537 987597 5845a8ab8 5045b05abb30 01984a8aba45
ab4a45b34941314 2512852b8458 04b0b345b2b151b 0250592b5458b85 9452b3 25a352345384 5a2524420 3a235a385458019
5a2524192942 845853351 045105 845853905035 945 4b749b9ab 0834979b79ab 1ab1b414074b 3143481a474bab4 4b79b492b912
9749b791b2b1083 b74b42240 b74b42834324 29a279237749 9a7974a27870207 37a3a274a1a040a 1a2874 491417713
491417081871 403743 487 9a8ab8 30939bb9a 01a0a88ab 31ab3a 12b1b99b8 30939b1292b9 02b80b 32b 23828aa89 9a2092
23828a0181a8 1a2 138918 091 038 -
"""
# Edge -> (di, dj, dk, axis) of the voxel it starts at, and its axis.
_EDGES = [(0, 0, 0, 0), (1, 0, 0, 1), (0, 1, 0, 0), (0, 0, 0, 1), (0, 0, 1, 0), (1, 0, 1, 1), (0, 1, 1, 0), (0, 0, 1, 1),
          (0, 0, 0, 2), (1, 0, 0, 2), (1, 1, 0, 2), (0, 1, 0, 2)]


def _fma(a, b, c):
    """a * b + c of 32-bit values with one rounding (the product is exact in 64 bits)."""
    return (np.asarray(a, np.float64) * np.asarray(b, np.float64) + np.asarray(c, np.float64)).astype(np.float32)


def _shifted_min(d, axis, reach):
    best = d.copy()
    for s in range(1, reach + 1):
        lo, hi = [slice(None)] * 3, [slice(None)] * 3
        lo[axis], hi[axis] = slice(None, -s), slice(s, None)
        np.minimum(best[tuple(lo)], d[tuple(hi)] + s * s, out=best[tuple(lo)])
        np.minimum(best[tuple(hi)], d[tuple(lo)] + s * s, out=best[tuple(hi)])
    return best


def _unsmoothed(xyz, rad, voxel):
    """Welded vertices as whole multiples of 0.001 A, in their order, and all triangles.  Which corners are inside and which
    multiple a vertex goes to are decided in 32 bits, as the mesh format has it: another type would number the vertices
    differently where one lies on a tie."""
    f = np.float32
    dx, probe, max_r = f(voxel), f(1.4), rad.max()
    low, high = xyz.min(0), xyz.max(0)
    reach = f(f((high - low).max() + f(2) * max_r) + f(4) * probe)
    origin = (low - max_r - probe).astype(f)
    G, R = int(np.ceil(reach / dx)), int(np.ceil(probe / dx))
    cells = max(0, G - 2 * R - 1)
    at = [_fma(np.arange(G + 1), dx, origin[c]) for c in range(3)]
    out, inner = np.ones((G, G, G), bool), np.zeros((G, G, G), bool)
    for p, r in zip(xyz, rad):
        near, core = f(f(probe + r) ** 2), f(f(r - dx) ** 2) if r > dx else f(-1)
        box = []
        for c in range(3):
            i = [int((p[c] + s * (probe + r) - origin[c]) / dx) for s in (-1, 1)]
            box.append(slice(max(0, i[0] - 1), min(G - 1, i[1] + 3)))
        ex, ey, ez = (at[c][box[c]] - p[c] for c in range(3))
        xy = _fma(ey[None, :], ey[None, :], (ex * ex)[:, None])
        d2 = _fma(ez[None, None, :], ez[None, None, :], xy[:, :, None])
        out[tuple(box)] &= ~(d2 < near)
        inner[tuple(box)] |= d2 < core
    d = np.where(out, 0, 9999).astype(np.int32)
    for axis in (2, 1, 0):
        d = _shifted_min(d, axis, R)
    far = d > 3 * R * R
    value = (float(probe) - float(dx) * np.sqrt(np.where(far, 0, d))).astype(f)
    value[far | inner] = -dx
    value[out] = probe
    neg = value < 0
    key, slot, base = [], [], 0
    E = cells + 1
    for axis in range(3):
        ext = [cells if c == axis else E for c in range(3)]
        here = tuple(slice(0, e) for e in ext)
        there = tuple(slice(1, e + 1) if c == axis else slice(0, e) for c, e in enumerate(ext))
        idx = np.argwhere(neg[here] != neg[there])
        a, b = value[here][tuple(idx.T)], value[there][tuple(idx.T)]
        t = -a / (b - a)
        p = np.stack([at[c][idx[:, c]] for c in range(3)], 1)
        p[:, axis] = _fma(t, at[axis][idx[:, axis] + 1] - p[:, axis], p[:, axis])
        m = (p / f(0.001)).astype(np.float64)
        key.append(np.trunc(m + np.copysign(0.5, m)).astype(np.int64))
        of = np.full((E + 1, E + 1, E + 1), -1, np.int64)
        of[tuple(idx.T)] = base + np.arange(len(idx))
        base += len(idx)
        slot.append(of)
    quantum, rank = np.unique(np.concatenate(key), axis=0, return_inverse=True)
    rank = rank.reshape(-1)
    c = neg[:cells + 1, :cells + 1, :cells + 1]
    cube = np.zeros((cells, cells, cells), np.int32)
    for bit, (i, j, k) in enumerate([(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]):
        cube |= c[i:i + cells, j:j + cells, k:k + cells].astype(np.int32) << bit
    table = [[] if t == "-" else [int(x, 16) for x in t] for t in _TABLE.split()]
    tri, order = [], []
    for case in range(1, 255):
        where = np.argwhere(cube == case)
        if not len(where) or not table[case]:
            continue
        corner = np.empty((len(where), len(table[case])), np.int64)
        for k, e in enumerate(table[case]):
            di, dj, dk, axis = _EDGES[e]
            corner[:, k] = slot[axis][where[:, 0] + di, where[:, 1] + dj, where[:, 2] + dk]
        n = len(table[case]) // 3
        tri.append(rank[corner].reshape(-1, 3))
        cell = (where[:, 0] * cells + where[:, 1]) * cells + where[:, 2]
        order.append((cell[:, None] * 8 + np.arange(n)).reshape(-1))
    if not tri:
        return quantum, np.zeros((0, 3), np.int64)
    return quantum, np.concatenate(tri)[np.argsort(np.concatenate(order), kind="stable")]


def _smoothed(vertices, triangles, passes):
    """Each vertex in turn goes to the mean of its triangles' other corners, which may have moved already."""
    near = [[] for _ in range(len(vertices))]
    for a, b, c in triangles.tolist():
        near[a] += (b, c)
        near[b] += (a, c)
        near[c] += (a, b)
    x, y, z = (vertices[:, k].tolist() for k in range(3))
    for _ in range(passes):
        for v, of in enumerate(near):
            n = len(of)
            x[v], y[v], z[v] = sum([x[u] for u in of]) / n, sum([y[u] for u in of]) / n, sum([z[u] for u in of]) / n
    return np.array([x, y, z]).T


def exact(case, seed):
    """The vertices; triangles and atom ids are whole numbers.  Meshes that numpy takes longer than some seconds for have no value here."""
    if case["call"] not in ("compute", "reference_api", "device", "host"):
        return None
    xyz, rad = _atoms(case, seed)[0]
    voxels = (float(np.ptp(xyz, axis=0).max()) + 9.2) ** 3 / case["voxel"] ** 3
    if voxels > 6e6 or _mesh_size(case["atoms"], case["voxel"], case.get("shape")) * (1 + case["passes"]) > 4e5:
        return None
    quantum, tri = _unsmoothed(xyz, rad, case["voxel"])
    v = _smoothed(quantum * 0.001, tri, case["passes"])
    if case["call"] == "host":
        return [(v, None, None, None)]
    return (v, None, None) if case["call"] == "reference_api" else (v, None, None, None)
