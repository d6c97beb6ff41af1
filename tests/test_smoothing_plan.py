"""The slab plan that a smoothing pass gets (CPU, through qses_debug_smoothing_plan).

The kernel's CTAs take slabs from a counter in the plan's order; a slab waits for lower slabs of its
own molecule, so every wait ends if those come earlier in the order.  A slab's state has to fit a
CTA's shared memory (11 904 vertices), a molecule may have more slabs than there are CTAs, and the
table has to hold them all.
"""
import ctypes

import numpy as np
import pytest

from quickses_gb300 import _lib as L

CAP = 11904


def _plan(nv, mol_off=None, depth=None, target=4096, wave=0, pmax=152):
    lib = L.lib()
    launch = (ctypes.c_uint * 6)()
    nm = 1 if mol_off is None else len(mol_off) - 1
    mo = None if mol_off is None else np.ascontiguousarray(mol_off, np.uint32)
    dp = None if depth is None else np.ascontiguousarray(depth, np.int32)
    args = [nv, None if mo is None else mo.ctypes.data, None if dp is None else dp.ctypes.data, nm, 512, target, wave, pmax,
            launch]
    assert lib.qses_debug_smoothing_plan(*args, None, 0) == L.QSES_OK
    ctas, smax, qcap, wsize, waves, words = list(launch)
    assert words == 2 * qcap + 2 and ctas == min(pmax, qcap)
    table = np.zeros(waves * words, np.uint32)
    assert lib.qses_debug_smoothing_plan(*args, table.ctypes.data, table.size) == L.QSES_OK
    out = []
    for t in table.reshape(waves, words).astype(np.int64):
        Q = int(t[0])
        assert 1 <= Q <= qcap
        out.append((t[1:Q + 2], t[qcap + 2:qcap + 2 + Q]))
    return smax, out


def _check(nv, mol_off, target, smax, waves):
    assert smax <= min(max(target, 256), CAP)
    at = 0
    for bnd, order in waves:
        assert bnd[0] == at and (np.diff(bnd) > 0).all() and np.diff(bnd).max() <= smax
        assert np.array_equal(np.sort(order), np.arange(len(order)))
        place = np.argsort(order)
        first = np.maximum(mol_off[np.searchsorted(mol_off, bnd[:-1], side="right") - 1], at)
        for q in np.nonzero(bnd[:-1] > first)[0]:  # not the first of its molecule: behind the slab before it
            assert place[q - 1] < place[q]
        last = np.searchsorted(mol_off, bnd[1:] - 1, side="right") - 1
        several = first < np.maximum(mol_off[last], at)  # more than one molecule in the slab: whole ones
        assert (bnd[:-1][several] == first[several]).all()
        assert (bnd[1:][several] == np.minimum(mol_off[last + 1], bnd[-1])[several]).all()
        at = bnd[-1]
    assert at == nv


@pytest.mark.parametrize("nv", [1, 255, 256, 257, 29_938, CAP, CAP + 1, 2 * CAP, 2 * CAP + 1, 3_540_690, 138_371_232])
@pytest.mark.parametrize("target", [1, 256, 4096, 11_903, CAP, CAP + 1, 25_000])
def test_one_molecule(nv, target):
    smax, waves = _plan(nv, target=target)
    _check(nv, np.array([0, nv]), target, smax, waves)
    (bnd, order), = waves
    t = min(max(target, 256), CAP)
    # as many slabs as the target asks for, however many CTAs there are, of one size and in order
    S = -(-nv // -(-nv // t))
    assert np.array_equal(bnd[:-1], np.arange(0, nv, S)) and np.array_equal(order, np.arange(len(order)))


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("target", [256, 1000, 5376, CAP, 25_000])
def test_batches(seed, target):
    rng = np.random.default_rng(seed)
    nm = int(rng.integers(2, 250))
    sizes = np.exp(rng.uniform(0.0, np.log(400_000), nm)).astype(np.int64)
    sizes[rng.random(nm) < 0.05] = 0
    sizes[0] = max(sizes[0], 1)
    mol_off = np.concatenate([[0], np.cumsum(sizes)])
    nv = int(mol_off[-1])
    depth = rng.integers(1, 700, nm)
    for wave in (0, max(target, nv // 5), max(target, nv // 2 + 1)):
        smax, waves = _plan(nv, mol_off, depth, target=target, wave=wave, pmax=int(rng.integers(1, 600)))
        _check(nv, mol_off, target, smax, waves)


def test_invalid():
    launch = (ctypes.c_uint * 6)()
    lib = L.lib()
    assert lib.qses_debug_smoothing_plan(0, None, None, 1, 512, 4096, 0, 152, launch, None, 0) == L.QSES_ERR_INVALID_ARG
    assert lib.qses_debug_smoothing_plan(10, None, None, 1, 512, 4096, 0, 0, launch, None, 0) == L.QSES_ERR_INVALID_ARG
    assert lib.qses_debug_smoothing_plan(10, None, None, 2, 512, 4096, 0, 152, launch, None, 0) == L.QSES_ERR_INVALID_ARG
    one = np.zeros(1, np.uint32)
    assert lib.qses_debug_smoothing_plan(10, None, None, 1, 512, 4096, 0, 152, launch, one.ctypes.data, 1) == L.QSES_ERR_INVALID_ARG
