// Neighbour-cell key per atom (hashAtoms + spaceToGrid + flatten3DTo1D, Kernels.cu:119-131,
// 185-216).
//
// This translation unit is compiled with -use_fast_math, like the reference, and spells the
// cell coordinate as the same expression (p - o) / cell truncated to int, so the compiler
// emits the same approximate division.  That matters: the grid origin is min - maxR - probe,
// which puts the atom with the smallest coordinate of each axis exactly on a cell boundary,
// where the approximate quotient (just below the integer) and the IEEE one (exactly the
// integer) pick different cells.  The cell key only orders the atoms (the sorted order
// behind API_getAtomIdPerVert); which atoms the field sees does not depend on it.
#include "kernels.h"

namespace qses {

// Cells beyond the grid's, which the bounds rule out for atoms that are somewhere, are clamped: the
// cell table has no others.
__device__ __forceinline__ unsigned atom_key(const QGrid &g, const float *__restrict__ xyz, unsigned a) {
    auto cell = [&](float p, float o) { return min(max((int)((p - o) / g.cell), 0), g.gnb - 1); };
    const int cx = cell(xyz[3 * a], g.ox), cy = cell(xyz[3 * a + 1], g.oy), cz = cell(xyz[3 * a + 2], g.oz);
    return (unsigned)(g.gnb * g.gnb * cx + g.gnb * cy + cz);
}
__global__ void k_atom_hash(QGrid g, const float *__restrict__ xyz, unsigned n, unsigned *__restrict__ key) {
    unsigned a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a < n) key[a] = atom_key(g, xyz, a);
}

// Few atoms, in one launch: every block has all keys, with the atoms' numbers below them, in shared
// memory, and a group of 8 lanes counts the ones before its atom - the atom's place in the stable
// order of the keys - and the ones in the cells before.  cells: zeroed.  Key, histogram, digit passes
// and gather are 5 or 6 launches with a wait for each: 200 atoms 48 us, 28 so; 1 000 52 and 31; 5 000
// still 10 us more.
__global__ void __launch_bounds__(256) k_atoms_few(QGrid g, const float *__restrict__ xyz, const float *__restrict__ r,
                                                   unsigned n, unsigned *__restrict__ skey, unsigned *__restrict__ sidx,
                                                   float4 *__restrict__ atoms, uint2 *__restrict__ cells) {
    __shared__ uint4 s_key[kFewAtoms / 4];
    const unsigned n32 = (n + 31) / 32 * 32;
    for (unsigned a = threadIdx.x; a < n32; a += 256)
        ((unsigned *)s_key)[a] = a < n ? atom_key(g, xyz, a) * kFewAtoms + a : 0xffffffffu;
    __syncthreads();
    const unsigned a = blockIdx.x * 32 + (threadIdx.x >> 3), sub = threadIdx.x & 7;
    const unsigned me = ((const unsigned *)s_key)[min(a, n - 1)], cell = me / kFewAtoms, cell0 = cell * kFewAtoms;
    unsigned before = 0, lower = 0;
    for (unsigned q = sub; q < n32 / 4; q += 8) {
        const uint4 k = s_key[q];
        before += (k.x < me) + (k.y < me) + (k.z < me) + (k.w < me);
        lower += (k.x < cell0) + (k.y < cell0) + (k.z < cell0) + (k.w < cell0);
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        before += __shfl_xor_sync(0xffffffffu, before, o);
        lower += __shfl_xor_sync(0xffffffffu, lower, o);
    }
    if (sub != 0 || a >= n) return;
    skey[before] = cell;
    sidx[before] = a;
    atoms[before] = make_float4(xyz[3 * a], xyz[3 * a + 1], xyz[3 * a + 2], r[a]);
    if (before == lower) cells[cell].x = before;
    atomicMax(&cells[cell].y, before + 1);
}

// Batch form: the key of an atom of molecule m is offset by m's first cell, so one stable
// sort orders every molecule's atoms exactly as its own sort would, molecule after molecule.
__global__ void k_atom_hash_batch(QBatch b, const float *__restrict__ xyz, unsigned n, unsigned *__restrict__ key) {
    unsigned a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n) return;
    const unsigned m = qses_find(b.atom_off, b.n_mol, a);
    key[a] = b.mols[m].cell_off + atom_key(b.mols[m].g, xyz, a);
}

void launch_atom_hash(const QGrid &g, const float *xyz, unsigned n, unsigned *key, cudaStream_t s) {
    k_atom_hash<<<(n + 255) / 256, 256, 0, s>>>(g, xyz, n, key);
}
void launch_atoms_few(const QGrid &g, const float *xyz, const float *r, unsigned n, unsigned *skey, unsigned *sidx,
                      float4 *atoms, uint2 *cells, cudaStream_t s) {
    k_atoms_few<<<(n + 31) / 32, 256, 0, s>>>(g, xyz, r, n, skey, sidx, atoms, cells);
}
void launch_atom_hash_batch(const QBatch &b, const float *xyz, unsigned n, unsigned *key, cudaStream_t s) {
    k_atom_hash_batch<<<(n + 255) / 256, 256, 0, s>>>(b, xyz, n, key);
}

}  // namespace qses
