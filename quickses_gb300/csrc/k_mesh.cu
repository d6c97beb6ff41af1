// Marching cubes, vertex weld, closest atom, degenerate filter and the neighbour lists' corners.
//
//  k_mc_count     per (x, y) row of cells: triangle count and active-edge count
//                 (countVertexPerCell, MarchingCubes.cu:571-658, single-slice cell range),
//                 and for each word of a row what the words before it have
//  k_mc_emit      triangles in cell linear order x*G^2 + y*G + z and one quantised key per
//                 active edge (generateTriangleVerticesSMEM + groupVertices,
//                 MarchingCubes.cu:736-862).  The sign of 32 voxels is one word, so cube
//                 indices and edge activity are bit ops.
//  k_weld         unique quantised positions in lexicographic order (CudaSurf.cu:444-457), plane by
//                 plane; k_weld_number and the radix sort for meshes that crowd a plane
//  k_closest      closest atom per welded vertex (closestAtomPerVertex, Kernels.cu:547-604)
//  k_tri_filter   drop triangles with a repeated index (CudaSurf.cu:820-829)
//  k_csr_*        neighbour lists in triangle order (getNeighboorsVertices,
//                 SmoothMesh.cpp:45-123) for the Gauss-Seidel dataflow (k_smooth.cu)
#include <algorithm>
#include <cfloat>
#include <cstdlib>
#include <cstring>

#include "device_common.cuh"

#include "kernels.h"
#include "mc_tables.h"
#include "prims.h"

namespace qses {

__constant__ unsigned long long c_mc[256] = QSES_MC_TABLE_INIT;

__device__ __forceinline__ unsigned ld_sign(const unsigned *__restrict__ sign, const QGrid &g, int i, int j, int w) {
    if (i >= g.G || j >= g.G || w >= g.W) return 0u;
    return __ldg(&sign[((size_t)i * g.G + j) * g.W + w]);
}

// The sign words of row (i + a, j + b), zero past the grid.
struct SignRow {
    const unsigned *p;
    unsigned there;  // all ones if the row exists
    __device__ __forceinline__ SignRow(const unsigned *__restrict__ row, const QGrid &g, int i, int j, int a, int b) {
        const bool ok = i + a < g.G && j + b < g.G;
        p = row + (ok ? (size_t)(a * g.G + b) * g.W : (size_t)0);
        there = ok ? 0xffffffffu : 0u;
    }
    // word w < W, and bit 0 of the next one
    __device__ __forceinline__ unsigned word(int w) const { return __ldg(p + w) & there; }
    __device__ __forceinline__ unsigned next(int w, int W) const { return w + 1 < W ? __ldg(p + w + 1) & there : 0u; }
};

__device__ __forceinline__ unsigned cube_index(unsigned b, unsigned c0, unsigned c1, unsigned c2, unsigned c3,
                                               unsigned c4, unsigned c5, unsigned c6, unsigned c7) {
    return ((c0 >> b) & 1u) | (((c1 >> b) & 1u) << 1) | (((c2 >> b) & 1u) << 2) | (((c3 >> b) & 1u) << 3) |
           (((c4 >> b) & 1u) << 4) | (((c5 >> b) & 1u) << 5) | (((c6 >> b) & 1u) << 6) | (((c7 >> b) & 1u) << 7);
}

__device__ __forceinline__ unsigned warp_sum(unsigned v) { return __reduce_add_sync(0xffffffffu, v); }

// round(p / 0.001) (groupVertices, MarchingCubes.cu:859).  Division by a constant with one
// multiplication and one correction (Markstein, IBM J. Res. Dev. 34, 1990): the rounded quotient is
// that of p / 0.001f for every |p| up to 16384, the coordinates a grid may have (all floats tried).
__device__ __forceinline__ int quantum(float p) {
    constexpr float r = 1.0f / QSES_WELD_TOL;
    const float q = __fmul_rn(p, r);
    return (int)roundf(__fmaf_rn(__fmaf_rn(-q, QSES_WELD_TOL, p), r, q));
}
// Quantised key of the vertex on edge (i, j, k) -> (i, j, k) + e_axis.
__device__ __forceinline__ unsigned long long edge_key(const QGrid &g, const unsigned char *__restrict__ codes,
                                                       const float *__restrict__ lut, int i, int j, int k, int ax) {
    const size_t base = ((size_t)i * g.G + j) * g.Gp + k;
    const size_t step = ax == 0 ? (size_t)g.G * g.Gp : (ax == 1 ? (size_t)g.Gp : (size_t)1);
    const float fa = __ldg(lut + __ldg(codes + base)), fb = __ldg(lut + __ldg(codes + base + step));
    const float t = __fdiv_rn(-fa, __fsub_rn(fb, fa));  // vertexInterp (MarchingCubes.cu:731-734)
    float p[3] = {vox(i, g.dx, g.ox), vox(j, g.dx, g.oy), vox(k, g.dx, g.oz)};
    const float from = ax == 0 ? p[0] : (ax == 1 ? p[1] : p[2]);
    const float to = vox((ax == 0 ? i : (ax == 1 ? j : k)) + 1, g.dx, ax == 0 ? g.ox : (ax == 1 ? g.oy : g.oz));
    const float at = __fmaf_rn(t, __fsub_rn(to, from), from);
#pragma unroll
    for (int c = 0; c < 3; c++)
        if (c == ax) p[c] = at;
    if (g.off[0] | g.off[1] | g.off[2]) {  // a slice box: + offset * dx (MarchingCubes.cu:841-848)
#pragma unroll
        for (int c = 0; c < 3; c++) p[c] = __fadd_rn(p[c], __fmul_rn((float)g.off[c], g.dx));
    }
    const unsigned x = (unsigned)(quantum(p[0]) - (int)g.bx), y = (unsigned)(quantum(p[1]) - (int)g.by),
                   z = (unsigned)(quantum(p[2]) - (int)g.bz);
    return ((unsigned long long)x << 42) | ((unsigned long long)y << 21) | z;
}

// Lanes per owner row: the row's words (voxels 0..Gc) rounded up to a power of two, at
// most 32, so a warp covers 32 / lanes rows of a small grid at once.
__host__ __device__ __forceinline__ int mc_lanes(int Gc) {
    const int Wc = (Gc + 32) / 32;
    int L = 1;
    while (L < Wc && L < 32) L <<= 1;
    return L;
}

// Inclusive scan over aligned groups of Lg lanes (Lg a power of two, warp-uniform).
__device__ __forceinline__ unsigned grp_incl_scan(unsigned v, int sub, int Lg) {
    for (int o = 1; o < Lg; o <<= 1) {
        const unsigned a = __shfl_up_sync(0xffffffffu, v, o, Lg);
        if (sub >= o) v += a;
    }
    return v;
}

// Bits [a, b) of a 32-bit word, the bounds clamped to [0, 32].
__device__ __forceinline__ unsigned bits_in(int a, int b) {
    a = max(a, 0);
    b = min(b, 32);
    if (a >= b) return 0u;
    const unsigned below_b = b == 32 ? 0xffffffffu : ((1u << b) - 1u);
    return below_b & ~((1u << a) - 1u);
}

// Which edges and cells of row (i, j) and word w are in the emitted range [clo, chi) per axis (the
// whole grid: [0, Gc)).  A row's +x edges are used when a cell of the range has them (x in
// [clo, chi), y in [clo, chi]), likewise +y; its +z edges when x and y are in [clo, chi].
struct McRange {
    int lox, hix, loy, hiy, loz, hiz;
    __device__ __forceinline__ explicit McRange(const QGrid &g)
        : lox(g.clo[0]), hix(g.chi[0]), loy(g.clo[1]), hiy(g.chi[1]), loz(g.clo[2]), hiz(g.chi[2]) {}
    __device__ __forceinline__ bool xr(int a, int b) const { return a >= lox && a < hix && b >= loy && b <= hiy; }
    __device__ __forceinline__ bool yr(int a, int b) const { return a >= lox && a <= hix && b >= loy && b < hiy; }
    __device__ __forceinline__ bool zr(int a, int b) const { return a >= lox && a <= hix && b >= loy && b <= hiy; }
    __device__ __forceinline__ bool cells(int a, int b) const { return a >= lox && a < hix && b >= loy && b < hiy; }
    __device__ __forceinline__ unsigned kv(int kb) const { return bits_in(loz - kb, hiz - kb + 1); }  // voxels in [loz, hiz]
    __device__ __forceinline__ unsigned kc(int kb) const { return bits_in(loz - kb, hiz - kb); }  // cells, z edges in [loz, hiz)
};

// One owner row (i, j) of a molecule's grid per group of Lg lanes; every lane of the warp
// calls this (groups whose row is past the end pass valid = false and write nothing).  Bound by
// instruction issue: 664^3 0.112 ms, 0.101 with the rows' addresses worked out once and words
// without a change of sign passed over; 1738^3 1.44 and 1.27.
// words[row * Wc + w]: what the row's words before w have, edges in bits 0-15 (3 a voxel at most)
// and triangles in bits 16-30 (5 a cell), and bit 31 if word w has any itself.
template <bool FULL>
__device__ __forceinline__ void mc_count_row(const QGrid &g, long long row, bool valid, int Lg,
                                             const unsigned *__restrict__ sign, const unsigned long long *s_tab,
                                             uint2 *__restrict__ rowCount, unsigned *__restrict__ words) {
    // FULL: one row per warp (Lg = 32, every group valid), known at compile time.
    if (FULL) {
        Lg = 32;
        valid = true;
    }
    const int sub = (int)(threadIdx.x & 31) & (Lg - 1);
    const int Gc = g.Gc, E = Gc + 1;
    if (!valid) row = 0;
    const int i = (int)(row / E), j = (int)(row % E);
    const McRange in(g);
    const int Wc = (Gc + 32) / 32;  // words holding voxels 0..Gc
    const unsigned *own = sign + ((size_t)i * g.G + j) * g.W;
    const SignRow r00(own, g, i, j, 0, 0), r10(own, g, i, j, 1, 0), r01(own, g, i, j, 0, 1), r11(own, g, i, j, 1, 1);
    unsigned carry = 0;
    for (int w0 = 0; w0 < Wc; w0 += Lg) {
        const int w = w0 + sub;
        const bool act = valid && w < Wc;
        const int kb = w * 32;
        const unsigned kv = act ? in.kv(kb) : 0u, kc = act ? in.kc(kb) : 0u;
        unsigned n = 0;
        unsigned S00 = 0, S10 = 0, S01 = 0, S11 = 0, P00 = 0, P10 = 0, P01 = 0, P11 = 0;
        if (act) {
            S00 = r00.word(w), S10 = r10.word(w), S01 = r01.word(w), S11 = r11.word(w);
            P00 = (S00 >> 1) | (r00.next(w, g.W) << 31), P10 = (S10 >> 1) | (r10.next(w, g.W) << 31);
            P01 = (S01 >> 1) | (r01.next(w, g.W) << 31), P11 = (S11 >> 1) | (r11.next(w, g.W) << 31);
        }
        const unsigned mixed = (S00 ^ S10) | (S00 ^ S11) | (S00 ^ S01) | (S00 ^ P00) | (S00 ^ P10) | (S00 ^ P11) | (S00 ^ P01);
        if (__any_sync(0xffffffffu, mixed)) {  // else none of the warp's words has an edge
            const unsigned X00 = in.xr(i, j) ? (S00 ^ S10) & kv : 0u;
            const unsigned Y00 = in.yr(i, j) ? (S00 ^ S01) & kv : 0u;
            const unsigned Z00 = in.zr(i, j) ? (S00 ^ P00) & kc : 0u;
            n = __popc(X00) + __popc(Y00) + __popc(Z00);
            if (in.cells(i, j))
                for (unsigned m = mixed & kc; m; m &= m - 1u) {
                    const unsigned b = __ffs(m) - 1;
                    n += (unsigned)(s_tab[cube_index(b, S00, S10, S11, S01, P00, P10, P11, P01)] >> 60) << 16;
                }
        }
        const unsigned incl = grp_incl_scan(n, sub, Lg);
        if (act) words[(size_t)row * Wc + w] = (carry + incl - n) | (n ? 0x80000000u : 0u);
        carry += __shfl_sync(0xffffffffu, incl, Lg - 1, Lg);
    }
    if (valid && sub == 0) rowCount[row] = make_uint2(carry >> 16, carry & 0xffffu);
}

__global__ void __launch_bounds__(256, 4) k_mc_count(QGrid g, const unsigned *__restrict__ sign,
                                                     uint2 *__restrict__ rowCount, unsigned *__restrict__ words, int lanes) {
    __shared__ unsigned long long s_tab[256];
    s_tab[threadIdx.x] = c_mc[threadIdx.x];
    __syncthreads();
    const int E = g.Gc + 1, Lg = lanes;
    const long long first = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * (32 / Lg), nrow = (long long)E * E;
    if (first >= nrow) return;  // the whole warp
    const long long row = first + (threadIdx.x & 31) / Lg;
    mc_count_row<false>(g, row, row < nrow, Lg, sign, s_tab, rowCount, words);
}

// Batch form: rows are numbered molecule after molecule, so one scan over all rows gives
// every molecule's triangles and edge slots contiguous ranges in molecule order.  Each warp
// takes one unit of 32 / Lg rows of one molecule (units numbered by mc_unit_off).
__global__ void __launch_bounds__(256, 4) k_mc_count_batch(QBatch b, const unsigned *__restrict__ sign,
                                                           uint2 *__restrict__ rowCount, unsigned *__restrict__ words) {
    __shared__ unsigned long long s_tab[256];
    s_tab[threadIdx.x] = c_mc[threadIdx.x];
    __syncthreads();
    const unsigned unit = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= __ldg(b.mc_unit_off + b.n_mol)) return;  // the whole warp
    const unsigned m = qses_find(b.mc_unit_off, b.n_mol, unit);
    const QMol &mol = b.mols[m];
    const QGrid g = mol.g;
    const int Lg = mc_lanes(g.Gc);
    const unsigned r0 = mol.row_off, nrow = (unsigned)(g.Gc + 1) * (unsigned)(g.Gc + 1);
    const unsigned row = (unit - __ldg(b.mc_unit_off + m)) * (32u / Lg) + (threadIdx.x & 31) / Lg;
    if (Lg == 32)  // warp-uniform
        mc_count_row<true>(g, (long long)row, true, 32, sign + mol.mask_off, s_tab, rowCount + r0, words + mol.mask_off);
    else
        mc_count_row<false>(g, (long long)row, row < nrow, Lg, sign + mol.mask_off, s_tab, rowCount + r0,
                            words + mol.mask_off);
}

// The emission.  A warp takes `chunk` consecutive words of the grid, collects the ones that have
// edges or triangles and works on 32 of them at a time: a lane per word for its masks and slots,
// then a lane per edge and a lane per cell of all of them together, whichever rows they are in.
// What consecutive words emit is contiguous, so keys and corners go out in whole lines, the corners
// by way of shared memory.
//
// Bound by instruction issue: 664^3 (4 160 000 edges, 8 310 000 triangles) takes 126 M warp
// instructions at 1.9 a cycle, 16 warps an SM.  Rows dealt to 4 or 32 lanes, each corner's slot from
// the words' masks and stored by itself: 0.74 ms there (568 M instructions), 0.24 so; 1738^3
// (138 000 000 edges) 13.0 and 4.6; 85^3 0.025 and 0.020.  Blocks of 8 warps wait for their slowest
// (0.26, 4.9); of 1 or 2 they load the table more often than that gains.
constexpr int kEmitRec = 9;    // uint4 a lane's record takes (8 used; odd, for the banks)
constexpr int kEmitQueue = 160;  // words waiting: 31 and 4 x 32 more
constexpr int kEmitWarps = 4;
struct EmitSmem {
    uint4 rec[32 * kEmitRec];
    unsigned slot[12 * 32];  // a cell's 12 edges, per lane
    unsigned out[32 * 15];   // corners of up to 32 cells
    unsigned short queue[kEmitQueue];
};

// The edge or cell of rank r: the largest b with at most r below it.
template <typename F> __device__ __forceinline__ unsigned bit_of_rank(F below, unsigned r) {
    unsigned b = 0;
#pragma unroll
    for (unsigned step = 16; step > 0; step >>= 1)
        if (below((1u << (b + step)) - 1u) <= r) b += step;
    return b;
}
// The lane whose items include item e: the largest with first <= e.
__device__ __forceinline__ unsigned lane_of_item(unsigned first, unsigned e) {
    unsigned lo = 0;
#pragma unroll
    for (unsigned step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, first, lo + step) <= e) lo += step;
    return lo;
}

// Up to 32 words (has: this lane's is one), in ascending order by lane: `at` words from row row0's start.
__device__ __forceinline__ void emit_words(const QGrid &g, const unsigned *__restrict__ sign,
                                           const unsigned char *__restrict__ codes, const float *__restrict__ lut,
                                           const unsigned *__restrict__ words, const uint2 *__restrict__ rowBase,
                                           unsigned *__restrict__ tri, unsigned long long *__restrict__ vkey,
                                           const unsigned long long *s_tab, EmitSmem &sm, bool has, unsigned row0, unsigned at) {
    const unsigned lane = threadIdx.x & 31;
    const int E = g.Gc + 1, Wc = (g.Gc + 32) / 32;
    unsigned nedge = 0, ncell = 0;
    if (has) {
        const unsigned row = row0 + at / (unsigned)Wc;
        const int w = (int)(at % (unsigned)Wc), i = (int)(row / (unsigned)E), j = (int)(row % (unsigned)E);
        const McRange in(g);
        const unsigned kv = in.kv(32 * w), kc = in.kc(32 * w);
        auto L = [&](int a, int b, int ww) { return ld_sign(sign, g, i + a, j + b, ww); };
        const unsigned S00 = L(0, 0, w), S10 = L(1, 0, w), S01 = L(0, 1, w), S11 = L(1, 1, w);
        const unsigned N00 = L(0, 0, w + 1), N10 = L(1, 0, w + 1), N01 = L(0, 1, w + 1), N11 = L(1, 1, w + 1);
        const unsigned S20 = L(2, 0, w), S21 = L(2, 1, w), S02 = L(0, 2, w), S12 = L(1, 2, w), N20 = L(2, 0, w + 1);
        const unsigned P00 = (S00 >> 1) | (N00 << 31), P10 = (S10 >> 1) | (N10 << 31);
        const unsigned P01 = (S01 >> 1) | (N01 << 31), P11 = (S11 >> 1) | (N11 << 31);
        // edges owned by the row and by the rows (i, j + 1), (i + 1, j) and (i + 1, j + 1)
        const unsigned X00 = in.xr(i, j) ? (S00 ^ S10) & kv : 0u, Y00 = in.yr(i, j) ? (S00 ^ S01) & kv : 0u;
        const unsigned Z00 = in.zr(i, j) ? (S00 ^ P00) & kc : 0u;
        const unsigned X01 = in.xr(i, j + 1) ? (S01 ^ S11) & kv : 0u, Y01 = in.yr(i, j + 1) ? (S01 ^ S02) & kv : 0u;
        const unsigned Z01 = in.zr(i, j + 1) ? (S01 ^ P01) & kc : 0u;
        const unsigned X10 = in.xr(i + 1, j) ? (S10 ^ S20) & kv : 0u, Y10 = in.yr(i + 1, j) ? (S10 ^ S11) & kv : 0u;
        const unsigned Z10 = in.zr(i + 1, j) ? (S10 ^ P10) & kc : 0u;
        const unsigned X11 = in.xr(i + 1, j + 1) ? (S11 ^ S21) & kv : 0u, Y11 = in.yr(i + 1, j + 1) ? (S11 ^ S12) & kv : 0u;
        const unsigned Z11 = in.zr(i + 1, j + 1) ? (S11 ^ P11) & kc : 0u;
        // the +x edge of voxel 32 w + 32 of row (i + 1, j)
        const unsigned xn = in.xr(i + 1, j) && 32 * w + 32 <= in.hiz && 32 * w + 32 >= in.loz ? (N10 ^ N20) & 1u : 0u;
        const bool nj = j + 1 < E, ni = i + 1 < E;
        auto first = [&](unsigned r) { return __ldg(&rowBase[r].y) + (__ldg(words + (size_t)r * Wc + w) & 0xffffu); };
        const uint2 own = __ldg(rowBase + row);
        const unsigned pre = __ldg(words + (size_t)row * Wc + w);
        const unsigned e0 = own.y + (pre & 0xffffu), e1 = nj ? first(row + 1) : 0u, e2 = ni ? first(row + E) : 0u,
                       e3 = ni && nj ? first(row + E + 1) : 0u;
        const unsigned cellm = !in.cells(i, j) ? 0u
                               : ((S00 ^ S10) | (S00 ^ S11) | (S00 ^ S01) | (S00 ^ P00) | (S00 ^ P10) | (S00 ^ P11) | (S00 ^ P01)) & kc;
        uint4 *my = sm.rec + lane * kEmitRec;
        my[0] = make_uint4(S00, S10, S11, S01);
        my[1] = make_uint4(P00, P10, P11, P01);
        my[2] = make_uint4(X00, Y00, Z00, e0);
        my[3] = make_uint4(X01, Y01, Z01, e1);
        my[4] = make_uint4(X10, Y10, Z10, e2);
        my[5] = make_uint4(X11, Y11, Z11, e3);
        my[6] = make_uint4(cellm, xn | ((unsigned)w << 1), (unsigned)i, (unsigned)j);
        if (lane == 0) my[7].x = own.x + ((pre >> 16) & 0x7fffu);
        nedge = __popc(X00) + __popc(Y00) + __popc(Z00);
        ncell = __popc(cellm);
    }
    __syncwarp();
    // the words' own edges, in voxel order, x then y then z within a voxel
    {
        const unsigned incl = warp_incl_scan(nedge), total = __shfl_sync(0xffffffffu, incl, 31), from = incl - nedge;
        const unsigned base = sm.rec[2].w;
        for (unsigned e0 = 0; e0 < total; e0 += 32) {
            const unsigned e = e0 + lane, lo = lane_of_item(from, e);
            const unsigned r = e - __shfl_sync(0xffffffffu, from, lo);
            if (e >= total) continue;
            const uint4 o = sm.rec[lo * kEmitRec + 2], id = sm.rec[lo * kEmitRec + 6];
            auto below = [&](unsigned lt) { return (unsigned)(__popc(o.x & lt) + __popc(o.y & lt) + __popc(o.z & lt)); };
            const unsigned b = bit_of_rank(below, r);
            const unsigned q = r - below((1u << b) - 1u), x = (o.x >> b) & 1u, y = (o.y >> b) & 1u;
            const int ax = q < x ? 0 : (q < x + y ? 1 : 2);
            vkey[(size_t)base + e] = edge_key(g, codes, lut, (int)id.z, (int)id.w, (int)(32 * (id.y >> 1) + b), ax);
        }
    }
    // the words' cells in order, corners as edge slots
    {
        const unsigned incl = warp_incl_scan(ncell), total = __shfl_sync(0xffffffffu, incl, 31), from = incl - ncell;
        unsigned *out = tri + 3ull * sm.rec[7].x;
        for (unsigned c0 = 0; c0 < total; c0 += 32) {
            const unsigned c = c0 + lane, lo = lane_of_item(from, c);
            const unsigned r = c - __shfl_sync(0xffffffffu, from, lo);
            unsigned long long corners = 0;
            if (c < total) {
                const uint4 *R = sm.rec + lo * kEmitRec;
                const uint4 s = R[0], p = R[1], id = R[6];
                const unsigned b = bit_of_rank([&](unsigned lt) { return (unsigned)__popc(id.x & lt); }, r), lt = (1u << b) - 1u;
                corners = s_tab[cube_index(b, s.x, s.y, s.z, s.w, p.x, p.y, p.z, p.w)];
                // the rows' edges before voxel b; the next voxel's follow behind this one's
                auto before = [&](const uint4 &o) { return o.w + __popc(o.x & lt) + __popc(o.y & lt) + __popc(o.z & lt); };
                auto bit = [&](unsigned v) { return (v >> b) & 1u; };
                const uint4 o0 = R[2], o1 = R[3], o2 = R[4], o3 = R[5];
                const unsigned a0 = before(o0), a1 = before(o1), a2 = before(o2), a3 = before(o3);
                const unsigned z0 = a0 + bit(o0.x) + bit(o0.y), z1 = a1 + bit(o1.x) + bit(o1.y),
                               z2 = a2 + bit(o2.x) + bit(o2.y), z3 = a3 + bit(o3.x) + bit(o3.y);
                const unsigned n0 = z0 + bit(o0.z), n1 = z1 + bit(o1.z), n2 = z2 + bit(o2.z);
                unsigned *S = sm.slot + lane;  // by the table's edge number (MarchingCubes.cu:814-825)
                S[0] = a0;
                S[32] = a2 + bit(o2.x);
                S[64] = a1;
                S[96] = a0 + bit(o0.x);
                S[128] = n0;
                S[160] = n2 + (b < 31 ? (o2.x >> (b + 1)) & 1u : id.y & 1u);
                S[192] = n1;
                S[224] = n0 + bit(p.x ^ p.y);
                S[256] = z0;
                S[288] = z2;
                S[320] = z3;
                S[352] = z1;
            }
            const unsigned nt = (unsigned)(corners >> 60), ti = warp_incl_scan(nt);
            const unsigned n3 = 3 * __shfl_sync(0xffffffffu, ti, 31);
            unsigned *o = sm.out + 3 * (ti - nt);
            for (unsigned t = 0; t < nt; t++, corners >>= 12, o += 3)
#pragma unroll
                for (unsigned v = 0; v < 3; v++) o[v] = sm.slot[(((unsigned)corners >> (4 * v)) & 15u) * 32 + lane];
            __syncwarp();
            for (unsigned q = lane; q < n3; q += 32) out[q] = sm.out[q];
            out += n3;
            __syncwarp();
        }
    }
    __syncwarp();
}

template <bool BATCH>
__global__ void __launch_bounds__(32 * kEmitWarps, 6) k_mc_emit(QGrid g1, QBatch b, const unsigned *__restrict__ sign,
                                                                const unsigned char *__restrict__ codes,
                                                                const float *__restrict__ lut,
                                                                const unsigned *__restrict__ words,
                                                                const uint2 *__restrict__ rowBase,
                                                                unsigned *__restrict__ tri,
                                                                unsigned long long *__restrict__ vkey, unsigned chunk,
                                                                unsigned units) {
    extern __shared__ uint4 s_emit[];
    __shared__ unsigned long long s_tab[256];
    for (unsigned k = threadIdx.x; k < 256; k += 32 * kEmitWarps) s_tab[k] = c_mc[k];
    __syncthreads();
    EmitSmem &sm = ((EmitSmem *)s_emit)[threadIdx.x >> 5];
    const unsigned unit = blockIdx.x * kEmitWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (unit >= units) return;  // the whole warp
    const unsigned m = BATCH ? qses_find(b.emit_off, b.n_mol, unit) : 0u;
    const QGrid &g = BATCH ? b.mols[m].g : g1;
    if (BATCH) {
        const QMol &mol = b.mols[m];
        sign += mol.mask_off, codes += mol.code_off, words += mol.mask_off, rowBase += mol.row_off, lut = b.lut + 256ull * m;
    }
    const unsigned long long all = (unsigned long long)(g.Gc + 1) * (g.Gc + 1) * ((g.Gc + 32) / 32);
    const unsigned long long w0 = (unsigned long long)(BATCH ? unit - __ldg(b.emit_off + m) : unit) * chunk;
    const unsigned n = (unsigned)min((unsigned long long)chunk, all - w0);
    const unsigned Wc = (unsigned)(g.Gc + 32) / 32, row0 = (unsigned)(w0 / Wc), off = (unsigned)(w0 - (unsigned long long)row0 * Wc);
    unsigned have = 0;  // words in the queue
    for (unsigned k = 0; k < n; k += 128) {
        unsigned v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] = k + 32 * q + lane < n ? __ldg(words + w0 + k + 32 * q + lane) : 0u;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const unsigned some = __ballot_sync(0xffffffffu, v[q] >> 31);
            if (v[q] >> 31) sm.queue[have + __popc(some & ((1u << lane) - 1u))] = (unsigned short)(k + 32 * q + lane);
            have += __popc(some);
        }
        __syncwarp();
        const bool flush = k + 128 >= n;  // the last: whatever is there
        unsigned at = 0;
        while (have - at >= 32 || (flush && at < have)) {
            const bool has = at + lane < have;
            emit_words(g, sign, codes, lut, words, rowBase, tri, vkey, s_tab, sm, has, row0,
                       off + (has ? sm.queue[at + lane] : 0));
            at = min(at + 32, have);
        }
        const unsigned left = have - at;  // below 32
        const unsigned short keep = lane < left ? sm.queue[at + lane] : 0;
        __syncwarp();
        if (lane < left) sm.queue[lane] = keep;
        have = left;
        __syncwarp();
    }
}

// ------------------------------------------------------------------ weld

// The weld: unique quantised positions in lexicographic order, in one kernel, a CTA per grid plane
// (x layer).  The edges of owner rows i come in contiguous slots and their keys lie between the
// planes i and i + 1: a layer's vertices are those on plane i (every y and z edge, and x edges of
// either side quantised onto it) and the x edges between it and the next.  The CTA counts its
// layer's keys into bins that follow the key order - y ranges for the plane, x ranges and within
// them y ranges for the rest - scatters them, ranks each key among its bin's few, and with the
// number of vertices of the layers before (decoupled look-back) numbers them.  A grid has at most
// 4096 layers and a layer of a small molecule is a few hundred keys: then latency bounds it, the
// phases' dozen barriers and the launch; a layer of a large one is bound by the comparisons within
// the bins and their loads.
//
// A radix sort of all keys (7 or 8 passes over 24 B, flags, scan, scatter) took the weld with its
// corner remap 0.14 ms at 30 000 edges, 0.83 at 4 160 000, 24.1 at 138 000 000 (0.03, 0.20 and 6.6 so,
// 1.1 of the last the remap).  A warp sorting each bin of 8 to 32 in registers instead of the
// comparisons: 0.57 and 18.4.
constexpr int kWeldT = 1024;
constexpr unsigned kWeldCap = 4096;  // bins at most, of either sort
constexpr unsigned long long kWeldFirst = 1ull << 63;  // the first of equal keys: the vertex
// What k_weld takes on itself.  A CTA needs some 8 ns for a key of its layer and 0.11 ns for a
// comparison within its bins, all CTAs together a 300th of that.
struct WeldLimits {
    // A layer of more comparisons than this, and than 256 for each key, is heavy: were all so, they would
    // take as long as the sort.
    static constexpr unsigned long long kHeavy = 393216;
    unsigned keys;                  // of a layer and the one before it
    unsigned long long pairs, all;  // comparisons of a layer; of the heavy ones together
    __device__ __forceinline__ explicit WeldLimits(unsigned ne)
        : keys(16384u + ne / 32), pairs(kHeavy + ne), all(20000000ull + 32ull * ne) {
        if (ne < kWeldSortMin) keys = ~0u, pairs = all = ~0ull;  // cannot crowd a layer
    }
    static __device__ __forceinline__ bool heavy(unsigned long long work, unsigned n) {
        return work > kHeavy && work > 256ull * n;
    }
};
constexpr unsigned kWeldX = 4096;       // x ranges of a layer at most: quanta, for voxels up to 4 A
// Quantised x of grid plane i, as edge_key has it for the edges in the plane.
__device__ __forceinline__ unsigned plane_quantum(const QGrid &g, int i) {
    float p = vox(i, g.dx, g.ox);
    if (g.off[0] | g.off[1] | g.off[2]) p = __fadd_rn(p, __fmul_rn((float)g.off[0], g.dx));
    return (unsigned)(quantum(p) - (int)g.bx);
}
// In place: exclusive sums of x[0, n), by the whole block; the total is returned.  squares (may be
// null, zeroed): the sum of the squares in units of 64, what a thread has over a multiple dropped.
template <int NT>
__device__ __forceinline__ unsigned block_excl_sums(unsigned *x, unsigned n, unsigned *s_tmp, unsigned *squares = nullptr) {
    const unsigned per = (n + NT - 1) / NT, lo = min(threadIdx.x * per, n), hi = min(lo + per, n);
    unsigned sum = 0, total;
    unsigned long long sq = 0;
    for (unsigned k = lo; k < hi; k++) {
        sum += x[k];
        if (squares) sq += (unsigned long long)x[k] * x[k];
    }
    if (squares) {
        // a warp's share ends at 2^32 pairs: no overflow, and above every limit
        const unsigned warp = warp_sum((unsigned)min(sq >> 6, 0x3ffffffull));
        if ((threadIdx.x & 31) == 0 && warp) atomicAdd(squares, min(warp, 0x3ffffffu));
    }
    unsigned run = block_excl_scan<NT>(sum, total, s_tmp);
    for (unsigned k = lo; k < hi; k++) {
        const unsigned c = x[k];
        x[k] = run;
        run += c;
    }
    __syncthreads();
    return total;
}

// A mesh may crowd a layer, though: a face normal to x has all its edges in one or two of them, one
// normal to y and a fibre along z put a plane's into few y ranges, and a layer's work is one CTA's and
// grows with the square of a bin's keys.  A layer that would take longer than sorting all keys does
// (WeldLimits) gives up and says so in total->y, and the caller sorts them (launch_weld_sorted), which
// takes 0.12 ms and 0.17 ns a key whatever the shape.  What the other layers did is lost then, and
// bounded by the same limits.  A flat sheet of 40 000 atoms at 0.4 A (530 000 edges) normal to x takes
// 0.33 ms, 31.2 with bins alone and 0.23 if it were sorted at once; one of 1 000 000 (18 000 000 edges)
// normal to y 5.1, 28.9 and 3.2.
template <bool BATCH>
__global__ void __launch_bounds__(kWeldT, 2) k_weld(QGrid g1, QBatch b, unsigned cap,
                                                    const unsigned long long *__restrict__ vkey,
                                                    const uint2 *__restrict__ rowBase, unsigned ne, unsigned layers,
                                                    const unsigned *__restrict__ edge_off, unsigned long long *skey,
                                                    unsigned *sslot, unsigned *__restrict__ vmap,
                                                    float *__restrict__ vq, unsigned *__restrict__ vmol,
                                                    unsigned *__restrict__ vtx_off, uint2 *__restrict__ total,
                                                    unsigned long long *status, unsigned *ticket,
                                                    unsigned long long *work, int *err) {
    extern __shared__ unsigned s_bin[];  // 2 x (2 cap + 2) and kWeldX / 2
    __shared__ unsigned s_tmp[kWeldT / 32], s_tile, s_pushed, s_before;
    __shared__ unsigned s_squares;
    __shared__ unsigned long long s_all;
    if (threadIdx.x == 0) {
        s_squares = 0;
        s_tile = atomicAdd(ticket, 1u);  // layers in the order CTAs start, so that every wait ends
        s_pushed = 0;
    }
    __syncthreads();
    const unsigned tile = s_tile, m = BATCH ? qses_find(b.layer_off, b.n_mol, tile) : 0u;
    const QGrid &g = BATCH ? b.mols[m].g : g1;
    const unsigned i = BATCH ? tile - __ldg(b.layer_off + m) : tile, E = (unsigned)g.Gc + 1;
    const uint2 *rows = rowBase + (BATCH ? b.mols[m].row_off : 0u);
    const unsigned s1 = rows[(size_t)i * E].y;
    unsigned s0 = i ? rows[(size_t)(i - 1) * E].y : s1;
    unsigned s2 = i + 1 < E ? rows[(size_t)(i + 1) * E].y : BATCH ? __ldg(edge_off + m + 1) : ne;
    const WeldLimits limits(ne);
    bool crowded = s2 - s0 > limits.keys;
    if (crowded) s0 = s2 = s1;
    const unsigned X0 = plane_quantum(g, (int)i), X1 = plane_quantum(g, (int)i + 1);
    const unsigned Rq = (unsigned)g.Rq;
    unsigned *cur = s_bin, *uniq = s_bin + 2 * cap + 2;
    unsigned short *x_at = (unsigned short *)(uniq + 2 * cap + 2);
    // y ranges of the plane
    unsigned sy = 0, sx = 0, sq = 0;
    while ((Rq >> sy) + 1 > cap) sy++;
    const unsigned np = (Rq >> sy) + 1;
    // x ranges above it
    while (((X1 - X0) >> sx) + 1 > kWeldX) sx++;
    const unsigned nx = ((X1 - X0) >> sx) + 1;
    // Field values are few, so x takes a tenth of its quanta.  Each that some 4096 of the layer's
    // keys fall on gets bins for y ranges; what lies between two of them is one bin.  Even ranges
    // would put 90 keys into a bin of the largest grids: 22.0 ms instead of 8.6 (0.26 and 0.24).
    for (unsigned k = threadIdx.x; k < nx; k += kWeldT) s_bin[k] = 0;
    __syncthreads();
    const unsigned step = (s2 - s1) / 4096 + 1;
    for (unsigned long long s = s1 + threadIdx.x * step; s < s2; s += kWeldT * step) {
        const unsigned X = (unsigned)(__ldg(vkey + s) >> 42);
        if (X > X0) s_bin[min((X - X0) >> sx, nx - 1)] = 1;
    }
    __syncthreads();
    for (unsigned k = threadIdx.x; k < nx; k += kWeldT) x_at[k] = (unsigned short)s_bin[k];
    const unsigned used = block_excl_sums<kWeldT>(s_bin, nx, s_tmp);
    const bool split = sx == 0 && 4 * used <= cap;  // else a bin for each used x and the ones up to it
    while (split && (Rq >> sq) + 1 > cap / (used + 1) - 1) sq++;
    const unsigned nq = split ? (Rq >> sq) + 1 : 0, nbin = np + min((used + 1) * (nq + 1), cap + 1);
    for (unsigned k = threadIdx.x; k < nx; k += kWeldT) x_at[k] = (unsigned short)(2 * s_bin[k] + x_at[k]);
    __syncthreads();
    // a key's bin: any map that follows the key order serves
    auto bin_of = [&](unsigned long long key) {
        const unsigned X = (unsigned)(key >> 42), Y = (unsigned)(key >> 21) & 0x1fffffu;
        if (X <= X0) return min(Y >> sy, np - 1);
        const unsigned x = x_at[min((X - X0) >> sx, nx - 1)];
        return min(np + (x >> 1) * (nq + 1) + (split && (x & 1) ? 1 + min(Y >> sq, nq - 1) : 0), nbin - 1);
    };
    // The keys of owner rows i lie in [X0, X1] (planes are 0.15 A and more apart, and rounding
    // moves a position by a few quanta at most): those at X1 and above are the next layer's.
    auto mine = [&](unsigned slot, unsigned long long key) {
        const unsigned X = (unsigned)(key >> 42);
        return slot < s1 ? X >= X0 : X < X1 || i + 1 == E;
    };
    for (unsigned k = threadIdx.x; k <= nbin; k += kWeldT) cur[k] = uniq[k] = 0;
    __syncthreads();
    // count
    unsigned below = 0;
    for (unsigned s = s0 + threadIdx.x; s < s2; s += kWeldT) {
        const unsigned long long key = __ldg(vkey + s);
        if (!mine(s, key)) continue;
        atomicAdd(&cur[bin_of(key)], 1u);
        below += s < s1;
    }
    if (below) atomicAdd(&s_pushed, below);
    __syncthreads();
    unsigned n = block_excl_sums<kWeldT>(cur, nbin, s_tmp, &s_squares);
    const unsigned long long pairs = 64ull * s_squares;
    if (limits.heavy(pairs, n)) {  // seldom; the sum passes its limit for the last to add to it, if not before
        if (threadIdx.x == 0) s_all = atomicAdd(work, pairs) + pairs;
        __syncthreads();
        crowded |= s_all > limits.all;
    }
    crowded |= pairs > limits.pairs;
    if (crowded) {
        s0 = s2 = s1;
        n = 0;
    }
    // scatter: the layer's keys to [base, base + n) (the ones before it are the slots before s1 less
    // those pushed up into this layer), bin after bin; cur[k] becomes the end of bin k
    const unsigned base = s1 - s_pushed;
    for (unsigned s = s0 + threadIdx.x; s < s2; s += kWeldT) {
        const unsigned long long key = __ldg(vkey + s);
        if (!mine(s, key)) continue;
        const unsigned q = base + atomicAdd(&cur[bin_of(key)], 1u);
        if (q < ne) {
            skey[q] = key;
            sslot[q] = s;
        }
    }
    __syncthreads();
    // the first of equal keys is the vertex; distinct keys per bin
    for (unsigned q = threadIdx.x; q < n; q += kWeldT) {
        const unsigned long long key = skey[base + q];
        const unsigned k = bin_of(key), lo = k ? cur[k - 1] : 0u;
        bool first = true;
#pragma unroll 4
        for (unsigned p = lo; p < q; p++) first &= (skey[base + p] & ~kWeldFirst) != key;
        if (first) {
            skey[base + q] = key | kWeldFirst;
            atomicAdd(&uniq[k], 1u);
        }
    }
    __syncthreads();
    const unsigned distinct = block_excl_sums<kWeldT>(uniq, nbin, s_tmp);
    if (threadIdx.x < 32) {
        const unsigned long long sum = look_back(status, tile, distinct | (crowded ? 1ull << 32 : 0ull), err);
        const unsigned before = (unsigned)sum;
        if (threadIdx.x == 0) {
            s_before = before;
            if (BATCH && i == 0) vtx_off[m] = before;
            if (tile == layers - 1) {
                *total = make_uint2(before + distinct, (unsigned)(sum >> 32) + crowded);
                if (BATCH) vtx_off[b.n_mol] = before + distinct;
            }
        }
    }
    __syncthreads();
    const unsigned before = s_before;
    for (unsigned q = threadIdx.x; q < n; q += kWeldT) {
        const unsigned long long own = skey[base + q], key = own & ~kWeldFirst;
        const unsigned k = bin_of(key), lo = k ? cur[k - 1] : 0u, hi = cur[k];
        unsigned rank = before + uniq[k];
#pragma unroll 4
        for (unsigned p = lo; p < hi; p++) rank += (skey[base + p] ^ kWeldFirst) < key;
        vmap[sslot[base + q]] = rank;
        if (own != key && rank < ne) {
            const long long mx = (long long)(key >> 42) + g.bx, my = (long long)((key >> 21) & 0x1fffffu) + g.by,
                            mz = (long long)(key & 0x1fffffu) + g.bz;
            vq[3ull * rank] = __fmul_rn((float)mx, QSES_WELD_TOL);
            vq[3ull * rank + 1] = __fmul_rn((float)my, QSES_WELD_TOL);
            vq[3ull * rank + 2] = __fmul_rn((float)mz, QSES_WELD_TOL);
            if (BATCH) vmol[rank] = m;
        }
    }
}

// The weld by sorting all keys, for meshes that crowd a few layers: the sorted keys' first ones
// marked, numbered by a scan, and sent to their slots.  Batch: the keys are put together anew with
// the molecule above its positions, which sorts the molecules one after another (bits: of a position).
__global__ void k_weld_tag(QBatch b, unsigned long long *__restrict__ vkey, const unsigned *__restrict__ edge_off,
                           unsigned n, int bits) {
    const unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const unsigned m = qses_find(edge_off, b.n_mol, s);
    const unsigned long long R = (unsigned long long)b.mols[m].g.Rq, key = vkey[s];
    vkey[s] = (unsigned long long)m << bits | (((key >> 42) * R + ((key >> 21) & 0x1fffffu)) * R + (key & 0x1fffffu));
}
__global__ void k_weld_flags(const unsigned long long *__restrict__ skey, unsigned n, uint2 *__restrict__ flags) {
    const unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) flags[p] = make_uint2(p == 0 || skey[p] != skey[p - 1] ? 1u : 0u, 0u);
}
template <bool BATCH>
__global__ void k_weld_number(QGrid g1, QBatch b, const unsigned long long *__restrict__ skey,
                              const unsigned *__restrict__ sslot, const uint2 *__restrict__ excl, unsigned n, int bits,
                              unsigned *__restrict__ vmap, float *__restrict__ vq, unsigned *__restrict__ vmol) {
    const unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const unsigned long long key = skey[p];
    const bool first = p == 0 || key != skey[p - 1];
    const unsigned rank = excl[p].x - (first ? 0u : 1u);
    vmap[sslot[p]] = rank;
    if (!first) return;
    const unsigned m = BATCH ? (unsigned)(key >> bits) : 0u;
    const QGrid &g = BATCH ? b.mols[m].g : g1;
    unsigned long long x, y, z;
    if (BATCH) {
        const unsigned long long at = key & ((1ull << bits) - 1ull), R = (unsigned long long)g.Rq;
        x = at / (R * R), y = at / R % R, z = at % R;
        vmol[rank] = m;
    } else {
        x = key >> 42, y = (key >> 21) & 0x1fffffu, z = key & 0x1fffffu;
    }
    vq[3ull * rank] = __fmul_rn((float)((long long)x + g.bx), QSES_WELD_TOL);
    vq[3ull * rank + 1] = __fmul_rn((float)((long long)y + g.by), QSES_WELD_TOL);
    vq[3ull * rank + 2] = __fmul_rn((float)((long long)z + g.bz), QSES_WELD_TOL);
}

// out[m] = excl[at[m]] for at[m] < n, else the scan total: the first scanned element of
// each molecule's range gives that molecule's offset in the compacted output.
__global__ void k_gather_offsets(const uint2 *__restrict__ excl, const unsigned *__restrict__ at, unsigned n_mol,
                                 unsigned n, const uint2 *__restrict__ total, unsigned *__restrict__ outx,
                                 unsigned *__restrict__ outy) {
    unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m > n_mol) return;
    const unsigned a = at[m];
    const uint2 v = a < n ? excl[a] : *total;
    if (outx) outx[m] = v.x;
    if (outy) outy[m] = v.y;
}

// Corners from edge slots to vertices.  Bound by the gathers, so each thread has four under way:
// 832 000 000 corners in 1.1 ms, one to a thread took 3.2.
// crowded (may be null): set if the weld gave up; the slots then stay.
__global__ void k_remap(unsigned *__restrict__ tri, size_t n3, const unsigned *__restrict__ vmap,
                        const unsigned *__restrict__ crowded) {
    const size_t q = 4 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
    const bool keep = crowded && __ldg(crowded);
    if (q + 4 <= n3) {
        uint4 t = *(const uint4 *)(tri + q);
        if (keep) return;
        t.x = __ldg(vmap + t.x), t.y = __ldg(vmap + t.y), t.z = __ldg(vmap + t.z), t.w = __ldg(vmap + t.w);
        *(uint4 *)(tri + q) = t;
    } else if (!keep) {
        for (size_t e = q; e < n3; e++) tri[e] = vmap[tri[e]];
    }
}

// ------------------------------------------------------------ closest atom

// The closest atom among the 27 cells around a point, the first in cell order of equally close ones
// (-1 without any): the least (distance, index) in whatever order they are searched, for the atoms
// are in cell order.  The up to three cells of an (x, y) column are one run of atoms.  The point's
// own column comes first, then the nearer neighbours, and what lies beyond the best distance so far
// is passed over; a warp's vertices have about the same x and y and mostly agree on that.  Cells are
// taken 0.01 A wider than they are: coordinates and cell numbers are rounded, by 0.004 A at most.
//
// Bound by instruction issue: 3 540 000 vertices in 0.17 ms (148 M warp instructions at 2.9 a cycle),
// 138 000 000 in 5.8; all 27 cells one by one took 0.30 (270 M) and 10.5, cell by cell in the order
// of closeness 0.27 and 9.8, for each lane wants other cells then.
__device__ __forceinline__ int closest_atom(const QGrid &g, const float4 *__restrict__ atoms, const uint2 *__restrict__ cells,
                                            float qx, float qy, float qz) {
    const float rx = __fsub_rn(qx, g.ox), ry = __fsub_rn(qy, g.oy), rz = __fsub_rn(qz, g.oz);
    const int cx = __float2int_rz(__fdiv_rn(rx, g.cell)), cy = __float2int_rz(__fdiv_rn(ry, g.cell)),
              cz = __float2int_rz(__fdiv_rn(rz, g.cell));
    int best = -1;
    float bestd = FLT_MAX;
    // A point outside the cells searches all of them (its clamped neighbours).
    const bool in = min(cx, min(cy, cz)) >= 0 && max(cx, max(cy, cz)) < g.gnb;
    // how far off the neighbour on the lower and on the upper side is at least, squared
    auto gaps = [&](float r, int c) {
        const float f = r - (float)c * g.cell, lo = fmaxf(f - 0.01f, 0.0f), hi = fmaxf(g.cell - f - 0.01f, 0.0f);
        return in ? make_float2(lo * lo, hi * hi) : make_float2(0.0f, 0.0f);
    };
    const float2 gx = gaps(rx, cx), gy = gaps(ry, cy), gz = gaps(rz, cz);
    const int nx = gx.x < gx.y ? -1 : 1, ny = gy.x < gy.y ? -1 : 1;
    const int z0 = min(max(cz, 0), g.gnb - 1), zm = min(max(cz - 1, 0), g.gnb - 1), zp = min(max(cz + 1, 0), g.gnb - 1);
    for (int a = 0; a < 3; a++) {
        const float lx = a == 0 ? 0.0f : (a == 1 ? fminf(gx.x, gx.y) : fmaxf(gx.x, gx.y));
        if (lx > bestd) break;
        const int xx = min(max(cx + (a == 0 ? 0 : (a == 1 ? nx : -nx)), 0), g.gnb - 1);
        for (int b = 0; b < 3; b++) {
            const float l = lx + (b == 0 ? 0.0f : (b == 1 ? fminf(gy.x, gy.y) : fmaxf(gy.x, gy.y)));
            if (l > bestd) break;
            const int yy = min(max(cy + (b == 0 ? 0 : (b == 1 ? ny : -ny)), 0), g.gnb - 1);
            const uint2 *col = cells + ((size_t)xx * g.gnb + yy) * g.gnb;
            const uint2 none = make_uint2(0u, 0u), r0 = col[z0], rm = l + gz.x <= bestd ? col[zm] : none,
                        rp = l + gz.y <= bestd ? col[zp] : none;  // an empty cell is (0, 0)
            const unsigned from = rm.y ? rm.x : (r0.y ? r0.x : rp.x), to = max(rm.y, max(r0.y, rp.y));
            for (unsigned s = from; s < to; s++) {
                const float4 at = atoms[s];
                const float ex = __fsub_rn(at.x, qx), ey = __fsub_rn(at.y, qy), ez = __fsub_rn(at.z, qz);
                const float d2 = __fmaf_rn(ez, ez, __fmaf_rn(ey, ey, __fmul_rn(ex, ex)));
                if (d2 < bestd || (d2 == bestd && (int)s < best)) {
                    bestd = d2;
                    best = (int)s;
                }
            }
        }
    }
    return best;
}

__global__ void k_closest(QGrid g, const float *__restrict__ vq, unsigned nv, const float4 *__restrict__ atoms,
                          const uint2 *__restrict__ cells, const unsigned *__restrict__ sorted_to_input,
                          int *__restrict__ asorted, int *__restrict__ ainput) {
    unsigned v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    const int best = closest_atom(g, atoms, cells, vq[3ull * v], vq[3ull * v + 1], vq[3ull * v + 2]);
    asorted[v] = best;
    ainput[v] = best >= 0 ? (int)sorted_to_input[best] : -1;
}
__global__ void k_closest_batch(QBatch b, const float *__restrict__ vq, const unsigned *__restrict__ vmol,
                                unsigned nv, const float4 *__restrict__ atoms, const uint2 *__restrict__ cells,
                                const unsigned *__restrict__ sorted_to_input, int *__restrict__ asorted,
                                int *__restrict__ ainput) {
    unsigned v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    const QMol &mol = b.mols[vmol[v]];
    const int best = closest_atom(mol.g, atoms, cells + mol.cell_off, vq[3ull * v], vq[3ull * v + 1], vq[3ull * v + 2]);
    asorted[v] = best >= 0 ? best - (int)mol.atom_off : -1;
    ainput[v] = best >= 0 ? (int)sorted_to_input[best] - (int)mol.atom_off : -1;
}

// Drops the triangles with a repeated corner in one pass: a block's 4096 triangles stay in
// registers, the kept ones go to shared memory in order and from there, behind those of the blocks
// before (look-back), to whole lines of `out`.  Batch: molecules flagged QSES_FLAG_KEEP_DEGENERATE
// keep every triangle, corners become molecule-local vertex ids and kept_off receives each
// molecule's first kept triangle.  `out` may be `tri`: a block writes behind the kept triangles of the
// blocks before it, which have read theirs when they publish their counts, and never past its own.
// Bound by memory, 24 B a triangle, and by the look-back that
// orders the blocks: 1024 triangles each took 2.7 ms for 277 000 000, 2048 2.1, 4096 1.9; a flag per
// triangle, a scan of the flags and a copy 5.2.  8 310 000: 0.19 -> 0.07 ms.
constexpr int kFiltT = 512, kFiltN = 8, kFiltTile = kFiltN * kFiltT;
template <bool BATCH>
__global__ void __launch_bounds__(kFiltT) k_tri_filter(QBatch b, const unsigned *tri, unsigned nt,
                                                       unsigned *out, unsigned *__restrict__ kept_off,
                                                       uint2 *__restrict__ total, unsigned long long *status,
                                                       unsigned *ticket, int *err) {
    __shared__ unsigned s_out[3 * kFiltTile];
    __shared__ unsigned s_tmp[kFiltT / 32], s_tile, s_before;
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const unsigned tile = s_tile, t0 = tile * kFiltTile + kFiltN * threadIdx.x;
    unsigned c[3 * kFiltN], m[kFiltN], keep = 0;
    if (t0 + kFiltN <= nt) {
        const uint4 *q = (const uint4 *)(tri + 3ull * t0);
#pragma unroll
        for (int r = 0; r < 3 * kFiltN / 4; r++) {
            const uint4 v = q[r];
            c[4 * r] = v.x, c[4 * r + 1] = v.y, c[4 * r + 2] = v.z, c[4 * r + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int r = 0; r < 3 * kFiltN; r++) c[r] = t0 + r / 3 < nt ? tri[3ull * t0 + r] : 0u;
    }
    unsigned at = BATCH && t0 < nt ? qses_find(b.tri_off, b.n_mol, t0) : 0u;
#pragma unroll
    for (int r = 0; r < kFiltN; r++) {
        if (t0 + r >= nt) continue;
        if (BATCH)
            while (__ldg(b.tri_off + at + 1) <= t0 + r) at++;
        m[r] = at;
        const unsigned x = c[3 * r], y = c[3 * r + 1], z = c[3 * r + 2];
        keep |= ((x != y && y != z && x != z) || (BATCH && (b.mols[at].flags & QSES_FLAG_KEEP_DEGENERATE))) << r;
    }
    unsigned n;
    const unsigned lo = block_excl_scan<kFiltT>(__popc(keep), n, s_tmp);
    if (threadIdx.x < 32) {
        const unsigned before = (unsigned)look_back(status, tile, n, err);
        if (threadIdx.x == 0) {
            s_before = before;
            if (tile == gridDim.x - 1) *total = make_uint2(before + n, 0u);
        }
    }
    unsigned k = lo;
#pragma unroll
    for (int r = 0; r < kFiltN; r++)
        if (keep >> r & 1) {
            const unsigned v0 = BATCH ? __ldg(b.vtx_off + m[r]) : 0u;
            s_out[3 * k] = c[3 * r] - v0, s_out[3 * k + 1] = c[3 * r + 1] - v0, s_out[3 * k + 2] = c[3 * r + 2] - v0;
            k++;
        }
    __syncthreads();
    const unsigned before = s_before;
    if (BATCH) {  // molecules that start at one of the thread's triangles, or behind the last
#pragma unroll
        for (int r = 0; r < kFiltN; r++)
            if (t0 + r < nt)
                for (int q = (int)m[r]; q >= 0 && __ldg(b.tri_off + q) == t0 + r; q--)
                    kept_off[q] = before + lo + __popc(keep & ((1u << r) - 1u));
        if (tile == gridDim.x - 1 && threadIdx.x == 0)
            for (int q = (int)b.n_mol; q >= 0 && __ldg(b.tri_off + q) == nt; q--) kept_off[q] = before + n;
    }
    if (before <= nt - min(n, nt))
        for (unsigned q = threadIdx.x; q < 3 * n; q += kFiltT) out[3ull * before + q] = s_out[q];
}

// --------------------------------------------------------------- smoothing

// Neighbour lists without a sort.  count: occurrences of each vertex among the 3T triangle
// corners (start[v].x, later scanned); scatter: each corner q is written into its vertex's
// range at a position taken with an atomic (start[v].y, zero after the scan), so the order
// within a range is arbitrary (k_gs_lists sorts it).
// The count also clears the smoothing's counters, for the kernels after it.
__global__ void k_csr_count(const unsigned *__restrict__ tri, size_t n3, uint2 *__restrict__ start,
                            unsigned *__restrict__ zero, unsigned nzero) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n3) atomicAdd(&start[tri[q]].x, 1u);
    for (size_t z = q; z < nzero; z += (size_t)gridDim.x * blockDim.x) zero[z] = 0u;
}

__global__ void k_csr_scatter(const unsigned *__restrict__ tri, size_t n3, uint2 *__restrict__ start,
                              unsigned *__restrict__ occ) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n3) return;
    const unsigned v = tri[q];
    // offset and position with one 64-bit atomic: 24 900 000 corners 0.16 ms, 0.20 with a load more
    const unsigned long long old = atomicAdd((unsigned long long *)&start[v], 1ull << 32);
    occ[(unsigned)old + (unsigned)(old >> 32)] = (unsigned)q;
}

__global__ void k_from_float4(const float4 *__restrict__ v4, unsigned nv, float *__restrict__ v3) {
    unsigned v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < nv) {
        const float4 q = v4[v];
        v3[3ull * v] = q.x; v3[3ull * v + 1] = q.y; v3[3ull * v + 2] = q.z;
    }
}

// ------------------------------------------------------------ launchers

static inline unsigned nblk(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

int mc_rows_per_warp(int Gc) { return 32 / mc_lanes(Gc); }
void launch_mc_count(const QGrid &g, const unsigned *sign, uint2 *rowCount, unsigned *words, cudaStream_t s) {
    const size_t rows = (size_t)(g.Gc + 1) * (g.Gc + 1);
    // Narrow groups put more rows in flight per warp: 664^3 grid 0.248 ms with whole-warp rows, 0.127
    // with 2 lanes; 502^3 0.105 and 0.074.
    const int L = (g.Gc + 32) / 32 >= 8 ? 2 : mc_lanes(g.Gc);
    k_mc_count<<<nblk(rows, 8 * (32 / L)), 256, 0, s>>>(g, sign, rowCount, words, L);
}
void launch_mc_count_batch(const QBatch &b, unsigned units, const unsigned *sign, uint2 *rowCount, unsigned *words,
                           cudaStream_t s) {
    k_mc_count_batch<<<nblk(units, 8), 256, 0, s>>>(b, sign, rowCount, words);
}
unsigned long long mc_words(int Gc) { return (unsigned long long)(Gc + 1) * (Gc + 1) * ((Gc + 32) / 32); }
// Words a warp of the emission takes: as many as leave every SM a few blocks, but more than 128 only
// on grids of 65 536 times as many.  A surface normal to x is in a fiftieth of the chunks, all of whose
// words have edges: 530 000 of them in 520^3 take 0.80 ms by 512 words, 0.23 by 128, 0.09 by 32.  Chunks
// with a few such words each want to be large, for a warp works on 32 at a time: 664^3 0.25, 0.25 and
// 0.45, a shell of 1 000 000 atoms (2 171^3) 7.3, 8.6 and 18.2.
unsigned mc_emit_chunk(unsigned long long words) {
    const unsigned long long small = std::min(words / 8192, 128ull), large = std::min(words / 65536, 512ull);
    return (unsigned)((std::max(std::max(small, large), 1ull) + 31) / 32 * 32);
}
template <bool BATCH>
static cudaError_t emit_with(const QGrid &g, const QBatch &b, const unsigned *sign, const unsigned char *codes,
                             const float *lut, const unsigned *words, const uint2 *rowBase, unsigned *tri,
                             unsigned long long *vkey, unsigned chunk, unsigned units, cudaStream_t s) {
    const cudaError_t e = cudaFuncSetAttribute((const void *)k_mc_emit<BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(kEmitWarps * sizeof(EmitSmem)));
    if (e != cudaSuccess) return e;
    k_mc_emit<BATCH><<<nblk(units, kEmitWarps), 32 * kEmitWarps, kEmitWarps * sizeof(EmitSmem), s>>>(
        g, b, sign, codes, lut, words, rowBase, tri, vkey, chunk, units);
    return cudaGetLastError();
}
cudaError_t launch_mc_emit(const QGrid &g, const unsigned *sign, const unsigned char *codes, const float *lut,
                           const unsigned *words, const uint2 *rowBase, unsigned *tri, unsigned long long *vkey,
                           cudaStream_t s) {
    const unsigned long long all = mc_words(g.Gc);
    const unsigned chunk = mc_emit_chunk(all);
    return emit_with<false>(g, QBatch{}, sign, codes, lut, words, rowBase, tri, vkey, chunk,
                            (unsigned)((all + chunk - 1) / chunk), s);
}
cudaError_t launch_mc_emit_batch(const QBatch &b, unsigned chunk, unsigned units, const unsigned *sign,
                                 const unsigned char *codes, const unsigned *words, const uint2 *rowBase, unsigned *tri,
                                 unsigned long long *vkey, cudaStream_t s) {
    return emit_with<true>(QGrid{}, b, sign, codes, nullptr, words, rowBase, tri, vkey, chunk, units, s);
}
size_t weld_tmp_bytes(unsigned layers) { return 256 + 8ull * layers; }
template <bool BATCH>
static cudaError_t weld_with(const QGrid &g, const QBatch &b, const unsigned long long *vkey, const uint2 *rowBase,
                             unsigned ne, unsigned layers, const unsigned *edge_off, unsigned long long *skey,
                             unsigned *sslot, unsigned *vmap, float *vq, unsigned *vmol, unsigned *vtx_off, uint2 *total,
                             void *tmp, int *err, cudaStream_t s) {
    // A bin of either sort for each key of an average layer: a key is compared with its whole bin.
    // Half or twice as many bins take the same time, 8192 at most (one CTA per SM) 9.3 ms for 8.6.
    const unsigned per = ne / layers, cap = per < 1024 ? 1024 : per > kWeldCap ? kWeldCap : per;
    static_assert(4 * 1024 + 4 >= kWeldX, "the x marks lie where the bins will");
    const size_t smem = 8ull * (2 * cap + 2) + 2 * kWeldX;
    cudaError_t e = cudaFuncSetAttribute((const void *)k_weld<BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         8 * (2 * kWeldCap + 2) + 2 * kWeldX);
    if (e == cudaSuccess) e = cudaMemsetAsync(tmp, 0, weld_tmp_bytes(layers), s);
    if (e != cudaSuccess) return e;
    k_weld<BATCH><<<layers, kWeldT, smem, s>>>(g, b, cap, vkey, rowBase, ne, layers, edge_off, skey, sslot, vmap, vq, vmol,
                                               vtx_off, total, (unsigned long long *)((char *)tmp + 256), (unsigned *)tmp,
                                               (unsigned long long *)((char *)tmp + 128), err);
    return cudaGetLastError();
}
cudaError_t launch_weld(const QGrid &g, const unsigned long long *vkey, const uint2 *rowBase, unsigned ne,
                        unsigned long long *skey, unsigned *sslot, unsigned *vmap, float *vq, uint2 *total, void *tmp,
                        int *err, cudaStream_t s) {
    return weld_with<false>(g, QBatch{}, vkey, rowBase, ne, (unsigned)g.Gc + 1, nullptr, skey, sslot, vmap, vq, nullptr,
                            nullptr, total, tmp, err, s);
}
cudaError_t launch_weld_batch(const QBatch &b, unsigned layers, const unsigned long long *vkey, const uint2 *rowBase,
                              unsigned ne, const unsigned *edge_off, unsigned long long *skey, unsigned *sslot,
                              unsigned *vmap, float *vq, unsigned *vmol, unsigned *vtx_off, uint2 *total, void *tmp, int *err,
                              cudaStream_t s) {
    return weld_with<true>(QGrid{}, b, vkey, rowBase, ne, layers, edge_off, skey, sslot, vmap, vq, vmol, vtx_off, total, tmp,
                           err, s);
}
template <bool BATCH>
static cudaError_t weld_sorted_with(const QGrid &g, const QBatch &b, unsigned long long *vkey, unsigned long long *skey,
                                    unsigned *sslot, unsigned ne, const unsigned *edge_off, int bits, unsigned *vmap,
                                    float *vq, unsigned *vmol, unsigned *vtx_off, uint2 *total, int *err,
                                    cudaStream_t s, int *launches) {
    // Positions come last, so their memory is the sort's and the scan's workspace until then.  An even
    // number of passes ends where it began: the other key buffer then holds the marks.
    const int key_bits = BATCH ? bits + bits_for(b.n_mol - 1) : 63, even = (key_bits + 15) / 16 * 16;
    if (ne < kWeldSortMin || key_bits > 64 ||
        12ull * ne < std::max(radix_sort_tmp_bytes<unsigned long long>(ne, even), scan_u2_tmp_bytes(ne)))
        return cudaErrorInvalidValue;
    if (BATCH) k_weld_tag<<<nblk(ne, 256), 256, 0, s>>>(b, vkey, edge_off, ne, bits);
    int alt = 0;
    cudaError_t e = radix_sort<unsigned long long>(vkey, skey, sslot, vmap, ne, even, true, vq, err, s, launches, &alt);
    if (e != cudaSuccess) return e;
    uint2 *flags = (uint2 *)skey;
    k_weld_flags<<<nblk(ne, 256), 256, 0, s>>>(vkey, ne, flags);
    e = scan_u2(flags, flags, ne, total, vq, err, s, launches);
    if (e != cudaSuccess) return e;
    k_weld_number<BATCH><<<nblk(ne, 256), 256, 0, s>>>(g, b, vkey, sslot, flags, ne, bits, vmap, vq, vmol);
    if (BATCH) launch_gather_offsets(flags, edge_off, b.n_mol, ne, total, vtx_off, nullptr, s);
    *launches += BATCH ? 4 : 2;
    return cudaGetLastError();
}
cudaError_t launch_weld_sorted(const QGrid &g, unsigned long long *vkey, unsigned long long *skey, unsigned *sslot,
                               unsigned ne, unsigned *vmap, float *vq, uint2 *total, int *err, cudaStream_t s,
                               int *launches) {
    return weld_sorted_with<false>(g, QBatch{}, vkey, skey, sslot, ne, nullptr, 0, vmap, vq, nullptr, nullptr, total, err, s,
                                   launches);
}
cudaError_t launch_weld_sorted_batch(const QBatch &b, unsigned long long *vkey, unsigned long long *skey, unsigned *sslot,
                                     unsigned ne, const unsigned *edge_off, int bits, unsigned *vmap, float *vq,
                                     unsigned *vmol, unsigned *vtx_off, uint2 *total, int *err, cudaStream_t s,
                                     int *launches) {
    return weld_sorted_with<true>(QGrid{}, b, vkey, skey, sslot, ne, edge_off, bits, vmap, vq, vmol, vtx_off, total, err, s,
                                  launches);
}
void launch_gather_offsets(const uint2 *excl, const unsigned *at, unsigned n_mol, unsigned n, const uint2 *total,
                           unsigned *outx, unsigned *outy, cudaStream_t s) {
    k_gather_offsets<<<nblk(n_mol + 1, 256), 256, 0, s>>>(excl, at, n_mol, n, total, outx, outy);
}
void launch_closest_batch(const QBatch &b, const float *vq, const unsigned *vmol, unsigned nv, const float4 *atoms,
                          const uint2 *cells, const unsigned *sorted_to_input, int *asorted, int *ainput,
                          cudaStream_t s) {
    k_closest_batch<<<nblk(nv, 128), 128, 0, s>>>(b, vq, vmol, nv, atoms, cells, sorted_to_input, asorted, ainput);
}
void launch_remap(unsigned *tri, size_t n3, const unsigned *vmap, const unsigned *crowded, cudaStream_t s) {
    k_remap<<<nblk((n3 + 3) / 4, 256), 256, 0, s>>>(tri, n3, vmap, crowded);
}
void launch_closest(const QGrid &g, const float *vq, unsigned nv, const float4 *atoms, const uint2 *cells,
                    const unsigned *sorted_to_input, int *asorted, int *ainput, cudaStream_t s) {
    k_closest<<<nblk(nv, 128), 128, 0, s>>>(g, vq, nv, atoms, cells, sorted_to_input, asorted, ainput);
}
size_t tri_filter_tmp_bytes(unsigned nt) { return 256 + 8 * (((size_t)nt + kFiltTile - 1) / kFiltTile); }
template <bool BATCH>
static cudaError_t filter_with(const QBatch &b, const unsigned *tri, unsigned nt, unsigned *out, unsigned *kept_off,
                               uint2 *total, void *tmp, int *err, cudaStream_t s) {
    const cudaError_t e = cudaMemsetAsync(tmp, 0, tri_filter_tmp_bytes(nt), s);
    if (e != cudaSuccess) return e;
    k_tri_filter<BATCH><<<nblk(nt, kFiltTile), kFiltT, 0, s>>>(b, tri, nt, out, kept_off, total,
                                                                (unsigned long long *)((char *)tmp + 256), (unsigned *)tmp, err);
    return cudaGetLastError();
}
cudaError_t launch_tri_filter(const unsigned *tri, unsigned nt, unsigned *out, uint2 *total, void *tmp, int *err,
                              cudaStream_t s) {
    return filter_with<false>(QBatch{}, tri, nt, out, nullptr, total, tmp, err, s);
}
cudaError_t launch_tri_filter_batch(const QBatch &b, const unsigned *tri, unsigned nt, unsigned *out, unsigned *kept_off,
                                    uint2 *total, void *tmp, int *err, cudaStream_t s) {
    return filter_with<true>(b, tri, nt, out, kept_off, total, tmp, err, s);
}
void launch_csr_count(const unsigned *tri, size_t n3, uint2 *start, unsigned *zero, unsigned nzero, cudaStream_t s) {
    k_csr_count<<<nblk(n3, 256), 256, 0, s>>>(tri, n3, start, zero, nzero);
}
void launch_csr_scatter(const unsigned *tri, size_t n3, uint2 *start, unsigned *occ, cudaStream_t s) {
    k_csr_scatter<<<nblk(n3, 256), 256, 0, s>>>(tri, n3, start, occ);
}
void launch_from_float4(const float4 *v4, unsigned nv, float *v3, cudaStream_t s) {
    k_from_float4<<<nblk(nv, 256), 256, 0, s>>>(v4, nv, v3);
}
}  // namespace qses
