// Marching cubes, vertex weld, closest atom, degenerate filter and Laplacian smoothing.
//
//  k_mc<false>    per (x, y) row of cells: triangle count and active-edge count
//                 (countVertexPerCell, MarchingCubes.cu:571-658, single-slice cell range)
//  k_mc<true>     the same rows again: triangles in cell linear order x*G^2 + y*G + z and
//                 one quantised key per active edge (generateTriangleVerticesSMEM +
//                 groupVertices, MarchingCubes.cu:736-862).  One warp per row; the sign of
//                 32 voxels is one word, so cube indices and edge activity are bit ops.
//  k_weld         unique quantised positions in lexicographic order (CudaSurf.cu:444-457)
//  k_closest      closest atom per welded vertex (closestAtomPerVertex, Kernels.cu:547-604)
//  k_tri_filter   drop triangles with a repeated index (CudaSurf.cu:820-829)
//  k_csr_*        neighbour lists in triangle order (getNeighboorsVertices,
//                 SmoothMesh.cpp:45-123) for the Gauss-Seidel dataflow (k_smooth.cu)
#include <cfloat>
#include <cstdlib>
#include <cstring>

#include "device_common.cuh"

#include "kernels.h"
#include "mc_tables.h"

namespace qses {

__constant__ unsigned long long c_mc[256] = QSES_MC_TABLE_INIT;

// Owner of each cube edge relative to the cell: bit0 di, bit1 dj, bit2 dk, bits3-4 axis.
// Edges follow MarchingCubes.cu:814-825 with corners as in :625-632.
constexpr unsigned long long kEdgeOwner =
    (0ull << 0) | (9ull << 5) | (2ull << 10) | (8ull << 15) | (4ull << 20) | (13ull << 25) | (6ull << 30) |
    (12ull << 35) | (16ull << 40) | (17ull << 45) | (19ull << 50) | (18ull << 55);

__device__ __forceinline__ unsigned ld_sign(const unsigned *__restrict__ sign, const QGrid &g, int i, int j, int w) {
    if (i >= g.G || j >= g.G || w >= g.W) return 0u;
    return __ldg(&sign[((size_t)i * g.G + j) * g.W + w]);
}

__device__ __forceinline__ unsigned cube_index(unsigned b, unsigned c0, unsigned c1, unsigned c2, unsigned c3,
                                               unsigned c4, unsigned c5, unsigned c6, unsigned c7) {
    return ((c0 >> b) & 1u) | (((c1 >> b) & 1u) << 1) | (((c2 >> b) & 1u) << 2) | (((c3 >> b) & 1u) << 3) |
           (((c4 >> b) & 1u) << 4) | (((c5 >> b) & 1u) << 5) | (((c6 >> b) & 1u) << 6) | (((c7 >> b) & 1u) << 7);
}

__device__ __forceinline__ unsigned warp_sum(unsigned v) { return __reduce_add_sync(0xffffffffu, v); }

// Quantised key of the vertex on edge (i, j, k) -> (i, j, k) + e_axis.
__device__ unsigned long long edge_key(const QGrid &g, const unsigned char *__restrict__ codes, const float *lut,
                                       int i, int j, int k, int ax) {
    const size_t base = ((size_t)i * g.G + j) * g.Gp + k;
    const size_t step = ax == 0 ? (size_t)g.G * g.Gp : (ax == 1 ? (size_t)g.Gp : (size_t)1);
    const float fa = lut[__ldg(codes + base)], fb = lut[__ldg(codes + base + step)];
    const float t = __fdiv_rn(-fa, __fsub_rn(fb, fa));  // vertexInterp (MarchingCubes.cu:731-734)
    float p[3] = {vox(i, g.dx, g.ox), vox(j, g.dx, g.oy), vox(k, g.dx, g.oz)};
    const float o[3] = {g.ox, g.oy, g.oz};
    const int idx[3] = {i, j, k};
#pragma unroll
    for (int c = 0; c < 3; c++)
        if (c == ax) p[c] = __fmaf_rn(t, __fsub_rn(vox(idx[c] + 1, g.dx, o[c]), p[c]), p[c]);
    if (g.off[0] | g.off[1] | g.off[2]) {  // a slice box: + offset * dx (MarchingCubes.cu:841-848)
#pragma unroll
        for (int c = 0; c < 3; c++) p[c] = __fadd_rn(p[c], __fmul_rn((float)g.off[c], g.dx));
    }
    // groupVertices: round(v / 0.001) (MarchingCubes.cu:859)
    long long mx = (long long)roundf(__fdiv_rn(p[0], QSES_WELD_TOL));
    long long my = (long long)roundf(__fdiv_rn(p[1], QSES_WELD_TOL));
    long long mz = (long long)roundf(__fdiv_rn(p[2], QSES_WELD_TOL));
    return ((unsigned long long)(mx - g.bx) << 42) | ((unsigned long long)(my - g.by) << 21) | (unsigned long long)(mz - g.bz);
}

__device__ __forceinline__ unsigned sel4(int o, unsigned a, unsigned b, unsigned c, unsigned d) {
    return o == 0 ? a : (o == 1 ? b : (o == 2 ? c : d));
}

// Lanes per owner row: the row's words (voxels 0..Gc) rounded up to a power of two, at
// most 32, so a warp covers 32 / lanes rows of a small grid at once.
__host__ __device__ __forceinline__ int mc_lanes(int Gc) {
    const int Wc = (Gc + 32) / 32;
    int L = 1;
    while (L < Wc && L < 32) L <<= 1;
    return L;
}

// Sum / inclusive scan over aligned groups of Lg lanes (Lg a power of two, warp-uniform).
__device__ __forceinline__ unsigned grp_sum(unsigned v, int Lg) {
    if (Lg == 32) return __reduce_add_sync(0xffffffffu, v);
    for (int o = Lg >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, Lg);
    return v;
}
__device__ __forceinline__ unsigned grp_incl_scan(unsigned v, int sub, int Lg) {
    for (int o = 1; o < Lg; o <<= 1) {
        const unsigned a = __shfl_up_sync(0xffffffffu, v, o, Lg);
        if (sub >= o) v += a;
    }
    return v;
}

// One owner row (i, j) of a molecule's grid per group of Lg lanes; every lane of the warp
// calls this (groups whose row is past the end pass valid = false and write nothing).
// Bits [a, b) of a 32-bit word, the bounds clamped to [0, 32].
__device__ __forceinline__ unsigned bits_in(int a, int b) {
    a = max(a, 0);
    b = min(b, 32);
    if (a >= b) return 0u;
    const unsigned below_b = b == 32 ? 0xffffffffu : ((1u << b) - 1u);
    return below_b & ~((1u << a) - 1u);
}

// Words per lane record of the triangle pass (34 used; an odd stride spreads the lanes'
// writes over the shared-memory banks).
constexpr int kRecW = 35;

template <bool EMIT, bool FULL>
__device__ __forceinline__ void mc_row(const QGrid &g, long long row, bool valid, int Lg,
                                       const unsigned *__restrict__ sign, const unsigned char *__restrict__ codes,
                                       const float *lut, const unsigned long long *s_tab,
                                       uint2 *__restrict__ rowCount, const uint2 *__restrict__ rowBase,
                                       unsigned *__restrict__ tri, unsigned long long *__restrict__ vkey,
                                       unsigned *s_rec) {
    // FULL: one row per warp (Lg = 32, every group valid), known at compile time.
    if (FULL) {
        Lg = 32;
        valid = true;
    }
    const int sub = (int)(threadIdx.x & 31) & (Lg - 1);
    const int Gc = g.Gc, E = Gc + 1;
    if (!valid) row = 0;
    const int i = (int)(row / E), j = (int)(row % E);
    // Emitted cells: [clo, chi) per axis (the whole grid: [0, Gc)).  A row's +x edges are
    // used when a cell of the range has them (x in [clo, chi), y in [clo, chi]), likewise +y;
    // its +z edges when x and y are in [clo, chi].
    const int lox = g.clo[0], hix = g.chi[0], loy = g.clo[1], hiy = g.chi[1], loz = g.clo[2], hiz = g.chi[2];
    auto xr = [&](int a, int b) { return a >= lox && a < hix && b >= loy && b <= hiy; };
    auto yr = [&](int a, int b) { return a >= lox && a <= hix && b >= loy && b < hiy; };
    auto zr = [&](int a, int b) { return a >= lox && a <= hix && b >= loy && b <= hiy; };
    const bool cellsRow = valid && i >= lox && i < hix && j >= loy && j < hiy;
    const int Wc = (Gc + 32) / 32;  // words holding voxels 0..Gc

    unsigned triBase = 0, eb0 = 0, eb1 = 0, eb2 = 0, eb3 = 0;  // owners (0,0) (0,1) (1,0) (1,1)
    if (EMIT && valid) {
        triBase = rowBase[row].x;
        eb0 = rowBase[row].y;
        if (j + 1 <= Gc) eb1 = rowBase[(size_t)i * E + j + 1].y;
        if (i + 1 <= Gc) eb2 = rowBase[(size_t)(i + 1) * E + j].y;
        if (i + 1 <= Gc && j + 1 <= Gc) eb3 = rowBase[(size_t)(i + 1) * E + j + 1].y;
    }
    unsigned triCarry = 0, ec0 = 0, ec1 = 0, ec2 = 0, ec3 = 0;
    for (int w0 = 0; w0 < Wc; w0 += Lg) {
        const int w = w0 + sub;
        const bool act = valid && w < Wc;
        const int kb = w * 32;
        unsigned kv = 0u, kc = 0u;
        if (act) {
            kv = bits_in(loz - kb, hiz - kb + 1);  // voxels in [loz, hiz]
            kc = bits_in(loz - kb, hiz - kb);      // cells / z-edges in [loz, hiz)
        }
        const bool nxt = act && (kb + 32 <= hiz) && (kb + 32 >= loz);
        auto L = [&](int a, int b, int ww) { return act ? ld_sign(sign, g, i + a, j + b, ww) : 0u; };
        const unsigned S00 = L(0, 0, w), S10 = L(1, 0, w), S01 = L(0, 1, w), S11 = L(1, 1, w);
        const unsigned N00 = L(0, 0, w + 1), N10 = L(1, 0, w + 1), N01 = L(0, 1, w + 1), N11 = L(1, 1, w + 1);
        const unsigned P00 = (S00 >> 1) | (N00 << 31), P10 = (S10 >> 1) | (N10 << 31);
        const unsigned P01 = (S01 >> 1) | (N01 << 31), P11 = (S11 >> 1) | (N11 << 31);
        const unsigned X00 = xr(i, j) ? (S00 ^ S10) & kv : 0u;
        const unsigned Y00 = yr(i, j) ? (S00 ^ S01) & kv : 0u;
        const unsigned Z00 = zr(i, j) ? (S00 ^ P00) & kc : 0u;
        const unsigned c00 = __popc(X00) + __popc(Y00) + __popc(Z00);
        unsigned cellm = 0u, ntri = 0u, nt0 = 0u, nt1 = 0u, nt2 = 0u;  // nt bit k of each active cell
        if (cellsRow) {
            cellm = ((S00 ^ S10) | (S00 ^ S11) | (S00 ^ S01) | (S00 ^ P00) | (S00 ^ P10) | (S00 ^ P11) |
                     (S00 ^ P01)) & kc;
            for (unsigned m = cellm; m; m &= m - 1u) {
                unsigned b = __ffs(m) - 1;
                const unsigned nt = (unsigned)(s_tab[cube_index(b, S00, S10, S11, S01, P00, P10, P11, P01)] >> 60);
                ntri += nt;
                if (EMIT) {
                    nt0 |= (nt & 1u) << b;
                    nt1 |= ((nt >> 1) & 1u) << b;
                    nt2 |= ((nt >> 2) & 1u) << b;
                }
            }
        }
        if (!EMIT) {
            triCarry += grp_sum(ntri, Lg);
            ec0 += grp_sum(c00, Lg);
            continue;
        }
        // Edges owned by the three neighbouring rows, for triangle corners.
        const unsigned S20 = L(2, 0, w), S21 = L(2, 1, w), S02 = L(0, 2, w), S12 = L(1, 2, w);
        const unsigned N20 = L(2, 0, w + 1), N21 = L(2, 1, w + 1), N02 = L(0, 2, w + 1), N12 = L(1, 2, w + 1);
        const unsigned X01 = xr(i, j + 1) ? (S01 ^ S11) & kv : 0u;
        const unsigned Y01 = yr(i, j + 1) ? (S01 ^ S02) & kv : 0u;
        const unsigned Z01 = zr(i, j + 1) ? (S01 ^ P01) & kc : 0u;
        const unsigned X10 = xr(i + 1, j) ? (S10 ^ S20) & kv : 0u;
        const unsigned Y10 = yr(i + 1, j) ? (S10 ^ S11) & kv : 0u;
        const unsigned Z10 = zr(i + 1, j) ? (S10 ^ P10) & kc : 0u;
        const unsigned X11 = xr(i + 1, j + 1) ? (S11 ^ S21) & kv : 0u;
        const unsigned Y11 = yr(i + 1, j + 1) ? (S11 ^ S12) & kv : 0u;
        const unsigned Z11 = zr(i + 1, j + 1) ? (S11 ^ P11) & kc : 0u;
        const unsigned c01 = __popc(X01) + __popc(Y01) + __popc(Z01);
        const unsigned c10 = __popc(X10) + __popc(Y10) + __popc(Z10);
        const unsigned c11 = __popc(X11) + __popc(Y11) + __popc(Z11);
        // Activity of the x/y edges of voxel kb+32 (bit 0 of the next word).
        const unsigned xn0 = (nxt && xr(i, j)) ? ((N00 ^ N10) & 1u) : 0u, yn0 = (nxt && yr(i, j)) ? ((N00 ^ N01) & 1u) : 0u;
        const unsigned xn1 = (nxt && xr(i, j + 1)) ? ((N01 ^ N11) & 1u) : 0u, yn1 = (nxt && yr(i, j + 1)) ? ((N01 ^ N02) & 1u) : 0u;
        const unsigned xn2 = (nxt && xr(i + 1, j)) ? ((N10 ^ N20) & 1u) : 0u, yn2 = (nxt && yr(i + 1, j)) ? ((N10 ^ N11) & 1u) : 0u;
        const unsigned xn3 = (nxt && xr(i + 1, j + 1)) ? ((N11 ^ N21) & 1u) : 0u, yn3 = (nxt && yr(i + 1, j + 1)) ? ((N11 ^ N12) & 1u) : 0u;

        const unsigned p0 = grp_incl_scan(c00, sub, Lg) - c00, p1 = grp_incl_scan(c01, sub, Lg) - c01;
        const unsigned p2 = grp_incl_scan(c10, sub, Lg) - c10, p3 = grp_incl_scan(c11, sub, Lg) - c11;
        const unsigned tp = grp_incl_scan(ntri, sub, Lg) - ntri;

        // Vertices owned by this row, in voxel order, x then y then z within a voxel: edge e of
        // the group's words goes to slot eb0 + ec0 + e.  The few words a surface crosses hold
        // all of a row's edges, so the edges are dealt out over the group's lanes: lane `sub`
        // takes e = sub, sub + Lg, ..., finds the owning lane (largest L with p0[L] <= e) and
        // the voxel and axis of the edge inside that lane's word.
        {
            const unsigned etot = grp_sum(c00, Lg);
            const unsigned emax = FULL ? etot : __reduce_max_sync(0xffffffffu, etot);  // warp-uniform
            const int gbase = (int)(threadIdx.x & 31) & ~(Lg - 1);
            for (unsigned eb = 0; eb < emax; eb += (unsigned)Lg) {
                const unsigned e = eb + (unsigned)sub;
                int lo = 0;
                for (int step = Lg >> 1; step > 0; step >>= 1) {
                    const unsigned pl = __shfl_sync(0xffffffffu, p0, gbase + lo + step);
                    if (pl <= e) lo += step;
                }
                const unsigned Xo = __shfl_sync(0xffffffffu, X00, gbase + lo);
                const unsigned Yo = __shfl_sync(0xffffffffu, Y00, gbase + lo);
                const unsigned Zo = __shfl_sync(0xffffffffu, Z00, gbase + lo);
                const unsigned po = __shfl_sync(0xffffffffu, p0, gbase + lo);
                if (e < etot) {
                    const unsigned r = e - po;  // rank of the edge inside the owner's word
                    int b = 0;                  // its voxel: the largest b with fewer than r+1 edges below
                    for (int step = 16; step > 0; step >>= 1) {
                        const unsigned lt = (1u << (b + step)) - 1u;
                        if ((unsigned)(__popc(Xo & lt) + __popc(Yo & lt) + __popc(Zo & lt)) <= r) b += step;
                    }
                    const unsigned lt = (1u << b) - 1u;
                    unsigned qa = r - (unsigned)(__popc(Xo & lt) + __popc(Yo & lt) + __popc(Zo & lt));
                    int ax = 2;
                    if ((Xo >> b) & 1u) {
                        if (qa == 0) ax = 0;
                        else qa--;
                    }
                    if (ax == 2 && ((Yo >> b) & 1u) && qa == 0) ax = 1;
                    const int k = (w0 + lo) * 32 + b;
                    vkey[eb0 + ec0 + e] = edge_key(g, codes, lut, i, j, k, ax);
                }
            }
        }
        // Triangles in cell order, corners as pre-weld vertex slots.  The few words a surface
        // crosses hold all of a row's cells, so the row's active cells are dealt out over the
        // group's lanes: every lane publishes its word's sign words, edge masks, slot bases and
        // per-cell triangle counts, and lane `sub` takes the row's active cells sub, sub + Lg,
        // ...; a cell's first triangle is its word's first plus the counts of the cells below.
        {
            unsigned *my = s_rec + (threadIdx.x & 31) * kRecW;
            my[0] = S00; my[1] = S10; my[2] = S11; my[3] = S01;
            my[4] = P00; my[5] = P10; my[6] = P11; my[7] = P01;
            my[8] = X00; my[9] = Y00; my[10] = Z00; my[11] = X01; my[12] = Y01; my[13] = Z01;
            my[14] = X10; my[15] = Y10; my[16] = Z10; my[17] = X11; my[18] = Y11; my[19] = Z11;
            my[20] = eb0 + ec0 + p0; my[21] = eb1 + ec1 + p1; my[22] = eb2 + ec2 + p2; my[23] = eb3 + ec3 + p3;
            my[24] = c00; my[25] = c01; my[26] = c10; my[27] = c11;
            my[28] = xn0 | (yn0 << 1) | (xn1 << 2) | (yn1 << 3) | (xn2 << 4) | (yn2 << 5) | (xn3 << 6) | (yn3 << 7);
            my[29] = nt0; my[30] = nt1; my[31] = nt2; my[32] = cellm; my[33] = triBase + triCarry + tp;
            __syncwarp();
            const unsigned nc = __popc(cellm);
            const unsigned cp = grp_incl_scan(nc, sub, Lg) - nc;
            const unsigned ctot = grp_sum(nc, Lg);
            const unsigned cmax = FULL ? ctot : __reduce_max_sync(0xffffffffu, ctot);  // warp-uniform
            const int gbase = (int)(threadIdx.x & 31) & ~(Lg - 1);
            for (unsigned cb = 0; cb < cmax; cb += (unsigned)Lg) {
                const unsigned ci = cb + (unsigned)sub;
                int lo = 0;
                for (int step = Lg >> 1; step > 0; step >>= 1) {
                    const unsigned pl = __shfl_sync(0xffffffffu, cp, gbase + lo + step);
                    if (pl <= ci) lo += step;
                }
                const unsigned po = __shfl_sync(0xffffffffu, cp, gbase + lo);
                if (ci < ctot) {
                    const unsigned *R = s_rec + (gbase + lo) * kRecW;
                    const unsigned cm = R[32], r = ci - po;
                    int b = 0;  // the r-th active cell of the owner's word: the largest b with r cells below
                    for (int step = 16; step > 0; step >>= 1)
                        if ((unsigned)__popc(cm & ((1u << (b + step)) - 1u)) <= r) b += step;
                    const unsigned lt = (1u << b) - 1u;
                    const unsigned ts = R[33] + __popc(R[29] & lt) + 2u * __popc(R[30] & lt) + 4u * __popc(R[31] & lt);
                    const unsigned long long e = s_tab[cube_index(b, R[0], R[1], R[2], R[3], R[4], R[5], R[6], R[7])];
                    const unsigned nt = (unsigned)(e >> 60);
                    for (unsigned q = 0; q < 3 * nt; q++) {
                        const unsigned edge = (unsigned)(e >> (4 * q)) & 15u;
                        const unsigned own = (unsigned)(kEdgeOwner >> (5 * edge)) & 31u;
                        const int o = (int)((own & 1u) * 2 + ((own >> 1) & 1u));  // (di, dj) -> owner index
                        const unsigned dk = (own >> 2) & 1u, ax = own >> 3;
                        const unsigned Xo = R[8 + 3 * o], Yo = R[9 + 3 * o], Zo = R[10 + 3 * o];
                        unsigned slot = R[20 + o];
                        const unsigned vb = (unsigned)b + dk;
                        if (vb < 32) {
                            const unsigned lt2 = (1u << vb) - 1u;
                            slot += __popc(Xo & lt2) + __popc(Yo & lt2) + __popc(Zo & lt2);
                            if (ax >= 1) slot += (Xo >> vb) & 1u;
                            if (ax >= 2) slot += (Yo >> vb) & 1u;
                        } else {
                            slot += R[24 + o];
                            if (ax >= 1) slot += (R[28] >> (2 * o)) & 1u;
                            if (ax >= 2) slot += (R[28] >> (2 * o + 1)) & 1u;
                        }
                        tri[3ull * ts + q] = slot;
                    }
                }
            }
            __syncwarp();  // the records are read before the next words' are written
        }
        triCarry += grp_sum(ntri, Lg);
        ec0 += grp_sum(c00, Lg);
        ec1 += grp_sum(c01, Lg);
        ec2 += grp_sum(c10, Lg);
        ec3 += grp_sum(c11, Lg);
    }
    if (!EMIT && valid && sub == 0) rowCount[row] = make_uint2(triCarry, ec0);
}

// Resident CTAs per SM: the emit is latency-bound, so four CTAs (64 registers, a few spilled)
// beat three: whole-warp rows 0.89 -> 0.82 ms on a 664^3 grid, 4-lane rows 0.780 -> 0.750 ms.
template <bool EMIT, bool FULL>
__global__ void __launch_bounds__(256, 4) k_mc(QGrid g, const unsigned *__restrict__ sign,
                                            const unsigned char *__restrict__ codes, const float *__restrict__ lut,
                                            uint2 *__restrict__ rowCount, const uint2 *__restrict__ rowBase,
                                            unsigned *__restrict__ tri, unsigned long long *__restrict__ vkey,
                                            int lanes) {
    __shared__ unsigned long long s_tab[256];
    __shared__ float s_lut[256];
    __shared__ unsigned s_rec[EMIT ? 8 * 32 * kRecW : 1];  // per warp: one record per lane
    s_tab[threadIdx.x] = c_mc[threadIdx.x];
    if (EMIT) s_lut[threadIdx.x] = lut[threadIdx.x];
    __syncthreads();
    const int E = g.Gc + 1, Lg = FULL ? 32 : lanes;
    const long long first = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * (32 / Lg), nrow = (long long)E * E;
    if (first >= nrow) return;  // the whole warp
    const long long row = first + (threadIdx.x & 31) / Lg;
    mc_row<EMIT, FULL>(g, row, row < nrow, Lg, sign, codes, s_lut, s_tab, rowCount, rowBase, tri, vkey,
                       s_rec + (EMIT ? (threadIdx.x >> 5) * 32 * kRecW : 0));
}

// Batch form: rows are numbered molecule after molecule, so one scan over all rows gives
// every molecule's triangles and edge slots contiguous ranges in molecule order.  Each warp
// takes one unit of 32 / Lg rows of one molecule (units numbered by mc_unit_off).
// Four resident CTAs per SM (7.17 -> 5.68 ms for the emit of 256 molecules against two).
template <bool EMIT>
__global__ void __launch_bounds__(256, 4) k_mc_batch(QBatch b, const unsigned *__restrict__ sign,
                                                  const unsigned char *__restrict__ codes, uint2 *__restrict__ rowCount,
                                                  const uint2 *__restrict__ rowBase, unsigned *__restrict__ tri,
                                                  unsigned long long *__restrict__ vkey) {
    __shared__ unsigned long long s_tab[256];
    __shared__ unsigned s_rec[EMIT ? 8 * 32 * kRecW : 1];  // per warp: one record per lane
    s_tab[threadIdx.x] = c_mc[threadIdx.x];
    __syncthreads();
    unsigned *rec = s_rec + (EMIT ? (threadIdx.x >> 5) * 32 * kRecW : 0);
    const unsigned unit = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= __ldg(b.mc_unit_off + b.n_mol)) return;  // the whole warp
    const unsigned m = qses_find(b.mc_unit_off, b.n_mol, unit);
    const QMol &mol = b.mols[m];
    const QGrid g = mol.g;
    // the batch keeps the words-per-row width (narrow groups, as the single-molecule
    // launches use, measured slower here: emit 5.68 -> 6.12 ms on a 256-molecule batch)
    const int Lg = mc_lanes(g.Gc);
    const unsigned r0 = mol.row_off, nrow = (unsigned)(g.Gc + 1) * (unsigned)(g.Gc + 1);
    const unsigned row = (unit - __ldg(b.mc_unit_off + m)) * (32u / Lg) + (threadIdx.x & 31) / Lg;
    if (Lg == 32)  // warp-uniform
        mc_row<EMIT, true>(g, (long long)row, true, 32, sign + mol.mask_off, codes + mol.code_off,
                           b.lut + 256ull * m, s_tab, rowCount + r0, rowBase + r0, tri, vkey, rec);
    else
        mc_row<EMIT, false>(g, (long long)row, row < nrow, Lg, sign + mol.mask_off, codes + mol.code_off,
                            b.lut + 256ull * m, s_tab, rowCount + r0, rowBase + r0, tri, vkey, rec);
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
// corner remap 0.14 ms at 30 000 edges, 0.83 at 3 700 000, 24.1 at 138 000 000 (0.03, 0.20 and 6.6 so,
// 1.1 of the last the remap).  A warp sorting each bin of 8 to 32 in registers instead of the
// comparisons: 0.57 and 18.4.
constexpr int kWeldT = 1024;
constexpr unsigned kWeldCap = 4096;  // bins at most, of either sort
constexpr unsigned long long kWeldFirst = 1ull << 63;  // the first of equal keys: the vertex
constexpr unsigned kWeldX = 4096;       // x ranges of a layer at most: quanta, for voxels up to 4 A
// Quantised x of grid plane i, as edge_key has it for the edges in the plane.
__device__ __forceinline__ unsigned plane_quantum(const QGrid &g, int i) {
    float p = vox(i, g.dx, g.ox);
    if (g.off[0] | g.off[1] | g.off[2]) p = __fadd_rn(p, __fmul_rn((float)g.off[0], g.dx));
    return (unsigned)((long long)roundf(__fdiv_rn(p, QSES_WELD_TOL)) - g.bx);
}
// In place: exclusive sums of x[0, n), by the whole block; the total is returned.
template <int NT>
__device__ __forceinline__ unsigned block_excl_sums(unsigned *x, unsigned n, unsigned *s_tmp) {
    const unsigned per = (n + NT - 1) / NT, lo = min(threadIdx.x * per, n), hi = min(lo + per, n);
    unsigned sum = 0, total;
    for (unsigned k = lo; k < hi; k++) sum += x[k];
    unsigned run = block_excl_scan<NT>(sum, total, s_tmp);
    for (unsigned k = lo; k < hi; k++) {
        const unsigned c = x[k];
        x[k] = run;
        run += c;
    }
    __syncthreads();
    return total;
}

template <bool BATCH>
__global__ void __launch_bounds__(kWeldT, 2) k_weld(QGrid g1, QBatch b, unsigned cap,
                                                    const unsigned long long *__restrict__ vkey,
                                                    const uint2 *__restrict__ rowBase, unsigned ne, unsigned layers,
                                                    const unsigned *__restrict__ edge_off, unsigned long long *skey,
                                                    unsigned *sslot, unsigned *__restrict__ vmap,
                                                    float *__restrict__ vq, unsigned *__restrict__ vmol,
                                                    unsigned *__restrict__ vtx_off, uint2 *__restrict__ total,
                                                    unsigned long long *status, unsigned *ticket, int *err) {
    extern __shared__ unsigned s_bin[];  // 2 x (2 cap + 2) and kWeldX / 2
    __shared__ unsigned s_tmp[kWeldT / 32], s_tile, s_pushed, s_before;
    if (threadIdx.x == 0) {
        s_tile = atomicAdd(ticket, 1u);  // layers in the order CTAs start, so that every wait ends
        s_pushed = 0;
    }
    __syncthreads();
    const unsigned tile = s_tile, m = BATCH ? qses_find(b.layer_off, b.n_mol, tile) : 0u;
    const QGrid &g = BATCH ? b.mols[m].g : g1;
    const unsigned i = BATCH ? tile - __ldg(b.layer_off + m) : tile, E = (unsigned)g.Gc + 1;
    const uint2 *rows = rowBase + (BATCH ? b.mols[m].row_off : 0u);
    const unsigned s1 = rows[(size_t)i * E].y, s0 = i ? rows[(size_t)(i - 1) * E].y : s1;
    const unsigned s2 = i + 1 < E ? rows[(size_t)(i + 1) * E].y : BATCH ? __ldg(edge_off + m + 1) : ne;
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
    const unsigned n = block_excl_sums<kWeldT>(cur, nbin, s_tmp);
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
        const unsigned before = (unsigned)look_back(status, tile, distinct, err);
        if (threadIdx.x == 0) {
            s_before = before;
            if (BATCH && i == 0) vtx_off[m] = before;
            if (tile == layers - 1) {
                *total = make_uint2(before + distinct, 0u);
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
__global__ void k_remap(unsigned *__restrict__ tri, size_t n3, const unsigned *__restrict__ vmap) {
    const size_t q = 4 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (q + 4 <= n3) {
        uint4 t = *(const uint4 *)(tri + q);
        t.x = __ldg(vmap + t.x), t.y = __ldg(vmap + t.y), t.z = __ldg(vmap + t.z), t.w = __ldg(vmap + t.w);
        *(uint4 *)(tri + q) = t;
    } else {
        for (size_t e = q; e < n3; e++) tri[e] = vmap[tri[e]];
    }
}

// ------------------------------------------------------------ closest atom

__global__ void k_closest(QGrid g, const float *__restrict__ vq, unsigned nv, const float4 *__restrict__ atoms,
                          const uint2 *__restrict__ cells, const unsigned *__restrict__ sorted_to_input,
                          int *__restrict__ asorted, int *__restrict__ ainput) {
    unsigned v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    const float qx = vq[3ull * v], qy = vq[3ull * v + 1], qz = vq[3ull * v + 2];
    const int cx = __float2int_rz(__fdiv_rn(__fsub_rn(qx, g.ox), g.cell));
    const int cy = __float2int_rz(__fdiv_rn(__fsub_rn(qy, g.oy), g.cell));
    const int cz = __float2int_rz(__fdiv_rn(__fsub_rn(qz, g.oz), g.cell));
    int best = -1;
    float bestd = FLT_MAX;
    for (int a = -1; a <= 1; a++) {
        const int xx = min(max(cx + a, 0), g.gnb - 1);
        for (int b = -1; b <= 1; b++) {
            const int yy = min(max(cy + b, 0), g.gnb - 1);
            for (int d = -1; d <= 1; d++) {
                const int zz = min(max(cz + d, 0), g.gnb - 1);
                const uint2 rg = cells[((size_t)xx * g.gnb + yy) * g.gnb + zz];
                for (unsigned s = rg.x; s < rg.y; s++) {
                    const float4 at = atoms[s];
                    const float ex = __fsub_rn(at.x, qx), ey = __fsub_rn(at.y, qy), ez = __fsub_rn(at.z, qz);
                    const float d2 = __fmaf_rn(ez, ez, __fmaf_rn(ey, ey, __fmul_rn(ex, ex)));
                    if (d2 < bestd) {
                        bestd = d2;
                        best = (int)s;
                    }
                }
            }
        }
    }
    asorted[v] = best;
    ainput[v] = best >= 0 ? (int)sorted_to_input[best] : -1;
}

// Batch form: molecule from the vertex, atom ids local to the molecule.
__global__ void k_closest_batch(QBatch b, const float *__restrict__ vq, const unsigned *__restrict__ vmol,
                                unsigned nv, const float4 *__restrict__ atoms, const uint2 *__restrict__ cells,
                                const unsigned *__restrict__ sorted_to_input, int *__restrict__ asorted,
                                int *__restrict__ ainput) {
    unsigned v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    const QMol &mol = b.mols[vmol[v]];
    const QGrid g = mol.g;
    const uint2 *mcells = cells + mol.cell_off;
    const float qx = vq[3ull * v], qy = vq[3ull * v + 1], qz = vq[3ull * v + 2];
    const int cx = __float2int_rz(__fdiv_rn(__fsub_rn(qx, g.ox), g.cell));
    const int cy = __float2int_rz(__fdiv_rn(__fsub_rn(qy, g.oy), g.cell));
    const int cz = __float2int_rz(__fdiv_rn(__fsub_rn(qz, g.oz), g.cell));
    int best = -1;
    float bestd = FLT_MAX;
    for (int a = -1; a <= 1; a++) {
        const int xx = min(max(cx + a, 0), g.gnb - 1);
        for (int bb = -1; bb <= 1; bb++) {
            const int yy = min(max(cy + bb, 0), g.gnb - 1);
            for (int d = -1; d <= 1; d++) {
                const int zz = min(max(cz + d, 0), g.gnb - 1);
                const uint2 rg = mcells[((size_t)xx * g.gnb + yy) * g.gnb + zz];
                for (unsigned s = rg.x; s < rg.y; s++) {
                    const float4 at = atoms[s];
                    const float ex = __fsub_rn(at.x, qx), ey = __fsub_rn(at.y, qy), ez = __fsub_rn(at.z, qz);
                    const float d2 = __fmaf_rn(ez, ez, __fmaf_rn(ey, ey, __fmul_rn(ex, ex)));
                    if (d2 < bestd) {
                        bestd = d2;
                        best = (int)s;
                    }
                }
            }
        }
    }
    asorted[v] = best >= 0 ? best - (int)mol.atom_off : -1;
    ainput[v] = best >= 0 ? (int)sorted_to_input[best] - (int)mol.atom_off : -1;
}

// ------------------------------------------------------ degenerate filter

// Drops the triangles with a repeated corner in one pass: a block's 4096 triangles stay in
// registers, the kept ones go to shared memory in order and from there, behind those of the blocks
// before (look-back), to whole lines of `out`.  Batch: molecules flagged QSES_FLAG_KEEP_DEGENERATE
// keep every triangle, corners become molecule-local vertex ids and kept_off receives each
// molecule's first kept triangle.  Bound by memory, 24 B a triangle, and by the look-back that
// orders the blocks: 1024 triangles each took 2.7 ms for 277 000 000, 2048 2.1, 4096 1.9; a flag per
// triangle, a scan of the flags and a copy 5.2.  7 400 000: 0.19 -> 0.07 ms.
constexpr int kFiltT = 512, kFiltN = 8, kFiltTile = kFiltN * kFiltT;
template <bool BATCH>
__global__ void __launch_bounds__(kFiltT) k_tri_filter(QBatch b, const unsigned *__restrict__ tri, unsigned nt,
                                                       unsigned *__restrict__ out, unsigned *__restrict__ kept_off,
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
__global__ void k_csr_count(const unsigned *__restrict__ tri, size_t n3, uint2 *__restrict__ start) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n3) atomicAdd(&start[tri[q]].x, 1u);
}

__global__ void k_csr_scatter(const unsigned *__restrict__ tri, size_t n3, uint2 *__restrict__ start,
                              unsigned *__restrict__ occ) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n3) return;
    const unsigned v = tri[q];
    const unsigned k = atomicAdd(&start[v].y, 1u);
    occ[start[v].x + k] = (unsigned)q;
}

__global__ void k_to_float4(const float *__restrict__ v3, unsigned nv, float4 *__restrict__ v4) {
    unsigned v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < nv) v4[v] = make_float4(v3[3ull * v], v3[3ull * v + 1], v3[3ull * v + 2], 0.0f);
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
// Lanes per row of the single-molecule count and emit (the per-row totals do not depend on
// it, so the two may differ).  Narrow groups put more rows in flight per warp; measured on
// GB300 (count / emit ms): 664^3 grid 0.248 / 0.821 with whole-warp rows, 0.127 / 0.780
// with 2 / 4 lanes; 502^3 0.105 / 0.404 -> 0.074 / 0.370; 85^3 emit 0.029 -> 0.023 with 8.
static int mc_lanes_for(int Gc, bool emit) {
    const int Wc = (Gc + 32) / 32;
    if (Wc >= 8) return emit ? 4 : 2;
    return emit ? 8 : mc_lanes(Gc);
}
void launch_mc_count(const QGrid &g, const unsigned *sign, uint2 *rowCount, cudaStream_t s) {
    size_t rows = (size_t)(g.Gc + 1) * (g.Gc + 1);
    const int L = mc_lanes_for(g.Gc, false);
    if (L == 32)
        k_mc<false, true><<<nblk(rows, 8), 256, 0, s>>>(g, sign, nullptr, nullptr, rowCount, nullptr, nullptr,
                                                         nullptr, 32);
    else
        k_mc<false, false><<<nblk(rows, 8 * (32 / L)), 256, 0, s>>>(g, sign, nullptr, nullptr,
                                                                    rowCount, nullptr, nullptr, nullptr, L);
}
void launch_mc_emit(const QGrid &g, const unsigned *sign, const unsigned char *codes, const float *lut,
                    const uint2 *rowBase, unsigned *tri, unsigned long long *vkey, cudaStream_t s) {
    size_t rows = (size_t)(g.Gc + 1) * (g.Gc + 1);
    const int L = mc_lanes_for(g.Gc, true);
    if (L == 32)
        k_mc<true, true><<<nblk(rows, 8), 256, 0, s>>>(g, sign, codes, lut, nullptr, rowBase, tri, vkey, 32);
    else
        k_mc<true, false><<<nblk(rows, 8 * (32 / L)), 256, 0, s>>>(g, sign, codes, lut, nullptr,
                                                                   rowBase, tri, vkey, L);
}
void launch_mc_count_batch(const QBatch &b, unsigned units, const unsigned *sign, uint2 *rowCount, cudaStream_t s) {
    k_mc_batch<false><<<nblk(units, 8), 256, 0, s>>>(b, sign, nullptr, rowCount, nullptr, nullptr, nullptr);
}
void launch_mc_emit_batch(const QBatch &b, unsigned units, const unsigned *sign, const unsigned char *codes,
                          const uint2 *rowBase, unsigned *tri, unsigned long long *vkey, cudaStream_t s) {
    k_mc_batch<true><<<nblk(units, 8), 256, 0, s>>>(b, sign, codes, nullptr, rowBase, tri, vkey);
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
                                               vtx_off, total, (unsigned long long *)((char *)tmp + 256), (unsigned *)tmp, err);
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
void launch_gather_offsets(const uint2 *excl, const unsigned *at, unsigned n_mol, unsigned n, const uint2 *total,
                           unsigned *outx, unsigned *outy, cudaStream_t s) {
    k_gather_offsets<<<nblk(n_mol + 1, 256), 256, 0, s>>>(excl, at, n_mol, n, total, outx, outy);
}
void launch_closest_batch(const QBatch &b, const float *vq, const unsigned *vmol, unsigned nv, const float4 *atoms,
                          const uint2 *cells, const unsigned *sorted_to_input, int *asorted, int *ainput,
                          cudaStream_t s) {
    k_closest_batch<<<nblk(nv, 128), 128, 0, s>>>(b, vq, vmol, nv, atoms, cells, sorted_to_input, asorted, ainput);
}
void launch_remap(unsigned *tri, size_t n3, const unsigned *vmap, cudaStream_t s) {
    k_remap<<<nblk((n3 + 3) / 4, 256), 256, 0, s>>>(tri, n3, vmap);
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
void launch_csr_count(const unsigned *tri, size_t n3, uint2 *start, cudaStream_t s) {
    k_csr_count<<<nblk(n3, 256), 256, 0, s>>>(tri, n3, start);
}
void launch_csr_scatter(const unsigned *tri, size_t n3, uint2 *start, unsigned *occ, cudaStream_t s) {
    k_csr_scatter<<<nblk(n3, 256), 256, 0, s>>>(tri, n3, start, occ);
}
void launch_to_float4(const float *v3, unsigned nv, float4 *v4, cudaStream_t s) {
    k_to_float4<<<nblk(nv, 256), 256, 0, s>>>(v3, nv, v4);
}
void launch_from_float4(const float4 *v4, unsigned nv, float *v3, cudaStream_t s) {
    k_from_float4<<<nblk(nv, 256), 256, 0, s>>>(v4, nv, v3);
}
}  // namespace qses
