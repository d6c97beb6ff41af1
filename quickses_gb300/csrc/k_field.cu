// Atom grid and SES distance field.
//
//  k_atom_minmax  bbox + largest radius for the grid sizing (getMinMax, CudaSurf.cu:149-174)
//  k_atom_hash    (k_hash.cu) neighbour-cell key per atom
//  k_atom_gather  cell-sorted xyzr + cell start/end (sortCell, Kernels.cu:306-341)
//  k_sas          SAS classification, 8x8 rows x 32 voxels per CTA, atoms staged in shared
//                 memory, row intervals found analytically and verified with the exact
//                 per-voxel predicate (computeInOrOut / probeIntersection, Kernels.cu:344-475)
//  k_edt          probe refine as an exact windowed squared distance transform over the
//                 outside bitmask (distanceFieldRefine, Kernels.cu:478-545)
//
// Field values are stored as one byte per voxel: n in [0, 3R^2] is the squared voxel
// distance to the nearest outside voxel (value probe - dx*sqrt(n)), 253 = border voxel
// with no outside voxel in its window (-dx), 254 = inside (-dx), 255 = outside (probe).
#include "device_common.cuh"
#include "kernels.h"
#include "prims.h"

namespace qses {

// ---------------------------------------------------------------- atoms

__device__ __forceinline__ unsigned enc_f(float f) {
    unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// A coordinate or radius that is not a number bounds nothing, as on the host and in the reference.
// 200 000 atoms 5 us; with the atomics of every warp in global memory 26.
__global__ void k_atom_minmax(const float *__restrict__ xyz, const float *__restrict__ r, unsigned n,
                              unsigned *mm /* 7, zeroed: complements of min xyz; max xyz, max r (order-preserving encodings) */) {
    unsigned lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[4] = {0u, 0u, 0u, 0u};
    for (size_t a = (size_t)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += (size_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const float x = xyz[3 * a + c];
            if (x != x) continue;
            const unsigned e = enc_f(x);
            lo[c] = min(lo[c], e);
            hi[c] = max(hi[c], e);
        }
        const float rad = r[a];
        if (rad == rad) hi[3] = max(hi[3], enc_f(rad));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            lo[c] = min(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
            hi[c] = max(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
        }
        hi[3] = max(hi[3], __shfl_xor_sync(0xffffffffu, hi[3], o));
    }
    __shared__ unsigned s_mm[7];
    if (threadIdx.x < 7) s_mm[threadIdx.x] = 0u;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        for (int c = 0; c < 3; c++) {
            atomicMax(&s_mm[c], ~lo[c]);
            atomicMax(&s_mm[3 + c], hi[c]);
        }
        atomicMax(&s_mm[6], hi[3]);
    }
    __syncthreads();
    if (threadIdx.x < 7) atomicMax(&mm[threadIdx.x], s_mm[threadIdx.x]);
}

__global__ void k_atom_gather(const float *__restrict__ xyz, const float *__restrict__ r,
                              const unsigned *__restrict__ skey, const unsigned *__restrict__ sidx, unsigned n,
                              float4 *__restrict__ atoms, uint2 *__restrict__ cells) {
    unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    unsigned a = sidx[s];
    atoms[s] = make_float4(xyz[3 * a], xyz[3 * a + 1], xyz[3 * a + 2], r[a]);
    unsigned k = skey[s];
    if (s == 0 || skey[s - 1] != k) cells[k].x = s;
    if (s == n - 1 || skey[s + 1] != k) cells[k].y = s + 1;
}

cudaError_t order_atoms(const QGrid &g, const float *xyz, const float *r, unsigned n, unsigned *key, unsigned *key2,
                        unsigned *idx, unsigned *idx2, int bits, float4 *atoms, uint2 *cells, size_t ncell, void *tmp,
                        int *err, cudaStream_t s, int *launches, int *alt) {
    *alt = 0;
    cudaError_t e = cudaMemsetAsync(cells, 0, 8 * ncell, s);
    if (e != cudaSuccess) return e;
    // in one launch while its n^2 comparisons are cheaper than the launches it saves, and a key and an
    // atom's number fit 32 bits
    if (n <= kFewAtoms && ncell < 0xffffffffull / kFewAtoms) {
        launch_atoms_few(g, xyz, r, n, key, idx, atoms, cells, s);
        if (launches) (*launches)++;
        return cudaGetLastError();
    }
    launch_atom_hash(g, xyz, n, key, s);
    e = radix_sort(key, key2, idx, idx2, n, bits, true, tmp, err, s, launches, alt);
    if (e != cudaSuccess) return e;
    launch_atom_gather(xyz, r, *alt ? key2 : key, *alt ? idx2 : idx, n, atoms, cells, s);
    if (launches) *launches += 2;
    return cudaGetLastError();
}

// ------------------------------------------------------------------ SAS

// The SAS pass is bound by instruction issue (3 a cycle): the candidates of a tile and, per row and
// atom, the interval's ends.  664^3, 50 000 atoms: 0.56 ms with a cell per thread in the search and
// every interval verified, 0.46 without the intervals a row has already, 0.40 with half a column of
// cells per thread; 1738^3 5.1, 5.2 and 3.8; 85^3 0.040 and 0.031.  512 candidates (12 KB) let as many
// blocks run as the registers do; 768 take 0.50.
constexpr int kSasTX = 8, kSasTY = 8, kSasNT = kSasTX * kSasTY, kSasCap = 512;

// Exact per-voxel test along a z row: fma(ez, ez, sxy) < t with ez = z(k) - az.
__device__ __forceinline__ bool zpred(float k, float az, float sxy, float t, float dx, float oz) {
    const float ez = __fsub_rn(__fmaf_rn(k, dx, oz), az);
    return __fmaf_rn(ez, ez, sxy) < t;
}

__device__ __forceinline__ unsigned span_bits(int a, int b) {  // bits a..b inclusive, 0 <= a <= b <= 31
    return (0xffffffffu >> (31 - (b - a))) << a;
}

__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// A z row's voxels, bit k of a word each: grid indices k0 .. klim.
struct ZRow {
    int k0, klim;
    float dx, oz, inv_dx;
};
// Adds to `word` the voxels of a z row whose squared distance to the atom (kc: its z as a voxel
// index) is below t.  They are an interval (the predicate is monotone in |k - kc|); its ends are
// estimated in closed form, and if `word` has it already with a voxel more at either end, that is
// all.  Else the ends are verified with the exact predicate, with a brute-force fallback if the
// estimate does not verify (so the estimate's square root need not be correctly rounded: one
// approximate instruction).  The estimate is good to a voxel while the rounding of t is small beside
// a voxel's square: below 100 A, by far.
__device__ __forceinline__ void add_zmask(unsigned &word, float az, float kc, float sxy, float t, const ZRow &z) {
    const float h = sqrt_approx(fmaxf(t - sxy, 0.0f)) * z.inv_dx;
    const float k0 = (float)z.k0, klim = (float)z.klim;
    const float lo = fmaxf(ceilf(kc - h), k0), hi = fminf(floorf(kc + h), klim);
    const int a = (int)lo - z.k0, b = (int)hi - z.k0;
    const int wa = max(a - 1, 0), wb = min(b + 1, z.klim - z.k0);
    if (t < 10000.0f) {
        if (wa > wb) return;
        const unsigned wide = span_bits(wa, wb);
        if ((word & wide) == wide) return;
    }
    auto at = [&](float k) { return zpred(k, az, sxy, t, z.dx, z.oz); };
    if (lo <= hi) {
        if (at(lo) & at(hi) & (lo == k0 || !at(lo - 1.0f)) & (hi == klim || !at(hi + 1.0f))) {
            word |= span_bits(a, b);
            return;
        }
    } else {
        const float c = fminf(fmaxf(rintf(kc), k0), klim);
        if (!at(c) & (c == k0 || !at(c - 1.0f)) & (c == klim || !at(c + 1.0f))) return;
    }
    for (int k = z.k0; k <= z.klim; k++)
        if (at((float)k)) word |= 1u << (k - z.k0);
}

// Row-interval classification of one z row against one atom (kc: its z as a voxel index).
__device__ __forceinline__ void sas_row_atom(float px, float py, const float4 &a, float tin, float kc, const ZRow &z,
                                             unsigned full, unsigned &sasw, unsigned &inw) {  // a.w: tsas
    const float ex = __fsub_rn(px, a.x), ey = __fsub_rn(py, a.y);
    const float sxy = __fmaf_rn(ey, ey, __fmul_rn(ex, ex));
    if (sxy < a.w && sasw != full) add_zmask(sasw, a.z, kc, sxy, a.w, z);
    if (sxy < tin && inw != full) add_zmask(inw, a.z, kc, sxy, tin, z);
}
__device__ __forceinline__ float voxel_index(float z, float oz, float inv_dx) {
    return fminf(fmaxf((z - oz) * inv_dx, -1.0e6f), 1.0e6f);
}

__device__ __forceinline__ void atom_thresholds(float r, const QGrid &g, float &tin, float &tsas) {
    float rin = __fsub_rn(r, g.dx);                        // d < r - dx  (Kernels.cu:377)
    tin = rin > 0.0f ? __fmul_rn(rin, rin) : -1.0f;
    float rs = __fadd_rn(g.probe, r);                      // d < probe + r  (Kernels.cu:380)
    tsas = __fmul_rn(rs, rs);
}

// One SAS tile: z-word w of the 8 x 8 rows starting at (i0, j0) = (8 ib, 8 jb), SPLIT threads to a row
// that share its candidates out.
template <int SPLIT>
__device__ __forceinline__ void sas_tile(const QGrid &g, int w, int jb, int ib, const float4 *__restrict__ atoms,
                                         const uint2 *__restrict__ cells, unsigned *__restrict__ inMask,
                                         unsigned *__restrict__ outMask) {
    __shared__ float4 s_a[kSasCap];  // x, y, z, threshold of probe + r
    __shared__ float2 s_t[kSasCap];  // threshold of r - dx, z as a voxel index
    __shared__ int s_n;
    const int j0 = jb * kSasTY, i0 = ib * kSasTX;
    constexpr int NT = kSasNT * SPLIT;
    const int t = threadIdx.x, row = t / SPLIT, i = i0 + row / kSasTY, j = j0 + row % kSasTY, k0 = w * 32;
    // Voxels with an index >= lim on an axis are never computed and stay outside: the last
    // layer G-1 (Kernels.cu:436-441) and, for a slice box, its own last layer and whatever
    // lies at or past the molecule grid's last layer.  Positions use the grid index
    // box index + off (gridToSpace of ijkOffset, Kernels.cu:427-446).
    const int G = g.G, lastx = g.lim[0] - 1, lasty = g.lim[1] - 1, lastz = g.lim[2] - 1;
    const int oi = g.off[0], oj = g.off[1], ok = g.off[2];
    const unsigned valid = (k0 + 32 <= G) ? 0xffffffffu : ((1u << (G - k0)) - 1u);
    const int fz = max(g.lim[2] - k0, 0);  // first forced-outside bit of this word
    const unsigned forced = fz >= 32 ? 0u : (valid & ~((1u << fz) - 1u));
    const int klim = min(k0 + 31, lastz);
    const float inv_dx = 1.0f / g.dx;
    unsigned sasw = 0, inw = 0;

    if (i0 <= lastx && j0 <= lasty && k0 <= lastz) {
        const float bx0 = vox(i0 + oi, g.dx, g.ox), bx1 = vox(min(i0 + kSasTX - 1, lastx) + oi, g.dx, g.ox);
        const float by0 = vox(j0 + oj, g.dx, g.oy), by1 = vox(min(j0 + kSasTY - 1, lasty) + oj, g.dx, g.oy);
        const float bz0 = vox(k0 + ok, g.dx, g.oz), bz1 = vox(klim + ok, g.dx, g.oz);
        const float ext = g.cell * 1.01f + g.dx;
        auto crange = [&](float lo, float hi, float o, int &c0, int &c1) {
            c0 = min(max((int)floorf((lo - ext - o) / g.cell), 0), g.gnb - 1);
            c1 = min(max((int)floorf((hi + ext - o) / g.cell), 0), g.gnb - 1);
        };
        int cx0, cx1, cy0, cy1, cz0, cz1;
        crange(bx0, bx1, g.ox, cx0, cx1);
        crange(by0, by1, g.oy, cy0, cy1);
        crange(bz0, bz1, g.oz, cz0, cz1);
        const int ncy = cy1 - cy0 + 1, ncz = cz1 - cz0 + 1, ncol = (cx1 - cx0 + 1) * ncy;
        // Stage every atom whose probe-inflated sphere can reach the tile (conservative box test).  A
        // thread takes half a column of cells, whose atoms are one run (an empty cell is (0, 0)).
        auto run = [&](int c) {
            const int cx = (c >> 1) / ncy, cy = (c >> 1) - cx * ncy;
            const int z0 = cz0 + (c & 1 ? ncz / 2 : 0), z1 = c & 1 ? cz1 + 1 : cz0 + ncz / 2;
            const uint2 *col = cells + ((size_t)(cx0 + cx) * g.gnb + (cy0 + cy)) * g.gnb;
            uint2 r = make_uint2(0xffffffffu, 0u);
            for (int z = z0; z < z1; z++) {
                const uint2 rg = __ldg(col + z);
                if (rg.y) r.x = min(r.x, rg.x);
                r.y = max(r.y, rg.y);
            }
            return r;
        };
        auto stage = [&](unsigned s) {
            const float4 a = __ldg(atoms + s);
            const float ddx = fmaxf(fmaxf(bx0 - a.x, a.x - bx1), 0.0f);
            const float ddy = fmaxf(fmaxf(by0 - a.y, a.y - by1), 0.0f);
            const float ddz = fmaxf(fmaxf(bz0 - a.z, a.z - bz1), 0.0f);
            const float rs = g.probe + a.w;
            if (!(ddx * ddx + ddy * ddy + ddz * ddz <= rs * rs * 1.001f + 1e-3f)) return;
            const int q = atomicAdd(&s_n, 1);
            if (q >= kSasCap) return;
            float tin, tsas;
            atom_thresholds(a.w, g, tin, tsas);
            s_a[q] = make_float4(a.x, a.y, a.z, tsas);
            s_t[q] = make_float2(tin, voxel_index(a.z, g.oz, inv_dx));
        };
        const float px = vox(i + oi, g.dx, g.ox), py = vox(j + oj, g.dx, g.oy);
        const ZRow z{k0 + ok, klim + ok, g.dx, g.oz, inv_dx};  // z range as grid indices
        const unsigned full = span_bits(0, klim - k0);
        auto classify = [&](int na) {
            if (i > lastx || j > lasty) return;
            for (int q = t % SPLIT; q < na; q += SPLIT) {
                const float2 u = s_t[q];
                sas_row_atom(px, py, s_a[q], u.x, u.y, z, full, sasw, inw);
            }
        };
        if (t == 0) s_n = 0;
        __syncthreads();
        for (int c = t; c < 2 * ncol; c += NT) {
            const uint2 r = run(c);
            for (unsigned s = r.x; s < r.y; s++) stage(s);
        }
        __syncthreads();
        if (s_n <= kSasCap) {
            classify(s_n);
        } else {
            // More than fit (crowded atoms, coarse voxels): all threads run through the columns
            // together and classify whenever there may be no room for another round.
            for (int c = 0; c < 2 * ncol; c++) {
                const uint2 r = run(c);
                for (unsigned s = r.x; s < r.y; s += NT) {
                    __syncthreads();
                    const int n = s_n > kSasCap ? 0 : s_n;  // the first round starts over
                    const bool flush = n > kSasCap - NT;
                    if (flush) classify(n);
                    __syncthreads();
                    if (t == 0) s_n = flush ? 0 : n;
                    __syncthreads();
                    if (s + t < r.y) stage(s + t);
                }
            }
            __syncthreads();
            classify(s_n);
        }
    }
#pragma unroll
    for (int o = 1; o < SPLIT; o <<= 1) {
        sasw |= __shfl_xor_sync(0xffffffffu, sasw, o);
        inw |= __shfl_xor_sync(0xffffffffu, inw, o);
    }
    if (i < G && j < G && t % SPLIT == 0) {
        unsigned outw, inw2;
        if (i > lastx || j > lasty) {
            outw = valid;
            inw2 = 0u;
        } else {
            outw = (~sasw & valid) | forced;
            inw2 = inw & ~forced;
        }
        size_t idx = ((size_t)i * G + j) * g.W + w;
        inMask[idx] = inw2;
        outMask[idx] = outw;
    }
}

template <int SPLIT>
__global__ void __launch_bounds__(kSasNT * SPLIT) k_sas(QGrid g, const float4 *__restrict__ atoms,
                                                const uint2 *__restrict__ cells, unsigned *__restrict__ inMask,
                                                unsigned *__restrict__ outMask) {
    sas_tile<SPLIT>(g, blockIdx.x, blockIdx.y, blockIdx.z, atoms, cells, inMask, outMask);
}

// ------------------------------------------------------------------ refine

constexpr int kEdtNT = 256;

// One refine tile: z-word w of the TX x TY rows starting at (TX ib, TY jb), with an R halo.
// Larger tiles re-read less halo per row (the z pass runs on (TX+2R)(TY+2R) rows for TX TY
// output rows) at the cost of shared memory (dynamic, edt_layout); the shape is chosen
// by the autotuner.
//
// Bound by instruction issue where there is a border, by the codes' bytes elsewhere.  664^3 (R = 7)
// 0.61 ms, 1738^3 (R = 3, most tiles without a border) 4.6.  With the z distances of all voxels in
// memory, written and read back with the halo, 0.67 and 7.6; with byte rows spread at each tap, taps
// one by one and codes voxel by voxel 0.83 and 7.6.

// Min-plus without the byte-SIMD add and min, which this GPU runs as several instructions each:
// four byte distances (255 = none) are spread over two words of 16-bit halves (one byte permute
// each), where the 16-bit add and min are one instruction, and stay so through the y and x passes.
// Real distances stay below 255 (y <= 2 R^2 = 162, x <= 3 R^2 = 243) and "none" at or above
// it; the taps at distance 0 bring it back to 255.
__device__ __forceinline__ unsigned spread_lo(unsigned w) { return __byte_perm(w, 0u, 0x4140); }  // bytes 0, 1
__device__ __forceinline__ unsigned spread_hi(unsigned w) { return __byte_perm(w, 0u, 0x4342); }  // bytes 2, 3
// The y pass of a tile: squared distances in the (y, z) plane, 8 voxels of a halo row's output at a
// time, from the z distances of its 2R + 1 neighbours, two at the same distance together.
__device__ __forceinline__ uint4 y_taps(const uint2 *g, int stride, int R) {  // g: of the row itself
    const uint2 c = g[0];
    uint4 v = make_uint4(spread_lo(c.x), spread_hi(c.x), spread_lo(c.y), spread_hi(c.y));
    unsigned d2 = 0x00010001u;
    for (int d = 1; d <= R; d++) {
        const uint2 m = g[-d * stride], p = g[d * stride];
        v.x = __vminu2(v.x, __vminu2(spread_lo(m.x), spread_lo(p.x)) + d2);
        v.y = __vminu2(v.y, __vminu2(spread_hi(m.x), spread_hi(p.x)) + d2);
        v.z = __vminu2(v.z, __vminu2(spread_lo(m.y), spread_lo(p.y)) + d2);
        v.w = __vminu2(v.w, __vminu2(spread_hi(m.y), spread_hi(p.y)) + d2);
        d2 += (unsigned)(2 * d + 1) * 0x00010001u;
    }
    return v;
}
// The x pass, the same over the y pass's rows.
__device__ __forceinline__ uint4 x_taps(const uint4 *h, int stride, int R) {
    uint4 v = h[0];
    unsigned d2 = 0x00010001u;
    for (int d = 1; d <= R; d++) {
        const uint4 m = h[-d * stride], p = h[d * stride];
        v.x = __vminu2(v.x, __vminu2(m.x, p.x) + d2);
        v.y = __vminu2(v.y, __vminu2(m.y, p.y) + d2);
        v.z = __vminu2(v.z, __vminu2(m.z, p.z) + d2);
        v.w = __vminu2(v.w, __vminu2(m.w, p.w) + d2);
        d2 += (unsigned)(2 * d + 1) * 0x00010001u;
    }
    return v;
}
// Voxels (4 bits) of two words of halves that are at or above a threshold (below: 0x8000 less it).
__device__ __forceinline__ unsigned at_least(unsigned lo, unsigned hi, unsigned below) {
    const unsigned a = (lo + below) & 0x80008000u, b = (hi + below) & 0x80008000u;
    return (a >> 15 & 1u) | (a >> 30) | (b >> 13 & 4u) | (b >> 28);
}

__device__ __forceinline__ unsigned nibble_bytes(unsigned nib) {  // 4 bits -> 0xff in each set bit's byte
    return ((nib * 0x00204081u) & 0x01010101u) * 0xffu;           // copies at bits 0, 7, 14, 21: no carries
}
// Squared z distances of one 32-voxel word c (bit = outside voxel) with its neighbouring
// words a (below) and d (above), one byte per voxel (<= R^2, 255 = none), four per output
// word.  Bit-parallel: the outside set grows by one voxel per step (two funnel shifts over
// the neighbouring words), and the voxels first covered at step k are at distance k.  The distances
// are collected as bit planes; four voxels' planes make a selector, and one byte permute looks up
// their squares (FAR: two, for distances above 6): some 100 instructions a word; writing the squares
// into the bytes step by step took 350.
template <bool FAR>
__device__ __forceinline__ void z_planes(unsigned a, unsigned c, unsigned d, int R, unsigned out[8]) {
    unsigned cov = c, p[4] = {0u, 0u, 0u, 0u};  // voxels with an outside voxel within k; bits of k
#pragma unroll
    for (int k = 1; k <= (FAR ? QSES_RMAX : 6); k++) {
        if (k > R) break;
        // bit b of the right funnel shift is voxel b + k, of the left one voxel b - k
        const unsigned nc = cov | __funnelshift_r(c, d, k) | __funnelshift_l(a, c, k);
        const unsigned nw = nc & ~cov;  // nearest outside voxel at distance k
        cov = nc;
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (k >> q & 1) p[q] |= nw;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) p[q] |= ~cov;  // none: 15, or 7 of the three planes
    // per four voxels the planes' nibbles side by side, even and odd groups; a 4 x 4 bit transpose
    // (two delta swaps, two groups at a time) turns them into the voxels' selectors
    const unsigned n = 0x0f0f0f0fu;
    const unsigned e01 = (p[0] & n) | ((p[1] & n) << 4), o01 = ((p[0] >> 4) & n) | (p[1] & ~n);
    const unsigned e23 = (p[2] & n) | (FAR ? (p[3] & n) << 4 : 0u), o23 = ((p[2] >> 4) & n) | (FAR ? p[3] & ~n : 0u);
#pragma unroll
    for (int j = 0; j < 4; j++) {  // voxels 8 j .. 8 j + 7
        const unsigned pick = (unsigned)j | (unsigned)(4 + j) << 4;
        unsigned x = __byte_perm(e01, e23, pick) & 0xffffu;
        x |= __byte_perm(o01, o23, pick) << 16;
        unsigned t = (x ^ (x >> 3)) & 0x0a0a0a0au;
        x ^= t ^ (t << 3);
        t = (x ^ (x >> 6)) & 0x00cc00ccu;
        x ^= t ^ (t << 6);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const unsigned sel = (h ? x >> 16 : x) & (FAR ? 0x7777u : 0xffffu);
            if (FAR) {
                const unsigned m = nibble_bytes((p[3] >> (8 * j + 4 * h)) & 0xfu);
                out[2 * j + h] = (__byte_perm(0x09040100u, 0x31241910u, sel) & ~m) |
                                 (__byte_perm(0x00005140u, 0xff000000u, sel) & m);
            } else {
                out[2 * j + h] = __byte_perm(0x09040100u, 0xff241910u, sel);
            }
        }
    }
}
__device__ __forceinline__ void z_word(unsigned a, unsigned c, unsigned d, int R, unsigned out[8]) {
    if ((a | c | d) == 0u || c == 0xffffffffu) {  // no outside voxel within 32, or all outside
#pragma unroll
        for (int k = 0; k < 8; k++) out[k] = c ? 0u : 0xffffffffu;
        return;
    }
    if (R <= 6)
        z_planes<false>(a, c, d, R, out);
    else
        z_planes<true>(a, c, d, R, out);
}

// Shared-memory layout of one refine tile for a window of R voxels: the halo rows' z distances, the
// y-pass rows, and the tile's in/out words.  Sized per launch, so a smaller window (a larger voxel)
// fits more CTAs per SM; the largest layout (R = QSES_RMAX) bounds every other.
struct EdtLayout {
    size_t h_off, in_off, ot_off, bytes;
};
__host__ __device__ __forceinline__ EdtLayout edt_layout(int TX, int TY, int R) {
    const size_t HX = (size_t)TX + 2 * R, HY = (size_t)TY + 2 * R;
    EdtLayout L;
    L.h_off = 32 * HX * HY;                     // [HX HY][32] z distances first
    L.in_off = L.h_off + 64 * HX * (size_t)TY;  // [HX][TY][32] y-pass rows, 16 bits
    L.ot_off = L.in_off + 4 * (size_t)TX * TY;
    L.bytes = L.ot_off + 4 * (size_t)TX * TY;
    return L;
}

template <int TX, int TY>
__device__ __forceinline__ void edt_tile(const QGrid &g, int w, int jb, int ib, const unsigned *__restrict__ inMask,
                                         const unsigned *__restrict__ outMask, unsigned char *__restrict__ codes,
                                         unsigned *__restrict__ signMask) {
    const EdtLayout L = edt_layout(TX, TY, g.R);
    extern __shared__ __align__(16) unsigned char edt_smem[];
    // squared z distances, one byte per voxel (255 = none)
    unsigned char (*s_g)[32] = reinterpret_cast<unsigned char (*)[32]>(edt_smem);
    uint4 *s_h = reinterpret_cast<uint4 *>(edt_smem + L.h_off);  // [HX][TY][4]
    unsigned *s_in = reinterpret_cast<unsigned *>(edt_smem + L.in_off);
    unsigned *s_ot = reinterpret_cast<unsigned *>(edt_smem + L.ot_off);
    const int j0 = jb * TY, i0 = ib * TX;
    const int R = g.R, G = g.G, W = g.W, t = threadIdx.x;
    const int HX = TX + 2 * R, HY = TY + 2 * R, k0 = w * 32;
    const unsigned valid = (k0 + 32 <= G) ? 0xffffffffu : ((1u << (G - k0)) - 1u);

    int anyb = 0;
    for (int q = t; q < TX * TY; q += kEdtNT) {
        int i = i0 + q / TY, j = j0 + q % TY;
        unsigned iw = 0u, ow = 0xffffffffu;
        if (i < G && j < G) {
            size_t idx = ((size_t)i * G + j) * W + w;
            iw = inMask[idx];
            ow = outMask[idx];
            anyb |= (valid & ~iw & ~ow) != 0u;
        }
        s_in[q] = iw;
        s_ot[q] = ow;
    }
    const int has_border = __syncthreads_or(anyb);
    int has_out = 0;
    if (has_border) {
        // z: squared distance (in voxels, <= R^2) to the nearest outside voxel along the row, a halo
        // row's 32 voxels per thread
        int any = 0;
        for (int q = t; q < HX * HY; q += kEdtNT) {
            const int i = i0 - R + q / HY, j = j0 - R + q % HY;
            unsigned a = 0u, c = 0u, d = 0u, out[8];
            if (i >= 0 && i < G && j >= 0 && j < G) {
                const unsigned *m = outMask + ((size_t)i * G + j) * W + w;
                if (w > 0) a = __ldg(m - 1);
                c = __ldg(m);
                if (w + 1 < W) d = __ldg(m + 1);
            }
            any |= (a | c | d) != 0u;
            z_word(a, c, d, R, out);
            uint4 *dst = reinterpret_cast<uint4 *>(s_g[q]);
            dst[0] = make_uint4(out[0], out[1], out[2], out[3]);
            dst[1] = make_uint4(out[4], out[5], out[6], out[7]);
        }
        has_out = __syncthreads_or(any);
    }
    if (has_border && has_out) {
        for (int q = t; q < HX * TY * 4; q += kEdtNT) {
            const int w8 = q & 3, y = (q >> 2) % TY, hx = (q >> 2) / TY;
            s_h[(hx * TY + y) * 4 + w8] = y_taps(reinterpret_cast<const uint2 *>(s_g[hx * HY + y + R]) + w8, 4, R);
        }
        __syncthreads();
    }
    // x: min over di of di^2 + h, then codes and sign bits; 4 threads per row, 8 voxels each
    // (TX TY / 64 rows per thread: the same trip count in every warp).
    for (int row = t >> 2; row < TX * TY; row += kEdtNT / 4) {
    const int part = t & 3, x = row / TY, y = row % TY, i = i0 + x, j = j0 + y;
    unsigned sgn = 0u;
    if (i < G && j < G) {
        const unsigned iw = s_in[row], ow = s_ot[row];
        // this thread's 8 voxels: squared distances where they are neither inside nor outside
        const unsigned o8 = ((ow | ~valid) >> (8 * part)) & 0xffu, i8 = (iw >> (8 * part)) & 0xffu & ~o8;
        uint4 v = make_uint4(0x00ff00ffu, 0x00ff00ffu, 0x00ff00ffu, 0x00ff00ffu);
        if (has_out) v = x_taps(s_h + ((x + R) * TY + y) * 4 + part, 4 * TY, R);
        const unsigned none = (unsigned)QSES_CODE_NONE * 0x00010001u;  // above every distance, below 255
        v.x = __vminu2(v.x, none), v.y = __vminu2(v.y, none), v.z = __vminu2(v.z, none), v.w = __vminu2(v.w, none);
        const unsigned below = (0x8000u - (unsigned)g.negmin) * 0x00010001u;
        sgn = ((at_least(v.x, v.y, below) | at_least(v.z, v.w, below) << 4 | i8) & ~o8) << (8 * part);
        auto codes4 = [&](unsigned lo, unsigned hi, unsigned o, unsigned in) {
            const unsigned om = nibble_bytes(o), im = nibble_bytes(in);  // IN = 254, OUT = 255
            return (__byte_perm(lo, hi, 0x6420) | om | im) & ~(im & 0x01010101u);
        };
        *(uint2 *)(codes + ((size_t)i * G + j) * g.Gp + k0 + part * 8) =
            make_uint2(codes4(v.x, v.y, o8 & 15u, i8 & 15u), codes4(v.z, v.w, o8 >> 4, i8 >> 4));
    }
    sgn |= __shfl_xor_sync(0xffffffffu, sgn, 1);
    sgn |= __shfl_xor_sync(0xffffffffu, sgn, 2);
    if (part == 0 && i < G && j < G) signMask[((size_t)i * G + j) * W + w] = sgn;
    }
}

// Four blocks an SM: with five (48 registers, as many as fit) 1738^3 takes 6.1 ms for 4.6, for more
// of them write their rows of codes at once.
template <int TX, int TY>
__global__ void __launch_bounds__(kEdtNT, 4) k_edt(QGrid g, const unsigned *__restrict__ inMask,
                                                const unsigned *__restrict__ outMask,
                                                unsigned char *__restrict__ codes, unsigned *__restrict__ signMask) {
    edt_tile<TX, TY>(g, blockIdx.x, blockIdx.y, blockIdx.z, inMask, outMask, codes, signMask);
}

// ------------------------------------------------------------ batched field

// Persistent CTAs take field tiles of every molecule of a batch from one work counter.
// A tile is decoded within its molecule exactly as the single-molecule grid would index it.
__device__ __forceinline__ bool next_tile(const QBatch &b, unsigned *counter, unsigned &m, int &w, int &jb, int &ib) {
    __shared__ unsigned s_item, s_m;
    __syncthreads();  // the previous tile's shared memory is no longer in use
    if (threadIdx.x == 0) {
        const unsigned it = atomicAdd(counter, 1u);
        s_item = it;
        s_m = it < __ldg(b.tile_off + b.n_mol) ? qses_find(b.tile_off, b.n_mol, it) : 0xffffffffu;
    }
    __syncthreads();
    m = s_m;
    if (m == 0xffffffffu) return false;
    const QGrid &g = b.mols[m].g;
    const unsigned loc = s_item - __ldg(b.tile_off + m), ny = (unsigned)(g.G + 7) / 8u;
    w = (int)(loc % (unsigned)g.W);
    jb = (int)((loc / (unsigned)g.W) % ny);
    ib = (int)(loc / ((unsigned)g.W * ny));
    return true;
}

__global__ void __launch_bounds__(kSasNT) k_sas_batch(QBatch b, const float4 *__restrict__ atoms,
                                                      const uint2 *__restrict__ cells, unsigned *__restrict__ inMask,
                                                      unsigned *__restrict__ outMask, unsigned *counter) {
    unsigned m;
    int w, jb, ib;
    while (next_tile(b, counter, m, w, jb, ib)) {
        const QMol mol = b.mols[m];
        sas_tile<1>(mol.g, w, jb, ib, atoms, cells + mol.cell_off, inMask + mol.mask_off, outMask + mol.mask_off);
    }
}

__global__ void __launch_bounds__(kEdtNT) k_edt_batch(QBatch b, const unsigned *__restrict__ inMask,
                                                      const unsigned *__restrict__ outMask,
                                                      unsigned char *__restrict__ codes,
                                                      unsigned *__restrict__ signMask, unsigned *counter) {
    unsigned m;
    int w, jb, ib;
    while (next_tile(b, counter, m, w, jb, ib)) {
        const QMol mol = b.mols[m];
        edt_tile<8, 8>(mol.g, w, jb, ib, inMask + mol.mask_off, outMask + mol.mask_off, codes + mol.code_off,
                       signMask + mol.mask_off);
    }
}

// ------------------------------------------------------------ launchers

void launch_atom_minmax(const float *xyz, const float *r, unsigned n, unsigned *mm, cudaStream_t s) {
    unsigned blocks = (n + 255) / 256;
    if (blocks > 608) blocks = 608;
    if (blocks == 0) blocks = 1;
    k_atom_minmax<<<blocks, 256, 0, s>>>(xyz, r, n, mm);
}
void launch_atom_gather(const float *xyz, const float *r, const unsigned *skey, const unsigned *sidx, unsigned n,
                        float4 *atoms, uint2 *cells, cudaStream_t s) {
    k_atom_gather<<<(n + 255) / 256, 256, 0, s>>>(xyz, r, skey, sidx, n, atoms, cells);
}
void launch_sas(const QGrid &g, const float4 *atoms, const uint2 *cells, unsigned *inMask, unsigned *outMask,
                cudaStream_t s) {
    const dim3 grid(g.W, (g.G + kSasTY - 1) / kSasTY, (g.G + kSasTX - 1) / kSasTX);
    // Small grids have a few blocks to an SM, and the time is a row's walk through its candidates:
    // 85^3 (363 tiles) 31 us with a thread to a row, 25, 19 and 16 with 2, 4 and 8.  From some thousand
    // tiles on all SMs are busy, and the shared rows verify more intervals: 171^3 (2 904 tiles) 28 us
    // with 1, 34 with 4; 301^3 57 and 102.
    if ((unsigned long long)grid.x * grid.y * grid.z <= 1000u)
        k_sas<8><<<grid, 8 * kSasNT, 0, s>>>(g, atoms, cells, inMask, outMask);
    else
        k_sas<1><<<grid, kSasNT, 0, s>>>(g, atoms, cells, inMask, outMask);
}
template <int TX, int TY>
static void launch_edt_shape(const QGrid &g, const unsigned *inMask, const unsigned *outMask, unsigned char *codes,
                             unsigned *signMask, cudaStream_t s) {
    static const bool attr = [] {
        return cudaFuncSetAttribute((const void *)k_edt<TX, TY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)edt_layout(TX, TY, QSES_RMAX).bytes) == cudaSuccess;
    }();
    (void)attr;
    const size_t smem = edt_layout(TX, TY, g.R).bytes;
    dim3 grid(g.W, (g.G + TY - 1) / TY, (g.G + TX - 1) / TX);
    k_edt<TX, TY><<<grid, kEdtNT, smem, s>>>(g, inMask, outMask, codes, signMask);
}

void launch_edt(const QGrid &g, const unsigned *inMask, const unsigned *outMask, unsigned char *codes,
                unsigned *signMask, cudaStream_t s, int shape) {
    // shape 0: 8 x 8 rows, 1: 16 x 8, 2: 16 x 16, 3: 32 x 16 (shared memory per CTA at R = 7: 27, 38,
    // 62 and 95 KB)
    switch (shape) {
        case 3: launch_edt_shape<32, 16>(g, inMask, outMask, codes, signMask, s); break;
        case 2: launch_edt_shape<16, 16>(g, inMask, outMask, codes, signMask, s); break;
        case 1: launch_edt_shape<16, 8>(g, inMask, outMask, codes, signMask, s); break;
        default: launch_edt_shape<8, 8>(g, inMask, outMask, codes, signMask, s); break;
    }
}
static unsigned persistent_blocks(const void *fn, int threads, unsigned items, size_t smem = 0) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
    unsigned blocks = (unsigned)(sms * (per_sm > 0 ? per_sm : 1));
    return items < blocks ? (items ? items : 1u) : blocks;
}
void launch_sas_batch(const QBatch &b, unsigned tiles, const float4 *atoms, const uint2 *cells, unsigned *inMask,
                      unsigned *outMask, unsigned *counter, cudaStream_t s) {
    k_sas_batch<<<persistent_blocks((const void *)k_sas_batch, kSasNT, tiles), kSasNT, 0, s>>>(
        b, atoms, cells, inMask, outMask, counter);
}
void launch_edt_batch(const QBatch &b, unsigned tiles, const unsigned *inMask, const unsigned *outMask,
                      unsigned char *codes, unsigned *signMask, unsigned *counter, cudaStream_t s) {
    const size_t smem = edt_layout(8, 8, QSES_RMAX).bytes;  // molecules of any window
    k_edt_batch<<<persistent_blocks((const void *)k_edt_batch, kEdtNT, tiles, smem), kEdtNT, smem, s>>>(
        b, inMask, outMask, codes, signMask, counter);
}

}  // namespace qses
