// Decoupled look-back scan and onesweep radix sort (Merrill & Garland 2016;
// Adinets & Merrill 2022), written for this project.
//
// The radix sort replaces QuickSES's thrust::sort calls (CudaSurf.cu:610-612 for the atom
// cell keys, :444-447 for the weld): one histogram kernel computes every digit's counts,
// then one kernel per 8-bit digit ranks a tile of keys in shared memory (warp match +
// per-warp digit counters, so equal digits keep input order), obtains the tile's global
// digit offsets through a decoupled look-back and scatters.  The look-back waits are
// bounded (QSES_ERR_TIMEOUT) and every scatter is bounds-checked.
#include "device_common.cuh"
#include "prims.h"

namespace qses {

// ------------------------------------------------------------------ scan
// A warp's 512 items are 8 rounds of 32 lanes x 2, so that loads and stores are whole lines.
// 3 540 000 items take 21 us, 25 us less than with a thread's 16 items one after the other and one
// lane looking back.
constexpr int kScanT = 256, kScanR = 8, kScanTile = kScanT * 2 * kScanR;

__device__ __forceinline__ unsigned long long pack31(uint2 v) {
    return (unsigned long long)(v.x & 0x7fffffffu) | ((unsigned long long)(v.y & 0x7fffffffu) << 31);
}
__device__ __forceinline__ uint2 unpack31(unsigned long long s) {
    return make_uint2((unsigned)(s & 0x7fffffffull), (unsigned)((s >> 31) & 0x7fffffffull));
}

__global__ void __launch_bounds__(kScanT) k_scan_u2(const uint2 *in, uint2 *out, unsigned n,
                                                    unsigned long long *status, unsigned *ticket,
                                                    uint2 *total, int *err) {
    __shared__ uint2 s_warp[kScanT / 32];
    __shared__ unsigned s_tile;
    __shared__ uint2 s_excl;
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const unsigned tile = s_tile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t base = (size_t)tile * kScanTile + (size_t)warp * (64 * kScanR) + 2 * lane;
    uint4 v[kScanR];
#pragma unroll
    for (int q = 0; q < kScanR; q++) {
        const size_t e = base + 64 * q;
        v[q] = e + 1 < n ? *(const uint4 *)(in + e) : make_uint4(0, 0, 0, 0);
        if (e + 1 == n) v[q].x = in[e].x, v[q].y = in[e].y;
    }
    uint2 run = make_uint2(0, 0), incl[kScanR];
#pragma unroll
    for (int q = 0; q < kScanR; q++) {
        incl[q] = add2(run, warp_incl_scan2(make_uint2(v[q].x + v[q].z, v[q].y + v[q].w)));
        run.x = __shfl_sync(0xffffffffu, incl[q].x, 31);
        run.y = __shfl_sync(0xffffffffu, incl[q].y, 31);
    }
    uint2 tot;
    const uint2 wexcl = block_excl_scan2<kScanT>(lane == 31 ? run : make_uint2(0, 0), tot, s_warp);
    if (warp == 0) {
        const uint2 excl = unpack31(look_back(status, tile, pack31(tot), err));
        if (lane == 0) {
            s_excl = excl;
            if (tile == gridDim.x - 1 && total) *total = add2(excl, tot);
        }
    }
    // of the warp: what the lanes before the last have (the last lane holds the warp's sum)
    const uint2 wbase = make_uint2(__shfl_sync(0xffffffffu, wexcl.x, 0), __shfl_sync(0xffffffffu, wexcl.y, 0));
    __syncthreads();
    const uint2 first = add2(s_excl, wbase);
#pragma unroll
    for (int q = 0; q < kScanR; q++) {
        const size_t e = base + 64 * q;
        const uint2 b = add2(first, incl[q]);  // after the pair
        const uint2 p1 = make_uint2(b.x - v[q].z, b.y - v[q].w), p0 = make_uint2(p1.x - v[q].x, p1.y - v[q].y);
        if (e + 1 < n)
            *(uint4 *)(out + e) = make_uint4(p0.x, p0.y, p1.x, p1.y);
        else if (e < n)
            out[e] = p0;
    }
}

size_t scan_u2_tmp_bytes(unsigned n) {
    size_t tiles = (n + kScanTile - 1) / kScanTile;
    return 256 + tiles * sizeof(unsigned long long);
}

cudaError_t scan_u2(const uint2 *in, uint2 *out, unsigned n, uint2 *d_total, void *tmp, int *d_err,
                    cudaStream_t s, int *launches, bool cleared) {
    unsigned tiles = (n + kScanTile - 1) / kScanTile;
    if (tiles == 0) {
        if (d_total) return cudaMemsetAsync(d_total, 0, sizeof(uint2), s);
        return cudaSuccess;
    }
    unsigned *ticket = (unsigned *)tmp;
    unsigned long long *status = (unsigned long long *)((char *)tmp + 256);
    if (!cleared) {
        const cudaError_t e = cudaMemsetAsync(tmp, 0, scan_u2_tmp_bytes(n), s);
        if (e != cudaSuccess) return e;
    }
    k_scan_u2<<<tiles, kScanT, 0, s>>>(in, out, n, status, ticket, d_total, d_err);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

// ------------------------------------------------------------ radix sort
constexpr int kRsT = 256, kRsW = kRsT / 32;
// Keys per thread: the tile is staged in shared memory before it is written out, so 64-bit keys take
// fewer (static shared memory stays under 48 KB).
template <typename K> constexpr int kRsItems = sizeof(K) == 8 ? 12 : 16;

template <typename K>
__global__ void __launch_bounds__(256) k_rs_hist(const K *keys, unsigned n, int npass, unsigned *hist) {
    __shared__ unsigned sh[sizeof(K) * 256];
    for (int q = threadIdx.x; q < npass * 256; q += 256) sh[q] = 0;
    __syncthreads();
    for (size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x; idx < n; idx += (size_t)gridDim.x * 256) {
        const K k = keys[idx];
        for (int p = 0; p < npass; p++) atomicAdd(&sh[p * 256 + (unsigned)((k >> (8 * p)) & 255)], 1u);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < npass * 256; q += 256)
        if (sh[q]) atomicAdd(&hist[q], sh[q]);
}

// One onesweep pass over a tile of kRsT x kRsItems keys: stable ranks by warp-level digit
// matching, the tile's offset per digit by decoupled look-back over tiles, then the tile is
// reordered by digit in shared memory so each digit's run is written out contiguously.
template <typename K>
__global__ void __launch_bounds__(kRsT) k_rs_pass(const K *__restrict__ kin, K *__restrict__ kout,
                                                  const unsigned *__restrict__ vin, unsigned *__restrict__ vout,
                                                  unsigned n, int shift, const unsigned *__restrict__ hist,
                                                  unsigned long long *status, unsigned *ticket, int *err) {
    constexpr int I = kRsItems<K>, TILE = kRsT * I;
    __shared__ unsigned s_wc[kRsW][256];
    __shared__ unsigned s_base[256], s_lstart[256];
    __shared__ unsigned s_tmp[kRsT / 32];
    __shared__ unsigned s_tile;
    __shared__ K s_key[TILE];
    __shared__ unsigned s_val[TILE];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(ticket, 1u);
    for (int q = tid; q < kRsW * 256; q += kRsT) (&s_wc[0][0])[q] = 0;
    __syncthreads();
    const unsigned tile = s_tile;
    const size_t tbase = (size_t)tile * TILE;
    const size_t wbase = tbase + (size_t)warp * (32 * I);

    K key[I];
    unsigned val[I], dig[I], rank[I];
#pragma unroll
    for (int it = 0; it < I; it++) {
        size_t idx = wbase + (size_t)it * 32 + lane;
        if (idx < n) {
            key[it] = kin[idx];
            val[it] = vin ? vin[idx] : (unsigned)idx;
            dig[it] = (unsigned)((key[it] >> shift) & 255);
        } else {
            key[it] = 0;
            val[it] = 0;
            dig[it] = 256;
        }
    }
    // Stable rank within the warp's contiguous segment, item by item in input order.
#pragma unroll
    for (int it = 0; it < I; it++) {
        const unsigned d = dig[it];
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const unsigned lower = peers & ((1u << lane) - 1u);
        const unsigned before = d < 256 ? s_wc[warp][d] : 0u;
        rank[it] = before + __popc(lower);
        __syncwarp();
        if (d < 256 && lower == 0) s_wc[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // Thread `tid` owns digit `tid`: exclusive prefix over warps, then the tile count.
    const unsigned d = tid;
    unsigned run = 0;
#pragma unroll
    for (int w = 0; w < kRsW; w++) {
        unsigned c = s_wc[w][d];
        s_wc[w][d] = run;
        run += c;
    }
    unsigned excl = 0;
    unsigned long long *st = status + (size_t)tile * 256 + d;
    if (tile == 0) {
        st_release(st, kFlagPre | run);
    } else {
        st_release(st, kFlagAgg | run);
        for (int j = (int)tile - 1; j >= 0; j--) {
            unsigned long long s = wait_status(status + (size_t)j * 256 + d, err);
            excl += (unsigned)(s & 0xffffffffull);
            if ((s >> 62) != 1) break;
        }
        st_release(st, kFlagPre | (unsigned long long)(excl + run));
    }
    unsigned htot, ltot;
    const unsigned dstart = block_excl_scan<kRsT>(hist[d], htot, s_tmp);
    const unsigned lstart = block_excl_scan<kRsT>(run, ltot, s_tmp);
    s_base[d] = dstart + excl;  // global position of this tile's first key of digit d
    s_lstart[d] = lstart;       // its position within the digit-sorted tile
    __syncthreads();
#pragma unroll
    for (int it = 0; it < I; it++) {
        const unsigned dd = dig[it];
        if (dd < 256) {
            const unsigned lp = s_lstart[dd] + s_wc[warp][dd] + rank[it];
            s_key[lp] = key[it];
            s_val[lp] = val[it];
        }
    }
    __syncthreads();
    // ltot keys of this tile, digit-sorted: consecutive threads write consecutive addresses.
    for (unsigned q = tid; q < ltot; q += kRsT) {
        const K k = s_key[q];
        const unsigned dd = (unsigned)((k >> shift) & 255);
        const unsigned pos = s_base[dd] + (q - s_lstart[dd]);
        if (pos < n) {
            kout[pos] = k;
            vout[pos] = s_val[q];
        }
    }
}

template <typename K> size_t radix_sort_tmp_bytes(unsigned n, int bits) {
    int npass = (bits + 7) / 8;
    size_t tiles = ((size_t)n + kRsT * kRsItems<K> - 1) / (kRsT * kRsItems<K>);
    return 256 + (size_t)(npass > 0 ? npass : 1) * 256 * (sizeof(unsigned) + tiles * sizeof(unsigned long long));
}

template <typename K>
cudaError_t radix_sort(K *keys, K *keys_alt, unsigned *vals, unsigned *vals_alt, unsigned n, int bits, bool identity,
                       void *tmp, int *d_err, cudaStream_t s, int *launches, int *in_alt, const K *keys_in) {
    *in_alt = 0;
    int npass = (bits + 7) / 8;
    if (npass > (int)sizeof(K)) npass = (int)sizeof(K);
    if (n == 0) return cudaSuccess;
    if (npass == 0) npass = 1;  // still materialise the values (identity case)
    constexpr unsigned kTile = kRsT * kRsItems<K>;
    unsigned tiles = (unsigned)(((size_t)n + kTile - 1) / kTile);
    unsigned *ticket = (unsigned *)tmp;
    unsigned *hist = (unsigned *)((char *)tmp + 256);
    unsigned long long *status = (unsigned long long *)((char *)hist + (size_t)npass * 256 * sizeof(unsigned));
    cudaError_t e = cudaMemsetAsync(tmp, 0, radix_sort_tmp_bytes<K>(n, bits), s);  // every pass's at once
    if (e != cudaSuccess) return e;
    unsigned hblocks = (n + 255) / 256;
    if (hblocks > 1216) hblocks = 1216;
    const K *first = keys_in ? keys_in : keys;
    k_rs_hist<K><<<hblocks, 256, 0, s>>>(first, n, npass, hist);
    if (launches) (*launches)++;
    const K *src = first;
    K *dst = keys_alt, *other = keys;  // passes after the first ping-pong between keys_alt and keys
    unsigned *vsrc = identity ? nullptr : vals, *vdst = vals_alt;
    for (int p = 0; p < npass; p++) {
        k_rs_pass<K><<<tiles, kRsT, 0, s>>>(src, dst, vsrc, vdst, n, 8 * p, hist + p * 256,
                                         status + (size_t)p * tiles * 256, ticket + p, d_err);
        if (launches) (*launches)++;
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        src = dst;
        K *tk = other; other = dst; dst = tk;
        unsigned *written = vdst;
        vdst = (written == vals_alt) ? vals : vals_alt;
        vsrc = written;
    }
    *in_alt = (npass & 1);
    return cudaSuccess;
}

template size_t radix_sort_tmp_bytes<unsigned>(unsigned, int);
template size_t radix_sort_tmp_bytes<unsigned long long>(unsigned, int);
template cudaError_t radix_sort<unsigned>(unsigned *, unsigned *, unsigned *, unsigned *, unsigned, int, bool, void *,
                                          int *, cudaStream_t, int *, int *, const unsigned *);
template cudaError_t radix_sort<unsigned long long>(unsigned long long *, unsigned long long *, unsigned *, unsigned *,
                                                    unsigned, int, bool, void *, int *, cudaStream_t, int *, int *,
                                                    const unsigned long long *);

}  // namespace qses
