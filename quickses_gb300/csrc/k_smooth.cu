// Exact Gauss-Seidel Laplacian smoothing (SmoothMesh.cpp:45-123) as a dataflow over slabs of
// vertex ids: a vertex is updated once every lower-id neighbour has been, exactly as the
// sequential loop would see them.  Persistent CTAs take the slabs from a device work queue.
#include <cstring>

#include "device_common.cuh"

#include "kernels.h"

namespace qses {

// Slab-partitioned Gauss-Seidel pass.  Vertex ids are split into contiguous slabs; every
// dependency edge goes from a lower to a higher id, so a chain of updates crosses each slab
// boundary at most once.  Inside a slab a vertex is one 16-byte record in shared memory - its
// position and a word with its readiness counter and its list's length - so that a chain step is
// one shared-memory gather, the sum, and one atomic per successor that returns all the next step
// needs.  L2 is touched only for the neighbour list (one 64-byte line, asked for while its
// vertex's lower neighbours are updated) and for neighbours in other slabs.
//
// What bounds it: the chain of dependent updates (5 332 levels on the 3 540 000-vertex mesh of
// 50 000 atoms at 0.2 A), not bytes.  Measured on GB300 with one chain of updates in one slab, a
// step takes 700 cycles - of them the gather, the rows and the sum in list order ~240, position
// store and fence 35, the successors' atomics 45, choosing and fetching the next ~150 - 1 050
// with a neighbour in another slab, and 500 more when the next vertex goes to another warp.  Per
// level a whole pass took 1.86 us with a warp per vertex, counters in shared memory and positions
// and lists in L2, and takes 1.0 us (9.89 -> 5.3 ms; 0.94 -> 0.41 ms on 30 000 vertices; 4.1 ->
// 1.7 ms on a batch of 16 molecules).  A slab's SM is saturated at ~43 cycles per vertex.
constexpr int kGsThreadsMax = 1024;
constexpr int kGsRecvWarps = 2;  // warps that watch the lower slabs' releases
constexpr unsigned kGsRow = 36;  // floats per component of a warp's row (32 used; offset banks)

// Shared-memory layout of a slab of at most smax vertices (bytes).
struct GsSmem {
    unsigned rec, pend, ring, bytes;
};
__host__ __device__ constexpr GsSmem gs_smem(unsigned smax) {
    GsSmem L{};
    L.rec = 0;                                       // records, and one of -0 that past-the-end entries read
    L.pend = L.rec + 16 * (smax + 1);                // 1 bit per vertex: waits for lower slabs
    L.ring = L.pend + 4 * ((smax + 62) / 32 + 1);    // 16-bit slab offsets of ready vertices
    L.bytes = (L.ring + 2 * (smax + 32) + 15) & ~15u;  // + one slot per warp past the last vertex
    return L;
}
static_assert(gs_smem(kGsSlabCap).bytes + 15 * 1024 <= 227 * 1024, "a slab's state fits a CTA");

// A record's word, built by k_gs_lists: bits 0-6 readiness counter (lower neighbours to come),
// bit 7 one of them is in a lower slab, bit 8 the list has more than 16 entries.  Lists of up to 16
// entries are at 16 v in the packed table, past-the-end entries naming record smax; bits 9-12 are
// their length in pairs.  Longer lists are in the neighbour table: bits 9-14 their length in
// pairs, bits 15-31 the offset in pairs from the slab's first entry, or kGsLost in bits 9-14 if
// either does not fit (the offsets table has both).
constexpr unsigned kGsPend = 0x80u, kGsLong = 0x100u, kGsLost = 63u;
__device__ __forceinline__ unsigned gs_first(unsigned word) { return (word >> 15) * 2u; }
__device__ __forceinline__ unsigned gs_len(unsigned word) { return ((word >> 9) & 63u) * 2u; }

// List entries.  Bit 31: in another slab; bit 30: higher id than the list's vertex; bit 29: no
// release (in a later wave, or named by an earlier entry of the list).  Below: the record (bit 31
// clear) or the vertex id.
constexpr unsigned kGsSucc = 2u, kGsFar = 6u;  // the top three bits of a successor here / in a higher slab

__device__ __forceinline__ void fence_cta() { asm volatile("fence.acq_rel.cta;" ::: "memory"); }

// A vertex position with its pass stamp in w, read and written as one 16-byte access: the
// stamp tells a reader whether the position is this pass's, so no fence orders the two.
__device__ __forceinline__ float4 ld_pos(const float4 *p) {
    float4 q;
    asm volatile("{\n\t.reg .b128 t;\n\t.reg .b64 lo, hi;\n\t"
                 "ld.relaxed.gpu.global.b128 t, [%4];\n\t"
                 "mov.b128 {lo, hi}, t;\n\tmov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
                 : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w)
                 : "l"(p)
                 : "memory");
    return q;
}
__device__ __forceinline__ void ld_pos_if(float4 &q, const float4 *p, bool go) {
    asm volatile("{\n\t.reg .pred g;\n\t.reg .b128 t;\n\t.reg .b64 lo, hi;\n\tsetp.ne.u32 g, %5, 0;\n\t"
                 "mov.b64 lo, {%0, %1};\n\tmov.b64 hi, {%2, %3};\n\tmov.b128 t, {lo, hi};\n\t"
                 "@g ld.relaxed.gpu.global.b128 t, [%4];\n\t"
                 "mov.b128 {lo, hi}, t;\n\tmov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
                 : "+f"(q.x), "+f"(q.y), "+f"(q.z), "+f"(q.w)
                 : "l"(p), "r"((unsigned)go)
                 : "memory");
}
__device__ __forceinline__ void st_pos(float4 *p, float4 q, bool go = true) {
    asm volatile("{\n\t.reg .pred g;\n\t.reg .b128 t;\n\t.reg .b64 lo, hi;\n\tsetp.ne.u32 g, %5, 0;\n\t"
                 "mov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\tmov.b128 t, {lo, hi};\n\t"
                 "@g st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "f"(q.x), "f"(q.y), "f"(q.z), "f"(q.w), "r"((unsigned)go)
                 : "memory");
}

// A record's position (its word may be counted down at the same time: a relaxed access).
__device__ __forceinline__ float4 ld_rec(unsigned p) {
    float4 q;
    asm volatile("ld.relaxed.cta.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w) : "r"(p) : "memory");
    return q;
}
__device__ __forceinline__ float ld_comp(unsigned p) {
    float x;
    asm volatile("ld.relaxed.cta.shared.f32 %0, [%1];" : "=f"(x) : "r"(p) : "memory");
    return x;
}
__device__ __forceinline__ void st_comp(unsigned p, float x, bool go) {
    asm volatile("{\n\t.reg .pred g;\n\tsetp.ne.u32 g, %2, 0;\n\t@g st.relaxed.cta.shared.f32 [%0], %1;\n\t}" ::"r"(p), "f"(x),
                 "r"((unsigned)go) : "memory");
}
// Counts the record at p down if `go`; the word before (0 if not).
__device__ __forceinline__ unsigned dec_rec(unsigned p, bool go) {
    unsigned old;
    asm volatile("{\n\t.reg .pred g;\n\tsetp.ne.u32 g, %2, 0;\n\tmov.u32 %0, 0;\n\t"
                 "@g atom.relaxed.cta.shared.add.u32 %0, [%1], -1;\n\t}"
                 : "=&r"(old) : "r"(p + 12u), "r"((unsigned)go) : "memory");
    return old;
}

// Asks for the sectors of a neighbour list without a register or a wait: an asynchronous copy
// of one word per sector into scratch that nobody reads (prefetch.global.L1 brings nothing into
// L1 on this GPU, and a plain load would be waited for by the next fence).
__device__ __forceinline__ void touch_l1(unsigned scratch, const unsigned *p, bool go) {
    asm volatile("{\n\t.reg .pred g;\n\tsetp.ne.u32 g, %2, 0;\n\t@g cp.async.ca.shared.global [%0], [%1], 4;\n\t}" ::"r"(scratch),
                 "l"(p), "r"((unsigned)go) : "memory");
}

__device__ __forceinline__ void red_ext(unsigned *ext, unsigned u, bool go) {
    asm volatile("{\n\t.reg .pred g;\n\tsetp.ne.u32 g, %2, 0;\n\t@g red.relaxed.gpu.global.add.u32 [%0], %1;\n\t}" ::"l"(ext + (u >> 2)),
                 "r"(0u - (1u << (8u * (u & 3u)))), "r"((unsigned)go) : "memory");
}
__device__ __forceinline__ void add_ext(unsigned *word, unsigned x) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(word), "r"(x) : "memory");
}
// This lane's entry of a list (what past-the-end entries read otherwise).
__device__ __forceinline__ unsigned ld_entry(const unsigned *p, bool go, unsigned other) {
    unsigned x = other;
    asm volatile("{\n\t.reg .pred g;\n\tsetp.ne.u32 g, %2, 0;\n\t@g ld.global.nc.u32 %0, [%1];\n\t}" : "+r"(x) : "l"(p), "r"((unsigned)go));
    return x;
}

// s / n for a whole n in [1, 126] with rn = 1/n correctly rounded: one multiplication and one
// correction by the exact residual give the correctly rounded quotient (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990; checked for every
// mantissa and every n up to 1 024) unless the quotient is subnormal (gs_tiny: it may be).
__device__ __forceinline__ float gs_div(float s, float n, float rn) {
    const float q = __fmul_rn(s, rn);
    return __fmaf_rn(__fmaf_rn(-q, n, s), rn, q);
}
__device__ __forceinline__ bool gs_tiny(float s) {  // 0 < |s| < 2^-100 (zero wraps round)
    return 2u * __float_as_uint(s) - 1u < 2u * 0x0d800000u - 1u;
}

// The slab's ready vertices: a ring in shared memory.  An idle warp takes the next ticket and
// watches the ring's slot of that number, so a vertex goes to the warp that has waited longest
// without any of them contending for it.
struct __align__(16) GsQueue {
    unsigned ticket, tail, done, stop;
};
__device__ __forceinline__ uint2 ld_queue(unsigned p) {  // ticket, tail
    uint2 x;
    asm volatile("ld.relaxed.cta.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x.x), "=r"(x.y) : "r"(p) : "memory");
    return x;
}
constexpr unsigned kGsEmpty = 0xffffu, kGsQuit = 0xfffeu;  // ring slots that hold no slab offset

// Each vertex enters the ring at most once: no wrap-around.  In two halves, so that a step can do
// other work between taking the slot and filling it; predicated, as a branch would end its block.
__device__ __forceinline__ unsigned gs_slot(unsigned tail, bool go) {
    unsigned t = 0;
    asm volatile("{\n\t.reg .pred g;\n\tsetp.ne.u32 g, %2, 0;\n\t@g atom.relaxed.cta.shared.add.u32 %0, [%1], 1;\n\t}"
                 : "+r"(t) : "r"(tail), "r"((unsigned)go) : "memory");
    return t;
}
__device__ __forceinline__ void gs_fill(unsigned ring, unsigned slot, unsigned k, bool go) {
    asm volatile("{\n\t.reg .pred g;\n\tsetp.ne.u32 g, %2, 0;\n\t@g st.relaxed.cta.shared.u16 [%0], %1;\n\t}" ::"r"(ring + 2 * slot),
                 "h"((unsigned short)k), "r"((unsigned)go) : "memory");
}
__device__ __forceinline__ void gs_push(unsigned tail, unsigned ring, unsigned k, bool go) {
    gs_fill(ring, gs_slot(tail, go), k, go);
}

__device__ __forceinline__ float add4(float s, float4 q) {
    return __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, q.x), q.y), q.z), q.w);
}

// A wait's clock.  It runs out spin_cycles after the last sign of progress: one that the waiter sees
// itself (restart) or an item taken from the counter since, by a CTA that has finished another.  So
// a wait behind a long queue of slabs lasts while they are being done, however slowly, and ends
// when none is, or at its next look after another wait has run out.
struct GsClock {
    long long since;
    unsigned taken;  // what the counter had at the last look
    __device__ __forceinline__ explicit GsClock(unsigned item) {
        since = clock64();
        taken = item + 1;
    }
    __device__ __forceinline__ void restart() { since = clock64(); }
    __device__ __forceinline__ bool out(const unsigned *next_slab, long long spin_cycles, const int *err) {
        const long long now = clock64();
        if (now - since <= spin_cycles) return false;
        unsigned k;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(k) : "l"(next_slab) : "memory");
        const bool none = k == taken;
        taken = k;
        since = now;
        return none || *(const volatile int *)err != 0;
    }
};

// Waits until slab p and the slabs of all its higher neighbours have had `pass` passes; false if
// that takes too long.
__device__ __forceinline__ bool gs_wait_pass(const GsOrder &ord, unsigned p, unsigned pass, GsClock clock,
                                             const unsigned *next_slab, long long spin_cycles, const int *err) {
    for (unsigned j = p; j <= ord.far[p]; j++) {
        while (ld_acquire_u32(&ord.done[j]) < pass) {
            if (clock.out(next_slab, spin_cycles, err)) return false;
            __nanosleep(200);
        }
        clock.restart();
    }
    return true;
}

// Several passes in one launch: a vertex's pass q needs its lower neighbours' pass q and its higher
// neighbours' pass q - 1, so pass q can follow pass q - 1 through the slabs a little behind it, and
// three passes take little longer than one (548 000 vertices: 4.77 ms launched one after another,
// 2.70 together, one alone 1.6).
// Item n of the passes of a wave: slabs by their place in the order, pass q of a place `lag` places
// behind pass q - 1, so that a place's items, and those of the places up to `lag` behind it, come
// after their previous passes.  items_before(t): the items whose place + lag q is below t.
struct GsItem {
    unsigned place, pass;
};
__device__ __forceinline__ unsigned long long gs_items_before(unsigned long long t, unsigned Q, unsigned passes,
                                                              unsigned lag) {
    const unsigned long long full = t >= Q ? min((unsigned long long)passes, (t - Q) / lag + 1) : 0;
    const unsigned long long part = t ? min((unsigned long long)passes, (t - 1) / lag + 1) : 0;
    return full * Q + (part - full) * t - (part > full ? lag * ((part * (part - 1) - full * (full - 1)) / 2) : 0);
}
__device__ __forceinline__ GsItem gs_item(unsigned n, unsigned Q, unsigned passes, unsigned lag) {
    if (passes == 1) return {n, 0u};
    unsigned long long lo = 0, hi = Q + (unsigned long long)lag * (passes - 1);  // before(lo) <= n < before(hi)
    while (hi - lo > 1) {
        const unsigned long long mid = (lo + hi) / 2;
        if (gs_items_before(mid, Q, passes, lag) <= n) lo = mid; else hi = mid;
    }
    const unsigned first = lo >= Q ? (unsigned)((lo - Q) / lag + 1) : 0u;  // passes that have places left at lo
    const unsigned pass = first + (unsigned)(n - gs_items_before(lo, Q, passes, lag));
    return {(unsigned)(lo - (unsigned long long)lag * pass), pass};
}

// What a warp spends its steps on, in clock cycles.
struct GsCycles {
    unsigned long long update = 0, release = 0, ids = 0, position = 0, fence = 0;
};
// The clock once x is there.
__device__ __forceinline__ long long clock_behind(unsigned x) {
    asm volatile("{\n\t.reg .b32 t;\n\tmov.b32 t, %0;\n\t}" ::"r"(x) : "memory");
    return clock64();
}
__device__ __forceinline__ long long clock_behind(float x) { return clock_behind(__float_as_uint(x)); }

// Persistent CTAs take the wave's slabs from a counter, in the table's order (a slab only
// waits for slabs taken before it, by CTAs that were running when they took them, so every
// wait ends without a co-residency guarantee).  Per slab the first two warps watch the release
// counters that lower slabs decrement (ext, one byte per vertex: neighbour entries in lower
// slabs still to come), the other warps update vertices.
// Table: Q, the Q + 1 slab bounds in id order (qcap + 1 slots), then the Q slab ids in the
// order they are taken.
// COUNT: the clock cycles of an update's parts are added up too (stats not null), which lengthens every
// step; a kernel of its own, for calls that ask for them.
// out (may be null): host memory that the last pass's positions go to as each slab is done, 3 floats
// a vertex.  Behind the kernel the copy of 44 MB took 0.22 ms of 8.2, that of 16 trajectory frames 0.16
// of 3.34.
template <bool COUNT>
__global__ void __launch_bounds__(kGsThreadsMax, 1)
    k_gs_flow(float4 *pos4, unsigned v0, unsigned nv, unsigned smax, const unsigned *__restrict__ table, unsigned qcap,
              unsigned *next_slab, const uint2 *__restrict__ start, const unsigned *__restrict__ nbr,
              const unsigned *__restrict__ word0, const unsigned *__restrict__ pack, unsigned *ext,
              const unsigned char *__restrict__ ext0, unsigned passes, unsigned stamp0, GsOrder ord, float *out, int *err,
              long long spin_cycles, unsigned long long *stats) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ GsQueue s_q;
    __shared__ unsigned s_slab, s_pass, s_item;
    // Per worker warp: the neighbours' coordinates, one row per component, summed in list order
    __shared__ __align__(16) float s_row[kGsThreadsMax / 32][3 * kGsRow];
    __shared__ unsigned s_void[32];  // target of touch_l1
    __shared__ float2 s_rcp[16];  // a packed list's length in pairs -> length, its reciprocal
    const GsSmem L = gs_smem(smax);
    float4 *rec = (float4 *)(s_dyn + L.rec);
    unsigned *pend = (unsigned *)(s_dyn + L.pend);
    volatile unsigned short *ring = (volatile unsigned short *)(s_dyn + L.ring);
    const unsigned rec_s = (unsigned)__cvta_generic_to_shared(rec), ring_s = (unsigned)__cvta_generic_to_shared(s_dyn + L.ring);
    const unsigned queue_s = (unsigned)__cvta_generic_to_shared(&s_q), tail_s = queue_s + 4;
    const unsigned T = blockDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned Q = min(__ldg(table), qcap);
    const unsigned *bnd = table + 1, *order = table + 2 + qcap;
    volatile unsigned *v_done = &s_q.done, *v_stop = &s_q.stop;
    const unsigned lag = passes > 1 ? *ord.lag : 1u;
    const unsigned v_scratch = (unsigned)__cvta_generic_to_shared(&s_void[lane]);
    unsigned long long polls = 0;
    GsCycles cyc;  // COUNT
    if (threadIdx.x == 0) {
        s_q.stop = 0;
        rec[smax] = make_float4(-0.0f, -0.0f, -0.0f, 0.0f);
    }
    if (threadIdx.x < 16) s_rcp[threadIdx.x] = make_float2(2.0f * threadIdx.x, __frcp_rn(2.0f * threadIdx.x));
    for (;;) {
        if (threadIdx.x == 0) {
            // a CTA whose wait ran out takes nothing more, or the others would see progress
            const unsigned k = s_q.stop ? 0xffffffffu : atomicAdd(next_slab, 1u);
            s_slab = 0xffffffffu;
            s_item = k;
            if (k < Q * passes) {
                const GsItem it = gs_item(k, Q, passes, lag);
                s_slab = __ldg(order + it.place);
                s_pass = it.pass;
                if (it.pass && !gs_wait_pass(ord, s_slab, it.pass, GsClock(k), next_slab, spin_cycles, err)) {
                    raise_error(err, QSES_ERR_TIMEOUT);
                    s_q.stop = 1;
                    s_slab = 0xffffffffu;
                }
            }
            s_q.ticket = 0; s_q.tail = 0; s_q.done = 0;
        }
        __syncthreads();
        const unsigned p = s_slab, pass = s_pass, stamp = stamp0 + pass;
        const float fstamp = __uint_as_float(stamp);
        if (p >= Q) break;  // uniform per CTA: no slab left (or an error stopped this CTA)
        const unsigned a = __ldg(bnd + p), b = __ldg(bnd + p + 1), len = b - a;
        if (a < v0 || b > nv || b <= a || len > smax) {  // uniform: a malformed table entry
            if (threadIdx.x == 0) raise_error(err, QSES_ERR_INTERNAL);
            break;
        }
        const unsigned a32 = a & ~31u, nword = (b - a32 + 31) / 32;  // words of ext bytes and pend bits
        const unsigned *list = nbr + 2 * (size_t)start[a].x;
        const unsigned *packs = pack + 16 * (size_t)a;
        for (unsigned k = threadIdx.x; k < len; k += T) {
            float4 q = ld_pos(pos4 + a + k);
            q.w = __uint_as_float(word0[a + k] & ~kGsPend);
            rec[k] = q;
        }
        for (unsigned k = threadIdx.x; k < len + 32; k += T) ring[k] = kGsEmpty;
        for (unsigned w = warp; w < nword; w += T / 32) {
            const unsigned v = a32 + 32 * w + lane;
            const unsigned m = __ballot_sync(0xffffffffu, v >= a && v < b && (word0[v] & kGsPend));
            if (lane == 0) pend[w] = m;
        }
        __syncthreads();
        for (unsigned k = threadIdx.x; k < len; k += T)
            gs_push(tail_s, ring_s, k, (word0[a + k] & 0x7fu) == 0);
        __syncthreads();

        if (warp < kGsRecvWarps) {
            // Receivers never update vertices, so arrivals are never stuck behind a chain.  A lane
            // watches 32 vertices at a time: the bytes of those still waiting; a byte at zero means
            // that every neighbour in a lower slab has been updated.
            unsigned idle_ns = 0, done_seen = 0;
            GsClock clock(s_item);
            for (;;) {
                const unsigned d = *v_done;
                if (__any_sync(0xffffffffu, d >= len || *v_stop)) break;
                polls++;
                bool any = false, left = false;
                for (unsigned w = warp * 32 + lane; w < nword; w += 32 * kGsRecvWarps) {
                    const unsigned m = pend[w];
                    if (!m) continue;
                    const unsigned *e = ext + (a32 >> 2) + 8 * w;
                    unsigned x[8], zero = 0;
                    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "l"(e) : "memory");
                    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7]) : "l"(e + 4) : "memory");
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        // 0x80 in each zero byte, then one bit per byte (the products do not overlap)
                        const unsigned z = ~(((x[j] & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x[j] | 0x7f7f7f7fu);
                        zero |= ((((z >> 7) * 0x01020408u) >> 24) & 0xfu) << (4 * j);
                    }
                    unsigned now = zero & m;
                    pend[w] = m & ~now;
                    left |= (m & ~now) != 0;
                    any |= now != 0;
                    for (; now; now &= now - 1) {
                        const unsigned k = a32 + 32 * w + (__ffs(now) - 1) - a;
                        const bool go = (dec_rec(rec_s + 16 * k, true) & 0x7fu) == 1u;
                        fence_cta();  // the neighbours' positions before the ring entry
                        gs_push(tail_s, ring_s, k, go);
                    }
                }
                any = __any_sync(0xffffffffu, any);
                left = __any_sync(0xffffffffu, left);
                if (!left) break;  // nobody here waits for a lower slab any more
                if (any || d != done_seen) clock.restart();
                done_seen = d;
                if (__any_sync(0xffffffffu, clock.out(next_slab, spin_cycles, err))) {
                    if (lane == 0) {
                        raise_error(err, QSES_ERR_TIMEOUT);
                        *v_stop = 1;
                    }
                    break;
                }
                idle_ns = any ? 0u : min(idle_ns + 20u, 200u);
                if (idle_ns) __nanosleep(idle_ns);
            }
            // The workers' own wait for a vertex ends with the slab or an error; it is watched here
            // once no arrival is expected any more.
            if (warp == 0) {
                clock.restart();
                unsigned seen = *v_done;
                while (true) {
                    const unsigned d = *v_done;
                    if (__any_sync(0xffffffffu, d >= len || *v_stop)) break;
                    if (d != seen) clock.restart();
                    seen = d;
                    if (__any_sync(0xffffffffu, clock.out(next_slab, spin_cycles, err))) {
                        if (lane == 0) {
                            raise_error(err, QSES_ERR_TIMEOUT);
                            *v_stop = 1;
                        }
                        break;
                    }
                    __nanosleep(500);
                }
            }
        } else {
            // Worker warps: a vertex per half warp, and on along the chain of vertices it releases.
            // The second half is in use only while more vertices are ready than warps wait for: 28
            // chains in a slab take 1 210 cycles a step on 14 warps that pair them, 1 850 on 28 that do
            // not (the shared-memory pipe is the limit, and a pair shares its instructions).  `i`,
            // `word` and `act` are a half's vertex at hand and whether there is one, `code` the lane's
            // entry of its list.
            float *row = s_row[warp];
            const unsigned hl = lane & 15u, half = lane & 16u;
            const float4 *crow = (const float4 *)(row + kGsRow * min(hl, 2u) + half);  // lanes past 2 repeat z
            const unsigned comp = rec_s + 4 * min(hl, 2u);
            unsigned i = smax, word = 0, code = smax, done = 0;
            bool act = false;
            // The step of the halves' vertices: sums, divisions, positions, then their successors of this
            // slab counted down; one that a half makes ready is its next vertex, others go to the ring.
            // The lists of all successors are asked for, for the steps that run them.  Halves that
            // `odd` says need more (a position still on its way, a quotient that may be subnormal)
            // release nothing and keep their vertex.  No branch: the step is one basic block (a branch
            // in it, taken or not, cost it 80-110 cycles), with predicated accesses instead.
            auto step = [&](bool &odd, bool &surplus) {
                const long long c0 = COUNT ? clock64() : 0, c1 = COUNT ? clock_behind(code) : 0;
                const float2 fr = s_rcp[(word >> 9) & 15u];
                float4 q = ld_rec(rec_s + 16 * min(code & 0x1fffffffu, smax));
                touch_l1(v_scratch, packs + 16 * (code & 0xffffu) + ((code >> 29) & 1u) * 8, (code >> 30) == 1u);
                const uint2 qt = ld_queue(queue_s);
                // Neighbours in other slabs: positions of this pass below (a release may overtake its
                // position), of the last one above.
                ld_pos_if(q, pos4 + (code & 0x1fffffffu), (int)code < 0);
                const long long c2 = COUNT ? clock_behind(q.x) : 0;
                const bool stale = (code >> 30) == 2u && __float_as_uint(q.w) != stamp;
                row[lane] = q.x; row[kGsRow + lane] = q.y; row[2 * kGsRow + lane] = q.z;
                __syncwarp();
                // Strictly in list order; entries past the list are -0: adding them changes no sum.
                const float4 q0 = crow[0], q1 = crow[1], q2 = crow[2], q3 = crow[3];
                const float sum = add4(add4(add4(add4(0.0f, q0), q1), q2), q3);
                odd = ((__ballot_sync(0xffffffffu, stale || gs_tiny(sum)) >> half) & 0xffffu) != 0u;
                const float at = gs_div(sum, fr.x, fr.y);
                const long long c3 = COUNT ? clock_behind(at) : 0;
                st_comp(comp + 16 * i, at, hl < 3 && act && !odd);
                __syncwarp();
                fence_cta();  // release: the position before the counters
                const long long c4 = COUNT ? clock64() : 0;
                const unsigned k = code & 0xffffu, old = dec_rec(rec_s + 16 * k, (code >> 29) == kGsSucc && !odd);
                const bool now = (old & 0x7fu) == 1u;
                const unsigned ready = (__ballot_sync(0xffffffffu, now) >> half) & 0xffffu;
                // Successors in higher slabs (none that belong to a later wave, which starts after this
                // one): the position for all, then their counters.
                const bool far = (code >> 29) == kGsFar && !odd;
                float4 r = ld_rec(rec_s + 16 * i);
                fence_cta();  // acquire: the next vertex's other neighbours
                const unsigned f = (31u - __clz(ready)) + half;
                const unsigned slot = gs_slot(tail_s, now && lane != f);
                const unsigned ni = __shfl_sync(0xffffffffu, k, f), nw = __shfl_sync(0xffffffffu, old, f);
                r.w = fstamp;
                st_pos(pos4 + a + i, r, far);  // every such lane the same
                red_ext(ext, code & 0x1fffffffu, far);
                done += act && !odd ? 1u : 0u;
                act = act && (odd || ready);
                i = ready ? ni : i;
                word = ready ? nw : word;
                code = ld_entry(packs + 16 * i + hl, act && !odd && !(word & kGsLong), odd ? code : smax);
                gs_fill(ring_s, slot, k, now && lane != f);
                surplus = !act && (int)(qt.y - qt.x) > 0;  // more vertices ready than warps wait for, and a half free
                if (COUNT) {
                    cyc.ids += c1 - c0, cyc.position += c2 - c1, cyc.fence += c4 - c3, cyc.update += c4 - c0;
                    cyc.release += clock_behind((unsigned)surplus) - c4;
                }
            };
            for (;;) {
                // Nothing at hand: wait for a vertex (the ring's slot of this warp's ticket).
                unsigned t = 0;
                if (lane == 0) t = atomicAdd(&s_q.ticket, 1u);
                t = min(__shfl_sync(0xffffffffu, t, 0), len + 31);
                unsigned got;
                for (unsigned it = 1;; it++) {
                    got = ring[t];
                    if (got != kGsEmpty) break;
                    if ((it & 63u) == 0 && (*v_stop || *v_done >= len)) {
                        got = kGsQuit;
                        break;
                    }
                    // the warps next in line look all the time, the others leave them the issue slots
                    if ((int)(t - *(volatile unsigned *)&s_q.tail) >= 4) __nanosleep(100);
                }
                if (got == kGsQuit) break;
                if (half == 0) {
                    act = true;
                    i = got;
                }
                done = 0;
                bool fresh = half == 0;  // the vertex at hand comes from the ring
                for (;;) {
                    fence_cta();  // acquire: the neighbours' positions behind the vertex
                    if (fresh) word = *(volatile unsigned *)&rec[i].w;
                    code = ld_entry(packs + 16 * i + hl, fresh && !(word & kGsLong), code);
                    bool odd = false, surplus = false;
                    if (!__any_sync(0xffffffffu, act && (word & kGsLong))) {
                        do {
                            step(odd, surplus);
                        } while (__ballot_sync(0xffffffffu, act) &&
                                 !__any_sync(0xffffffffu, surplus || odd || (act && (word & kGsLong))));
                    }
                    // A half at a time: long lists and odd vertices, without haste and by the whole warp.
                    for (unsigned h = 0; h < 32; h += 16) {
                        if (!__shfl_sync(0xffffffffu, (unsigned)(act && (odd || (word & kGsLong))), h)) continue;
                        const unsigned vi = __shfl_sync(0xffffffffu, i, h), vw = __shfl_sync(0xffffffffu, word, h);
                        unsigned n = gs_len(vw);
                        const unsigned *ids = packs + 16 * vi;
                        if (vw & kGsLong) {
                            ids = list + gs_first(vw);
                            if (n == 2 * kGsLost) {  // the list is where the offsets table says
                                const unsigned e = start[a + vi].x;
                                ids = nbr + 2 * (size_t)e;
                                n = 2 * (start[a + vi + 1].x - e);
                            }
                        }
                        const long long c0 = COUNT ? clock64() : 0;
                        float sum = 0.0f;
                        unsigned first = smax;
                        for (unsigned base = 0; base < n; base += 32) {
                            const unsigned cd = ld_entry(ids + base + lane, base + lane < n, smax);
                            if (base == 0) first = cd;
                            const long long ca = COUNT ? clock_behind(cd) : 0;
                            if (COUNT && base == 0) cyc.ids += ca - c0;
                            float4 q = ld_rec(rec_s + 16 * min(cd & 0x1fffffffu, smax));
                            const float4 *up = pos4 + (cd & 0x1fffffffu);
                            ld_pos_if(q, up, (int)cd < 0);
                            for (unsigned it = 0;; it++) {
                                const bool stale = (cd >> 30) == 2u && __float_as_uint(q.w) != stamp;
                                if (!__any_sync(0xffffffffu, stale)) break;
                                if (it == (1u << 20)) {
                                    if (lane == 0) raise_error(err, QSES_ERR_TIMEOUT);
                                    *v_stop = 1;
                                    break;
                                }
                                ld_pos_if(q, up, stale);
                            }
                            if (COUNT && base == 0) cyc.position += clock_behind(q.x) - ca;
                            __syncwarp();  // the rows are rewritten
                            row[lane] = q.x; row[kGsRow + lane] = q.y; row[2 * kGsRow + lane] = q.z;
                            __syncwarp();
                            const float4 *all = (const float4 *)(row + kGsRow * min(hl, 2u));
                            for (int j = 0; j < 8; j++) sum = add4(sum, all[j]);
                        }
                        const float at = __fdiv_rn(sum, (float)(int)n);
                        const long long c3 = COUNT ? clock_behind(at) : 0;
                        st_comp(comp + 16 * vi, at, lane < 3);
                        __syncwarp();
                        fence_cta();  // release: the position before the counters
                        const long long c4 = COUNT ? clock64() : 0;
                        if (COUNT) cyc.fence += c4 - c3, cyc.update += c4 - c0;
                        float4 r = ld_rec(rec_s + 16 * vi);
                        r.w = fstamp;
                        unsigned next = kGsEmpty, nw = 0;
                        for (unsigned base = 0; base < n; base += 32) {
                            const unsigned cd = base == 0 ? first : ld_entry(ids + base + lane, base + lane < n, smax);
                            const unsigned k = cd & 0xffffu, old = dec_rec(rec_s + 16 * k, (cd >> 29) == kGsSucc);
                            const bool now = (old & 0x7fu) == 1u;
                            const unsigned ready = __ballot_sync(0xffffffffu, now);
                            fence_cta();
                            unsigned f = 32;
                            if (ready && next == kGsEmpty) {
                                f = __ffs(ready) - 1;
                                next = __shfl_sync(0xffffffffu, k, f);
                                nw = __shfl_sync(0xffffffffu, old, f);
                            }
                            gs_push(tail_s, ring_s, k, now && lane != f);
                            st_pos(pos4 + a + vi, r, (cd >> 29) == kGsFar);
                            red_ext(ext, cd & 0x1fffffffu, (cd >> 29) == kGsFar);
                        }
                        if (COUNT) cyc.release += clock_behind(next) - c4;
                        if (half == h) {
                            done++;
                            act = next != kGsEmpty;
                            i = act ? next : i;
                            word = act ? nw : word;
                            code = ld_entry(packs + 16 * i + hl, act && !(word & kGsLong), smax);
                        }
                    }
                    // A free half takes a vertex that no warp waits for.
                    fresh = false;
                    const unsigned free = __ballot_sync(0xffffffffu, surplus && !act);
                    if (free) {
                        unsigned x = kGsEmpty;
                        const unsigned src = __ffs(free) - 1;  // one half at a time
                        if (lane == src) {
                            // a ticket only if its slot is sure to be filled
                            unsigned tk = *(volatile unsigned *)&s_q.ticket;
                            if ((int)(*(volatile unsigned *)&s_q.tail - tk) > 0 && atomicCAS(&s_q.ticket, tk, tk + 1) == tk)
                            {
                                for (unsigned it = 0; it < (1u << 20) && x == kGsEmpty; it++) x = ring[tk];
                                if (x == kGsEmpty) {
                                    raise_error(err, QSES_ERR_TIMEOUT);
                                    *v_stop = 1;
                                }
                            }
                        }
                        x = __shfl_sync(0xffffffffu, x, src);
                        if (x != kGsEmpty && x != kGsQuit && half == (src & 16u)) {
                            act = fresh = true;
                            i = x;
                        }
                    }
                    if (!__any_sync(0xffffffffu, act)) break;
                }
                done = __reduce_add_sync(0xffffffffu, hl == 0 ? done : 0u);
                if (stats && lane == 0) atomicAdd(stats + 4, (unsigned long long)done);
                done = __shfl_sync(0xffffffffu, lane == 0 ? atomicAdd(&s_q.done, done) + done : 0u, 0);
                if (done >= len) ring[*(volatile unsigned *)&s_q.tail + lane] = kGsQuit;  // the slab is done: so are the waiting warps
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        __syncthreads();
        if (*v_done >= len) {
            // the whole slab: its positions to the later waves, passes and the result
            for (unsigned k = threadIdx.x; k < len; k += T) {
                float4 q = rec[k];
                q.w = fstamp;
                st_pos(pos4 + a + k, q);
            }
            if (pass + 1 < passes) {
                // What the next pass starts with, added to counters that are at zero: other slabs count
                // down the neighbouring bytes of a word at the slab's ends, by atomics of whole words too.
                const unsigned *from = (const unsigned *)ext0;
                for (unsigned w = a / 4 + threadIdx.x; 4 * w < b; w += T) {
                    const unsigned below = 4 * w < a ? (1u << (8 * (a - 4 * w))) - 1u : 0u;
                    const unsigned upto = 4 * w + 4 > b ? (1u << (8 * (b - 4 * w))) - 1u : 0xffffffffu;
                    add_ext(ext + w, __ldg(from + w) & upto & ~below);
                }
            } else if (out)
                for (unsigned k = threadIdx.x; k < 3 * len; k += T) out[3ull * a + k] = ((const float *)(rec + k / 3))[k % 3];
        } else if (stats && threadIdx.x == 0) {
            atomicAdd(stats + 1, 1ull);  // unfinished slabs
        }
        __syncthreads();
        if (pass + 1 < passes && threadIdx.x == 0 && *v_done >= len) {
            __threadfence();  // the CTA's stores before the flag
            st_release_u32(&ord.done[p], pass + 1);
        }
    }  // next slab
    if (stats && threadIdx.x == 0) atomicMax(stats, polls);
    if (COUNT && stats && lane == 0 && warp >= kGsRecvWarps) {
        atomicAdd(stats + 2, cyc.update);
        atomicAdd(stats + 3, cyc.release);
        atomicAdd(stats + 5, cyc.ids);
        atomicAdd(stats + 6, cyc.position);
        atomicAdd(stats + 7, cyc.fence);
    }
}

// Where a vertex's lists end up, and the counts that make its word.
struct GsVertex {
    unsigned a, b;  // its slab's vertices
    unsigned v0, v1;
    unsigned loc, rem, far;  // distinct lower neighbours in the slab and below it; the highest above it
    // An entry in the pass's form; `again`: an earlier one names the same vertex.
    __device__ __forceinline__ unsigned take(unsigned v, unsigned u, bool again) {
        const bool here = u >= a && u < b;
        if (u < v && u >= v0 && !again) {  // below v0: an earlier wave, already final
            if (here) loc++; else rem++;
        }
        if (u >= b && u < v1) far = max(far, u);
        return (here ? u - a : u | 0x80000000u) | (u > v ? 0x40000000u : 0u) | (again || u >= v1 ? 0x20000000u : 0u);
    }
    __device__ __forceinline__ unsigned slab(const unsigned *__restrict__ table, unsigned v) {
        const unsigned *bnd = table + 1;
        unsigned lo = 0, hi = __ldg(table);  // bnd[lo] <= v < bnd[hi]
        while (hi - lo > 1) {
            const unsigned mid = (lo + hi) >> 1;
            if (__ldg(bnd + mid) <= v) lo = mid; else hi = mid;
        }
        a = __ldg(bnd + lo);
        b = __ldg(bnd + lo + 1);
        return lo;
    }
    // w: the word but for its counts.  A vertex is the weld of edges around one grid corner, so its
    // distinct neighbours lie on the 54 edges of 8 cells: both counts stay below their fields.
    __device__ __forceinline__ void write(unsigned v, unsigned lo, unsigned w, unsigned *__restrict__ word0,
                                          unsigned char *__restrict__ ext, unsigned char *__restrict__ ext0,
                                          const GsOrder &ord, int *err) const {
        if (rem > 255u || loc > 0x7eu) raise_error(err, QSES_ERR_INTERNAL);
        word0[v] = w | (loc + (rem ? 1u + kGsPend : 0u));
        ext[v] = (unsigned char)rem;
        if (ext0) {  // several passes in one launch
            ext0[v] = (unsigned char)rem;
            if (far) atomicMax(&ord.far[lo], far);
        }
    }
};

// The two other corners of corner q's triangle, in triangle order.
__device__ __forceinline__ uint2 gs_corners(const unsigned *__restrict__ tri, unsigned q) {
    const unsigned t = q / 3u, c = q - 3u * t;
    const unsigned x = tri[3ull * t], y = tri[3ull * t + 1], z = tri[3ull * t + 2];
    return make_uint2(c == 0 ? y : x, c == 2 ? y : z);
}

// Neighbour lists without a sort of all corners: occ holds each vertex's triangle corners in any
// order (k_csr_scatter); sorting a vertex's few restores triangle order exactly (the order
// getNeighboorsVertices appends in, SmoothMesh.cpp:45-66), and each adds the two other corners of
// its triangle.  Then the vertex's word (counting only distinct lower neighbours), its list in the
// form the pass reads, and the count of neighbours in lower slabs.  Vertices [v0, v1) form the
// slabs of the table (Q, then Q + 1 bounds in id order).  Neighbours below v0 belong to waves that
// finished before this one (final values); neighbours at or above v1 are read before their update.
// A thread per vertex; vertices of more than 8 corners are left to k_gs_lists_long, as a few of
// them among a warp's 32 hold up all (3 540 000 vertices, 10 % of them long: the whole list stage
// 1.19 ms with one kernel, 0.83 with two).
__global__ void __launch_bounds__(128) k_gs_lists(const float *__restrict__ vq, float4 *__restrict__ pos,
                                                  const unsigned *__restrict__ tri, const unsigned *__restrict__ occ,
                                                  const uint2 *__restrict__ start, unsigned v0, unsigned v1,
                                                  unsigned smax, const unsigned *__restrict__ table,
                                                  unsigned *__restrict__ word0, uint4 *__restrict__ pack,
                                                  unsigned char *__restrict__ ext, unsigned char *__restrict__ ext0,
                                                  GsOrder ord, unsigned *__restrict__ longs, int *err) {
    const unsigned v = v0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= v1) return;
    const unsigned o0 = start[v].x, m = start[v + 1].x - o0;  // corners
    pos[v] = make_float4(vq[3ull * v], vq[3ull * v + 1], vq[3ull * v + 2], 0.0f);
    if (m > 8) {
        longs[atomicAdd(ord.longs, 1u)] = v;
        return;
    }
    GsVertex g{0, 0, v0, v1, 0, 0, 0};
    const unsigned lo = g.slab(table, v);
    unsigned r[8];
#pragma unroll
    for (unsigned i = 0; i < 8; i++) r[i] = i < m ? occ[o0 + i] : 0xffffffffu;
#pragma unroll
    for (unsigned i = 1; i < 8; i++) {
#pragma unroll
        for (unsigned j = i; j > 0; j--) {
            const unsigned x = r[j - 1], y = r[j];
            r[j - 1] = min(x, y);
            r[j] = max(x, y);
        }
    }
    unsigned id[16];
#pragma unroll
    for (unsigned i = 0; i < 8; i++) {
        const uint2 e = i < m ? gs_corners(tri, r[i]) : make_uint2(0xffffffffu, 0xffffffffu);
        id[2 * i] = e.x;
        id[2 * i + 1] = e.y;
    }
    unsigned code[16];
#pragma unroll
    for (unsigned i = 0; i < 16; i++) {
        bool again = false;
#pragma unroll
        for (unsigned j = 0; j < i; j++) again |= id[j] == id[i];
        code[i] = i < 2 * m ? g.take(v, id[i], again) : smax;
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
        pack[4 * (size_t)v + j] = make_uint4(code[4 * j], code[4 * j + 1], code[4 * j + 2], code[4 * j + 3]);
    g.write(v, lo, m << 9, word0, ext, ext0, ord, err);
}

// The vertices of more than 8 corners: a warp each, a corner per lane, sorted by counting the
// smaller ones; a hash table finds the entries that name a vertex again; their lists go to the
// neighbour table at twice the vertex's offset.  At 0.2 A, where the surface runs through grid
// points, a tenth of the vertices have 9 to 28 corners: 336 000 of 3 540 000 in 0.225 ms (each entry
// compared with all before it: 0.286).
__global__ void __launch_bounds__(256) k_gs_lists_long(const unsigned *__restrict__ tri, unsigned *__restrict__ occ,
                                                       const uint2 *__restrict__ start, unsigned *__restrict__ nbr,
                                                       unsigned v0, unsigned v1, const unsigned *__restrict__ table,
                                                       unsigned *__restrict__ word0, unsigned char *__restrict__ ext,
                                                       unsigned char *__restrict__ ext0, GsOrder ord,
                                                       const unsigned *__restrict__ longs, int *err) {
    __shared__ unsigned s_q[8][32], s_id[8][64];
    __shared__ uint2 s_seen[8][128];  // hash table: an id, the first entry that has it
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, count = *ord.longs;
    unsigned *row = s_id[warp], *sq = s_q[warp];
    uint2 *seen = s_seen[warp];
    for (unsigned x = blockIdx.x * 8 + warp; x < count; x += gridDim.x * 8) {
        const unsigned v = longs[x], o0 = start[v].x, m = start[v + 1].x - o0;
        GsVertex g{0, 0, v0, v1, 0, 0, 0};
        const unsigned lo = g.slab(table, v);
        unsigned *list = nbr + 2 * (size_t)o0;
        if (m <= 32) {
#pragma unroll
            for (unsigned k = 0; k < 4; k++) seen[lane + 32 * k] = make_uint2(0xffffffffu, 0xffffffffu);
            const unsigned q = lane < m ? occ[o0 + lane] : 0xffffffffu;
            sq[lane] = q;
            __syncwarp();
            unsigned rank = 0;
            for (unsigned j = 0; j < m; j++) rank += sq[j] < q;
            if (lane < m) {
                const uint2 e = gs_corners(tri, q);
                row[2 * rank] = e.x;
                row[2 * rank + 1] = e.y;
            }
            __syncwarp();
            unsigned u[2], at[2];
#pragma unroll
            for (unsigned k = 0; k < 2; k++) {
                const unsigned e = lane + 32 * k;
                u[k] = e < 2 * m ? row[e] : 0u;
                at[k] = (u[k] * 2654435761u) >> 25;
                if (e >= 2 * m) continue;
                for (;;) {  // at most 64 ids: there is a free slot
                    const unsigned was = atomicCAS(&seen[at[k]].x, 0xffffffffu, u[k]);
                    if (was == 0xffffffffu || was == u[k]) break;
                    at[k] = (at[k] + 1u) & 127u;
                }
                atomicMin(&seen[at[k]].y, e);
            }
            __syncwarp();
#pragma unroll
            for (unsigned k = 0; k < 2; k++) {
                const unsigned e = lane + 32 * k;
                if (e < 2 * m) list[e] = g.take(v, u[k], seen[at[k]].y < e);
            }
            __syncwarp();  // the rows are rewritten for the next vertex
            g.loc = __reduce_add_sync(0xffffffffu, g.loc);
            g.rem = __reduce_add_sync(0xffffffffu, g.rem);
            g.far = __reduce_max_sync(0xffffffffu, g.far);
        } else if (lane == 0) {
            // insertion sort in place
            for (unsigned i = 1; i < m; i++) {
                const unsigned q = occ[o0 + i];
                unsigned j = i;
                while (j > 0 && occ[o0 + j - 1] > q) {
                    occ[o0 + j] = occ[o0 + j - 1];
                    j--;
                }
                occ[o0 + j] = q;
            }
            for (unsigned i = 0; i < m; i++) {
                const uint2 e = gs_corners(tri, occ[o0 + i]);
                list[2 * i] = e.x;
                list[2 * i + 1] = e.y;
            }
            for (unsigned i = 2 * m; i-- > 0;) {  // from the end: the entries before are still ids
                const unsigned u = list[i];
                bool again = false;
                for (unsigned j = 0; j < i; j++) again |= list[j] == u;
                list[i] = g.take(v, u, again);
            }
        }
        const unsigned o = o0 - start[g.a].x;
        if (lane == 0)
            g.write(v, lo, kGsLong | (o < (1u << 17) && m < kGsLost ? m << 9 | o << 15 : kGsLost << 9), word0, ext, ext0, ord,
                    err);
    }
}

// The slab of each slab's highest neighbour, and how many places of the order a slab's passes have
// to lie behind one another for all such neighbours to have had the pass before.  One CTA.
__global__ void __launch_bounds__(1024) k_gs_order(const unsigned *__restrict__ table, unsigned qcap, GsOrder ord) {
    __shared__ unsigned s_lag;
    const unsigned Q = min(__ldg(table), qcap);
    const unsigned *bnd = table + 1, *order = table + 2 + qcap;
    if (threadIdx.x == 0) s_lag = 0;
    for (unsigned x = threadIdx.x; x < Q; x += blockDim.x) ord.place[order[x]] = x;
    __syncthreads();
    unsigned lag = 0;
    for (unsigned q = threadIdx.x; q < Q; q += blockDim.x) {
        unsigned lo = q, hi = Q;  // bnd[lo] <= far < bnd[hi]
        const unsigned far = ord.far[q];
        if (far >= bnd[q])
            while (hi - lo > 1) {
                const unsigned mid = (lo + hi) >> 1;
                if (__ldg(bnd + mid) <= far) lo = mid; else hi = mid;
            }
        ord.far[q] = lo;
        const unsigned from = ord.place[q], to = ord.place[lo];
        if (to > from) lag = max(lag, to - from);
    }
    atomicMax(&s_lag, lag);
    __syncthreads();
    if (threadIdx.x == 0) *ord.lag = s_lag + 1;
}

// ------------------------------------------------------------ launchers

void launch_gs_lists(const float *vq, float4 *pos, const unsigned *tri, unsigned *occ, const uint2 *start, unsigned *nbr, unsigned v0, unsigned v1,
                     unsigned smax, const unsigned *table, unsigned *word0, uint4 *pack, unsigned char *ext,
                     unsigned char *ext0, const GsOrder &ord, unsigned *longs, int *err, cudaStream_t s) {
    k_gs_lists<<<(v1 - v0 + 127) / 128, 128, 0, s>>>(vq, pos, tri, occ, start, v0, v1, smax, table, word0, pack, ext, ext0, ord, longs,
                                                     err);
    // as many CTAs as fit the SMs, or as there can be vertices for
    const unsigned ctas = (v1 - v0 + 63) / 64;
    k_gs_lists_long<<<ctas < 1216u ? ctas : 1216u, 256, 0, s>>>(tri, occ, start, nbr, v0, v1, table, word0, ext, ext0, ord,
                                                                longs, err);
}
void launch_gs_order(const unsigned *table, unsigned qcap, const GsOrder &ord, cudaStream_t s) {
    k_gs_order<<<1, 1024, 0, s>>>(table, qcap, ord);
}

size_t gs_slab_smem(unsigned S) { return gs_smem(S).bytes; }

cudaError_t launch_gs_slab(float4 *pos, unsigned v0, unsigned nv, unsigned smax, const unsigned *table,
                           unsigned qcap, unsigned *next_slab, int P, int threads,
                           const uint2 *start, const unsigned *nbr, const unsigned *word0, const uint4 *pack, unsigned *ext,
                           const unsigned char *ext0, unsigned passes, unsigned stamp, const GsOrder &ord, int *err,
                           float *out, long long spin_cycles, unsigned long long *stats, bool cycles, cudaStream_t s) {
    if (smax == 0 || smax > kGsSlabCap) return cudaErrorInvalidValue;
    const size_t smem = gs_slab_smem(smax);
    // the same registers per thread at most, so as many blocks fit with COUNT
    const void *fn = stats && cycles ? (const void *)k_gs_flow<true> : (const void *)k_gs_flow<false>;
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gs_slab_smem(kGsSlabCap));
    void *args[] = {&pos, &v0, &nv, &smax, (void *)&table, &qcap, &next_slab, (void *)&start, (void *)&nbr,
                    (void *)&word0, (void *)&pack, &ext, (void *)&ext0, &passes, &stamp, (void *)&ord, &out, &err,
                    &spin_cycles, &stats};
    // A cooperative launch: every CTA resident from the start.  (A plain launch would also be
    // safe - a CTA only waits for slabs taken before its own, by CTAs that were running when
    // they took them - but its CTAs can then take the SMs the side stream's kernels wait for.)
    // With one CTA to an SM anyway, and slabs enough to keep most SMs busy, 18 worker warps instead of
    // 14: 3 540 000 vertices 5.43 -> 5.35 ms, 5 550 000 at 0.3 A 5.80 -> 5.64, three passes over 548 000
    // 2.70 -> 2.61 (22 warps 5.38, 5.69 and 2.61).  Two CTAs fit an SM with 512 threads only: 16 frames
    // 1.25 ms, with 640 1.35.
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int block = threads >= 1024 ? 1024 : P <= sms && 2 * P > sms ? 640 : 512;
    return cudaLaunchCooperativeKernel(fn, dim3(P), dim3(block), args, smem, s);
}
void gs_l2_window(int device, cudaStream_t s, const void *p, size_t bytes) {
    int max_persist = 0, max_window = 0;
    cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, device);
    cudaDeviceGetAttribute(&max_window, cudaDevAttrMaxAccessPolicyWindowSize, device);
    cudaStreamAttrValue attr;
    memset(&attr, 0, sizeof(attr));
    if (bytes > 0 && max_persist > 0 && max_window > 0) {
        const size_t window = bytes < (size_t)max_window ? bytes : (size_t)max_window;
        cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, (size_t)max_persist);
        attr.accessPolicyWindow.base_ptr = const_cast<void *>(p);
        attr.accessPolicyWindow.num_bytes = window;
        attr.accessPolicyWindow.hitRatio = window <= (size_t)max_persist ? 1.0f : (float)max_persist / (float)window;
        attr.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
        attr.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
        cudaStreamSetAttribute(s, cudaStreamAttributeAccessPolicyWindow, &attr);
    } else {
        attr.accessPolicyWindow.num_bytes = 0;
        cudaStreamSetAttribute(s, cudaStreamAttributeAccessPolicyWindow, &attr);
        cudaCtxResetPersistingL2Cache();
        cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, 0);
    }
    cudaGetLastError();  // the window is a hint: a refusal leaves the results unchanged
}

int gs_slab_max_blocks(int device, unsigned S, int threads) {
    const void *fn = (const void *)k_gs_flow<false>;
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gs_slab_smem(kGsSlabCap));
    int per_sm = 0, sms = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads >= 1024 ? 1024 : 512, gs_slab_smem(S));
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return per_sm * sms;
}

}  // namespace qses
