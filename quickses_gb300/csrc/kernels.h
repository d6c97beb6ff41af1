// Kernel launchers (host side).  Every launcher enqueues on the given stream only.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "qses_internal.h"

namespace qses {

void launch_atom_minmax(const float *xyz, const float *r, unsigned n, unsigned *mm, cudaStream_t s);
constexpr unsigned kFewAtoms = 8192;  // that are ordered in one launch
void launch_atoms_few(const QGrid &g, const float *xyz, const float *r, unsigned n, unsigned *skey, unsigned *sidx,
                      float4 *atoms, uint2 *cells, cudaStream_t s);
// Atoms and their input numbers in cell order (stable) and the cells' ranges; the sorted keys and
// numbers end up in (key, idx) or, with *alt, in (key2, idx2).
cudaError_t order_atoms(const QGrid &g, const float *xyz, const float *r, unsigned n, unsigned *key, unsigned *key2,
                        unsigned *idx, unsigned *idx2, int bits, float4 *atoms, uint2 *cells, size_t ncell, void *tmp,
                        int *err, cudaStream_t s, int *launches, int *alt);
void launch_atom_hash(const QGrid &g, const float *xyz, unsigned n, unsigned *key, cudaStream_t s);
void launch_atom_gather(const float *xyz, const float *r, const unsigned *skey, const unsigned *sidx, unsigned n,
                        float4 *atoms, uint2 *cells, cudaStream_t s);
void launch_sas(const QGrid &g, const float4 *atoms, const uint2 *cells, unsigned *inMask, unsigned *outMask,
                cudaStream_t s);
// shape: refine tile of 8 x 8 (0), 16 x 8 (1), 16 x 16 (2) or 32 x 16 (3) z-rows; the same
// codes for all.
void launch_edt(const QGrid &g, const unsigned *inMask, const unsigned *outMask, unsigned char *codes,
                unsigned *signMask, cudaStream_t s, int shape = 0);

// words: one per 32 voxels of an owner row, what its row's words before it have (k_mesh.cu).
void launch_mc_count(const QGrid &g, const unsigned *sign, uint2 *rowCount, unsigned *words, cudaStream_t s);
cudaError_t launch_mc_emit(const QGrid &g, const unsigned *sign, const unsigned char *codes, const float *lut,
                           const unsigned *words, const uint2 *rowBase, unsigned *tri, unsigned long long *vkey,
                           cudaStream_t s);
// Vertex ids (vmap, per edge slot), welded positions and their count from the edge keys in owner
// row order (rowBase: the scanned row counts).  skey, sslot: scratch, one entry per edge.  total->y:
// not 0 if the mesh crowds a layer (k_mesh.cu); the results are then launch_weld_sorted's, which
// overwrites vkey, and until it has run launch_remap leaves the corners alone (crowded: &total->y).
size_t weld_tmp_bytes(unsigned layers);
cudaError_t launch_weld(const QGrid &g, const unsigned long long *vkey, const uint2 *rowBase, unsigned ne,
                        unsigned long long *skey, unsigned *sslot, unsigned *vmap, float *vq, uint2 *total, void *tmp,
                        int *err, cudaStream_t s);
constexpr unsigned kWeldSortMin = 4096;  // edges
cudaError_t launch_weld_sorted(const QGrid &g, unsigned long long *vkey, unsigned long long *skey, unsigned *sslot,
                               unsigned ne, unsigned *vmap, float *vq, uint2 *total, int *err, cudaStream_t s,
                               int *launches);
void launch_remap(unsigned *tri, size_t n3, const unsigned *vmap, const unsigned *crowded, cudaStream_t s);
void launch_closest(const QGrid &g, const float *vq, unsigned nv, const float4 *atoms, const uint2 *cells,
                    const unsigned *sorted_to_input, int *asorted, int *ainput, cudaStream_t s);
// Triangles without a repeated corner, in order, to out (which may be tri); their number to *total.
size_t tri_filter_tmp_bytes(unsigned nt);
cudaError_t launch_tri_filter(const unsigned *tri, unsigned nt, unsigned *out, uint2 *total, void *tmp, int *err,
                              cudaStream_t s);
// Neighbour lists by counting: start (nv + 1 entries, zeroed) -> counts -> (scan) -> corner
// occurrences scattered per vertex into occ (n3), in any order.
void launch_csr_count(const unsigned *tri, size_t n3, uint2 *start, unsigned *zero, unsigned nzero, cudaStream_t s);
void launch_csr_scatter(const unsigned *tri, size_t n3, uint2 *start, unsigned *occ, cudaStream_t s);
// Slab table of one Gauss-Seidel wave (device words): [0] Q slabs, [1, Q + 2) their bounds in
// id order (qcap + 1 slots), [qcap + 2, qcap + 2 + Q) the slab ids in the order CTAs take them.
inline size_t gs_table_words(unsigned qcap) { return 2ull * qcap + 2; }
// Several passes in one launch: done (zeroed) passes of each slab, far (zeroed, then filled by
// launch_gs_lists with each slab's highest neighbour id and by launch_gs_order with its slab).
struct GsOrder {
    unsigned *lag, *longs;         // one value each; longs (zeroed): vertices with long lists
    unsigned *done, *far, *place;  // one per slab each
};
// The pass's lists from the occurrences: word0, pack (64 B) per vertex, lists of more than 16
// entries in nbr (2 n3) at twice the vertex's offset (k_smooth.cu); ext, ext0 (may be null): one
// byte per vertex, the neighbours in lower slabs still to come; longs: scratch, one per vertex.
void launch_gs_lists(const float *vq, float4 *pos, const unsigned *tri, unsigned *occ, const uint2 *start, unsigned *nbr, unsigned v0, unsigned v1,
                     unsigned smax, const unsigned *table, unsigned *word0, uint4 *pack, unsigned char *ext,
                     unsigned char *ext0, const GsOrder &ord, unsigned *longs, int *err, cudaStream_t s);
void launch_gs_order(const unsigned *table, unsigned qcap, const GsOrder &ord, cudaStream_t s);
size_t gs_slab_smem(unsigned S);
void launch_from_float4(const float4 *v4, unsigned nv, float *v3, cudaStream_t s);
// Gauss-Seidel passes over vertices [v0, nv) in the table's slabs (each at most smax
// vertices), taken by P persistent CTAs from *next_slab (zeroed).  passes > 1: that many passes,
// each following the one before through the slabs (ext0: the release counters a pass starts with).
// stamp: written to w of every position updated, one more for each pass (another value than any
// position holds before).  threads: 512 or 1024 per slab CTA.  cycles: those of an update's parts too
// (stats[2], [3] and [5]-[7]), which makes it slower.
cudaError_t launch_gs_slab(float4 *pos, unsigned v0, unsigned nv, unsigned smax, const unsigned *table,
                           unsigned qcap, unsigned *next_slab, int P, int threads,
                           const uint2 *start, const unsigned *nbr, const unsigned *word0, const uint4 *pack, unsigned *ext,
                           const unsigned char *ext0, unsigned passes, unsigned stamp, const GsOrder &ord, int *err,
                           float *out, long long spin_cycles, unsigned long long *stats, bool cycles, cudaStream_t s);
int gs_slab_max_blocks(int device, unsigned S, int threads);
constexpr long long kGsSpin = 4000000000ll;  // cycles without progress after which a wait gives up

// Gauss-Seidel launch shape: threads per slab CTA and the slab size aimed at (vertices);
// the result does not depend on it, only the time does.  The cache flags name policies of an
// earlier kernel that read positions through L2; the records in shared memory leave them nothing
// to choose, so they are accepted and, but for kGsPersistL2, without effect on a pass
// (gs_plan_for still splits by kGsSmemPos when no cap is given).
struct GsShape {
    int threads = 512;
    unsigned target = 16384;
    unsigned flags = 0;
    unsigned wave = 0;   // most vertices per slab-kernel launch (0: the whole mesh)
    unsigned cap = 0;    // largest slab (0: 8192 with kGsSmemPos, else 25 000)
};
constexpr unsigned kGsPersistL2 = 4;    // host side: keep the positions in persisting L2 lines
constexpr unsigned kGsSmemPos = 8;
constexpr unsigned kGsSmemPosMaxVerts = 8192;
constexpr unsigned kGsPair = 16;
constexpr unsigned kGsQuad = 32;
inline bool gs_flags_valid(unsigned f) { return f < 64 && (f & (kGsPair | kGsQuad)) != (kGsPair | kGsQuad); }
// Sets (bytes > 0) or clears the stream's L2 persistence window over [p, p + bytes); the
// set-aside is this process's context limit, restored when the window is cleared.
void gs_l2_window(int device, cudaStream_t s, const void *p, size_t bytes);
// Tuned shape for a mesh of nv vertices (batch: many molecules), or the default; biggest: the
// vertices of the largest molecule.
GsShape gs_shape(unsigned nv, bool batch, unsigned biggest, int passes);
void gs_shape_record(unsigned nv, bool batch, unsigned biggest, int passes, GsShape s);
void gs_shape_record_all(bool batch, GsShape s);  // for every such call
int gs_shape_candidates(GsShape *out, int max);
// Tuned refine tile shape (launch_edt `shape`) for grids of G voxels per axis, or the default.
int edt_shape(int G);
void edt_shape_record(int G, int shape);
constexpr int kEdtShapes = 4;
constexpr unsigned kGsSlabMaxVerts = 25000;
constexpr unsigned kGsSlabCap = 11904;  // vertices whose state fits a CTA's shared memory (18 B each)
constexpr unsigned kGsSlabTwo = 5376;   // ... fits twice into an SM's

// ---- batch forms (QBatch: per-molecule grids and offsets in device memory)
void launch_atom_hash_batch(const QBatch &b, const float *xyz, unsigned n, unsigned *key, cudaStream_t s);
void launch_sas_batch(const QBatch &b, unsigned tiles, const float4 *atoms, const uint2 *cells, unsigned *inMask,
                      unsigned *outMask, unsigned *counter, cudaStream_t s);
void launch_edt_batch(const QBatch &b, unsigned tiles, const unsigned *inMask, const unsigned *outMask,
                      unsigned char *codes, unsigned *signMask, unsigned *counter, cudaStream_t s);
// Owner rows a marching-cubes warp covers for a grid with Gc emitted cells per axis.
int mc_rows_per_warp(int Gc);
void launch_mc_count_batch(const QBatch &b, unsigned units, const unsigned *sign, uint2 *rowCount, unsigned *words,
                           cudaStream_t s);
// Words of a molecule's rows, and how many of them a warp of the emission takes (a batch: of the
// words of all; emit_off counts each molecule's in such chunks).
unsigned long long mc_words(int Gc);
unsigned mc_emit_chunk(unsigned long long words);
cudaError_t launch_mc_emit_batch(const QBatch &b, unsigned chunk, unsigned units, const unsigned *sign,
                                 const unsigned char *codes, const unsigned *words, const uint2 *rowBase, unsigned *tri,
                                 unsigned long long *vkey, cudaStream_t s);
// layers: owner planes (Gc + 1) of all molecules; vtx_off receives each molecule's first vertex.
cudaError_t launch_weld_batch(const QBatch &b, unsigned layers, const unsigned long long *vkey, const uint2 *rowBase,
                              unsigned ne, const unsigned *edge_off, unsigned long long *skey, unsigned *sslot,
                              unsigned *vmap, float *vq, unsigned *vmol, unsigned *vtx_off, uint2 *total, void *tmp, int *err,
                              cudaStream_t s);
// bits: of the largest position among the molecules' (with the molecules' numbers at most 64)
cudaError_t launch_weld_sorted_batch(const QBatch &b, unsigned long long *vkey, unsigned long long *skey, unsigned *sslot,
                                     unsigned ne, const unsigned *edge_off, int bits, unsigned *vmap, float *vq,
                                     unsigned *vmol, unsigned *vtx_off, uint2 *total, int *err, cudaStream_t s,
                                     int *launches);
void launch_gather_offsets(const uint2 *excl, const unsigned *at, unsigned n_mol, unsigned n, const uint2 *total,
                           unsigned *outx, unsigned *outy, cudaStream_t s);
void launch_closest_batch(const QBatch &b, const float *vq, const unsigned *vmol, unsigned nv, const float4 *atoms,
                          const uint2 *cells, const unsigned *sorted_to_input, int *asorted, int *ainput,
                          cudaStream_t s);
cudaError_t launch_tri_filter_batch(const QBatch &b, const unsigned *tri, unsigned nt, unsigned *out, unsigned *kept_off,
                                    uint2 *total, void *tmp, int *err, cudaStream_t s);

}  // namespace qses
