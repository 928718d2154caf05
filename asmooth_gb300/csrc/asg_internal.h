// asg_internal.h -- device data layout and kernel launchers shared by the
// translation units of libasmooth_gb300.so (not part of the public C ABI).
//
// Data layout in HBM (one particle set, N particles):
//   pos   float4[N]  x, y, z, w = input index (int bits)   -- Hilbert order
//   vel   float4[N]  vx, vy, vz, dens                        -- Hilbert order
//   igrp  int[N]                                             -- Hilbert order
//   rk    float[N], t33 float[N], idx33 int[N]               -- Hilbert order
// Blocked box tree over the sorted particles (TreeView): boxes of `leaf`
// consecutive particles, then of 32 consecutive boxes, level by level.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace asg {

// process-wide count of kernel launches made by this library
void count_launches(int k);

// Levels of the box tree: leaf = 1 and n = 2^31 - 1 need 7.
constexpr int TREE_LEVELS = 7;
struct TreeView {
    int n;                       // particles
    int leaf;                    // particles per leaf (1..32), the last leaf may hold fewer
    int nlev;                    // levels, level 0 = leaves; the top one has at most 32 boxes
    int cnt[TREE_LEVELS];        // boxes of each level: ceil(n / leaf), then ceil(below / 32)
    long long off[TREE_LEVELS];  // first box of each level in `box`
    const float4* box;           // two float4 per box: lo.x hi.x lo.y hi.y | lo.z hi.z 0 0
};
// the tree's shape for n particles (box not set), and the bytes of its boxes
TreeView tree_shape(int n, int leaf);
size_t tree_box_bytes(int n, int leaf);

// ---- index build (asg_index.cu) -------------------------------------------------
// Staged particles in input order, rec[2i] = x, y, z, igrp (int bits) and rec[2i + 1]
// = vx, vy, vz, dens, from reference Particle records (36 B), device arrays or
// mixed-precision positions (int32 cell index + 3 x uint16 offsets in cells of
// side cs), with the keys of the particles on a grid (keys may be null)
struct KeyGrid {
    float left, scale;  // cell = (x - left) * scale, clamped to 16 bits
    int hilbert;        // Hilbert order; Morton with ASG_SPACE_CURVE=morton
};
KeyGrid key_grid(float left, float right);
void launch_unpack_aos(const void* aos, int n, float4* rec, float* rk_in, const KeyGrid& grid,
                       uint64_t* keys, int* err, cudaStream_t s);
void launch_unpack_soa(const float* x, const float* v, const float* dens, const int* igrp, int n,
                       float4* rec, const KeyGrid& grid, uint64_t* keys, int* err, cudaStream_t s);
void launch_unpack_quant(const int* cell, const uint16_t* off, const float* v, int n, int grid,
                         float left, float cs, float4* rec, const KeyGrid& kgrid, uint64_t* keys,
                         int* err, cudaStream_t s);
// keys over the particles' own bounding cube (d_lohi: 2 ints of scratch)
void launch_own_keys(const float4* rec, int n, int* d_lohi, uint64_t* keys, cudaStream_t s);
// stable LSD radix sort of (keys, vals) on the low `bits` bits; iota: vals0 is not
// read, the values are the input positions; ping-pong buffers; returns which
// buffer (0/1) holds the result.  err |= ERR_SORT if a tile's look-back gives up.
size_t radix_sort_temp_bytes(int n);
int radix_sort32(uint32_t* keys0, int* vals0, uint32_t* keys1, int* vals1, int n, int bits, bool iota,
                 void* temp, int* err, cudaStream_t s);
int radix_sort(uint64_t* keys0, int* vals0, uint64_t* keys1, int* vals1, int n, int bits, bool iota,
               void* temp, int* err, cudaStream_t s);
// the staged particles in the order perm (pos.w: input index), and the boxes of t
// over them; rk_in may be null (0)
void launch_gather(int* perm, const float4* rec, const float* rk_in, const TreeView& t, float4* pos,
                   float4* vel, int* igrp, float* rk, cudaStream_t s);
void launch_iota(int* a, int n, cudaStream_t s);
// exclusive scan of uint32 counts (in place); temp from scan_temp_bytes
size_t scan_temp_bytes(size_t n);
void exclusive_scan_u32(uint32_t* data, size_t n, void* temp, cudaStream_t s);

// ---- neighbour search (asg_knn.cu) -------------------------------------------
// Leaves k_knn_t33 scanned, per 32-query bundle: word 0 = their count (-1 when
// more than KNN_LIST), then the leaf numbers.  k_dens_scatter visits these
// instead of walking the tree again, which takes long for the bundles at the edge
// of a halo, whose lists are the longest: with room for 96 leaves the density
// took 206 us on 377 k particles in NFW halos, for 128 211, 192 172, 256 171.
constexpr int KNN_LIST = 192;
inline size_t knn_list_words(int n) { return (size_t)((n + 31) / 32) * (KNN_LIST + 1); }
// t33, rk = sqrtf(t33), idx33 = -1 (no tie at the 33rd) or -2 (ties to resolve);
// blist (knn_list_words ints, or null) receives the scanned leaves; warps: 2 or
// 4 warps per block (tuning; leaves of 16 particles always run 1)
void launch_knn_t33(const float4* pos, const TreeView& t, float* t33, float* rk, int* idx33,
                    int* blist, int* err, cudaStream_t s, int warps = 2);
// idx33 = input index of the 33rd key, for flagged queries (all = 0) or every query;
// dexp (n ints, or null) and acc (n uint64) are prepared for launch_dens
void launch_knn_ties(const float4* pos, const TreeView& t, const float* t33, int* idx33,
                     int all, const int* blist, const float* rk, int* dexp, unsigned long long* acc,
                     int* err, cudaStream_t s);
// vel[j].w (dens) += the tent weights j receives as one of the 32 nearest;
// dexp and acc as launch_knn_ties prepared them; blist from launch_knn_t33 or null
void launch_dens(const float4* pos, const TreeView& t, const float* t33, const int* idx33,
                 const int* blist, const float* rk, const int* dexp, unsigned long long* acc,
                 float4* vel, cudaStream_t s);

// ---- mesh deposit (asg_deposit.cu) ---------------------------------------------
struct MeshJob {
    int nc;           // cells per dimension
    float dx;         // boxsize / nc (host float division, as the reference)
    float ncf;        // (float)nc
    int tiles[3];     // tiles per dimension (x, y, z)
    int tile_begin;   // first global tile id of this mesh
    float* mesh;      // 6*nc^3 floats (reference layout) or nc^3 (density only)
    double* partial;  // per-tile FP64 partial sums, 2 per tile (n, halo)
};
constexpr int MAX_MESHES = 8;
struct DepositParams {
    int n_jobs;
    MeshJob job[MAX_MESHES];
    float boxsize;
    float rbox;       // 1/boxsize rounded to nearest (for div_rn_by)
    int sign;
    int periodic;
    float offset[3];  // periodic: rank cube offset
    int density_only;
    int seg;          // most pairs per work item of the persistent deposit (tuning, > 0)
    int mma;          // the deposit engine: 1 the tensor cores, 0 the CUDA cores
    int wide;         // tensor cores, six channels: the wider tiles
    int shift[3];     // log2 of the tile edges in cells (deposit_tile_shape)
    int log_parts;    // log2 of the warps that make a bundle's entries (deposit_log_parts)
};
// the tile shape of the engine p.mma
void deposit_tile_shape(DepositParams& p);
// scratch of one deposit: particle records, entries (a bundle of 32 particles and
// those of them that touch a tile), work items
struct DepositScratch {
    float4* rec;          // [2n] x', y', z', h (-h: halo channel, 0: skipped) | dens, v
    uint32_t* count;      // [units+1] entries per part of a bundle, then their exclusive scan
    void* scan_tmp_n;     // scan scratch for units+1 entries
    uint2* entry;         // [entries] bundle, lane mask, as emitted
    uint2* list;          // [entries] the same in key order
    uint32_t* keys0;      // [entries] tile << 5 | image (periodic), else tile; ping-pong with keys1
    uint32_t* keys1;
    int* vals0;           // [entries] emission number, ping-pong with vals1
    int* vals1;
    uint32_t* first;      // [entries+1] first pair of each sorted entry
    void* scan_tmp_e;     // scan scratch for entries+1
    void* sort_tmp;       // radix sort scratch for the entries
    uint32_t* tentry;     // [T+1] first entry of each tile
    uint32_t* item_off;   // [T+1] exclusive scan of work items per tile
    uint32_t* merge;      // [T] tiles with several items
    uint32_t* item_tile;  // [items] tile of each work item
    void* scan_tmp_t;     // scan scratch for T+1 entries
    float* partial;       // [items] partial tiles of multi-segment tiles
    int* counters;        // 32 bytes: work counter of the persistent kernel, length of merge's
                          // front, number of pairs (64 bits), length of merge's back
};
size_t deposit_prep_bytes(int n);
// log2 of the warps that share the making of a bundle's entries (units = bundles << log_parts)
int deposit_log_parts(int n, bool periodic, long long total_tiles);
// pairs from which on six channels take the wider tiles
unsigned long long deposit_wide_pairs(int n);
size_t deposit_tile_bytes(int total_tiles);
size_t deposit_entry_bytes(uint32_t entries);
// the per-entry arrays of w inside one block of deposit_entry_bytes
void deposit_entry_layout(void* base, uint32_t entries, DepositScratch& w);
// the entries or pairs that a plan for n of them has room for: a sixteenth more
uint32_t deposit_headroom(uint32_t n);
// work items that `npairs` pairs make at most, with at most `most` pairs each
uint32_t deposit_max_items(int total_tiles, uint32_t npairs, int most, bool n_alone);
int deposit_default_mma();
size_t deposit_item_words(const DepositParams& p);  // of an item's partial tile
size_t deposit_partial_bytes(uint32_t items, size_t item_words);
// pass 1: particle records and entry counts; count[units] then holds the number
// of entries, counters[2..3] the number of pairs
void launch_deposit_prep(const float4* pos, const float4* vel, const int* igrp, const float* rk,
                         int n, const DepositParams& p, DepositScratch& w, int* err,
                         cudaStream_t s);
// pass 2: emit and sort the entries, deposit every (tile, segment), merge multi-segment tiles.
// padded = false: `entries` is the exact number (read back from count[units]);
// padded = true: it is the arrays' capacity, the number stays on the device
// (no host synchronisation, e.g. under stream capture) and a larger one sets ERR_CAP,
// as do more than max_items work items
void launch_deposit_run(int n, const DepositParams& p, int total_tiles, uint32_t entries,
                        uint32_t max_items, bool padded, DepositScratch& w, int* err, cudaStream_t s);
// totals: 2 doubles per mesh (n, halo), then scratch: deposit_totals_bytes
size_t deposit_totals_bytes(int n_nc);
void launch_deposit_totals(const DepositParams& p, int total_tiles, double* totals, cudaStream_t s);
void launch_normalise(float* mesh, int nc, float vol, cudaStream_t s);

// ---- FOF and SO halos (asg_fof.cu) -----------------------------------------------
void launch_fof_link(const float4* pos, const TreeView& t, float ll, int* parent, int* err,
                     cudaStream_t s);
void launch_fof_finish(const float4* pos, int n, int* parent, int* minin, int* mark,
                       cudaStream_t s);
void launch_fof_label(int n, const int* parent, const int* minin, const uint32_t* scan,
                      int* igrp_sorted, cudaStream_t s);
void launch_mark_halos(const float4* pos, const TreeView& t, const float* halos, int nh,
                       float left, float right, int* igrp, long long* counts, double* mass8,
                       cudaStream_t s);
void launch_count_labels(const int* igrp, int n, uint32_t* counts, cudaStream_t s);
void launch_keep_mask(uint32_t* counts, int ngrp, int threshold, cudaStream_t s);
void launch_relabel(int* igrp, int n, const uint32_t* scan, const uint32_t* keep, cudaStream_t s);

// ---- periodic buffer shell of a single-cube run (asg_shell.cu) ------------------------------
// base[b][d]: first slot of the copies of bin b sent in direction d (-1: none)
struct ShellPlan {
    int base[27][27];
};
void launch_shell_bins(const float4* rec, int n, float lt, float rt, uint32_t* keys0, int* vals0,
                       uint32_t* keys1, int* vals1, void* sort_tmp, uint32_t* start, uint32_t* end,
                       const uint32_t** keys, const int** order, int* err, cudaStream_t s);
// staged particles with all copies; rk and ark may both be null
void launch_shell_emit(const float4* rec, const float* rk, const uint32_t* keys, const int* order,
                       const uint32_t* start, int n, const ShellPlan& plan, float L, float4* arec,
                       float* ark, cudaStream_t s);
// keep -bf*L < x < L + bf*L, with keys; flags has n_all + 1 words and ends as the exclusive scan
void launch_shell_filter(const float4* arec, const float* ark, int n_all, float lo, float hi,
                         uint32_t* flags, void* scan_tmp, float4* rec, float* rk, const KeyGrid& grid,
                         uint64_t* out_keys, cudaStream_t s);

// ---- particle file payloads (asg_decode.cu) ----------------------------------------------
void launch_decode_xv(const float* xv, int n, const float* shift, float4* rec, int* err, cudaStream_t s);
size_t zip_scratch_bytes(int ncell);
// *start: first particle of every cell, ncell + 1 entries (the last = total)
void launch_zip_counts(const uint8_t* c8, const int* c32, int n32, int ncell, void* scratch,
                       uint32_t** start, int* err, cudaStream_t s);
void launch_zip_particles(const uint8_t* off, const int16_t* vq, const uint32_t* start, int ncell,
                          int nc, int n, int mesh_scale, float v_r2i, const float* shift,
                          float4* rec, cudaStream_t s);

// ---- FOF halo catalogue and file formats (asg_output.cu) ----------------------------------
// records {x[3], v[3], int nfof} of labels 1..nhalo with centre inside (0, boxsize)^3, label
// order, into out (device, 7*nhalo words) and *nlocal (device).  The particles are either
// sorted arrays (pos.w the caller's array index) or, with igrp null, staged records in the
// caller's order (pos = rec, vel = rec + 1).
size_t fof_catalogue_bytes(int n, int nhalo);
void launch_fof_catalogue(const float4* pos, const float4* vel, const int* igrp, int n,
                          int nhalo, float boxsize, void* scratch, float* out, uint32_t* nlocal,
                          int* err, cudaStream_t s);
int write_mesh_files(const char* base, int inode, const float* mesh, int nc);
int write_fof_file(const char* filename, const float* rec, int nlocal);

// ---- output (asg_index.cu) ------------------------------------------------------------
// write reference Particle records in input order from the sorted fields
void launch_pack_aos(const int* perm, const float4* pos, const float4* vel, const float* rk,
                     const int* igrp, int n, void* aos, cudaStream_t s);
// the same from staged records (rk may be null: 0)
void launch_pack_staged(const float4* rec, const float* rk, int n, void* aos, cudaStream_t s);
// sorted fields to input order (dens is vel.w); outputs may be null
void launch_scatter_fields(const int* perm, const float* rk, const float4* vel, const int* igrp,
                           int n, float* rk_out, float* dens_out, int* igrp_out, cudaStream_t s);

// ---- loading ahead (the allocation-free search) ----------------------------------------
// load the kernels that such a call can launch, whatever its particle count; false: a
// CUDA error
bool load_small_set_kernels();
bool load_search_kernels();

}  // namespace asg
