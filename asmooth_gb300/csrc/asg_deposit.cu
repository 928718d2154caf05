// asg_deposit.cu -- adaptive kernel deposit onto coarse meshes
// (assign_on_mesh, coarse_mesh.cpp:45-127; the periodic assign_on_global_mesh,
// global_mesh.cpp:25-123; the n-only assign_on_density_mesh, :212-269), the
// FP64 mass totals (mesh_total / check_total_mass, coarse_mesh.cpp:35-43,
// clumping_tree_main.cpp:578-600) and the write_mesh_separate normalisation
// (coarse_mesh.cpp:158-171).
//
// Per particle and per cell: the cell range [left, right) per axis is the
// reference's float expression ((x -+ h)/boxsize)*nc, and ker3 = (k0*k1)*k2 as
// in the reference; each 1-D weight k is the tent's integral over the cell,
// evaluated more accurately than the reference's ker_integ(s1, s1 + ds): the
// cell edges' offsets are fma(i, dx, -x)*hinv and the integral uses
// cancellation-free forms (tent_integral_rn).  The reference's float weights
// err by up to 1.1e-5 relative in a mesh cell against FP64 on the 256^3 cube
// (a halo particle's sliver weight in a thin cell); these stay near 1e-6.
//
// Sort by target tile, then gather; deterministic, no atomics on the mesh.
//  (1) k_dep_prep: one 32-byte record per particle (position, h, dens, v).  A
//      particle makes one (tile, image) pair per tile its exact cell range
//      touches; a bundle of 32 consecutive particles makes one entry (tile,
//      image, lane mask) per tile that any of them touches, counted here.
//  (2) k_entries: the entries, at offsets from an exclusive scan (so the emit
//      order is the particle order).
//  (3) a stable radix sort of the entries by key = tile << 5 | image (the tile
//      alone without periodic images) groups each tile's particles in particle
//      order; k_tile_items finds each tile's pairs and cuts them into work items.
//  (4) k_deposit_mma: a persistent kernel whose warps take work items and sum
//      the outer products of each item's pairs on the tensor cores
//      (k_deposit_items on the CUDA cores with ASG_DEPOSIT=simt);
//      k_merge_tiles adds the partial tiles of tiles with several items in item
//      order.
// n, c and halo are double-float (two-sum) sums; the FP64 totals are summed per
// pair.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "asg_common.cuh"
#include "asg_internal.h"

namespace asg {

constexpr int TS = 8;             // tile edge in cells of the CUDA-core engine
constexpr int TC = TS * TS * TS;   // cells of such a tile
// Tiles of the tensor-core engine, cells in x, y, z.  A pair costs the dense tile
// whatever it touches, so small tiles waste less on the narrow supports of halo
// particles and of coarse meshes, and their sums fit a warp; wide supports then
// reach more tiles.  All six channels: 8 x 4 x 4 (6.6 pairs per particle on the
// 256^3 step's three meshes; 4.5 with 8 x 8 x 8, 8.2 with 4 x 4 x 4).  n alone: 8
// x 8 x 8, whose one channel takes no more registers and whose meshes are the
// finest (on 160^3 cells for 512 k particles 13 pairs per particle, 33 with 8 x 4 x 4).
// WIDE: 8 x 8 x 4 for the six channels of wide supports (deposit_wide_pairs).
template <int NCH, bool WIDE>
struct TileShape {
    static constexpr int X = 8, Y = NCH == 1 || WIDE ? 8 : 4, Z = NCH == 1 ? 8 : 4;
    static constexpr int CELLS = X * Y * Z;
};
constexpr int PW = 9, PW_ALONE = 2;  // partial words per cell: all channels, n alone
__host__ __device__ inline int partial_words(const DepositParams& P) { return P.density_only ? PW_ALONE : PW; }
constexpr int IMG_BITS = 5;        // periodic images per pair: up to 3 x 3 x 3
// key bits of the image index: none without periodic images (every pair is
// image 0), so the pair sort needs fewer passes
__host__ __device__ inline int img_bits(const DepositParams& P) { return P.periodic ? IMG_BITS : 0; }
constexpr unsigned FULLM = 0xffffffffu;

// ---------------------------------------------------------------------------
// geometry helpers
// ---------------------------------------------------------------------------
struct TileGeo {
    int job, local, nc;
    int O[3], E[3];
};

__device__ __forceinline__ TileGeo tile_geo(const DepositParams& P, int tile)
{
    int jb = 0;
    while (jb + 1 < P.n_jobs && tile >= P.job[jb + 1].tile_begin) ++jb;
    const MeshJob& J = P.job[jb];
    TileGeo g;
    g.job = jb;
    g.local = tile - J.tile_begin;
    g.nc = J.nc;
    const int tx = g.local % J.tiles[0];
    const int ty = (g.local / J.tiles[0]) % J.tiles[1];
    const int tz = g.local / (J.tiles[0] * J.tiles[1]);
    g.O[0] = tx << P.shift[0]; g.O[1] = ty << P.shift[1]; g.O[2] = tz << P.shift[2];
    for (int a = 0; a < 3; ++a) g.E[a] = min(1 << P.shift[a], g.nc - g.O[a]);
    return g;
}

__device__ __forceinline__ int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

// cells [left, right) of one axis (unwrapped for the periodic mesh) and the
// mesh images k_lo .. k_lo+nk-1 whose shifted range meets [0, nc)
struct AxisRange {
    int left, right, k_lo, nk;
};

__device__ __forceinline__ AxisRange axis_range(float exlo, float exhi, const MeshJob& J, int nc,
                                                bool periodic)
{
    AxisRange r;
    const float fl = __fmul_rn(exlo, J.ncf);
    const float fr = __fmul_rn(exhi, J.ncf);
    if (!periodic) {  // coarse_mesh.cpp:72-75
        r.left = max(0, __float2int_rz(fl));
        r.right = min(nc, 1 + __float2int_rz(fr));
        r.k_lo = 0;
        r.nk = r.left < r.right ? 1 : 0;
    } else {  // global_mesh.cpp:66-69; cells wrap modulo nc (:85-87)
        r.left = (int)floorf(fl);
        r.right = 1 + (int)ceilf(fr);
        r.k_lo = floor_div(r.left, nc);
        r.nk = floor_div(r.right - 1, nc) - r.k_lo + 1;
    }
    return r;
}

// ---------------------------------------------------------------------------
// (1) per-particle records
// ---------------------------------------------------------------------------
constexpr int FLAG_HALO = 1;  // sign*igrp > 0: deposit into the halo channel
constexpr int FLAG_SKIP = 2;  // periodic particle outside [0, L) or a halo in an n-only mesh

// particle i's record as the deposit kernels use it: A = (x', 1/h), B = ((x'-h)/L,
// dens), Cc = ((x'+h)/L, vx), D = (vy, vz, flags)
__device__ __forceinline__ void load_dep_rec(const float4* __restrict__ rec, int i, float L,
                                             float rL, float4& A, float4& B, float4& Cc, float4& D)
{
    const float4 a = rec[2 * (size_t)i], b = rec[2 * (size_t)i + 1];
    const float h = fabsf(a.w);
    const int flags = (a.w < 0.0f ? FLAG_HALO : 0) | (h > 0.0f ? 0 : FLAG_SKIP);
    A = make_float4(a.x, a.y, a.z, __frcp_rn(h));  // 1/h correctly rounded
    B = make_float4(div_rn_by(__fsub_rn(a.x, h), L, rL), div_rn_by(__fsub_rn(a.y, h), L, rL),
                    div_rn_by(__fsub_rn(a.z, h), L, rL), b.x);
    Cc = make_float4(div_rn_by(__fadd_rn(a.x, h), L, rL), div_rn_by(__fadd_rn(a.y, h), L, rL),
                     div_rn_by(__fadd_rn(a.z, h), L, rL), b.y);
    D = make_float4(b.z, b.w, __int_as_float(flags), 0.0f);
}

// tiles of one axis touched by image k: [t0, t1] (empty when t0 > t1)
__device__ __forceinline__ void image_tiles(const AxisRange& r, int k, int nc, int shift, int& t0,
                                            int& t1)
{
    const int c0 = max(r.left - k * nc, 0), c1 = min(r.right - k * nc, nc);
    t0 = c0 >> shift;
    t1 = c1 > c0 ? (c1 - 1) >> shift : t0 - 1;
}

// Every entry (tile, image, mask) of the warp's 32 particles with cell-range edges
// lo and hi (per axis, / boxsize; live: the lane deposits): f(tile, image, mask),
// called by the whole warp, an entry's mask the lanes that touch the tile.  Per
// mesh and image the warp goes through the tiles of the union of its lanes' tile
// boxes; where that holds many more tiles than the lanes touch (particles far
// apart), through each lane's own tiles, one lane after another.  Either way the
// particles of a tile come in lane order.  SPLIT: of the warps with the same bundle
// (a power of two; a template, as reading their number costs 2% of a large deposit)
// each takes the rows of tiles whose y + z falls to it.
// count(entries, pairs) instead of f with COUNT: the lanes' own boxes give the pairs,
// and a row of tiles is one union of bit masks.
template <bool PERIODIC, bool SPLIT, bool COUNT, class F>
__device__ __forceinline__ void for_entries(const DepositParams& P, const float (&lo)[3],
                                            const float (&hi)[3], bool live, int part, int* err, F f)
{
    const int parts = SPLIT ? 1 << P.log_parts : 1;
    // the first row of tiles from y on, at z, that falls to this warp
    auto first_row = [&](int y, int z) { return SPLIT ? y + ((part - y - z) & (parts - 1)) : y; };
    for (int jb = 0; jb < P.n_jobs; ++jb) {
        const MeshJob& J = P.job[jb];
        const int nc = J.nc;
        AxisRange r[3];
        bool on = live;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            r[a] = axis_range(lo[a], hi[a], J, nc, PERIODIC);
            on = on && r[a].nk > 0;
        }
        if (PERIODIC && on && (r[0].nk > 3 || r[1].nk > 3 || r[2].nk > 3)) {  // wider than two mesh periods
            atomicOr(err, ERR_RANGE);
            on = false;
        }
        if (!__any_sync(FULLM, on)) continue;
        // one image of the mesh per axis (nx, ny, nz: the lane's 0th, 1st or 2nd), of
        // the lanes of `group`
        auto one_image = [&](bool group, int nx, int ny, int nz) {
            const int dk[3] = {nx, ny, nz};
            const int image = nz * 9 + ny * 3 + nx;
            int t0[3], t1[3];  // the lane's tiles
            bool in = group;
            unsigned own = 1;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                image_tiles(r[a], PERIODIC ? r[a].k_lo + dk[a] : 0, nc, P.shift[a], t0[a], t1[a]);
                in = in && (!PERIODIC || (dk[a] < r[a].nk && t0[a] <= t1[a]));
                own *= (unsigned)(t1[a] - t0[a] + 1);
            }
            unsigned lanes = PERIODIC ? __ballot_sync(FULLM, in) : ~0u;
            if (PERIODIC && !lanes) return;
            int u0[3], u1[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (!in) { t0[a] = INT_MAX; t1[a] = -1; }  // no tiles
                u0[a] = (int)__reduce_min_sync(FULLM, (unsigned)t0[a]);
                u1[a] = __reduce_max_sync(FULLM, t1[a]);
            }
            if (!in) own = 0;
            const unsigned touched = __reduce_add_sync(FULLM, min(own, 1u << 24));
            const unsigned wx = u1[0] - u0[0] + 1, wy = u1[1] - u0[1] + 1, wz = u1[2] - u0[2] + 1;
            if constexpr (COUNT) f(0u, !SPLIT || part == 0 ? own : 0u);
            if ((unsigned long long)(wx * wy) * wz <= 2ull * touched + 64) {
                // of 32 tiles from x on, those that the lane touches
                auto touches = [&](int x) {
                    const int a = max(t0[0] - x, 0), b = min(t1[0] - x, 31);
                    return a <= b ? (2u << (b & 31)) - (1u << (a & 31)) : 0u;
                };
                const unsigned first32 = COUNT ? touches(u0[0]) : 0u;
                for (int tz = u0[2]; tz <= u1[2]; ++tz) {
                    const bool inz = t0[2] <= tz && tz <= t1[2];
                    for (int ty = first_row(u0[1], tz); ty <= u1[1]; ty += parts) {
                        const bool iny = inz && t0[1] <= ty && ty <= t1[1];
                        if constexpr (COUNT) {
                            f((unsigned)__popc(__reduce_or_sync(FULLM, iny ? first32 : 0u)), 0u);
                            for (int tx = u0[0] + 32; tx <= u1[0]; tx += 32)
                                f((unsigned)__popc(__reduce_or_sync(FULLM, iny ? touches(tx) : 0u)), 0u);
                        } else {
                            int tile = J.tile_begin + (tz * J.tiles[1] + ty) * J.tiles[0] + u0[0];
                            for (int tx = u0[0]; tx <= u1[0]; ++tx, ++tile) {
                                const unsigned m = __ballot_sync(FULLM, iny && t0[0] <= tx && tx <= t1[0]);
                                if (m) f(tile, image, m);
                            }
                        }
                    }
                }
            } else {
                lanes = __ballot_sync(FULLM, in);
                while (lanes) {
                    const int l = __ffs(lanes) - 1;
                    lanes &= lanes - 1;
                    const int x0 = __shfl_sync(FULLM, t0[0], l), x1 = __shfl_sync(FULLM, t1[0], l);
                    const int y0 = __shfl_sync(FULLM, t0[1], l), y1 = __shfl_sync(FULLM, t1[1], l);
                    const int z0 = __shfl_sync(FULLM, t0[2], l), z1 = __shfl_sync(FULLM, t1[2], l);
                    for (int tz = z0; tz <= z1; ++tz)
                        for (int ty = first_row(y0, tz); ty <= y1; ty += parts)
                            if constexpr (COUNT)
                                f((unsigned)(x1 - x0 + 1), 0u);
                            else
                                for (int tx = x0; tx <= x1; ++tx)
                                    f(J.tile_begin + (tz * J.tiles[1] + ty) * J.tiles[0] + tx, image, 1u << l);
                }
            }
        };
        if constexpr (PERIODIC) {
            // The lanes of the same first image go together: their n-th images lie together,
            // while those of a lane that reaches over the mesh's edge and of its neighbour
            // that does not lie at opposite ends of the mesh, and a union of both is all of
            // it (262,144 particles on 383^3 cells 6.1 -> 5.0 ms, 13,840 on 95^3 485 -> 422
            // us).  All lanes together where the mesh has few tiles, as each group costs what
            // 128 tiles do (4096 particles on 31^3 92, in groups 96), and where the bundle's
            // particles are far apart (more than 8 groups).
            const int first = (r[0].k_lo & 1023) | (r[1].k_lo & 1023) << 10 | (r[2].k_lo & 1023) << 20;
            const unsigned same = __match_any_sync(FULLM, on ? first : -1);
            unsigned leaders = __ballot_sync(FULLM, on && (same & lanemask_lt()) == 0u);
            const bool together = __popc(leaders) > 8 || J.tiles[0] * J.tiles[1] * J.tiles[2] < 128 * parts;
            if (together) leaders &= 0u - leaders;
            for (; leaders; leaders &= leaders - 1) {
                const int lead = __shfl_sync(FULLM, first, __ffs(leaders) - 1);
                const bool group = on && (together || first == lead);
                int most[3];  // images per axis
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    most[a] = (int)__reduce_max_sync(FULLM, (unsigned)(group ? r[a].nk : 0));
                for (int nz = 0; nz < most[2]; ++nz)
                    for (int ny = 0; ny < most[1]; ++ny)
                        for (int nx = 0; nx < most[0]; ++nx) one_image(group, nx, ny, nz);
            }
        } else {
            one_image(on, 0, 0, 0);
        }
    }
}

// One 32-byte record per particle: (x', y', z', h') and (dens, vx, vy, vz),
// with x' the deposit position (plus the rank offset when periodic) and h' = h,
// -h when the particle deposits into the halo channel, 0 when it deposits
// nothing.  The cell-range edges (x' -+ h)/L and 1/h are recomputed from it
// where they are needed (load_dep_rec), with the same rounded operations.
// counts: the entries of each part of each bundle, then 0; *pairs += the pairs.
template <bool PERIODIC, bool SPLIT>
__global__ void k_dep_prep(const float4* __restrict__ pos, const float4* __restrict__ vel,
                           const int* __restrict__ igrp, const float* __restrict__ rk, int n,
                           const __grid_constant__ DepositParams P, float4* __restrict__ rec,
                           uint32_t* __restrict__ counts, unsigned long long* __restrict__ pairs,
                           int* err)
{
    grid_begin();
    __shared__ unsigned long long block_pairs;  // one atomic per block: 0.57 M on one word took 0.3 ms
    const int log_parts = SPLIT ? P.log_parts : 0;
    const int unit = (blockIdx.x * blockDim.x + threadIdx.x) / 32, part = unit & ((1 << log_parts) - 1);
    const int i = (unit >> log_parts) * 32 + (threadIdx.x & 31);
    const int bundles = (n + 31) / 32;
    if (threadIdx.x == 0) block_pairs = 0ull;
    if (blockIdx.x == 0 && threadIdx.x == 0) counts[bundles << log_parts] = 0u;
    __syncthreads();
    bool live = i < n;
    const int ii = live ? i : n - 1;
    const float4 p = pos[ii];
    const float4 v = vel[ii];
    const float h = rk[ii];
    const bool good = h > 0.0f && h < INFINITY;
    if (live && !good) atomicOr(err, ERR_ZERO_RK);
    const float L = P.boxsize;
    const bool halo = (P.sign * igrp[ii]) > 0;
    bool skip = !good || (P.density_only && halo);
    float x[3] = {p.x, p.y, p.z};
    if constexpr (PERIODIC) {  // global_mesh.cpp:52-61: skip outside the cube, then add the offset
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (x[a] < 0.0f || x[a] >= L) skip = true;
            x[a] = __fadd_rn(x[a], P.offset[a]);
        }
    }
    if (live && part == 0) {
        rec[2 * (size_t)i] = make_float4(x[0], x[1], x[2], skip ? 0.0f : (halo ? -h : h));
        rec[2 * (size_t)i + 1] = make_float4(v.w, v.x, v.y, v.z);
    }
    live = live && !skip;
    float lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {  // as load_dep_rec
        lo[a] = div_rn_by(__fsub_rn(x[a], h), L, P.rbox);
        hi[a] = div_rn_by(__fadd_rn(x[a], h), L, P.rbox);
    }
    uint32_t cnt = 0;
    unsigned long long np = 0;  // this lane's
    for_entries<PERIODIC, SPLIT, true>(P, lo, hi, live, part, err, [&](unsigned entries, unsigned pairs) {
        cnt += entries;
        np += pairs;
    });
    const unsigned np_lo = __reduce_add_sync(FULLM, (unsigned)np & 0xffffffu);
    const unsigned np_hi = __reduce_add_sync(FULLM, (unsigned)(np >> 24));
    if ((i & 31) == 0 && i < n) {
        counts[unit] = cnt;
        if (!SPLIT || part == 0) atomicAdd(&block_pairs, ((unsigned long long)np_hi << 24) + np_lo);
    }
    __syncthreads();
    if (threadIdx.x == 0 && block_pairs) atomicAdd(pairs, block_pairs);
}

// ---------------------------------------------------------------------------
// (2) entries
// ---------------------------------------------------------------------------
// Entries instead of pairs: consecutive particles mostly touch the same tiles, so
// an entry stands for about ten pairs, and what is sorted shrinks by as much: on
// the 256^3 step pairs, their sort and the tiles' bounds took 4.2 ms, entries with
// the same 2.0 ms.
// entry o is written only when o < cap (the entry arrays' capacity); one beyond
// it sets ERR_CAP instead
template <bool PERIODIC, bool SPLIT>
__global__ void k_entries(const float4* __restrict__ rec, int n, const __grid_constant__ DepositParams P,
                          const uint32_t* __restrict__ offs, uint32_t* __restrict__ keys,
                          uint2* __restrict__ entry, uint32_t cap, int* err)
{
    grid_begin();
    const int lane = threadIdx.x & 31;
    const int unit = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int log_parts = SPLIT ? P.log_parts : 0;
    const int i = (unit >> log_parts) * 32 + lane;
    if ((i & ~31) >= n) return;
    float4 a, b, c, d;
    load_dep_rec(rec, min(i, n - 1), P.boxsize, P.rbox, a, b, c, d);
    const bool live = i < n && !(__float_as_int(d.z) & FLAG_SKIP);
    const float lo[3] = {b.x, b.y, b.z}, hi[3] = {c.x, c.y, c.z};
    uint32_t o = offs[unit];    // the next group of up to 32 entries goes here
    int held = 0;               // entries held by the lanes below it
    uint32_t key = 0, mask = 0;
    auto store = [&]() {
        if (lane < held) {
            if (o + lane < cap) {
                keys[o + lane] = key;
                entry[o + lane] = make_uint2((uint32_t)(i >> 5), mask);
            } else {
                atomicOr(err, ERR_CAP);
            }
        }
        o += held;
        held = 0;
    };
    for_entries<PERIODIC, SPLIT, false>(P, lo, hi, live, unit & ((1 << log_parts) - 1), err, [&](int tile, int image, unsigned m) {
        if (lane == held) {
            key = PERIODIC ? ((uint32_t)tile << IMG_BITS) | (uint32_t)image : (uint32_t)tile;
            mask = m;
        }
        if (++held == 32) store();
    });
    store();
}

// entries [*count, cap) of a pre-sized array: key of tile T (past the last real
// tile), so they sort last and belong to no tile
__global__ void k_pad_entries(uint32_t* __restrict__ keys, uint2* __restrict__ entry,
                              const uint32_t* __restrict__ count, uint32_t cap, uint32_t pad_key)
{
    grid_begin();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cap || j < *count) return;
    keys[j] = pad_key;
    entry[j] = make_uint2(0u, 0u);
}

// the entries in key order, and their pair counts (then scanned in place, in 32 bits:
// a captured call whose pairs outgrew them sets ERR_CAP and has none)
__global__ void k_sorted_entries(const int* __restrict__ order, const uint2* __restrict__ entry,
                                 uint32_t count, const unsigned long long* __restrict__ pairs,
                                 uint2* __restrict__ list, uint32_t* __restrict__ first, int* err)
{
    grid_begin();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    const bool many = *pairs > (unsigned long long)INT_MAX;
    if (j == count) {
        first[j] = 0u;
        if (many) atomicOr(err, ERR_CAP);
    }
    if (j >= count) return;
    // not in order when the sort gave up: no pairs at all
    const uint2 e = many || (*err & ERR_SORT) ? make_uint2(0u, 0u) : entry[order[j]];
    list[j] = e;
    first[j] = (uint32_t)__popc(e.y);
}

constexpr int MERGE_FEW = 8;  // items of a tile that one warp merges by itself

// Pairs per work item, at most `most`.  An item is a serial chain for its warp, so
// a small set takes short items and all warps: a quarter of the pairs a warp
// would get if the items were dealt out evenly over 24 warps on 152 SMs, in steps
// of the 64 pairs between two flushes; half of them for n alone, whose larger
// partial tiles cost more to merge (the deposit of 512 k particles on 160^3 cells 381
// -> 363 us; with all channels a half costs 5% more on 1.2 to 2.5 M particles).  One
// item length of 4096 pairs left a set of 13,840 particles to 20 warps: 354 us
// against 18.
constexpr int ITEM_SHARE = 4 * 24 * 152;
__device__ __forceinline__ int deposit_seg(const int* __restrict__ counters, int most, bool n_alone)
{
    const unsigned long long pairs = *reinterpret_cast<const unsigned long long*>(counters + 2);
    const unsigned long long seg = (pairs / (n_alone ? ITEM_SHARE / 2 : ITEM_SHARE) + 64) & ~63ull;
    return (int)min(seg, (unsigned long long)most);
}

// tentry[t]: the first entry of tile t (tentry[T]: past the last real tile), by a
// search of the sorted keys, in parallel over the tiles, with seven probes a step: a
// chain of 6 loads for 200,000 entries instead of 18 (13 -> 10 us).  nitems: seg-pair
// work items per tile (at least one), nitems[T] = 0.
__device__ __forceinline__ uint32_t lower_bound(const uint32_t* __restrict__ keys, uint32_t n,
                                                uint64_t key)
{
    uint32_t lo = 0, hi = n;  // all keys before lo are below `key`, none from hi on
    for (;;) {
        const uint32_t w = hi - lo < 8 ? 1u : (hi - lo) / 8;
        uint32_t probe[7], below = 0;
#pragma unroll
        for (uint32_t u = 0; u < 7; ++u) {
            const uint32_t at = hi - lo < 8 ? lo + u : lo + w * (u + 1);
            probe[u] = at < hi ? keys[at] : 0xffffffffu;
        }
#pragma unroll
        for (uint32_t u = 0; u < 7; ++u) below += probe[u] < key && (hi - lo >= 8 || lo + u < hi) ? 1u : 0u;
        if (hi - lo < 8) return lo + below;
        const uint32_t next = lo + w * (below + 1);
        if (below > 0) lo = lo + w * below + 1;
        if (below < 7) hi = next;
    }
}
constexpr int TI_THREADS = 256, TI_TILES = TI_THREADS - 1;  // the last thread finds the next block's first
__global__ void k_tile_items(const uint32_t* __restrict__ keys, uint32_t count,
                             const uint32_t* __restrict__ first, int total_tiles, int ib, int most, bool n_alone,
                             uint32_t* __restrict__ tentry, uint32_t* __restrict__ nitems,
                             const int* __restrict__ counters)
{
    grid_begin();
    __shared__ uint32_t e[TI_THREADS];
    const int seg = deposit_seg(counters, most, n_alone);
    const long long tt = (long long)blockIdx.x * TI_TILES + threadIdx.x;
    const int t = (int)min(tt, (long long)total_tiles + 1);
    const uint32_t b = lower_bound(keys, count, (uint64_t)min(t, total_tiles) << ib);
    e[threadIdx.x] = b;
    __syncthreads();
    if (t > total_tiles || threadIdx.x == TI_TILES) return;
    tentry[t] = b;
    if (t == total_tiles) {
        nitems[t] = 0u;
        return;
    }
    // e[t + 1] < b only when the keys are not in order (the sort gave up)
    const uint32_t end = max(e[threadIdx.x + 1], b);
    const uint32_t c = first[end] - first[b];
    nitems[t] = max(1u, (c + (uint32_t)seg - 1) / (uint32_t)seg);
}

// item_tile[i]: the tile of item i; merge: the tiles with several items, those of
// up to MERGE_FEW from the front (counters[1] of them), those of more from the
// back (counters[4]).  More
// items than the arrays hold (a captured call whose pairs outgrew its capacity)
// set ERR_CAP; those that they hold run all the same, so each has its tile.
__global__ void k_item_list(const uint32_t* __restrict__ item_off, int total_tiles,
                            uint32_t max_items, uint32_t* __restrict__ item_tile,
                            uint32_t* __restrict__ merge, int* __restrict__ counters, int* err)
{
    grid_begin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total_tiles) return;
    const uint32_t i0 = item_off[t], i1 = item_off[t + 1];
    for (uint32_t i = i0; i < min(i1, max_items); ++i) item_tile[i] = (uint32_t)t;
    if (i1 > max_items) {
        atomicOr(err, ERR_CAP);
        return;
    }
    if (i1 - i0 > MERGE_FEW) merge[total_tiles - 1 - atomicAdd(counters + 4, 1)] = (uint32_t)t;
    else if (i1 - i0 > 1) merge[atomicAdd(counters + 1, 1)] = (uint32_t)t;
}

// The pairs of one work item, 32 at a time: lane l of chunk c has pair 32 c + l.
// A chunk spans at most 32 entries, which the lanes load together; the entries then
// place their particles one after another, a lane of the bundle each (about four
// entries a chunk; searching each pair's entry and bit took twice the instructions).
struct PairCursor {
    const uint2* list;
    const uint32_t* first;
    uint32_t at, end;  // the entry of the next chunk's first pair, the tile's last + 1
    uint32_t f;        // of entry at + lane, loaded a chunk ahead: its first pair
    uint2 e;           // and itself

    __device__ __forceinline__ void load()
    {
        const uint32_t mine = at + (threadIdx.x & 31);
        f = mine < end ? first[mine] : 0xffffffffu;
        e = mine < end ? list[mine] : make_uint2(0u, 0u);
    }

    // particle and entry number of pair j0 + lane (j0 from chunk to chunk 32 on);
    // lanes past j1 get -1.  box: 32 words of the warp's shared memory
    __device__ __forceinline__ int take(uint32_t j0, uint32_t j1, int2* box, uint32_t& which)
    {
        const int lane = threadIdx.x & 31;
        const uint32_t stop = min(j0 + 32u, j1);
        const int n = __popc(__ballot_sync(FULLM, f < stop));  // first[] rises: the lanes below n
        for (int k = 0; k < n; ++k) {
            const uint32_t start = __shfl_sync(FULLM, f, k), m = __shfl_sync(FULLM, e.y, k);
            const uint32_t w = __shfl_sync(FULLM, e.x, k);
            const uint32_t to = start + (uint32_t)__popc(m & lanemask_lt()) - j0;  // wraps before j0
            if ((m >> lane & 1u) && to < 32u) box[to] = make_int2((int)(w * 32u) + lane, k);
        }
        __syncwarp();
        const int2 got = box[lane];
        const uint32_t j = j0 + (uint32_t)lane;
        which = at + (uint32_t)got.y;
        // on to the last of these entries, or past it when its pairs end here
        if (n > 0) {
            const uint32_t last = __shfl_sync(FULLM, f + (uint32_t)__popc(e.y), n - 1);
            at += (uint32_t)(n - 1) + (last <= stop ? 1u : 0u);
        }
        load();
        __syncwarp();  // `box` may be written again
        return j < j1 ? got.x : -1;
    }
};
__device__ __forceinline__ PairCursor open_pairs(const uint2* __restrict__ list,
                                                 const uint32_t* __restrict__ first, uint32_t e0,
                                                 uint32_t e1, uint32_t j0)
{
    uint32_t lo = e0, hi = e1;  // the last entry in [e0, e1) that starts at or before pair j0
    while (hi - lo > 1) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (first[mid] <= j0) lo = mid; else hi = mid;
    }
    PairCursor c{list, first, lo, e1, 0u, make_uint2(0u, 0u)};
    c.load();
    return c;
}

// ---------------------------------------------------------------------------
// (4) persistent deposit of (tile, segment) work items
// ---------------------------------------------------------------------------
// One warp owns one work item and accumulates its tile in a private
// shared-memory copy; it adds the item's pairs one after another, its lanes
// spread over the pair's whole 3-D cell box.  Per cell the additions happen in
// pair order, so the sums are deterministic.
constexpr int DEP_WARPS = 2;                // warps per CTA (independent)
constexpr int WROW = 3 * TS + 1;            // staged 1-D weights per lane: [axis * TS + cell]

struct WarpTile {
    float4 a[TC];           // n_hi, n_lo, c_hi, c_lo
    float4 b[TC];           // vx, vy, vz, halo_hi
    float hl[TC];           // halo_lo
    float w[32][WROW];      // 1-D cell weights of the chunk's 32 pairs (odd row stride)
};

// cell slot in a WarpTile: rows of 8 cells rotated by (6y + 4z) mod 8, which
// spreads the 128-bit accesses of a small 3-D box over distinct bank groups
__device__ __forceinline__ int tile_slot(int x, int y, int z)
{
    return (z << 6) | (y << 3) | ((x + 6 * y + 4 * z) & (TS - 1));
}

// floor(c / d) = (c * m_d) >> 15 with m_d = ceil(2^15 / d), exactly for
// 0 <= c < 512 and 1 <= d <= 64 (checked for every c and d): a pair's box has
// at most 8^3 cells and nx * ny <= 64.  Integer multiply and shift, no
// conversions on the per-cell path.
#define ASG_M15(d) ((32768 + (d) - 1) / (d))
#define ASG_M8(b) ASG_M15(b + 1), ASG_M15(b + 2), ASG_M15(b + 3), ASG_M15(b + 4), \
    ASG_M15(b + 5), ASG_M15(b + 6), ASG_M15(b + 7), ASG_M15(b + 8)
__constant__ int c_m15[TS * TS + 1] = {0, ASG_M8(0), ASG_M8(8), ASG_M8(16), ASG_M8(24),
                                       ASG_M8(32), ASG_M8(40), ASG_M8(48), ASG_M8(56)};
#undef ASG_M8
#undef ASG_M15

__device__ __forceinline__ int small_div(int c, int m) { return (c * m) >> 15; }

// one particle's weight w3 into one cell: n and c as double-float, v as float
__device__ __forceinline__ void add_cell(WarpTile& S, int slot, float w3, float dens, float vx,
                                         float vy, float vz)
{
    float4 Aa = S.a[slot];
    float4 Bb = S.b[slot];
    two_sum_acc_nonneg(Aa.x, Aa.y, w3);
    const float pr = __fmul_rn(w3, dens);
    const float pe = fmaf(w3, dens, -pr);  // the exact rounding error of the product
    two_sum_acc_nonneg(Aa.z, Aa.w, pr);
    Aa.w = __fadd_rn(Aa.w, pe);
    Bb.x = fmaf(w3, vx, Bb.x);
    Bb.y = fmaf(w3, vy, Bb.y);
    Bb.z = fmaf(w3, vz, Bb.z);
    S.a[slot] = Aa;
    S.b[slot] = Bb;
}

// a halo particle's weight into the halo channel (double-float)
__device__ __forceinline__ void add_halo(WarpTile& S, int slot, float w3)
{
    float hh = S.b[slot].w, hl = S.hl[slot];
    two_sum_acc_nonneg(hh, hl, w3);
    S.b[slot].w = hh;
    S.hl[slot] = hl;
}

__device__ __forceinline__ void write_tile(const WarpTile& S, const DepositParams& P, const TileGeo& g,
                                           double& sn, double& sh, int lane)
{
    const MeshJob& J = P.job[g.job];
    const int nc = g.nc;
    const size_t nmesh = (size_t)nc * nc * nc;
    for (int e = lane; e < TC; e += 32) {
        const int lz = e >> 6, ly = (e >> 3) & (TS - 1), lx = e & (TS - 1);
        if (lx >= g.E[0] || ly >= g.E[1] || lz >= g.E[2]) continue;
        const int slot = tile_slot(lx, ly, lz);
        const float4 A = S.a[slot];
        const float4 B = S.b[slot];
        const float hl = S.hl[slot];
        const size_t idx = ((size_t)(g.O[2] + lz) * nc + (g.O[1] + ly)) * nc + (g.O[0] + lx);
        sn += (double)A.x + (double)A.y;
        sh += (double)B.w + (double)hl;
        J.mesh[idx] = __fadd_rn(A.x, A.y);
        if (!P.density_only) {
            J.mesh[nmesh + idx] = __fadd_rn(B.w, hl);
            J.mesh[2 * nmesh + idx] = __fadd_rn(A.z, A.w);
            J.mesh[3 * nmesh + 3 * idx] = B.x;
            J.mesh[3 * nmesh + 3 * idx + 1] = B.y;
            J.mesh[3 * nmesh + 3 * idx + 2] = B.z;
        }
    }
}

__global__ void __launch_bounds__(32 * DEP_WARPS)
k_deposit_items(const float4* __restrict__ rec, const __grid_constant__ DepositParams P,
                int total_tiles, const uint32_t* __restrict__ item_off,
                uint32_t max_items, const uint32_t* __restrict__ item_tile,
                const uint32_t* __restrict__ tentry, const uint32_t* __restrict__ ekeys,
                const uint2* __restrict__ list, const uint32_t* __restrict__ first,
                float* __restrict__ partial, double* __restrict__ item_tot, int* __restrict__ counters)
{
    grid_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    WarpTile& S = reinterpret_cast<WarpTile*>(smem_raw)[threadIdx.x >> 5];
    const bool periodic = P.periodic != 0;
    const uint32_t total_items = min(item_off[total_tiles], max_items);
    const int most = deposit_seg(counters, P.seg, P.density_only != 0);  // pairs per item

    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(counters, 1);
        item = __shfl_sync(FULLM, item, 0);
        if ((uint32_t)item >= total_items) break;
        const int tile = (int)item_tile[item];
        const TileGeo g = tile_geo(P, tile);
        const MeshJob& J = P.job[g.job];
        const int nc = g.nc;
        const int seg = item - (int)item_off[tile];
        const int nseg = (int)(item_off[tile + 1] - item_off[tile]);
        const uint32_t e0 = tentry[tile], e1 = max(tentry[tile + 1], e0);
        const uint32_t j0 = first[e0] + (uint32_t)(seg * most);
        const uint32_t j1 = min(first[e1], j0 + (uint32_t)most);
        PairCursor pairs = open_pairs(list, first, e0, e1, j0);

        for (int e = lane; e < TC; e += 32) {
            S.a[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            S.b[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            S.hl[e] = 0.f;
        }
        __syncwarp();

        for (uint32_t c0 = j0; c0 < j1; c0 += 32) {
            // ---- setup: one pair per lane: exact ranges of its image, 1-D weights ----
            // rect packs tile-relative [x0,x1) [y0,y1) [z0,z1) in 4-bit fields and
            // the halo flag in bit 24; 0 means no cells
            uint32_t rect = 0;
            float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
            {
                uint32_t which;
                const int i = pairs.take(c0, j1, reinterpret_cast<int2*>(S.w), which);
                if (i >= 0) {
                    const int combo = periodic ? (int)(ekeys[which] & ((1u << IMG_BITS) - 1u)) : 0;
                    const int dk[3] = {combo % 3, (combo / 3) % 3, combo / 9};
                    float4 A, B, Cc, D;
                    load_dep_rec(rec, i, P.boxsize, P.rbox, A, B, Cc, D);
                    const float xs[3] = {A.x, A.y, A.z};
                    const float lo[3] = {B.x, B.y, B.z};
                    const float hi[3] = {Cc.x, Cc.y, Cc.z};
                    const float hinv = A.w;
                    float* wl = S.w[lane];
                    uint32_t r = 0;
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        const AxisRange ar = axis_range(lo[a], hi[a], J, nc, periodic);
                        const int k = ar.k_lo + dk[a];
                        const int sh = k * nc + g.O[a];
                        const int r0 = max(ar.left - sh, 0), r1 = min(ar.right - sh, g.E[a]);
                        r |= (uint32_t)((r0 & 15) | ((max(r1, r0) & 15) << 4)) << (8 * a);
                        // cell t covers [fi*dx, (fi+1)*dx] for the unwrapped cell index
                        // fi = t + sh (exact float steps, |index| < 2^24); each edge's
                        // offset from the particle in units of h is fma(fi, dx, -x) * hinv
                        // (one rounding before the scaling; the reference's s1 and
                        // s1 + ds, coarse_mesh.cpp:80-90, round i*dx first)
                        float fi = (float)(r0 + sh);
                        float e0 = __fmul_rn(__fmaf_rn(fi, J.dx, -xs[a]), hinv);
                        for (int t = r0; t < r1; ++t) {
                            fi = __fadd_rn(fi, 1.0f);
                            const float e1 = __fmul_rn(__fmaf_rn(fi, J.dx, -xs[a]), hinv);
                            wl[a * TS + t] = tent_integral_rn(e0, e1);
                            e0 = e1;
                        }
                    }
                    rect = r | ((uint32_t)(__float_as_int(D.z) & FLAG_HALO) << 24);
                    val = make_float4(B.w, Cc.w, D.x, D.y);
                }
            }
            __syncwarp();
            // ---- the warp adds the chunk's pairs in order, lanes over each pair's cells ----
            const int cnt = (int)min(32u, j1 - c0);
            for (int p = 0; p < cnt; ++p) {
                const uint32_t rp = __shfl_sync(FULLM, rect, p);
                const int x0 = rp & 15, nx = ((rp >> 4) & 15) - x0;
                const int y0 = (rp >> 8) & 15, ny = ((rp >> 12) & 15) - y0;
                const int z0 = (rp >> 16) & 15, nz = ((rp >> 20) & 15) - z0;
                if (nx <= 0 || ny <= 0 || nz <= 0) continue;
                const float dens = __shfl_sync(FULLM, val.x, p);
                const float vx = __shfl_sync(FULLM, val.y, p);
                const float vy = __shfl_sync(FULLM, val.z, p);
                const float vz = __shfl_sync(FULLM, val.w, p);
                const int nxy = nx * ny, ncell = nxy * nz;
                const int rx = c_m15[nx], rxy = c_m15[nxy];
                const float* wp = S.w[p];
                const bool hal = (rp >> 24) != 0;
                if (!hal) {
                    for (int c = lane; c < ncell; c += 32) {
                        const int iz = small_div(c, rxy);
                        const int rem = c - iz * nxy;
                        const int iy = small_div(rem, rx);
                        const int gx = x0 + rem - iy * nx, gy = y0 + iy, gz = z0 + iz;
                        const float w3 = __fmul_rn(__fmul_rn(wp[gx], wp[TS + gy]), wp[2 * TS + gz]);
                        add_cell(S, tile_slot(gx, gy, gz), w3, dens, vx, vy, vz);
                    }
                } else {
                    for (int c = lane; c < ncell; c += 32) {
                        const int iz = small_div(c, rxy);
                        const int rem = c - iz * nxy;
                        const int iy = small_div(rem, rx);
                        const int gx = x0 + rem - iy * nx, gy = y0 + iy, gz = z0 + iz;
                        const float w3 = __fmul_rn(__fmul_rn(wp[gx], wp[TS + gy]), wp[2 * TS + gz]);
                        add_halo(S, tile_slot(gx, gy, gz), w3);
                    }
                }
                __syncwarp();  // the next pair may add to the same cells from other lanes
            }
            __syncwarp();  // the next chunk's setup overwrites S.w
        }

        // ---- write: final tile when alone, partial tile otherwise ----
        double sn = 0.0, sh = 0.0;
        if (nseg > 1) {
            float* pt = partial + (size_t)item * TC * partial_words(P);
            float nh = 0.f, nl = 0.f, hh = 0.f, hl = 0.f;  // the mass of the lane's cells
            for (int e = lane; e < TC; e += 32) {
                const int slot = tile_slot(e & (TS - 1), (e >> 3) & (TS - 1), e >> 6);
                const float4 A = S.a[slot];
                const float4 B = S.b[slot];
                two_sum_acc_nonneg(nh, nl, A.x);
                nl = __fadd_rn(nl, A.y);
                two_sum_acc_nonneg(hh, hl, B.w);
                hl = __fadd_rn(hl, S.hl[slot]);
                pt[e] = A.x; pt[TC + e] = A.y;
                if (P.density_only) continue;
                pt[2 * TC + e] = A.z; pt[3 * TC + e] = A.w;
                pt[4 * TC + e] = B.x; pt[5 * TC + e] = B.y; pt[6 * TC + e] = B.z;
                pt[7 * TC + e] = B.w; pt[8 * TC + e] = S.hl[slot];
            }
            sn = (double)nh + (double)nl;
            sh = (double)hh + (double)hl;
        } else {
            write_tile(S, P, g, sn, sh, lane);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sn += __shfl_down_sync(FULLM, sn, o);
            sh += __shfl_down_sync(FULLM, sh, o);
        }
        if (lane == 0) {
            double* mass = nseg > 1 ? item_tot + 2 * (size_t)item : J.partial + 2 * (size_t)g.local;
            mass[0] = sn;
            mass[1] = sh;
        }
        __syncwarp();  // the next item clears the tile
    }
}

// ---------------------------------------------------------------------------
// (4') the same work items on the tensor cores
// ---------------------------------------------------------------------------
// A pair's contribution to its tile is separable: weight wx[x] wy[y] wz[z]
// times the particle's value in each channel (n: 1, halo: 1, c: dens, v), so a
// tile is a sum of outer products, C[(x, y)][(channel, z)] = sum over pairs of
// A[(x, y)][p] B[p][(channel, z)] with A = wx wy (32 rows) and B = wz * value
// (two channels x 4 z per block of 8 columns): a GEMM with K = the item's
// pairs.  One warp runs it with mma.sync m16n8k8 (TF32 in, FP32 accumulate), 8
// pairs per K step, on 2 row blocks x 3 column blocks of fragments.  TF32 keeps
// 11 significant bits, so every operand is split into hi + lo TF32 parts and
// each K step issues lo*hi, hi*lo and hi*hi (the lo*lo term is below 2^-22
// relative), which gives each product to about 2^-21.  Every 64 pairs the
// fragments are added into per-lane double-float sums in shared memory and
// cleared, so the FP32 accumulation never carries more than 24 roundings.
// Lane (g, t) owns the cells x = g, z = 2 (t mod 2) + {0, 1}, every y, of the
// channels n, c, vy (t < 2) or halo, vx, vz (t >= 2), both in the fragments and
// in its sums, so the sums need no synchronisation.
// The FP64 mass totals do not come from the cells: each pair adds
// (sum wx)(sum wy)(sum wz), formed in double-float arithmetic, to its lane's
// double-float total.  A K step skips the row blocks (two y rows each) that none
// of its 8 pairs touches, and the columns of c and v when all are halo
// particles: their products are exact zeros.
//
// One warp per item and CTA: no barriers, and a warp that waits for its own
// loads or its mma.sync chains leaves the SM to 23 others (8 KB of shared memory
// each): 70% of issue slots busy against 48% with two warps per 8 x 8 x 8 item and
// 16 warps per SM.  Bound by instruction issue and, more than by the tensor cores, by
// the ALU pipe (half rate: selects, comparisons, min/max, integer), so roundings to
// TF32 and two-sums run on the FMA pipe, two values per instruction where they can:
// 9.22 -> 7.02 -> 6.29 ms on the 256^3 step's 120 M pairs (of the last part, packed
// two-sums in the flush and the placed entries took 0.20 ms, the splitting by FMAs
// 0.38, the centre cell outside the loop 0.07, entries loaded a chunk ahead 0.05); on
// 160^3 cells, n alone, 0.27 -> 0.23 ms for 512 k particles.  Two cells of an axis at
// a time in packed arithmetic gained nothing: the ALU part stays.
constexpr int MMA_FLUSH = 64;  // pairs between flushes of the fragments

template <int NCH, bool WIDE>
struct MmaWarp {
    static constexpr int R = 2 * TileShape<NCH, WIDE>::Y;  // cells per lane and column block
    // [words r, r + 1][lane]: R hi, R lo of n/halo; of c/vx; R of vy/vz (n alone: R hi, R lo)
    float2 acc[(NCH == 1 ? 2 : 5) * R / 2][32];
    __device__ __forceinline__ float sum(int r, int lane) const  // word r
    {
        return r & 1 ? acc[r >> 1][lane].y : acc[r >> 1][lane].x;
    }
    // per pair of the chunk: wx | wy | wz | n, halo (1 or 0), dens, vx, vy, vz (n alone:
    // padding); the row lengths spread a K step's four rows over all banks
    float w[32][NCH == 1 ? 28 : WIDE ? 40 : 24];
};

__device__ __forceinline__ uint32_t tf32_rna(float x)
{
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
// x = hi + lo: hi = x rounded to TF32 (11 significant bits), lo = x - hi
// (exact in FP32) passed with its FP32 bits: the tensor core reads the TF32
// part of an operand register, so lo enters truncated to 11 significant bits,
// an error below 2^-11 |lo| <= 2^-23 |x|
__device__ __forceinline__ void tf32_split(float x, uint32_t& hi, uint32_t& lo)
{
    hi = tf32_rna(x);
    lo = __float_as_uint(__fsub_rn(x, __uint_as_float(hi)));
}
// tf32_split of two weights (|x| <= 1: no overflow) on the FMA pipe, which has room
// where the ALU pipe of the integer rounding has none: hi by the splitting with the
// constant 2^13 + 1 (T. J. Dekker, "A floating-point technique for extending the
// available precision", Numer. Math. 18, 1971), also x rounded to 11 bits
__device__ __forceinline__ void tf32_split_x2(f32x2 x, uint32_t& h0, uint32_t& h1, uint32_t& l0, uint32_t& l1)
{
    const f32x2 c = mul2_rn(x, pack2(8193.0f, 8193.0f));
    const f32x2 hi = add2_rn(c, sub2_rn(x, c));
    const f32x2 lo = sub2_rn(x, hi);
    h0 = __float_as_uint(lo2(hi));
    h1 = __float_as_uint(hi2(hi));
    l0 = __float_as_uint(lo2(lo));
    l1 = __float_as_uint(hi2(lo));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// product of two double-floats (hi, lo) in FP32 arithmetic (two_prod by FMA)
__device__ __forceinline__ void df_mul_df(float& hi, float& lo, float bh, float bl)
{
    const float p = __fmul_rn(hi, bh);
    const float e = fmaf(hi, bh, -p);
    const float l = fmaf(hi, bl, fmaf(lo, bh, e));
    const float s = __fadd_rn(p, l);
    lo = __fsub_rn(l, __fsub_rn(s, p));
    hi = s;
}

// tent_integral_rn as selections, with the same operations where they matter and
// so the same bits.  For a cell on one side of the centre with its nearer edge at
// distance p and its farther one at q: (q - p)(1 - (p + q)/2), or (1 - p)^2/2 when
// the support ends inside it, 0 when it lies beyond; q - p and p + q are |b - a| and
// |a + b| to the bit (sign changes are exact), 1 - t/2 is one FMA because t/2 is
// exact.  The cell around the centre (a < 0 < b) is tent_centre_rn.
__device__ __forceinline__ float tent_side_rn(float a, float b)
{
    const float p = fminf(fabsf(a), fabsf(b)), q = fmaxf(fabsf(a), fabsf(b));
    const float u = __saturatef(__fsub_rn(1.0f, p));  // p >= 0
    const float tail = __fmul_rn(__fmul_rn(0.5f, u), u);
    const float mid = __fmul_rn(__fsub_rn(b, a), __fmaf_rn(-0.5f, fabsf(__fadd_rn(a, b)), 1.0f));
    return q >= 1.0f ? tail : mid;
}
__device__ __forceinline__ float tent_centre_rn(float a, float b)
{
    const float t = fminf(b, 1.0f), s = fminf(-a, 1.0f);  // F(1) = 1/2 exactly
    return __fadd_rn(__fmul_rn(t, __fmaf_rn(-0.5f, t, 1.0f)), __fmul_rn(s, __fmaf_rn(-0.5f, s, 1.0f)));
}

template <int NCH, bool WIDE>
__global__ void __launch_bounds__(32, WIDE ? 14 : 24)
k_deposit_mma(const float4* __restrict__ rec, const __grid_constant__ DepositParams P, int total_tiles,
              const uint32_t* __restrict__ item_off, uint32_t max_items,
              const uint32_t* __restrict__ item_tile, const uint32_t* __restrict__ tentry,
              const uint32_t* __restrict__ ekeys, const uint2* __restrict__ list,
              const uint32_t* __restrict__ first, float* __restrict__ partial,
              double* __restrict__ item_tot, int* __restrict__ counters)
{
    grid_begin();
    using Shape = TileShape<NCH, WIDE>;
    constexpr int MX = Shape::X, MY = Shape::Y, MZ = Shape::Z, MC = Shape::CELLS;
    constexpr int NB = NCH == 1 ? 1 : 3;  // column blocks: n (8 z) or n halo | c vx | vy vz (4 z each)
    constexpr int RB = MY / 2;            // row blocks: 8 x and 2 y
    constexpr int R = 4 * RB;             // cells per lane and column block
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MmaWarp<NCH, WIDE>& S = *reinterpret_cast<MmaWarp<NCH, WIDE>*>(smem_raw);
    const int lane = threadIdx.x;
    const int g = lane >> 2, t = lane & 3;
    const bool periodic = P.periodic != 0;
    const uint32_t total_items = min(item_off[total_tiles], max_items);
    const int most = deposit_seg(counters, P.seg, P.density_only != 0);  // pairs per item

    int item = 0;
    if (lane == 0) item = atomicAdd(counters, 1);
    item = __shfl_sync(FULLM, item, 0);
    while ((uint32_t)item < total_items) {
        int next = 0;  // the next item's number arrives while this one runs
        if (lane == 0) next = atomicAdd(counters, 1);
        const int tile = (int)item_tile[item];
        const TileGeo geo = tile_geo(P, tile);
        const MeshJob& J = P.job[geo.job];
        const int nc = geo.nc;
        const float rdx = __fmul_rn(J.ncf, P.rbox);  // about 1 / dx
        const int i0 = (int)item_off[tile], nseg = (int)item_off[tile + 1] - i0;
        const uint32_t e0 = tentry[tile], e1 = max(tentry[tile + 1], e0);
        const uint32_t j0 = first[e0] + (uint32_t)((item - i0) * most);
        const uint32_t j1 = min(first[e1], j0 + (uint32_t)most);
        PairCursor pairs = open_pairs(list, first, e0, e1, j0);

#pragma unroll
        for (int k = 0; k < (int)(sizeof(S.acc) / sizeof(S.acc[0])); ++k) S.acc[k][lane] = make_float2(0.f, 0.f);
        float C[RB][NB][4];
#pragma unroll
        for (int m = 0; m < RB; ++m)
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int i = 0; i < 4; ++i) C[m][b][i] = 0.f;
        float tn_hi = 0.f, tn_lo = 0.f, th_hi = 0.f, th_lo = 0.f;  // this lane's pairs' totals

        // adds the fragments into the lane's sums and clears them, two words at a time
        auto flush = [&]() {
#pragma unroll
            for (int m = 0; m < RB; ++m)
#pragma unroll
                for (int i = 0; i < 4; i += 2) {
                    const int r = (4 * m + i) / 2;
#pragma unroll
                    for (int b = 0; b < (NB < 2 ? NB : 2); ++b) {
                        f32x2* hi = reinterpret_cast<f32x2*>(&S.acc[R * b + r][lane]);
                        f32x2* lo = reinterpret_cast<f32x2*>(&S.acc[R * b + R / 2 + r][lane]);
                        f32x2 h = *hi, l = *lo;
                        two_sum_acc_x2(h, l, pack2(C[m][b][i], C[m][b][i + 1]));
                        *hi = h;
                        *lo = l;
                    }
                    if constexpr (NB > 2) {
                        f32x2* v = reinterpret_cast<f32x2*>(&S.acc[2 * R + r][lane]);
                        *v = add2_rn(*v, pack2(C[m][2][i], C[m][2][i + 1]));
                    }
#pragma unroll
                    for (int b = 0; b < NB; ++b) C[m][b][i] = C[m][b][i + 1] = 0.f;
                }
        };

        int since_flush = 0;
        for (uint32_t c0 = j0; c0 < j1; c0 += 32) {
            // ---- setup: one pair per lane: its image's cell range, 1-D weights
            // (zero outside the range), channel values and FP64 mass.  The cells
            // of an axis that some lane touches are taken by all lanes together ----
            uint32_t rows = 0;  // the y rows the pair touches
            bool halo = false;
            {
                uint32_t which;
                const int i = pairs.take(c0, j1, reinterpret_cast<int2*>(S.w), which);
                float* wl = S.w[lane];
                float4* wz4 = reinterpret_cast<float4*>(wl);
#pragma unroll
                for (int k = 0; k < (MX + MY + MZ) / 4; ++k) wz4[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                float4 A = make_float4(0.f, 0.f, 0.f, 0.f), B = A, Cc = A, D = A;
                int combo = 0;
                if (i >= 0) {
                    load_dep_rec(rec, i, P.boxsize, P.rbox, A, B, Cc, D);
                    if (periodic) combo = (int)(ekeys[which] & ((1u << IMG_BITS) - 1u));
                }
                halo = (__float_as_int(D.z) & FLAG_HALO) != 0;
                const int dk[3] = {combo % 3, (combo / 3) % 3, combo / 9};
                const float xs[3] = {A.x, A.y, A.z};
                const float lo[3] = {B.x, B.y, B.z};
                const float hi[3] = {Cc.x, Cc.y, Cc.z};
                const float hinv = A.w;
                float mh = 0.0f, ml = 0.0f;  // product of the three 1-D sums (double-float)
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    constexpr int at[3] = {0, MX, MX + MY};
                    const AxisRange ar = axis_range(lo[a], hi[a], J, nc, periodic);
                    const int sh = (ar.k_lo + dk[a]) * nc + geo.O[a];
                    int r0 = max(ar.left - sh, 0), r1 = min(ar.right - sh, geo.E[a]);
                    if (i < 0 || r1 <= r0) r0 = r1 = 0;
                    const int any0 = (int)__reduce_min_sync(FULLM, (unsigned)(r1 > r0 ? r0 : MX));
                    const int any1 = (int)__reduce_max_sync(FULLM, (unsigned)r1);
                    // the cell around the particle, by the signs of its edges (an FMA's
                    // sign is exact; the guess is off by one at most)
                    int fc = __float2int_rd(__fmul_rn(xs[a], rdx));
                    {
                        const float f = (float)fc;
                        fc += (__fmaf_rn(__fadd_rn(f, 1.0f), J.dx, -xs[a]) < 0.0f ? 1 : 0) -
                              (__fmaf_rn(f, J.dx, -xs[a]) >= 0.0f ? 1 : 0);
                    }
                    const float ff = (float)fc;
                    const float ca = __fmul_rn(__fmaf_rn(ff, J.dx, -xs[a]), hinv);
                    const float cb = __fmul_rn(__fmaf_rn(__fadd_rn(ff, 1.0f), J.dx, -xs[a]), hinv);
                    const float wc = tent_centre_rn(ca, cb);
                    const int centre = ca < 0.0f && cb > 0.0f ? (int)((unsigned)fc - (unsigned)sh) : -1;
                    // cell c covers [fi*dx, (fi+1)*dx] with fi = c + sh (see k_deposit_items)
                    float fi = (float)(any0 + sh);
                    float e0 = __fmul_rn(__fmaf_rn(fi, J.dx, -xs[a]), hinv);
                    float sh_ = 0.f, sl_ = 0.f;
                    const unsigned len = (unsigned)(r1 - r0);
                    for (int c = any0; c < any1; ++c) {
                        fi = __fadd_rn(fi, 1.0f);
                        const float e1 = __fmul_rn(__fmaf_rn(fi, J.dx, -xs[a]), hinv);
                        float wv = tent_side_rn(e0, e1);
                        wv = c == centre ? wc : wv;
                        wv = (unsigned)(c - r0) < len ? wv : 0.0f;
                        wl[at[a] + c] = wv;
                        two_sum_acc(sh_, sl_, wv);
                        e0 = e1;
                    }
                    if (a == 0) { mh = sh_; ml = sl_; }
                    else df_mul_df(mh, ml, sh_, sl_);
                    if (a == 1) rows = ((1u << r1) - 1u) & ~((1u << r0) - 1u);
                }
                // a halo particle counts in the halo channel only
                if constexpr (NCH > 1)
                {
                    wz4[(MX + MY + MZ) / 4] = halo ? make_float4(0.f, 1.f, 0.f, 0.f) : make_float4(1.f, 0.f, B.w, Cc.w);
                    *reinterpret_cast<float2*>(wl + MX + MY + MZ + 4) =
                        halo ? make_float2(0.f, 0.f) : make_float2(D.x, D.y);
                }
                if (!halo) {
                    two_sum_acc(tn_hi, tn_lo, mh);
                    tn_lo = __fadd_rn(tn_lo, ml);
                } else {
                    two_sum_acc(th_hi, th_lo, mh);
                    th_lo = __fadd_rn(th_lo, ml);
                }
            }
            __syncwarp();
            // ---- K steps of 8 pairs: pairs 8s + t and 8s + t + 4 for this lane ----
            const int cnt = (int)min(32u, j1 - c0);
            for (int s8 = 0; s8 < cnt; s8 += 8) {
                const unsigned krows =
                    __reduce_or_sync(FULLM, (unsigned)(lane - s8) < 8u ? rows : 0u);
                const float* wa = S.w[s8 + t];
                const float* wb = S.w[s8 + t + 4];
                const float xa = wa[g], xb = wb[g];
                const float za = wa[MX + MY + (NCH == 1 ? g : g & 3)];
                const float zb = wb[MX + MY + (NCH == 1 ? g : g & 3)];
                uint32_t bh[NB][2], bl[NB][2];
                if constexpr (NCH == 1) {
                    tf32_split_x2(pack2(za, zb), bh[0][0], bh[0][1], bl[0][0], bl[0][1]);
                } else {
                    // n, halo: a weight times 1 or 0
                    const int at = MX + MY + MZ + (g >> 2);
                    tf32_split_x2(pack2(__fmul_rn(za, wa[at]), __fmul_rn(zb, wb[at])), bh[0][0], bh[0][1],
                                  bl[0][0], bl[0][1]);
#pragma unroll
                    for (int b = 1; b < NB; ++b) {
                        tf32_split(__fmul_rn(za, wa[at + 2 * b]), bh[b][0], bl[b][0]);
                        tf32_split(__fmul_rn(zb, wb[at + 2 * b]), bh[b][1], bl[b][1]);
                    }
                }
                // two row blocks at a time, those this K step touches, both in one
                // block of code when both do; the passes run over all live
                // accumulators, so the independent accumulation chains interleave
#pragma unroll
                for (int h = 0; h < RB; h += 2) {
                    const float4 ya = *reinterpret_cast<const float4*>(wa + MX + 2 * h);
                    const float4 yb = *reinterpret_cast<const float4*>(wb + MX + 2 * h);
                    auto blocks = [&](auto use0, auto use1) {
                        constexpr bool U[2] = {decltype(use0)::value, decltype(use1)::value};
                        uint32_t ah[2][4], al[2][4];
#pragma unroll
                        for (int m = 0; m < 2; ++m) {
                            if (!U[m]) continue;
                            tf32_split_x2(mul2_rn(pack2(xa, xa), m ? pack2(ya.z, ya.w) : pack2(ya.x, ya.y)),
                                          ah[m][0], ah[m][1], al[m][0], al[m][1]);
                            tf32_split_x2(mul2_rn(pack2(xb, xb), m ? pack2(yb.z, yb.w) : pack2(yb.x, yb.y)),
                                          ah[m][2], ah[m][3], al[m][2], al[m][3]);
                        }
#pragma unroll
                        for (int m = 0; m < 2; ++m)
#pragma unroll
                            for (int b = 0; b < NB; ++b)
                                if (U[m]) mma_tf32(C[h + m][b], al[m], bh[b][0], bh[b][1]);
#pragma unroll
                        for (int m = 0; m < 2; ++m)
#pragma unroll
                            for (int b = 0; b < NB; ++b)
                                if (U[m]) mma_tf32(C[h + m][b], ah[m], bl[b][0], bl[b][1]);
#pragma unroll
                        for (int m = 0; m < 2; ++m)
#pragma unroll
                            for (int b = 0; b < NB; ++b)
                                if (U[m]) mma_tf32(C[h + m][b], ah[m], bh[b][0], bh[b][1]);
                    };
                    const bool r0 = (krows >> (2 * h) & 3u) != 0, r1 = (krows >> (2 * h) & 12u) != 0;
                    if (r0 && r1) blocks(std::true_type{}, std::true_type{});
                    else if (r0) blocks(std::true_type{}, std::false_type{});
                    else if (r1) blocks(std::false_type{}, std::true_type{});
                }
            }
            since_flush += 32;
            if (since_flush >= MMA_FLUSH) {
                flush();
                since_flush = 0;
            }
            __syncwarp();  // the next chunk's setup overwrites S.w
        }
        if (since_flush > 0) flush();

        // ---- this item's FP64 mass, then the tile (final) or the partial tile ----
        double sn = (double)tn_hi + (double)tn_lo, shl = (double)th_hi + (double)th_lo;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sn += __shfl_down_sync(FULLM, sn, o);
            shl += __shfl_down_sync(FULLM, shl, o);
        }
        const bool low = NCH == 1 || t < 2;  // the lane's channels: n, c, vy, else halo, vx, vz
        if (nseg > 1) {
            float* pt = partial + (size_t)item * MC * (NCH == 1 ? PW_ALONE : PW);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int y = r >> 1, z = 2 * (NCH == 1 ? t : t & 1) + (r & 1);
                const int e = (z * MY + y) * MX + g;
                pt[(low ? 0 : 7) * MC + e] = S.sum(r, lane);
                pt[(low ? 1 : 8) * MC + e] = S.sum(R + r, lane);
                if constexpr (NCH > 1) {
                    if (low) {
                        pt[2 * MC + e] = S.sum(2 * R + r, lane);
                        pt[3 * MC + e] = S.sum(3 * R + r, lane);
                    } else {
                        pt[4 * MC + e] = __fadd_rn(S.sum(2 * R + r, lane), S.sum(3 * R + r, lane));
                    }
                    pt[(low ? 5 : 6) * MC + e] = S.sum(4 * R + r, lane);
                }
            }
            if (lane == 0) {
                item_tot[2 * (size_t)item] = sn;
                item_tot[2 * (size_t)item + 1] = shl;
            }
        } else {
            const size_t nmesh = (size_t)nc * nc * nc;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int y = r >> 1, z = 2 * (NCH == 1 ? t : t & 1) + (r & 1);
                if (g >= geo.E[0] || y >= geo.E[1] || z >= geo.E[2]) continue;
                const size_t idx = ((size_t)(geo.O[2] + z) * nc + (geo.O[1] + y)) * nc + (geo.O[0] + g);
                J.mesh[(low ? 0 : nmesh) + idx] = __fadd_rn(S.sum(r, lane), S.sum(R + r, lane));
                if constexpr (NCH > 1) {
                    J.mesh[low ? 2 * nmesh + idx : 3 * nmesh + 3 * idx] =
                        __fadd_rn(S.sum(2 * R + r, lane), S.sum(3 * R + r, lane));
                    J.mesh[3 * nmesh + 3 * idx + (low ? 1 : 2)] = S.sum(4 * R + r, lane);
                }
            }
            if (lane == 0) {
                J.partial[2 * (size_t)geo.local] = sn;
                J.partial[2 * (size_t)geo.local + 1] = shl;
            }
        }
        item = __shfl_sync(FULLM, next, 0);
    }
}

// ---------------------------------------------------------------------------
// (5) merge the partial tiles of multi-segment tiles, in segment order
// ---------------------------------------------------------------------------
// A warp takes 128 cells, four neighbours per lane.  It merges a tile of up to
// MERGE_FEW items by itself, in item order; for a tile of more, a CTA's 8 warps add
// an eighth of the items each and the eight sums are added in order (n, c and halo
// as double-floats throughout).  One thread per cell over all items was a chain of
// loads: 73 us for the 36 tiles of about 36 items of a 13,840-particle set, so 14.  Where
// nearly all pairs fall into few tiles, a CTA for all cells of each was the chain: n alone
// of 300,000 particles in one Gaussian clump 641 -> 247 us.
// item_tot: the FP64 mass of every item.
constexpr int MERGE_WARPS = 8;
static_assert(MERGE_WARPS <= 32, "one lane per warp's mass");

struct MergeSums {
    float s[PW][4];  // n hi, lo; c hi, lo; v; halo hi, lo of four cells
    __device__ __forceinline__ MergeSums()
    {
#pragma unroll
        for (int q = 0; q < PW; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[q][i] = 0.f;
    }
    // adds the words at x, word q at x[q * stride]
    __device__ __forceinline__ void add(const float* __restrict__ x, size_t stride, bool all)
    {
        float4 v[PW];
#pragma unroll
        for (int q = 0; q < PW; ++q)
            v[q] = q < 2 || all ? *reinterpret_cast<const float4*>(x + q * stride)
                                : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            auto at = [&](int q) { return i == 0 ? v[q].x : i == 1 ? v[q].y : i == 2 ? v[q].z : v[q].w; };
            two_sum_acc(s[0][i], s[1][i], at(0));
            s[1][i] = __fadd_rn(s[1][i], at(1));
            if (all) {
                two_sum_acc(s[2][i], s[3][i], at(2));
                s[3][i] = __fadd_rn(s[3][i], at(3));
#pragma unroll
                for (int q = 4; q < 7; ++q) s[q][i] = __fadd_rn(s[q][i], at(q));
                two_sum_acc(s[7][i], s[8][i], at(7));
                s[8][i] = __fadd_rn(s[8][i], at(8));
            }
        }
    }
};

__global__ void __launch_bounds__(32 * MERGE_WARPS)
k_merge_tiles(const __grid_constant__ DepositParams P, int total_tiles,
              const uint32_t* __restrict__ item_off, const uint32_t* __restrict__ merge,
              const int* __restrict__ counters, const float* __restrict__ partial,
              const double* __restrict__ item_tot)
{
    grid_begin();
    __shared__ __align__(16) float sums[MERGE_WARPS][PW][128];
    __shared__ double mass[2][MERGE_WARPS];
    const int cells = 1 << (P.shift[0] + P.shift[1] + P.shift[2]);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool all = !P.density_only;
    const int words = partial_words(P);
    const int few = counters[1], many = counters[4];

    // items [a0, a1) of cells [e, e + 3]
    auto sum_items = [&](int a0, int a1, int e, MergeSums& m) {
        for (int it = a0; it < a1; ++it)
            m.add(partial + (size_t)it * cells * words + e, (size_t)cells, all);
    };
    auto store = [&](const TileGeo& g, int e, const MergeSums& m) {
        const MeshJob& J = P.job[g.job];
        const size_t nc = (size_t)g.nc, nmesh = nc * nc * nc;
        const int ly = (e >> P.shift[0]) & ((1 << P.shift[1]) - 1), lz = e >> (P.shift[0] + P.shift[1]);
        if (ly >= g.E[1] || lz >= g.E[2]) return;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int lx = (e & ((1 << P.shift[0]) - 1)) + i;
            if (lx >= g.E[0]) return;
            const size_t idx = ((size_t)(g.O[2] + lz) * nc + (g.O[1] + ly)) * nc + (g.O[0] + lx);
            J.mesh[idx] = __fadd_rn(m.s[0][i], m.s[1][i]);
            if (all) {
                J.mesh[nmesh + idx] = __fadd_rn(m.s[7][i], m.s[8][i]);
                J.mesh[2 * nmesh + idx] = __fadd_rn(m.s[2][i], m.s[3][i]);
#pragma unroll
                for (int q = 0; q < 3; ++q) J.mesh[3 * nmesh + 3 * idx + q] = m.s[4 + q][i];
            }
        }
    };
    // the mass of items [a0, a1), to lane 0
    auto sum_mass = [&](int a0, int a1, double& sn, double& sh) {
        sn = sh = 0.0;
        for (int it = a0 + lane; it < a1; it += 32) {
            sn += item_tot[2 * (size_t)it];
            sh += item_tot[2 * (size_t)it + 1];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sn += __shfl_down_sync(FULLM, sn, o);
            sh += __shfl_down_sync(FULLM, sh, o);
        }
    };

    // ---- tiles of many items first, a CTA each, or for each 128 cells of few such tiles ----
    const int shares = many <= (int)gridDim.x / (cells / 128) ? cells / 128 : 1;
    for (int k = blockIdx.x; k < many * shares; k += gridDim.x) {
        const int tile = (int)merge[total_tiles - 1 - k / shares], share = k % shares;
        const int i0 = (int)item_off[tile], i1 = (int)item_off[tile + 1];
        const int a0 = i0 + (int)((long long)(i1 - i0) * w / MERGE_WARPS);
        const int a1 = i0 + (int)((long long)(i1 - i0) * (w + 1) / MERGE_WARPS);
        const TileGeo g = tile_geo(P, tile);
        double sn, sh;
        for (int c = 4 * lane + 128 * share; c < cells; c += 128 * shares) {
            MergeSums m;
            sum_items(a0, a1, c, m);
#pragma unroll
            for (int q = 0; q < PW; ++q)
                *reinterpret_cast<float4*>(&sums[w][q][4 * lane]) =
                    make_float4(m.s[q][0], m.s[q][1], m.s[q][2], m.s[q][3]);
            __syncthreads();
            if (w == 0) {
                for (int o = 1; o < MERGE_WARPS; ++o) m.add(&sums[o][0][4 * lane], 128, all);
                store(g, c, m);
            }
            __syncthreads();  // sums is written again
        }
        if (share) continue;
        sum_mass(a0, a1, sn, sh);
        if (lane == 0) {
            mass[0][w] = sn;
            mass[1][w] = sh;
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            double m = 0.0;
            for (int o = 0; o < MERGE_WARPS; ++o) m += mass[threadIdx.x][o];
            P.job[g.job].partial[2 * (size_t)g.local + threadIdx.x] = m;
        }
        __syncthreads();  // mass is written again
    }
    // ---- the others, a warp each ----
    for (int k = (int)blockIdx.x + (int)gridDim.x * w; k < few; k += (int)gridDim.x * MERGE_WARPS) {
        const int tile = (int)merge[k];
        const int i0 = (int)item_off[tile], i1 = (int)item_off[tile + 1];
        const TileGeo g = tile_geo(P, tile);
        double sn, sh;
        for (int c = 4 * lane; c < cells; c += 128) {
            MergeSums m;
            sum_items(i0, i1, c, m);
            store(g, c, m);
        }
        sum_mass(i0, i1, sn, sh);
        if (lane == 0) {
            P.job[g.job].partial[2 * (size_t)g.local] = sn;
            P.job[g.job].partial[2 * (size_t)g.local + 1] = sh;
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
size_t deposit_prep_bytes(int n) { return 32 * (size_t)n; }

// A warp goes through a bundle's tiles one after another: with few bundles and wide
// supports on a fine mesh, few warps had a long way (64 particles with supports of 120
// cells of a 256^3 mesh 8.8 ms, a thread per particle 0.8, 32 warps per bundle 0.6).
// As many as make 4096 warps, whose counts one scan launch takes: 13,840 particles on
// a mesh of 6 cells per mean separation 391 us with 1, 281 with 8; 32,768 647, 577 with
// 2.  Above that, and where the meshes hold few tiles (256 per warp), a bundle's
// fixed cost (ranges, unions) is most of it: 32,768 on 32^3 cells 82 us with 1, 87 with
// 8.  A periodic mesh has more tiles and images per bundle: 8192 warps (131,072
// particles at 6 cells 2.71, 2.57 ms with 2) and 128 tiles; a bundle of particles far
// apart goes through all images (64 on 24^3 cells 294 us with 1, 146 with 4).
int deposit_log_parts(int n, bool periodic, long long total_tiles)
{
    const long long bundles = ((long long)n + 31) / 32;
    const bool far_apart = bundles <= 32;
    const long long most = std::min(total_tiles / (!periodic ? 256 : far_apart ? 16 : 128),
                                    far_apart ? 32ll : std::min(16ll, (periodic ? 8192 : 4095) / bundles));
    int log_parts = 0;
    while ((2ll << log_parts) <= most) ++log_parts;
    return log_parts;
}

void deposit_tile_shape(DepositParams& p)
{
    const bool small = p.mma && !p.density_only;
    p.shift[0] = 3;
    p.shift[1] = small && !p.wide ? 2 : 3;
    p.shift[2] = small ? 2 : 3;
}

size_t deposit_tile_bytes(int total_tiles)
{
    // tentry, item_off, merge (+1 each) and their scan scratch
    const size_t T1 = (size_t)total_tiles + 1;
    return 4 * T1 * 3 + scan_temp_bytes(T1) + 256;
}

// keys and values of the sort (ping-pong), entries as emitted and in key order, and
// the first pair of each with its scan scratch
size_t deposit_entry_bytes(uint32_t entries)
{
    const size_t E = (size_t)entries + 2;
    return (4 + 4 + 8) * 2 * E + 4 * E + scan_temp_bytes(E) + 256;
}

void deposit_entry_layout(void* base, uint32_t entries, DepositScratch& w)
{
    const size_t E = ((size_t)entries + 2) & ~size_t(1);  // entry and list stay 8-byte aligned
    w.entry = static_cast<uint2*>(base);
    w.list = w.entry + E;
    w.keys0 = reinterpret_cast<uint32_t*>(w.list + E);
    w.keys1 = w.keys0 + E;
    w.vals0 = reinterpret_cast<int*>(w.keys1 + E);
    w.vals1 = w.vals0 + E;
    w.first = reinterpret_cast<uint32_t*>(w.vals1 + E);
    w.scan_tmp_e = w.first + E;
}

static int key_bits(int total_tiles, int ib)
{
    int b = 0;
    while ((1 << b) < total_tiles) ++b;
    return b + ib;
}

// Above this many pairs with 8 x 4 x 4 tiles, six channels go through the preparation
// again with 8 x 8 x 4 ones: wide supports fill the tiles, and a pair's weights are
// formed for twice the cells.
// 262,144 particles at 6 cells per mean separation (182 pairs per particle) 3.91 ->
// 3.79 ms, in halos 3.81 -> 3.55, periodic 5.09 -> 4.66; at 4 cells (75) 1.46 and 1.45, at
// 2 (28) 0.39 and 0.49.  Below 8 M pairs the second preparation and the longer items of
// fewer warps are not made up: 13,840 particles at 6 cells 0.28 and 0.36 ms, 32,768
// 0.56 both, 65,536 1.06 both and periodic 1.50 -> 1.46.
unsigned long long deposit_wide_pairs(int n)
{
    return std::max(64ull * (unsigned long long)n, 8ull << 20);
}

// the default deposit engine: 1 the tensor cores, 0 the CUDA cores
// (ASG_DEPOSIT=simt, a comparison knob; a context's tuner may choose)
int deposit_default_mma()
{
    static const int m = [] {
        const char* e = std::getenv("ASG_DEPOSIT");
        return e && std::strcmp(e, "simt") == 0 ? 0 : 1;
    }();
    return m;
}

// per-item FP64 masses after the partial tiles of deposit_max_items items
static double* deposit_item_totals(float* partial, uint32_t items, const DepositParams& p)
{
    const size_t off = ((size_t)items * deposit_item_words(p) * sizeof(float) + 15) & ~size_t(15);
    return reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(partial) + off);
}

// a persistent kernel: as many CTAs as fit on every SM at once, its dynamic
// shared memory allowed once per device (function attributes are per device).  The
// kernel is a template argument: kernels of one signature share a function's statics
template <auto Kern, class... Args>
static void launch_persistent(int dev, int sms, int threads, size_t smem, cudaStream_t s, Args... args)
{
    static std::atomic<unsigned long long> attr_set{0};  // one bit per device, per kernel
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(attr_set.load() & bit)) {
        cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(Kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        attr_set.fetch_or(bit);
    }
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, Kern, threads, smem);
    launch(Kern, sms * (per_sm > 0 ? per_sm : 1), threads, smem, s, args...);
}

void launch_deposit_prep(const float4* pos, const float4* vel, const int* igrp, const float* rk,
                         int n, const DepositParams& p, DepositScratch& w, int* err,
                         cudaStream_t s)
{
    const int units = (n + 31) / 32 << p.log_parts;
    cudaMemsetAsync(w.counters, 0, 32, s);
    auto kern = p.periodic ? (p.log_parts ? k_dep_prep<true, true> : k_dep_prep<true, false>)
                           : (p.log_parts ? k_dep_prep<false, true> : k_dep_prep<false, false>);
    launch(kern, (units + 7) / 8, 256, 0, s, pos, vel, igrp, rk, n, p, w.rec, w.count,
           reinterpret_cast<unsigned long long*>(w.counters + 2), err);
    exclusive_scan_u32(w.count, (size_t)units + 1, w.scan_tmp_n, s);
    count_launches(1);
}

void launch_deposit_run(int n, const DepositParams& p, int total_tiles, uint32_t entries,
                        uint32_t max_items, bool padded, DepositScratch& w, int* err, cudaStream_t s)
{
    const int T = total_tiles, units = (n + 31) / 32 << p.log_parts;
    auto kern = p.periodic ? (p.log_parts ? k_entries<true, true> : k_entries<true, false>)
                           : (p.log_parts ? k_entries<false, true> : k_entries<false, false>);
    launch(kern, (units + 7) / 8, 256, 0, s, w.rec, n, p, w.count, w.keys0, w.entry, entries, err);
    count_launches(1);
    if (padded && entries > 0) {  // `entries` is the capacity; the count itself is the last of `count`
        launch(k_pad_entries, (entries + 255) / 256, 256, 0, s, w.keys0, w.entry, w.count + units, entries,
                                                            (uint32_t)T << img_bits(p));
        count_launches(1);
    }
    const int cur = radix_sort32(w.keys0, w.vals0, w.keys1, w.vals1, (int)entries,
                                 key_bits(padded ? T + 1 : T, img_bits(p)), true, w.sort_tmp, err, s);
    const uint32_t* keys = cur ? w.keys1 : w.keys0;
    launch(k_sorted_entries, entries / 256 + 1, 256, 0, s, cur ? w.vals1 : w.vals0, w.entry, entries,
           reinterpret_cast<const unsigned long long*>(w.counters + 2), w.list, w.first, err);
    exclusive_scan_u32(w.first, (size_t)entries + 1, w.scan_tmp_e, s);
    launch(k_tile_items, T / TI_TILES + 1, TI_THREADS, 0, s, keys, entries, w.first, T, img_bits(p), p.seg,
           p.density_only != 0, w.tentry,
                                             w.item_off, w.counters);
    exclusive_scan_u32(w.item_off, (size_t)T + 1, w.scan_tmp_t, s);
    launch(k_item_list, (T + 255) / 256, 256, 0, s, w.item_off, T, max_items, w.item_tile, w.merge,
                                                w.counters, err);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    double* item_tot = deposit_item_totals(w.partial, max_items, p);
    if (p.mma) {
        auto run = [&](auto nch, auto wide) {
            constexpr int N = decltype(nch)::value;
            constexpr bool W = decltype(wide)::value;
            launch_persistent<k_deposit_mma<N, W>>(dev, sms, 32, sizeof(MmaWarp<N, W>), s, w.rec, p, T, w.item_off,
                                                   max_items, w.item_tile, w.tentry, keys, w.list, w.first,
                                                   w.partial, item_tot, w.counters);
        };
        using One = std::integral_constant<int, 1>;
        using Six = std::integral_constant<int, 6>;
        if (p.density_only) run(One{}, std::false_type{});
        else if (p.wide) run(Six{}, std::true_type{});
        else run(Six{}, std::false_type{});
    } else {
        launch_persistent<k_deposit_items>(dev, sms, 32 * DEP_WARPS, DEP_WARPS * sizeof(WarpTile), s, w.rec, p,
                                           T, w.item_off, max_items, w.item_tile, w.tentry, keys, w.list,
                                           w.first, w.partial, item_tot, w.counters);
    }
    launch(k_merge_tiles, 4 * sms, 32 * MERGE_WARPS, 0, s, p, T, w.item_off, w.merge, w.counters,
                                                       w.partial, item_tot);
    count_launches(5);
}

// (the sort numbers entries with 31 bits)
uint32_t deposit_headroom(uint32_t n) { return (uint32_t)std::min((uint64_t)n + n / 16 + 4096, (uint64_t)INT_MAX); }

// Work items that `npairs` pairs or fewer make: a partial one per tile, and as many
// full ones as deposit_seg leaves, of 64 pairs at least.  (Room for ITEM_SHARE whatever
// the pairs took 76 MB for the smallest deposit of six channels, 303 for n alone.)
uint32_t deposit_max_items(int total_tiles, uint32_t npairs, int most, bool n_alone)
{
    const uint32_t share = n_alone ? ITEM_SHARE / 2 : ITEM_SHARE;
    return (uint32_t)total_tiles + std::max(std::min(share, npairs / 64), npairs / (uint32_t)most) + 2;
}

size_t deposit_item_words(const DepositParams& p)
{
    return (size_t)partial_words(p) << (p.shift[0] + p.shift[1] + p.shift[2]);
}

// partial tiles of multi-item tiles, then each item's FP64 mass (2 doubles)
size_t deposit_partial_bytes(uint32_t items, size_t item_words)
{
    return (((size_t)items * item_words * sizeof(float) + 15) & ~size_t(15)) + 16 * (size_t)items;
}

// FP64 totals of every mesh from its tiles' partial sums: block (b, mesh) adds a
// fixed slice of the tiles; with one block per mesh into out, else into scratch
// for the second launch (one block per mesh over the REDUCE_BLOCKS sums), which
// takes 12 us for the 150 k tiles of the 256^3 step (one block per mesh: 85 us for
// a quarter as many).
constexpr int REDUCE_BLOCKS = 64, REDUCE_MIN = 8192;
__global__ void __launch_bounds__(256)
k_reduce_partials(const __grid_constant__ DepositParams P, const double* __restrict__ in,
                  double* __restrict__ out)
{
    grid_begin();
    __shared__ double r[2][256];
    const int k = blockIdx.y, B = gridDim.x;
    const MeshJob& J = P.job[k];
    const double* src = in ? in + 2 * (size_t)k * REDUCE_BLOCKS : J.partial;
    const int count = in ? REDUCE_BLOCKS : J.tiles[0] * J.tiles[1] * J.tiles[2];
    double a = 0.0, b = 0.0;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < count; i += B * 256) {
        a += src[2 * (size_t)i];
        b += src[2 * (size_t)i + 1];
    }
    r[0][threadIdx.x] = a;
    r[1][threadIdx.x] = b;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            r[0][threadIdx.x] += r[0][threadIdx.x + o];
            r[1][threadIdx.x] += r[1][threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x < 2) out[2 * ((size_t)k * B + blockIdx.x) + threadIdx.x] = r[threadIdx.x][0];
}

size_t deposit_totals_bytes(int n_nc) { return 16 * (size_t)n_nc * (1 + REDUCE_BLOCKS); }

void launch_deposit_totals(const DepositParams& p, int total_tiles, double* totals, cudaStream_t s)
{
    const unsigned k = (unsigned)p.n_jobs;
    if (total_tiles <= REDUCE_MIN) {
        launch(k_reduce_partials, dim3(1, k), 256, 0, s, p, nullptr, totals);
        count_launches(1);
        return;
    }
    double* part = totals + 2 * p.n_jobs;
    launch(k_reduce_partials, dim3(REDUCE_BLOCKS, k), 256, 0, s, p, nullptr, part);
    launch(k_reduce_partials, dim3(1, k), 256, 0, s, p, part, totals);
    count_launches(2);
}

// write_mesh_separate normalisation (coarse_mesh.cpp:158-171), in place
__global__ void k_normalise(float* __restrict__ mesh, size_t nmesh, float vol)
{
    grid_begin();
    const size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nmesh) return;
    float* n = mesh;
    float* halo = mesh + nmesh;
    float* c = halo + nmesh;
    float* v = c + nmesh;
    const float nj = n[j];
    if (nj > 0.0f) {
        c[j] = __fmul_rn(c[j], __fdiv_rn(vol, __fmul_rn(nj, nj)));
        v[3 * j] = __fdiv_rn(v[3 * j], nj);
        v[3 * j + 1] = __fdiv_rn(v[3 * j + 1], nj);
        v[3 * j + 2] = __fdiv_rn(v[3 * j + 2], nj);
    } else {
        c[j] = 0.0f;
        v[3 * j] = v[3 * j + 1] = v[3 * j + 2] = 0.0f;
    }
    n[j] = __fmul_rn(nj, 8.0f);
    halo[j] = __fmul_rn(halo[j], 8.0f);
}

void launch_normalise(float* mesh, int nc, float vol, cudaStream_t s)
{
    const size_t nmesh = (size_t)nc * nc * nc;
    launch(k_normalise, (unsigned)((nmesh + 255) / 256), 256, 0, s, mesh, nmesh, vol);
    count_launches(1);
}

}  // namespace asg
