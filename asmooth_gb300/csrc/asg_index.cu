// asg_index.cu -- the spatial index that replaces KDTreeSimple
// (kdtree_balanced.cpp:212-296): particles are put in 48-bit Hilbert order
// (16 bits per axis; Morton order with ASG_SPACE_CURVE=morton) by a stable LSD
// radix sort (each 8-bit digit pass is a counting sort: per-tile
// digit histograms built with warp-aggregated shared-memory atomics, one
// exclusive scan, a stable scatter), then the boxes of the blocked tree
// (TreeView) are reduced level by level.
//
// Determinism: the sort is stable and starts from input order, so equal keys
// stay in input-index order; the tree is a pure function of the sorted keys.
#include <atomic>
#include <cstdlib>
#include <cstring>

#include "asg_common.cuh"
#include "asg_internal.h"

namespace asg {

// ---------------------------------------------------------------------------
// unpack + space-filling-curve keys
// ---------------------------------------------------------------------------
struct ParticleRec {  // struct Particle (basic_types.h:10-15), 36 bytes
    float x[3], v[3];
    float dens, rk;
    int igrp;
};
static_assert(sizeof(ParticleRec) == 36, "Particle record must be 36 bytes");

__global__ void k_unpack_aos(const ParticleRec* __restrict__ aos, int n, float4* __restrict__ pos,
                             float4* __restrict__ vel, int* __restrict__ igrp,
                             float* __restrict__ rkin, int* err)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* r = reinterpret_cast<const float*>(aos + i);
    const float x = r[0], y = r[1], z = r[2];
    if (!(isfinite(x) && isfinite(y) && isfinite(z))) atomicOr(err, ERR_NONFINITE);
    pos[i] = make_float4(x, y, z, __int_as_float(i));
    vel[i] = make_float4(r[3], r[4], r[5], r[6]);
    igrp[i] = reinterpret_cast<const int*>(r)[8];
    rkin[i] = r[7];
}

__global__ void k_unpack_soa(const float* __restrict__ x3, const float* __restrict__ v3,
                             const float* __restrict__ dens, const int* __restrict__ ig, int n,
                             float4* __restrict__ pos, float4* __restrict__ vel,
                             int* __restrict__ igrp, float* __restrict__ rkin, int* err)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = x3[3 * (size_t)i], y = x3[3 * (size_t)i + 1], z = x3[3 * (size_t)i + 2];
    if (!(isfinite(x) && isfinite(y) && isfinite(z))) atomicOr(err, ERR_NONFINITE);
    pos[i] = make_float4(x, y, z, __int_as_float(i));
    const float d = dens ? dens[i] : 0.0f;
    vel[i] = v3 ? make_float4(v3[3 * (size_t)i], v3[3 * (size_t)i + 1], v3[3 * (size_t)i + 2], d)
                : make_float4(0.f, 0.f, 0.f, d);
    igrp[i] = ig ? ig[i] : 0;
    rkin[i] = 0.0f;
}

// Mixed-precision input: one int32 cell index c = (cz * grid + cy) * grid + cx
// and three uint16 offsets per particle.  Each coordinate decodes as
//   x = (left + cs * cx) + off * unit,   unit = cs / 65536,
// every product and sum rounded to nearest in this order (the host decode in
// the Python package does the same float32 operations).
__global__ void k_unpack_quant(const int* __restrict__ cell, const uint16_t* __restrict__ off,
                               const float* __restrict__ v3, int n, int grid, float left, float cs,
                               float unit, float4* __restrict__ pos, float4* __restrict__ vel,
                               int* __restrict__ igrp, float* __restrict__ rkin, int* err)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = cell[i];
    const int g2 = grid * grid;
    if (c < 0 || (long long)c >= (long long)g2 * grid) {
        atomicOr(err, ERR_BADCELL);
        c = 0;
    }
    const int cx = c % grid, cy = (c / grid) % grid, cz = c / g2;
    const float x = __fadd_rn(__fadd_rn(left, __fmul_rn(cs, (float)cx)),
                              __fmul_rn((float)off[3 * (size_t)i], unit));
    const float y = __fadd_rn(__fadd_rn(left, __fmul_rn(cs, (float)cy)),
                              __fmul_rn((float)off[3 * (size_t)i + 1], unit));
    const float z = __fadd_rn(__fadd_rn(left, __fmul_rn(cs, (float)cz)),
                              __fmul_rn((float)off[3 * (size_t)i + 2], unit));
    pos[i] = make_float4(x, y, z, __int_as_float(i));
    vel[i] = v3 ? make_float4(v3[3 * (size_t)i], v3[3 * (size_t)i + 1], v3[3 * (size_t)i + 2], 0.0f)
                : make_float4(0.f, 0.f, 0.f, 0.f);
    igrp[i] = 0;
    rkin[i] = 0.0f;
}

void launch_unpack_quant(const int* cell, const uint16_t* off, const float* v, int n, int grid,
                         float left, float cs, float4* pos_in, float4* vel_in, int* igrp_in,
                         float* rk_in, int* err, cudaStream_t s)
{
    if (n <= 0) return;
    const float unit = cs / 65536.0f;
    k_unpack_quant<<<(n + 255) / 256, 256, 0, s>>>(cell, off, v, n, grid, left, cs, unit, pos_in,
                                                    vel_in, igrp_in, rk_in, err);
    count_launches(1);
}

void launch_unpack_aos(const void* aos, int n, float4* pos_in, float4* vel_in, int* igrp_in,
                       float* rk_in, int* err, cudaStream_t s)
{
    if (n <= 0) return;
    k_unpack_aos<<<(n + 255) / 256, 256, 0, s>>>((const ParticleRec*)aos, n, pos_in, vel_in,
                                                  igrp_in, rk_in, err);
    count_launches(1);
}

void launch_unpack_soa(const float* x, const float* v, const float* dens, const int* igrp, int n,
                       float4* pos_in, float4* vel_in, int* igrp_in, float* rk_in, int* err,
                       cudaStream_t s)
{
    if (n <= 0) return;
    k_unpack_soa<<<(n + 255) / 256, 256, 0, s>>>(x, v, dens, igrp, n, pos_in, vel_in, igrp_in,
                                                  rk_in, err);
    count_launches(1);
}

// order-preserving float <-> int map for atomicMin/atomicMax on floats
__device__ __forceinline__ int fkey(float f)
{
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float fkey_inv(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

__global__ void k_bounds_init(int* lohi)
{
    lohi[0] = 0x7fffffff;
    lohi[1] = (int)0x80000000;
}

__global__ void k_bounds(const float4* __restrict__ pos, int n, int* lohi)
{
    float lo = INFINITY, hi = -INFINITY;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 p = pos[i];
        lo = fminf(lo, fminf(p.x, fminf(p.y, p.z)));
        hi = fmaxf(hi, fmaxf(p.x, fmaxf(p.y, p.z)));
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_down_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_down_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(lohi, fkey(lo));
        atomicMax(lohi + 1, fkey(hi));
    }
}

// space-filling-curve key of each particle: 16 bits per axis over [left,
// right), with the bounds either given (lohi == nullptr) or read from
// k_bounds' output; Hilbert order, or Morton order with hilbert == 0
__global__ void k_space_keys(const float4* __restrict__ pos, int n, float left, float right,
                             const int* __restrict__ lohi, uint64_t prefix, int hilbert,
                             uint64_t* __restrict__ keys, int* __restrict__ vals)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (lohi) {
        left = fkey_inv(lohi[0]);
        right = fkey_inv(lohi[1]);
    }
    const float w = right - left;
    const float scale = w > 0.0f ? 65536.0f / w : 1.0f;
    const float4 p = pos[i];
    auto cell = [&](float c) -> uint32_t {
        float t = (c - left) * scale;
        t = fminf(fmaxf(t, 0.0f), 65535.0f);
        return (uint32_t)t;
    };
    const uint32_t cx = cell(p.x), cy = cell(p.y), cz = cell(p.z);
    const uint64_t k = hilbert ? hilbert_key48(cx, cy, cz)
                               : spread3(cx) | (spread3(cy) << 1) | (spread3(cz) << 2);
    keys[i] = (prefix << 48) | k;
    vals[i] = i;
}

// ASG_SPACE_CURVE=morton selects Morton order (a tuning and comparison knob)
static int use_hilbert()
{
    static const int h = [] {
        const char* e = std::getenv("ASG_SPACE_CURVE");
        return (e && std::strcmp(e, "morton") == 0) ? 0 : 1;
    }();
    return h;
}

void launch_space_keys(const float4* pos_in, int n, float left, float right, int* d_lohi,
                       uint64_t key_prefix, uint64_t* keys, int* vals, cudaStream_t s)
{
    if (n <= 0) return;
    if (d_lohi) {
        k_bounds_init<<<1, 1, 0, s>>>(d_lohi);
        k_bounds<<<min((n + 255) / 256, 1216), 256, 0, s>>>(pos_in, n, d_lohi);
        count_launches(2);
    }
    k_space_keys<<<(n + 255) / 256, 256, 0, s>>>(pos_in, n, left, right, d_lohi, key_prefix,
                                                  use_hilbert(), keys, vals);
    count_launches(1);
}

// ---------------------------------------------------------------------------
// exclusive scan (uint32)
// ---------------------------------------------------------------------------
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(uint32_t* data, size_t n, uint32_t* sums)
{
    __shared__ uint32_t warp_tot[32];
    const size_t base = (size_t)blockIdx.x * SCAN_TILE + (size_t)threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS];
    uint32_t t = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        v[k] = (base + k < n) ? data[base + k] : 0u;
        t += v[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = warp_tot[lane];
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        warp_tot[lane] = wi - w;  // exclusive warp offsets
        if (lane == 31 && sums) sums[blockIdx.x] = wi;
    }
    __syncthreads();
    uint32_t run = warp_tot[warp] + inc - t;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        if (base + k < n) data[base + k] = run;
        run += v[k];
    }
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_add(uint32_t* data, size_t n, const uint32_t* offs)
{
    const uint32_t o = offs[blockIdx.x];
    const size_t base = (size_t)blockIdx.x * SCAN_TILE;
    for (int k = threadIdx.x; k < SCAN_TILE; k += SCAN_THREADS)
        if (base + k < n) data[base + k] += o;
}

size_t scan_temp_bytes(size_t n)
{
    size_t total = 0;
    while (n > 1) {
        n = (n + SCAN_TILE - 1) / SCAN_TILE;
        total += n;
    }
    return (total + 64) * sizeof(uint32_t);
}

void exclusive_scan_u32(uint32_t* data, size_t n, void* temp, cudaStream_t s)
{
    if (n == 0) return;
    const size_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    uint32_t* sums = (uint32_t*)temp;
    k_scan_tiles<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(data, n, nb > 1 ? sums : nullptr);
    count_launches(1);
    if (nb > 1) {
        exclusive_scan_u32(sums, nb, sums + nb, s);
        k_scan_add<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(data, n, sums);
        count_launches(1);
    }
}

// ---------------------------------------------------------------------------
// stable LSD radix sort, 8-bit digits
// ---------------------------------------------------------------------------
#ifndef ASG_RS_ROUNDS
#define ASG_RS_ROUNDS 8
#endif
constexpr int RS_THREADS = 256;
constexpr int RS_ROUNDS = ASG_RS_ROUNDS;  // elements per thread of a tile
constexpr int RS_TILE = RS_THREADS * RS_ROUNDS;

template <class K>
__global__ void __launch_bounds__(RS_THREADS) k_rs_count(const K* __restrict__ keys, int n,
                                                         int shift, uint32_t* __restrict__ counts,
                                                         int ntiles)
{
    __shared__ uint32_t hist[256];
    hist[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * RS_TILE;
    const unsigned lane = threadIdx.x & 31;
    for (int r = 0; r < RS_ROUNDS; ++r) {
        const int i = base + r * RS_THREADS + threadIdx.x;
        const bool valid = i < n;
        const unsigned d = valid ? (unsigned)((keys[i] >> shift) & 255u) : 256u;
        // warp-aggregated atomics: one shared-memory add per distinct digit
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        if (valid && lane == (unsigned)(__ffs(peers) - 1)) atomicAdd(&hist[d], __popc(peers));
    }
    __syncthreads();
    counts[(size_t)threadIdx.x * ntiles + blockIdx.x] = hist[threadIdx.x];
}

// Stable scatter of one 8-bit digit.  A block takes a tile of RS_TILE elements;
// warp w ranks its own contiguous RS_ROUNDS x 32 elements with per-warp digit
// counters (no block barrier while ranking), one block-level scan turns the
// counters into positions of the tile in digit order, the tile is placed in
// shared memory in that order, and written out so that consecutive threads
// store consecutive addresses within each digit's run.  Order is kept: within
// a digit, elements stay in (warp, round, lane) = input order.
template <class K>
struct RsScatterSmem {
    K key[RS_TILE];
    int val[RS_TILE];
    uint32_t wcnt[RS_THREADS / 32][256];  // per-warp digit counts, then offsets
    uint32_t lstart[256];                 // first slot of each digit in the tile
    uint32_t gstart[256];                 // the digit's first output position for this tile
};

template <class K>
__global__ void __launch_bounds__(RS_THREADS) k_rs_scatter(const K* __restrict__ kin,
                                                           const int* __restrict__ vin,
                                                           K* __restrict__ kout,
                                                           int* __restrict__ vout, int n,
                                                           int shift,
                                                           const uint32_t* __restrict__ offs,
                                                           int ntiles)
{
    extern __shared__ __align__(16) unsigned char rs_smem[];
    RsScatterSmem<K>& S = *reinterpret_cast<RsScatterSmem<K>*>(rs_smem);
    const int tid = threadIdx.x, warp = tid >> 5;
    const unsigned lane = tid & 31, lt = lanemask_lt();
    const int base = blockIdx.x * RS_TILE;
#pragma unroll
    for (int w = 0; w < RS_THREADS / 32; ++w) S.wcnt[w][tid] = 0u;
    S.gstart[tid] = offs[(size_t)tid * ntiles + blockIdx.x];
    __syncthreads();
    // ---- rank: this warp's elements base + warp*32*ROUNDS + r*32 + lane ----
    K k[RS_ROUNDS];
    int v[RS_ROUNDS];
    uint32_t pos[RS_ROUNDS];  // position among this warp's elements of the same digit
    const int wbase = base + warp * 32 * RS_ROUNDS;
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
        const int i = wbase + r * 32 + (int)lane;
        const bool valid = i < n;
        k[r] = valid ? kin[i] : (K)0;
        v[r] = valid ? vin[i] : 0;
        const unsigned d = valid ? (unsigned)((k[r] >> shift) & 255u) : 256u;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const uint32_t before = valid ? S.wcnt[warp][d] : 0u;
        pos[r] = before + __popc(peers & lt);
        __syncwarp();
        if (valid && (peers & lt) == 0u) S.wcnt[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // ---- per digit (thread = digit): offsets of the warps, then the tile's scan ----
    {
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < RS_THREADS / 32; ++w) {
            const uint32_t c = S.wcnt[w][tid];
            S.wcnt[w][tid] = sum;
            sum += c;
        }
        // exclusive scan of the 256 digit totals (one per thread)
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if ((int)lane >= o) inc += y;
        }
        __shared__ uint32_t wsum[RS_THREADS / 32];
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        uint32_t woff = 0;
        for (int w = 0; w < warp; ++w) woff += wsum[w];
        S.lstart[tid] = woff + inc - sum;
    }
    __syncthreads();
    // ---- place the tile in digit order ----
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
        const int i = wbase + r * 32 + (int)lane;
        if (i < n) {
            const unsigned d = (unsigned)((k[r] >> shift) & 255u);
            const uint32_t slot = S.lstart[d] + S.wcnt[warp][d] + pos[r];
            S.key[slot] = k[r];
            S.val[slot] = v[r];
        }
    }
    __syncthreads();
    // ---- write out: slot j of digit d goes to gstart[d] + (j - lstart[d]) ----
    const int cnt = min(RS_TILE, n - base);
    for (int j = tid; j < cnt; j += RS_THREADS) {
        const K kk = S.key[j];
        const unsigned d = (unsigned)((kk >> shift) & 255u);
        const uint32_t dst = S.gstart[d] + ((uint32_t)j - S.lstart[d]);
        kout[dst] = kk;
        vout[dst] = S.val[j];
    }
}

size_t radix_sort_temp_bytes(int n)
{
    const size_t ntiles = (size_t)(n + RS_TILE - 1) / RS_TILE;
    const size_t nc = 256 * ntiles;
    return nc * sizeof(uint32_t) + scan_temp_bytes(nc) + 256;
}

template <class K>
static int radix_sort_t(K* keys0, int* vals0, K* keys1, int* vals1, int n, int bits, void* temp,
                        cudaStream_t s)
{
    if (n <= 1) return 0;
    const int ntiles = (n + RS_TILE - 1) / RS_TILE;
    static std::atomic<unsigned long long> attr_set{0};  // one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (!(attr_set.load() & (1ull << (dev & 63)))) {
        cudaFuncSetAttribute(k_rs_scatter<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(RsScatterSmem<K>));
        attr_set.fetch_or(1ull << (dev & 63));
    }
    uint32_t* counts = (uint32_t*)temp;
    void* stemp = (void*)(counts + (size_t)256 * ntiles);
    K* kb[2] = {keys0, keys1};
    int* vb[2] = {vals0, vals1};
    int cur = 0;
    for (int shift = 0; shift < bits; shift += 8) {
        k_rs_count<K><<<ntiles, RS_THREADS, 0, s>>>(kb[cur], n, shift, counts, ntiles);
        exclusive_scan_u32(counts, (size_t)256 * ntiles, stemp, s);
        k_rs_scatter<K><<<ntiles, RS_THREADS, sizeof(RsScatterSmem<K>), s>>>(
            kb[cur], vb[cur], kb[cur ^ 1], vb[cur ^ 1], n, shift, counts, ntiles);
        count_launches(2);
        cur ^= 1;
    }
    return cur;
}

int radix_sort(uint64_t* keys0, int* vals0, uint64_t* keys1, int* vals1, int n, int bits,
               void* temp, cudaStream_t s)
{
    return radix_sort_t<uint64_t>(keys0, vals0, keys1, vals1, n, bits, temp, s);
}

int radix_sort32(uint32_t* keys0, int* vals0, uint32_t* keys1, int* vals1, int n, int bits,
                 void* temp, cudaStream_t s)
{
    return radix_sort_t<uint32_t>(keys0, vals0, keys1, vals1, n, bits, temp, s);
}

__global__ void k_gather(const int* __restrict__ perm, const float4* __restrict__ pos_in,
                         const float4* __restrict__ vel_in, const int* __restrict__ igrp_in,
                         const float* __restrict__ rk_in, int n, float4* __restrict__ pos,
                         float4* __restrict__ vel, int* __restrict__ igrp, float* __restrict__ rk)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int o = perm[i];
    pos[i] = pos_in[o];
    vel[i] = vel_in[o];
    igrp[i] = igrp_in[o];
    rk[i] = rk_in[o];
}

void launch_gather_sorted(const int* perm, const float4* pos_in, const float4* vel_in,
                          const int* igrp_in, const float* rk_in, int n, float4* pos, float4* vel,
                          int* igrp, float* rk, cudaStream_t s)
{
    if (n <= 0) return;
    k_gather<<<(n + 255) / 256, 256, 0, s>>>(perm, pos_in, vel_in, igrp_in, rk_in, n, pos, vel,
                                              igrp, rk);
    count_launches(1);
}

__global__ void k_iota(int* a, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = i;
}
void launch_iota(int* a, int n, cudaStream_t s)
{
    if (n <= 0) return;
    k_iota<<<(n + 255) / 256, 256, 0, s>>>(a, n);
    count_launches(1);
}

__global__ void k_check_rk(const float* __restrict__ rk, int n, int* err)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float h = rk[i];
    if (!(h > 0.0f && h < INFINITY)) atomicOr(err, ERR_ZERO_RK);
}
void launch_check_rk(const float* rk, int n, int* err, cudaStream_t s)
{
    if (n <= 0) return;
    k_check_rk<<<(n + 255) / 256, 256, 0, s>>>(rk, n, err);
    count_launches(1);
}

// ---------------------------------------------------------------------------
// blocked box tree (TreeView)
// ---------------------------------------------------------------------------
TreeView tree_shape(int n, int leaf)
{
    TreeView t{};
    t.n = n;
    t.leaf = leaf;
    long long c = ((long long)n + leaf - 1) / leaf, off = 0;
    for (;;) {
        t.cnt[t.nlev] = (int)c;
        t.off[t.nlev] = off;
        off += c;
        ++t.nlev;
        if (c <= 32) break;
        c = (c + 31) / 32;
    }
    return t;
}

size_t tree_box_bytes(int n, int leaf)
{
    const TreeView t = tree_shape(n, leaf);
    return 32 * (size_t)(t.off[t.nlev - 1] + t.cnt[t.nlev - 1]);
}

// union of the boxes of the lanes of each aligned group of G lanes
template <int G>
__device__ __forceinline__ void group_box(float (&r)[6])
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 6; ++a) {
            const float v = __shfl_xor_sync(0xffffffffu, r[a], o);
            r[a] = a < 3 ? fminf(r[a], v) : fmaxf(r[a], v);
        }
}
__device__ __forceinline__ void store_box(float4* box, size_t id, const float (&r)[6])
{
    box[2 * id] = make_float4(r[0], r[1], r[2], r[3]);
    box[2 * id + 1] = make_float4(r[4], r[5], 0.0f, 0.0f);
}

// level 0: G lanes (16, or 32 for leaves of more particles) per leaf, one
// coalesced load per lane
template <int G>
__global__ void k_leaf_boxes(const float4* __restrict__ pos, int n, int leaf, int nleaf,
                             float4* __restrict__ box)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long id = t / G;
    const int r = (int)(t % G);
    const bool live = id < nleaf;
    const long long i = min(id * leaf + min(r, leaf - 1), (long long)n - 1);
    const float4 p = pos[live ? i : 0];
    float b[6] = {p.x, p.y, p.z, p.x, p.y, p.z};
    group_box<G>(b);
    if (live && r == 0) store_box(box, (size_t)id, b);
}

// one level up: a warp per box, a child per lane
__global__ void k_up_boxes(const float4* __restrict__ below, int nbelow, float4* __restrict__ box,
                           int nbox)
{
    const long long id = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    if (id >= nbox) return;
    const long long c = min(id * 32 + (threadIdx.x & 31), (long long)nbelow - 1);
    const float4 u = below[2 * c], v = below[2 * c + 1];
    float b[6] = {u.x, u.y, u.z, u.w, v.x, v.y};
    group_box<32>(b);
    if ((threadIdx.x & 31) == 0) store_box(box, (size_t)id, b);
}

void launch_tree_boxes(const float4* pos, const TreeView& t, cudaStream_t s)
{
    if (t.n <= 0) return;
    float4* box = const_cast<float4*>(t.box);
    const int g = t.leaf <= 16 ? 16 : 32;
    const unsigned nb = (unsigned)(((long long)t.cnt[0] * g + 255) / 256);
    if (g == 16) k_leaf_boxes<16><<<nb, 256, 0, s>>>(pos, t.n, t.leaf, t.cnt[0], box);
    else k_leaf_boxes<32><<<nb, 256, 0, s>>>(pos, t.n, t.leaf, t.cnt[0], box);
    for (int l = 1; l < t.nlev; ++l)
        k_up_boxes<<<(unsigned)(((long long)t.cnt[l] * 32 + 255) / 256), 256, 0, s>>>(
            box + 2 * t.off[l - 1], t.cnt[l - 1], box + 2 * t.off[l], t.cnt[l]);
    count_launches(t.nlev);
}

// ---------------------------------------------------------------------------
// output in input order
// ---------------------------------------------------------------------------
__global__ void k_pack_aos(const int* __restrict__ perm, const float4* __restrict__ pos,
                           const float4* __restrict__ vel, const float* __restrict__ rk,
                           const float* __restrict__ dens, const int* __restrict__ igrp, int n,
                           ParticleRec* __restrict__ aos)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int o = perm ? perm[i] : i;  // no perm: the arrays are in output order
    const float4 p = pos[i], v = vel[i];
    float* r = reinterpret_cast<float*>(aos + o);
    r[0] = p.x; r[1] = p.y; r[2] = p.z;
    r[3] = v.x; r[4] = v.y; r[5] = v.z;
    r[6] = dens ? dens[i] : v.w;
    r[7] = rk ? rk[i] : 0.0f;
    reinterpret_cast<int*>(r)[8] = igrp[i];
}

void launch_pack_aos(const int* perm, const float4* pos, const float4* vel, const float* rk,
                     const float* dens, const int* igrp, int n, void* aos, cudaStream_t s)
{
    if (n <= 0) return;
    k_pack_aos<<<(n + 255) / 256, 256, 0, s>>>(perm, pos, vel, rk, dens, igrp, n,
                                                (ParticleRec*)aos);
    count_launches(1);
}

__global__ void k_scatter_fields(const int* __restrict__ perm, const float* __restrict__ rk,
                                 const float* __restrict__ dens, const int* __restrict__ igrp,
                                 int n, float* rk_out, float* dens_out, int* igrp_out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int o = perm[i];
    if (rk_out) rk_out[o] = rk[i];
    if (dens_out) dens_out[o] = dens[i];
    if (igrp_out) igrp_out[o] = igrp[i];
}

void launch_scatter_fields(const int* perm, const float* rk, const float* dens, const int* igrp,
                           int n, float* rk_out, float* dens_out, int* igrp_out, cudaStream_t s)
{
    if (n <= 0) return;
    k_scatter_fields<<<(n + 255) / 256, 256, 0, s>>>(perm, rk, dens, igrp, n, rk_out, dens_out,
                                                      igrp_out);
    count_launches(1);
}

}  // namespace asg
