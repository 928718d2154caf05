// asg_index.cu -- the spatial index that replaces KDTreeSimple
// (kdtree_balanced.cpp:212-296): particles are put in 48-bit Hilbert order
// (16 bits per axis; Morton order with ASG_SPACE_CURVE=morton) by a stable LSD
// radix sort (one pass over the data per 8-bit digit; small sets in one launch), then the boxes of the
// blocked tree (TreeView) are reduced level by level.
//
// Determinism: the sort is stable and starts from input order, so equal keys
// stay in input-index order; the tree is a pure function of the sorted keys.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>

#include <cooperative_groups.h>

#include "asg_common.cuh"
#include "asg_internal.h"
#include "asg_keys.cuh"

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

// A staged particle is 32 bytes, one memory sector: x, y, z, igrp (int bits) and vx,
// vy, vz, dens, so that putting the particles in curve order reads one random
// sector each (four when the fields were staged apart: 1.32 against 0.42 ms for
// 18.3 M particles).  The unpack kernels also form each particle's key.
__device__ __forceinline__ void store_staged(float4* __restrict__ rec, int i, float x, float y, float z,
                                             int igrp, float vx, float vy, float vz, float dens)
{
    rec[2 * (size_t)i] = make_float4(x, y, z, __int_as_float(igrp));
    rec[2 * (size_t)i + 1] = make_float4(vx, vy, vz, dens);
}

__global__ void k_unpack_aos(const ParticleRec* __restrict__ aos, int n, float4* __restrict__ rec,
                             float* __restrict__ rkin, KeyGrid grid, uint64_t* __restrict__ keys,
                             int* err)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* r = reinterpret_cast<const float*>(aos + i);
    const float x = r[0], y = r[1], z = r[2];
    if (!(isfinite(x) && isfinite(y) && isfinite(z))) atomicOr(err, ERR_NONFINITE);
    store_staged(rec, i, x, y, z, reinterpret_cast<const int*>(r)[8], r[3], r[4], r[5], r[6]);
    rkin[i] = r[7];
    if (keys) keys[i] = space_key(grid, x, y, z);
}

__global__ void k_unpack_soa(const float* __restrict__ x3, const float* __restrict__ v3,
                             const float* __restrict__ dens, const int* __restrict__ ig, int n,
                             float4* __restrict__ rec, KeyGrid grid, uint64_t* __restrict__ keys,
                             int* err)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = x3[3 * (size_t)i], y = x3[3 * (size_t)i + 1], z = x3[3 * (size_t)i + 2];
    if (!(isfinite(x) && isfinite(y) && isfinite(z))) atomicOr(err, ERR_NONFINITE);
    float v[3] = {0.f, 0.f, 0.f};
    if (v3)
#pragma unroll
        for (int a = 0; a < 3; ++a) v[a] = v3[3 * (size_t)i + a];
    store_staged(rec, i, x, y, z, ig ? ig[i] : 0, v[0], v[1], v[2], dens ? dens[i] : 0.0f);
    if (keys) keys[i] = space_key(grid, x, y, z);
}

// Mixed-precision input: one int32 cell index c = (cz * grid + cy) * grid + cx
// and three uint16 offsets per particle.  Each coordinate decodes as
//   x = (left + cs * cx) + off * unit,   unit = cs / 65536,
// every product and sum rounded to nearest in this order (the host decode in
// the Python package does the same float32 operations).
__global__ void k_unpack_quant(const int* __restrict__ cell, const uint16_t* __restrict__ off,
                               const float* __restrict__ v3, int n, int grid, float left, float cs,
                               float unit, float4* __restrict__ rec, KeyGrid kgrid,
                               uint64_t* __restrict__ keys, int* err)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = cell[i];
    const int g2 = grid * grid;
    if (c < 0 || (long long)c >= (long long)g2 * grid) {
        atomicOr(err, ERR_BADCELL);
        c = 0;
    }
    const int cc[3] = {c % grid, (c / grid) % grid, c / g2};
    float x[3], v[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int a = 0; a < 3; ++a)
        x[a] = __fadd_rn(__fadd_rn(left, __fmul_rn(cs, (float)cc[a])),
                         __fmul_rn((float)off[3 * (size_t)i + a], unit));
    if (v3)
#pragma unroll
        for (int a = 0; a < 3; ++a) v[a] = v3[3 * (size_t)i + a];
    store_staged(rec, i, x[0], x[1], x[2], 0, v[0], v[1], v[2], 0.0f);
    keys[i] = space_key(kgrid, x[0], x[1], x[2]);
}

void launch_unpack_quant(const int* cell, const uint16_t* off, const float* v, int n, int grid,
                         float left, float cs, float4* rec, const KeyGrid& kgrid, uint64_t* keys,
                         int* err, cudaStream_t s)
{
    if (n <= 0) return;
    const float unit = cs / 65536.0f;
    launch(k_unpack_quant, (n + 255) / 256, 256, 0, s, cell, off, v, n, grid, left, cs, unit, rec, kgrid,
                                                    keys, err);
    count_launches(1);
}

void launch_unpack_aos(const void* aos, int n, float4* rec, float* rk_in, const KeyGrid& grid,
                       uint64_t* keys, int* err, cudaStream_t s)
{
    if (n <= 0) return;
    launch(k_unpack_aos, (n + 255) / 256, 256, 0, s, (const ParticleRec*)aos, n, rec, rk_in, grid, keys, err);
    count_launches(1);
}

void launch_unpack_soa(const float* x, const float* v, const float* dens, const int* igrp, int n,
                       float4* rec, const KeyGrid& grid, uint64_t* keys, int* err, cudaStream_t s)
{
    if (n <= 0) return;
    launch(k_unpack_soa, (n + 255) / 256, 256, 0, s, x, v, dens, igrp, n, rec, grid, keys, err);
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
    grid_begin();
    lohi[0] = 0x7fffffff;
    lohi[1] = (int)0x80000000;
}

__global__ void k_bounds(const float4* __restrict__ rec, int n, int* lohi)
{
    grid_begin();
    float lo = INFINITY, hi = -INFINITY;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 p = rec[2 * (size_t)i];
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

// keys over the particles' own bounding cube, from k_bounds' output
__global__ void k_space_keys(const float4* __restrict__ rec, int n, const int* __restrict__ lohi,
                             int hilbert, uint64_t* __restrict__ keys)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    KeyGrid g;
    g.left = fkey_inv(lohi[0]);
    const float w = fkey_inv(lohi[1]) - g.left;
    g.scale = w > 0.0f ? 65536.0f / w : 1.0f;
    g.hilbert = hilbert;
    const float4 p = rec[2 * (size_t)i];
    keys[i] = space_key(g, p.x, p.y, p.z);
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

KeyGrid key_grid(float left, float right)
{
    KeyGrid g;
    g.left = left;
    const float w = right - left;
    g.scale = w > 0.0f ? 65536.0f / w : 1.0f;
    g.hilbert = use_hilbert();
    return g;
}

void launch_own_keys(const float4* rec, int n, int* d_lohi, uint64_t* keys, cudaStream_t s)
{
    if (n <= 0) return;
    launch(k_bounds_init, 1, 1, 0, s, d_lohi);
    launch(k_bounds, min((n + 255) / 256, 1216), 256, 0, s, rec, n, d_lohi);
    launch(k_space_keys, (n + 255) / 256, 256, 0, s, rec, n, d_lohi, use_hilbert(), keys);
    count_launches(3);
}

// ---------------------------------------------------------------------------
// exclusive scan (uint32)
// ---------------------------------------------------------------------------
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(uint32_t* data, size_t n, uint32_t* sums)
{
    grid_begin();
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

// adds each tile's offset: the sum of the tiles before it, which the block forms
// itself when they are few (scanned == 0: offs holds the tiles' sums), one launch less
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_add(uint32_t* data, size_t n, const uint32_t* offs,
                                                           int scanned)
{
    grid_begin();
    __shared__ uint32_t warp_tot[32];
    uint32_t o;
    if (scanned) {
        o = offs[blockIdx.x];
    } else {
        const uint32_t v = threadIdx.x < blockIdx.x ? offs[threadIdx.x] : 0u;
        const uint32_t w = __reduce_add_sync(0xffffffffu, v);
        if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = w;
        __syncthreads();
        o = __reduce_add_sync(0xffffffffu, warp_tot[threadIdx.x & 31]);
    }
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
    launch(k_scan_tiles, (unsigned)nb, SCAN_THREADS, 0, s, data, n, nb > 1 ? sums : nullptr);
    count_launches(1);
    if (nb > 1) {
        const bool few = nb <= SCAN_THREADS;
        if (!few) exclusive_scan_u32(sums, nb, sums + nb, s);
        launch(k_scan_add, (unsigned)nb, SCAN_THREADS, 0, s, data, n, sums, few ? 0 : 1);
        count_launches(1);
    }
}

// ---------------------------------------------------------------------------
// stable LSD radix sort: one pass over the data per digit
// ---------------------------------------------------------------------------
// k_rs_hist counts every digit of every key once and scans the counts;
// k_rs_pass then sorts one digit, each block ranking one tile and finding the
// tile's place by looking back over the counts that the tiles before it publish
// (the single-pass scan with decoupled look-back of D. Merrill and M. Garland,
// NVIDIA Technical Report NVR-2016-002, and the sort built on it by A. Adinets
// and D. Merrill, "Onesweep", arXiv:2206.01784).  A pass reads and writes each
// element once, 170 us for 18.3 M 64-bit keys with values; a count, a scan of
// the counts and a scatter per digit took 300 us and five launches instead of one.
// A digit has 8 bits, or 9 where that saves a pass.
constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_BACK = 8;          // tile states read at a time
constexpr int RS_POLLS = 1 << 22;  // look-back polls after which a block gives up (ERR_SORT)
template <class K>
constexpr int RS_ROUNDS = sizeof(K) == 8 ? 12 : 16;  // elements per thread of a tile
template <class K>
constexpr int RS_TILE = RS_THREADS * RS_ROUNDS<K>;
constexpr int RS_PASSES = 8;

// the sort's scratch: words [0, RS_PASSES) the passes' tile counters, [RS_PASSES]
// the histogram blocks done, then RS_PASSES x 512 digit starts, then each pass's
// tile states
constexpr size_t RS_HEAD = 16, RS_HIST = RS_PASSES * 512;

// a tile's published count of one digit: flag 1 with the tile's own count, 2 with
// the count of all tiles up to it (0: not yet known)
template <class S>
struct RsState {
    static constexpr int SHIFT = sizeof(S) * 8 - 2;
    static constexpr S OWN = (S)1 << SHIFT, ALL = (S)2 << SHIFT, COUNT = OWN - 1;
};

// tile states are written and polled by running blocks
__device__ __forceinline__ uint32_t state_load(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t state_load(const uint64_t* p)
{
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void state_store(uint32_t* p, uint32_t v)
{
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" : : "l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void state_store(uint64_t* p, uint64_t v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" : : "l"(p), "l"(v) : "memory");
}

template <class K>
__global__ void __launch_bounds__(RS_THREADS)
k_rs_hist(const K* __restrict__ keys, int n, int passes, int bits, uint32_t* __restrict__ head)
{
    grid_begin();
    __shared__ uint32_t h[RS_HIST];
    __shared__ bool last;
    const int bins = 1 << bits, tid = threadIdx.x;
    uint32_t* hist = head + RS_HEAD;
    for (int i = tid; i < passes << bits; i += RS_THREADS) h[i] = 0u;
    __syncthreads();
    const unsigned lane = tid & 31;
    for (long long i0 = (long long)blockIdx.x * RS_THREADS; i0 < n; i0 += (long long)gridDim.x * RS_THREADS) {
        const long long i = i0 + tid;
        const bool valid = i < n;
        const K k = valid ? keys[i] : (K)0;
        const unsigned act = __ballot_sync(0xffffffffu, valid);
        if (!valid) continue;
        for (int p = 0; p < passes; ++p) {
            const unsigned d = (unsigned)(k >> (p * bits)) & (unsigned)(bins - 1);
            // neighbours often share their high digits: one add for the warp then
            const unsigned first = __shfl_sync(act, d, __ffs(act) - 1);
            if (__all_sync(act, d == first)) {
                if (lane == (unsigned)(__ffs(act) - 1)) atomicAdd(&h[(p << bits) + d], __popc(act));
            } else {
                atomicAdd(&h[(p << bits) + d], 1u);
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < passes << bits; i += RS_THREADS)
        if (h[i]) atomicAdd(hist + i, h[i]);
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(head + RS_PASSES, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    // the last block: exclusive scan of each pass's counts, a warp per pass, a lane
    // over bins / 32 neighbours
    __threadfence();
    for (int p = tid >> 5; p < passes; p += RS_WARPS) {
        uint32_t* c = hist + (p << bits) + lane * (bins >> 5);
        uint32_t v[16], sum = 0;
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            v[u] = u < bins >> 5 ? __ldcg(c + u) : 0u;
            sum += v[u];
        }
        uint32_t run = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, run, o);
            if ((int)lane >= o) run += y;
        }
        run -= sum;
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            if (u < bins >> 5) c[u] = run;
            run += v[u];
        }
    }
}

template <class K, int BITS>
struct RsSmem {
    K key[RS_TILE<K>];
    int val[RS_TILE<K>];
    uint32_t wcnt[RS_WARPS][1 << BITS];  // per-warp digit counts, then offsets
    uint32_t lstart[1 << BITS];          // first slot of each digit in the tile
    uint32_t gstart[1 << BITS];          // the digit's first output position for this tile
    uint32_t wsum[RS_WARPS];
    int tile;
};

// One digit, stable.  A block takes the next tile; warp w ranks its own contiguous
// ROUNDS x 32 elements with per-warp digit counters (no block barrier while
// ranking), the tile's digit counts are published, one block-level scan turns
// the counters into positions of the tile in digit order, the tile is placed in
// shared memory in that order, and written out so that consecutive threads
// store consecutive addresses within each digit's run.  Order is kept: within a
// digit, elements stay in (warp, round, lane) = input order.  vin == nullptr: the
// values are the input positions.  Tiles are numbered in the order in which
// blocks start, so the tiles a block looks back at are running or done.
template <class K, int BITS, class S>
__global__ void __launch_bounds__(RS_THREADS, 3)
k_rs_pass(const K* __restrict__ kin, const int* __restrict__ vin, K* __restrict__ kout,
          int* __restrict__ vout, int n, int shift, uint32_t* __restrict__ ticket,
          const uint32_t* __restrict__ start, S* state, int* err)
{
    grid_begin();
    constexpr int BINS = 1 << BITS, PER = BINS / RS_THREADS;  // digits per thread, neighbours
    constexpr int ROUNDS = RS_ROUNDS<K>;
    extern __shared__ __align__(16) unsigned char rs_smem[];
    RsSmem<K, BITS>& M = *reinterpret_cast<RsSmem<K, BITS>*>(rs_smem);
    const int tid = threadIdx.x, warp = tid >> 5;
    const unsigned lane = tid & 31, lt = lanemask_lt();
    if (tid == 0) M.tile = (int)atomicAdd(ticket, 1u);
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w)
#pragma unroll
        for (int c = 0; c < PER; ++c) M.wcnt[w][tid + c * RS_THREADS] = 0u;
    __syncthreads();
    const int tile = M.tile;
    const long long base = (long long)tile * RS_TILE<K>;
    // ---- rank: this warp's elements base + warp*32*ROUNDS + r*32 + lane ----
    // An element's rank is the count of its digit before this round plus its place
    // among the lanes of equal digit; the first of them adds to the counter.  The
    // digit matches and the adds of all rounds are issued without waiting for one
    // another (a warp's shared-memory operations complete in order): waiting for
    // each round's counter was half of the pass's time.
    K k[ROUNDS];
    unsigned short pos[ROUNDS];  // position among this warp's elements of the same digit
    const long long wbase = base + warp * 32 * ROUNDS;
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const long long i = wbase + r * 32 + (int)lane;
        k[r] = i < n ? kin[i] : (K)0;
    }
    {
        unsigned peers[ROUNDS];
        uint32_t before[ROUNDS];
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            const bool valid = wbase + r * 32 + (int)lane < n;
            const unsigned d = (unsigned)(k[r] >> shift);
            if constexpr (sizeof(K) == 8) {  // by ballots: 170 against 185 us per pass of 18.3 M
                peers[r] = __ballot_sync(0xffffffffu, valid);
                peers[r] = valid ? peers[r] : ~peers[r];
#pragma unroll
                for (int b = 0; b < BITS; ++b) {
                    const bool set = (d >> b) & 1u;
                    const unsigned m = __ballot_sync(0xffffffffu, set);
                    peers[r] &= set ? m : ~m;
                }
            } else {  // with twice the elements in flight the match instruction is faster
                peers[r] = __match_any_sync(0xffffffffu, valid ? d & (BINS - 1) : (unsigned)BINS);
            }
        }
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            const bool valid = wbase + r * 32 + (int)lane < n;
            before[r] = 0u;
            if (valid && (peers[r] & lt) == 0u)
                before[r] = atomicAdd(&M.wcnt[warp][(unsigned)(k[r] >> shift) & (BINS - 1)],
                                      (uint32_t)__popc(peers[r]));
            __syncwarp();
        }
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r)
            pos[r] = (unsigned short)(__shfl_sync(0xffffffffu, before[r], __ffs(peers[r]) - 1) +
                                      __popc(peers[r] & lt));
    }
    int v[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const long long i = wbase + r * 32 + (int)lane;
        v[r] = i < n ? (vin ? vin[i] : (int)i) : 0;
    }
    __syncthreads();
    // ---- per digit: offsets of the warps, the tile's count published, the tile's scan ----
    uint32_t cnt[PER];
    uint32_t sum = 0;
#pragma unroll
    for (int c = 0; c < PER; ++c) {
        const int d = tid * PER + c;
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) {
            const uint32_t x = M.wcnt[w][d];
            M.wcnt[w][d] = run;
            run += x;
        }
        cnt[c] = run;
        state_store(state + (size_t)tile * BINS + d, (tile ? RsState<S>::OWN : RsState<S>::ALL) | (S)run);
        M.lstart[d] = sum;
        sum += run;
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if ((int)lane >= o) inc += y;
    }
    if (lane == 31) M.wsum[warp] = inc;
    __syncthreads();
    uint32_t woff = inc - sum;
    for (int w = 0; w < warp; ++w) woff += M.wsum[w];
#pragma unroll
    for (int c = 0; c < PER; ++c) M.lstart[tid * PER + c] += woff;
    __syncthreads();
    // ---- place the tile in digit order ----
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        if (wbase + r * 32 + (int)lane < n) {
            const unsigned d = (unsigned)(k[r] >> shift) & (BINS - 1);
            const uint32_t slot = M.lstart[d] + M.wcnt[warp][d] + pos[r];
            M.key[slot] = k[r];
            M.val[slot] = v[r];
        }
    }
    // ---- look back: the elements of each digit in the tiles before this one ----
#pragma unroll
    for (int c = 0; c < PER; ++c) {
        const int d = tid * PER + c;
        S before = 0;
        int polls = 0;
        for (int q = tile - 1; q >= 0;) {
            // the states of the next RS_BACK tiles at once: a chain of single loads
            // took longer than the tile's own work
            S x[RS_BACK];
#pragma unroll
            for (int u = 0; u < RS_BACK; ++u)
                x[u] = q - u >= 0 ? state_load(state + (size_t)(q - u) * BINS + d) : RsState<S>::ALL;
            bool ended = false;
#pragma unroll
            for (int u = 0; u < RS_BACK; ++u) {
                if (ended || !(x[u] >> RsState<S>::SHIFT)) {
                    ended = true;  // done, or not yet published: ask again from here
                } else {
                    before += x[u] & RsState<S>::COUNT;
                    --q;
                    if (x[u] & RsState<S>::ALL) {
                        ended = true;
                        q = -1;
                    }
                }
            }
            if (q >= 0 && ++polls >= RS_POLLS) {
                atomicOr(err, ERR_SORT);
                break;
            }
        }
        if (tile)
            state_store(state + (size_t)tile * BINS + d,
                        RsState<S>::ALL | ((before + (S)cnt[c]) & RsState<S>::COUNT));
        M.gstart[d] = start[d] + (uint32_t)before;
    }
    __syncthreads();
    // ---- write out: slot j of digit d goes to gstart[d] + (j - lstart[d]) ----
    const int live = (int)min((long long)RS_TILE<K>, n - base);
    for (int j = tid; j < live; j += RS_THREADS) {
        const K kk = M.key[j];
        const unsigned d = (unsigned)(kk >> shift) & (BINS - 1);
        const uint32_t dst = M.gstart[d] + ((uint32_t)j - M.lstart[d]);
        if (dst < (uint32_t)n) {  // always, unless a look-back gave up
            kout[dst] = kk;
            vout[dst] = M.val[j];
        }
    }
}

// ---- up to RSC_MAX elements: one launch on a cluster of 8 or 16 blocks ----
// Small sorts are bound by the latency of a pass (5 to 8 us each, and a histogram and
// a memset before them).  Here the elements stay in the cluster: block b holds
// positions [b T, (b + 1) T) in registers, ranks them as k_rs_pass does, the blocks read
// one another's digit counts, and every element goes straight to its new place in the
// shared memory of the block it belongs to.  Missing elements have all bits set and
// stay last.  Unpack, 48-bit sort and gather together: 4099 particles 54 -> 32 us,
// 13,840 61 -> 38, 32,768 64 -> 54; above that the cluster is slower (50,000: 67 and
// 79).  8 blocks up to 8192 elements (2 us less than 16), 16 above (13,840: 9 us less
// than 8).
constexpr int RSC_THREADS = 1024, RSC_WARPS = RSC_THREADS / 32, RSC_BINS = 256;
constexpr int RSC_MAX = 16 * RSC_THREADS * 2;

template <class K, int R>
struct RsCluster {
    K key[RSC_THREADS * R];
    int val[RSC_THREADS * R];
    uint32_t wcnt[RSC_WARPS][RSC_BINS];  // per-warp digit counts, then offsets in the quarter
    uint32_t part[4][RSC_BINS];          // per quarter of the warps: counts, then offsets
    uint32_t cnt[RSC_BINS];              // the block's digit counts, read by the cluster
    uint32_t gstart[RSC_BINS];           // the digit's first position for this block
    uint32_t wsum[RSC_BINS / 32];
};

template <class K, int R, int RSC_CTAS>
__global__ void __cluster_dims__(RSC_CTAS, 1, 1) __launch_bounds__(RSC_THREADS)
k_rs_cluster(const K* __restrict__ kin, const int* __restrict__ vin, K* __restrict__ kout,
             int* __restrict__ vout, int n, int passes)
{
    grid_begin();
    extern __shared__ __align__(16) unsigned char rs_smem[];
    using Mem = RsCluster<K, R>;
    Mem& M = *reinterpret_cast<Mem*>(rs_smem);
    auto cluster = cooperative_groups::this_cluster();
    constexpr int T = RSC_THREADS * R;
    const int tid = threadIdx.x, warp = tid >> 5, me = blockIdx.x;
    const unsigned lane = tid & 31, lt = lanemask_lt();
    const int mine = warp * 32 * R + (int)lane;  // + 32 r: the thread's elements of the block
    K k[R];
    int v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = me * T + mine + 32 * r;
        k[r] = i < n ? kin[i] : ~(K)0;
        v[r] = i < n ? (vin ? vin[i] : i) : 0;
    }
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
#pragma unroll
        for (int c = 0; c < RSC_BINS / 32; ++c) M.wcnt[warp][32 * c + lane] = 0u;
        __syncwarp();
        unsigned peers[R];
        uint32_t pos[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned d = (unsigned)(k[r] >> shift);
            peers[r] = ~0u;
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const bool set = (d >> b) & 1u;
                const unsigned m = __ballot_sync(0xffffffffu, set);
                peers[r] &= set ? m : ~m;
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            pos[r] = 0u;
            if ((peers[r] & lt) == 0u)
                pos[r] = atomicAdd(&M.wcnt[warp][(unsigned)(k[r] >> shift) & (RSC_BINS - 1)],
                                   (uint32_t)__popc(peers[r]));
            __syncwarp();
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            pos[r] = __shfl_sync(0xffffffffu, pos[r], __ffs(peers[r]) - 1) + __popc(peers[r] & lt);
        __syncthreads();
        // per digit: offsets of the warps within their quarter, of the quarters, the count
        {
            const int d = tid & (RSC_BINS - 1), quarter = tid / RSC_BINS;
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < RSC_WARPS / 4; ++w) {
                const uint32_t x = M.wcnt[quarter * (RSC_WARPS / 4) + w][d];
                M.wcnt[quarter * (RSC_WARPS / 4) + w][d] = run;
                run += x;
            }
            M.part[quarter][d] = run;
        }
        __syncthreads();
        if (tid < RSC_BINS) {
            uint32_t run = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t x = M.part[q][tid];
                M.part[q][tid] = run;
                run += x;
            }
            M.cnt[tid] = run;
        }
        cluster.sync();  // the counts are out; every block's elements are in registers
        uint32_t before = 0, all = 0, inc = 0;
        if (tid < RSC_BINS) {
#pragma unroll
            for (int c = 0; c < RSC_CTAS; ++c) {
                const uint32_t x = *cluster.map_shared_rank(&M.cnt[tid], c);
                before += c < me ? x : 0u;
                all += x;
            }
            inc = all;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if ((int)lane >= o) inc += y;
            }
            if (lane == 31) M.wsum[warp] = inc;
        }
        __syncthreads();
        if (tid < RSC_BINS) {
            uint32_t g = before + inc - all;
            for (int w = 0; w < warp; ++w) g += M.wsum[w];
            M.gstart[tid] = g;
        }
        __syncthreads();
        const bool last = p == passes - 1;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned d = (unsigned)(k[r] >> shift) & (RSC_BINS - 1);
            const uint32_t at = M.gstart[d] + M.part[warp / (RSC_WARPS / 4)][d] + M.wcnt[warp][d] + pos[r];
            if (last) {
                if (at < (uint32_t)n) {
                    kout[at] = k[r];
                    vout[at] = v[r];
                }
            } else {
                *cluster.map_shared_rank(&M.key[at % T], at / T) = k[r];
                *cluster.map_shared_rank(&M.val[at % T], at / T) = v[r];
            }
        }
        cluster.sync();  // all elements have arrived; at the end: all counts have been read
        if (!last) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                k[r] = M.key[mine + 32 * r];
                v[r] = M.val[mine + 32 * r];
            }
        }
    }
}

// sets the kernel up on the current device, once; false: it cannot run such a cluster
template <class K, int R, int CTAS>
static bool rs_cluster_ready()
{
    int dev = 0;
    cudaGetDevice(&dev);
    static std::atomic<unsigned long long> checked{0}, possible{0};  // one bit per device
    const unsigned long long bit = 1ull << (dev & 63);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CTAS);
    cfg.blockDim = dim3(RSC_THREADS);
    cfg.dynamicSmemBytes = sizeof(RsCluster<K, R>);
    if (!(checked.load() & bit)) {
        auto* f = k_rs_cluster<K, R, CTAS>;
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes);
        cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        int clusters = 0;
        cudaLaunchAttribute dims;
        dims.id = cudaLaunchAttributeClusterDimension;
        dims.val.clusterDim.x = CTAS;
        dims.val.clusterDim.y = dims.val.clusterDim.z = 1;
        cfg.attrs = &dims;
        cfg.numAttrs = 1;
        const bool ok = cudaOccupancyMaxActiveClusters(&clusters, f, &cfg) == cudaSuccess && clusters > 0;
        if (!ok) cudaGetLastError();
        if (ok) possible.fetch_or(bit);
        checked.fetch_or(bit);
    }
    return (possible.load() & bit) != 0;
}

template <class K, int R, int CTAS>
static bool rs_cluster_t(const K* kin, const int* vin, K* kout, int* vout, int n, int passes, cudaStream_t s)
{
    if (!rs_cluster_ready<K, R, CTAS>()) return false;
    launch(k_rs_cluster<K, R, CTAS>, CTAS, RSC_THREADS, sizeof(RsCluster<K, R>), s, kin, vin, kout, vout, n, passes);
    count_launches(1);
    return true;
}

// sorts up to RSC_MAX elements into keys1, vals1
template <class K>
static bool rs_cluster(const K* keys0, const int* vals0, K* keys1, int* vals1, int n, int passes, bool iota,
                       cudaStream_t s)
{
    const int* vin = iota ? nullptr : vals0;
    if (n <= 8 * RSC_THREADS) return rs_cluster_t<K, 1, 8>(keys0, vin, keys1, vals1, n, passes, s);
    if (n <= 16 * RSC_THREADS) return rs_cluster_t<K, 1, 16>(keys0, vin, keys1, vals1, n, passes, s);
    return rs_cluster_t<K, 2, 16>(keys0, vin, keys1, vals1, n, passes, s);
}

// 32-bit tile states hold counts below 2^30
static bool rs_wide(int n) { return n >= (1 << 30); }

size_t radix_sort_temp_bytes(int n)
{
    // as many passes as either key type takes: 6 digits of 8 bits over tiles of
    // the 64-bit keys, 4 of 9 bits over tiles of the 32-bit keys
    const size_t t64 = (size_t)n / RS_TILE<uint64_t> + 1, t32 = (size_t)n / RS_TILE<uint32_t> + 1;
    const size_t states = std::max(6 * 256 * t64, 4 * 512 * t32) * (rs_wide(n) ? 8 : 4);
    return 4 * (RS_HEAD + RS_HIST) + states + 256;
}

// allows k_rs_pass its shared memory on the current device, once
template <class K, int BITS, class S>
static void rs_pass_ready(int dev)
{
    static std::atomic<unsigned long long> attr_set{0};  // one bit per device
    if (attr_set.load() & (1ull << (dev & 63))) return;
    cudaFuncSetAttribute(k_rs_pass<K, BITS, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(RsSmem<K, BITS>));
    attr_set.fetch_or(1ull << (dev & 63));
}

template <class K, int BITS, class S>
static int radix_sort_t(K* keys0, int* vals0, K* keys1, int* vals1, int n, int passes, bool iota,
                        void* temp, int* err, cudaStream_t s)
{
    constexpr int BINS = 1 << BITS;
    const int ntiles = (int)(((long long)n + RS_TILE<K> - 1) / RS_TILE<K>);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    rs_pass_ready<K, BITS, S>(dev);
    uint32_t* head = static_cast<uint32_t*>(temp);
    S* state = reinterpret_cast<S*>(head + RS_HEAD + RS_HIST);
    const size_t per_pass = (size_t)ntiles * BINS;
    cudaMemsetAsync(temp, 0, 4 * (RS_HEAD + RS_HIST) + sizeof(S) * per_pass * passes, s);
    const int blocks = std::min(4 * sms, (int)(((long long)n + 8 * RS_THREADS - 1) / (8 * RS_THREADS)));
    launch(k_rs_hist<K>, blocks, RS_THREADS, 0, s, keys0, n, passes, BITS, head);
    K* kb[2] = {keys0, keys1};
    int* vb[2] = {vals0, vals1};
    int cur = 0;
    for (int p = 0; p < passes; ++p) {
        launch(k_rs_pass<K, BITS, S>, ntiles, RS_THREADS, sizeof(RsSmem<K, BITS>), s, 
            kb[cur], p == 0 && iota ? nullptr : vb[cur], kb[cur ^ 1], vb[cur ^ 1], n, p * BITS,
            head + p, head + RS_HEAD + p * BINS, state + per_pass * p, err);
        cur ^= 1;
    }
    count_launches(1 + passes);
    return cur;
}

int radix_sort(uint64_t* keys0, int* vals0, uint64_t* keys1, int* vals1, int n, int bits, bool iota,
               void* temp, int* err, cudaStream_t s)
{
    const int passes = n > 1 ? (bits + 7) / 8 : 0;
    if (passes == 0) {
        if (iota) launch_iota(vals0, n, s);
        return 0;
    }
    if (n <= RSC_MAX && rs_cluster(keys0, vals0, keys1, vals1, n, passes, iota, s)) return 1;
    return rs_wide(n) ? radix_sort_t<uint64_t, 8, uint64_t>(keys0, vals0, keys1, vals1, n, passes, iota, temp, err, s)
                      : radix_sort_t<uint64_t, 8, uint32_t>(keys0, vals0, keys1, vals1, n, passes, iota, temp, err, s);
}

int radix_sort32(uint32_t* keys0, int* vals0, uint32_t* keys1, int* vals1, int n, int bits, bool iota,
                 void* temp, int* err, cudaStream_t s)
{
    const int p8 = n > 1 ? (bits + 7) / 8 : 0, p9 = n > 1 ? (bits + 8) / 9 : 0;
    if (p8 == 0) {
        if (iota) launch_iota(vals0, n, s);
        return 0;
    }
    if (n <= RSC_MAX && rs_cluster(keys0, vals0, keys1, vals1, n, p8, iota, s)) return 1;
    if (p9 < p8)
        return rs_wide(n) ? radix_sort_t<uint32_t, 9, uint64_t>(keys0, vals0, keys1, vals1, n, p9, iota, temp, err, s)
                          : radix_sort_t<uint32_t, 9, uint32_t>(keys0, vals0, keys1, vals1, n, p9, iota, temp, err, s);
    return rs_wide(n) ? radix_sort_t<uint32_t, 8, uint64_t>(keys0, vals0, keys1, vals1, n, p8, iota, temp, err, s)
                      : radix_sort_t<uint32_t, 8, uint32_t>(keys0, vals0, keys1, vals1, n, p8, iota, temp, err, s);
}

__global__ void k_iota(int* a, int n)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = i;
}
void launch_iota(int* a, int n, cudaStream_t s)
{
    if (n <= 0) return;
    launch(k_iota, (n + 255) / 256, 256, 0, s, a, n);
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
    box[2 * id] = make_float4(r[0], r[3], r[1], r[4]);
    box[2 * id + 1] = make_float4(r[2], r[5], 0.0f, 0.0f);
}

// The particles in curve order, the boxes of their leaves and, LEAF16 (leaves of
// 16 particles), of the level above: a block holds 512 particles, the children of
// one box of level 1.  perm is a permutation unless the sort gave up (ERR_SORT):
// then its stray entries are replaced, so that nothing after reads or writes out
// of range.  rk_in == nullptr: no smoothing lengths yet, 0.
constexpr int GATHER_THREADS = 512;
template <bool LEAF16>
__global__ void __launch_bounds__(GATHER_THREADS)
k_gather(int* __restrict__ perm, const float4* __restrict__ rec, const float* __restrict__ rk_in, int n,
         float4* __restrict__ pos, float4* __restrict__ vel, int* __restrict__ igrp,
         float* __restrict__ rk, const __grid_constant__ TreeView t)
{
    grid_begin();
    const int i = blockIdx.x * GATHER_THREADS + threadIdx.x;
    const bool live = i < n;
    int o = live ? perm[i] : 0;
    if ((unsigned)o >= (unsigned)n) {
        o = i;
        perm[i] = i;
    }
    const float4 p = rec[2 * (size_t)o], v = rec[2 * (size_t)o + 1];
    if (live) {
        pos[i] = make_float4(p.x, p.y, p.z, __int_as_float(o));
        vel[i] = v;
        igrp[i] = __float_as_int(p.w);
        rk[i] = rk_in ? rk_in[o] : 0.0f;
    }
    if constexpr (LEAF16) {
        __shared__ float leaf[6][GATHER_THREADS / 16];
        float4* box = const_cast<float4*>(t.box);
        const float inf = INFINITY;
        float b[6] = {live ? p.x : inf, live ? p.y : inf, live ? p.z : inf,
                      live ? p.x : -inf, live ? p.y : -inf, live ? p.z : -inf};
        group_box<16>(b);
        if ((threadIdx.x & 15) == 0) {
            if (live) store_box(box, (size_t)(i >> 4), b);
#pragma unroll
            for (int a = 0; a < 6; ++a) leaf[a][threadIdx.x >> 4] = b[a];
        }
        if (t.nlev == 1) return;
        __syncthreads();
        if (threadIdx.x >= 32) return;
#pragma unroll
        for (int a = 0; a < 6; ++a) b[a] = leaf[a][threadIdx.x];
        group_box<32>(b);
        if (threadIdx.x == 0) store_box(box, (size_t)t.off[1] + blockIdx.x, b);
    }
}

// level 0: G lanes (16, or 32 for leaves of more particles) per leaf, one
// coalesced load per lane
template <int G>
__global__ void k_leaf_boxes(const float4* __restrict__ pos, int n, int leaf, int nleaf,
                             float4* __restrict__ box)
{
    grid_begin();
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
    grid_begin();
    const long long id = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    if (id >= nbox) return;
    const long long c = min(id * 32 + (threadIdx.x & 31), (long long)nbelow - 1);
    const float4 u = below[2 * c], v = below[2 * c + 1];
    float b[6] = {u.x, u.z, v.x, u.y, u.w, v.y};
    group_box<32>(b);
    if ((threadIdx.x & 31) == 0) store_box(box, (size_t)id, b);
}

void launch_gather(int* perm, const float4* rec, const float* rk_in, const TreeView& t, float4* pos,
                   float4* vel, int* igrp, float* rk, cudaStream_t s)
{
    if (t.n <= 0) return;
    float4* box = const_cast<float4*>(t.box);
    const unsigned nb = (unsigned)(((long long)t.n + GATHER_THREADS - 1) / GATHER_THREADS);
    int l = 2;
    if (t.leaf == 16) {
        launch(k_gather<true>, nb, GATHER_THREADS, 0, s, perm, rec, rk_in, t.n, pos, vel, igrp, rk, t);
        count_launches(1);
    } else {
        launch(k_gather<false>, nb, GATHER_THREADS, 0, s, perm, rec, rk_in, t.n, pos, vel, igrp, rk, t);
        const int g = t.leaf <= 16 ? 16 : 32;
        const unsigned lb = (unsigned)(((long long)t.cnt[0] * g + 255) / 256);
        if (g == 16) launch(k_leaf_boxes<16>, lb, 256, 0, s, pos, t.n, t.leaf, t.cnt[0], box);
        else launch(k_leaf_boxes<32>, lb, 256, 0, s, pos, t.n, t.leaf, t.cnt[0], box);
        count_launches(2);
        l = 1;
    }
    for (; l < t.nlev; ++l) {
        launch(k_up_boxes, (unsigned)(((long long)t.cnt[l] * 32 + 255) / 256), 256, 0, s, 
            box + 2 * t.off[l - 1], t.cnt[l - 1], box + 2 * t.off[l], t.cnt[l]);
        count_launches(1);
    }
}

// ---------------------------------------------------------------------------
// output in input order
// ---------------------------------------------------------------------------
__global__ void k_pack_aos(const int* __restrict__ perm, const float4* __restrict__ pos,
                           const float4* __restrict__ vel, const float* __restrict__ rk,
                           const int* __restrict__ igrp, int n, ParticleRec* __restrict__ aos)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int o = perm[i];
    const float4 p = pos[i], v = vel[i];
    float* r = reinterpret_cast<float*>(aos + o);
    r[0] = p.x; r[1] = p.y; r[2] = p.z;
    r[3] = v.x; r[4] = v.y; r[5] = v.z;
    r[6] = v.w;
    r[7] = rk[i];
    reinterpret_cast<int*>(r)[8] = igrp[i];
}

void launch_pack_aos(const int* perm, const float4* pos, const float4* vel, const float* rk,
                     const int* igrp, int n, void* aos, cudaStream_t s)
{
    if (n <= 0) return;
    launch(k_pack_aos, (n + 255) / 256, 256, 0, s, perm, pos, vel, rk, igrp, n,
                                                (ParticleRec*)aos);
    count_launches(1);
}

// staged records as Particle records, in their order
__global__ void k_pack_staged(const float4* __restrict__ rec, const float* __restrict__ rk, int n,
                              ParticleRec* __restrict__ aos)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = rec[2 * (size_t)i], v = rec[2 * (size_t)i + 1];
    float* r = reinterpret_cast<float*>(aos + i);
    r[0] = p.x; r[1] = p.y; r[2] = p.z;
    r[3] = v.x; r[4] = v.y; r[5] = v.z;
    r[6] = v.w;
    r[7] = rk ? rk[i] : 0.0f;
    reinterpret_cast<int*>(r)[8] = __float_as_int(p.w);
}

void launch_pack_staged(const float4* rec, const float* rk, int n, void* aos, cudaStream_t s)
{
    if (n <= 0) return;
    launch(k_pack_staged, (n + 255) / 256, 256, 0, s, rec, rk, n, (ParticleRec*)aos);
    count_launches(1);
}

// Sorted fields to input order; dens is vel.w.  The stores go to random places.  Where
// the fields together are larger than SCATTER_L2, they are written one at a time, each
// in slices of that size (the particles of input positions [first, first + count)), so
// that the L2 takes all stores to a sector before it goes to memory: rk and dens of
// 18.3 M particles 728 -> 314 us (80 and 96 MB; 60 MB, two slices each, 425; both
// fields in two slices 392), of 60 M, three slices each, 6.8 -> 3.1 ms.  A slice reads
// all its input again, so from more than SCATTER_SLICES on there is one.
// STREAM: loads that leave the L2 to the stores, from SCATTER_STREAM of fields on (rk
// and dens of 10 M particles 149 -> 136 us, all three 259 -> 198; rk of 5 M 34 and 39).  Without
// slices nothing waits for perm but the stores (rk of 18 M 131 -> 110 us).
constexpr long long SCATTER_L2 = 80LL << 20, SCATTER_STREAM = 40LL << 20;
constexpr int SCATTER_SLICES = 5;
template <bool SLICED, bool STREAM>
__global__ void k_scatter_fields(const int* __restrict__ perm, const float* __restrict__ rk,
                                 const float4* __restrict__ vel, const int* __restrict__ igrp,
                                 int n, int first, int count, float* rk_out, float* dens_out, int* igrp_out)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    auto load = [](auto* p) { return STREAM ? __ldcs(p) : *p; };
    const int o = load(perm + i);
    if (SLICED && (unsigned)(o - first) >= (unsigned)count) return;
    if (rk_out) rk_out[o] = load(rk + i);
    if (dens_out) dens_out[o] = __ldcs(&vel[i].w);
    if (igrp_out) igrp_out[o] = load(igrp + i);
}

void launch_scatter_fields(const int* perm, const float* rk, const float4* vel, const int* igrp,
                           int n, float* rk_out, float* dens_out, int* igrp_out, cudaStream_t s)
{
    if (n <= 0) return;
    const int fields = (rk_out != nullptr) + (dens_out != nullptr) + (igrp_out != nullptr);
    const long long bytes = 4LL * n, all = bytes * fields;
    auto run = [&](int slices, float* r, float* d, int* g) {
        const int count = (n + slices - 1) / slices;
        auto kern = slices > 1 ? k_scatter_fields<true, true>
                               : all > SCATTER_STREAM ? k_scatter_fields<false, true> : k_scatter_fields<false, false>;
        for (int k = 0; k < slices; ++k)
            launch(kern, (n + 255) / 256, 256, 0, s, perm, rk, vel, igrp, n, k * count, count, r, d, g);
        count_launches(slices);
    };
    if (all <= SCATTER_L2) {
        run(1, rk_out, dens_out, igrp_out);
        return;
    }
    int slices = (int)((bytes - 1) / SCATTER_L2) + 1;
    if (slices > SCATTER_SLICES) slices = 1;
    if (rk_out) run(slices, rk_out, nullptr, nullptr);
    if (dens_out) run(slices, nullptr, dens_out, nullptr);
    if (igrp_out) run(slices, nullptr, nullptr, igrp_out);
}

// every kernel that a device array of up to RSC_MAX particles goes through from the
// load to the outputs, but the search
bool load_small_set_kernels()
{
    bool ok = kernel_loaded(k_unpack_soa) && kernel_loaded(k_gather<true>) && kernel_loaded(k_up_boxes) &&
              kernel_loaded(k_scatter_fields<false, false>);
    const bool clusters[] = {rs_cluster_ready<uint64_t, 1, 8>(), rs_cluster_ready<uint64_t, 1, 16>(),
                             rs_cluster_ready<uint64_t, 2, 16>()};
    ok = ok && kernel_loaded(k_rs_cluster<uint64_t, 1, 8>) && kernel_loaded(k_rs_cluster<uint64_t, 1, 16>) &&
         kernel_loaded(k_rs_cluster<uint64_t, 2, 16>);
    if (!(clusters[0] && clusters[1] && clusters[2])) {
        int dev = 0;
        cudaGetDevice(&dev);
        ok = ok && kernel_loaded(k_rs_hist<uint64_t>) && kernel_loaded(k_rs_pass<uint64_t, 8, uint32_t>);
        rs_pass_ready<uint64_t, 8, uint32_t>(dev);
    }
    return ok;
}

}  // namespace asg
