// asg_knn.cu -- k=33 nearest neighbours, smoothing length and particle density
// (the loop at clumping_tree_main.cpp:418-430 over neighbor_search,
// nbr_search.cpp:61-127, with KNeighbors k=33 from k_neighbors.h:9-51).
//
// Definition implemented (order independent): for query p the neighbour set is
// the 33 particles with the smallest key (d2, input index), d2 evaluated with
// the reference's float expression.  rk = sqrtf(d2 of the 33rd); the 32
// smallest keys (the 33rd excluded, self included) receive the tent weight
// ker(p, q, 1/rk) in dens.
//
// Three warp-bundle kernels over the blocked box tree (asg_tree.cuh); a warp
// serves the 32 consecutive (Hilbert-ordered) particles of one bundle, one
// lane per particle, and scans a leaf when any lane's radius reaches its box:
//   k_knn_t33   per-lane sorted top-33 of d2 in registers, candidates queued
//               and merged by comparator networks (asg_knn_net.cuh)
//               -> t33 = 33rd smallest d2 (exact, with multiplicity)
//   k_knn_ties  exact-radius recount: L = #(d2 < t33), the tied indices
//               -> idx33 = input index of the 33rd key, rk = sqrtf(t33)
//   k_dens_scatter the bundle's queries are SOURCES q with their exact radii;
//               in each leaf a lane holds a receiver j and adds ker(q, j)
//               for the queries q whose 32-set holds j, as 64-bit fixed point
//               (per-receiver power-of-two scale, one integer atomic per
//               receiver and leaf): exact integer sums, so deterministic in
//               any order.  It visits the leaves k_knn_t33 recorded.
#include <climits>
#include <cstddef>
#include <type_traits>

#include "asg_common.cuh"
#include "asg_internal.h"
#include "asg_knn_net.cuh"
#include "asg_tree.cuh"

namespace asg {

constexpr int KNN_WARPS = 4;
// k_dens_scatter: four warps per block and four queries per turn of its loop, 6.47
// ms on the 256^3 step (two queries 6.57, one warp per block 6.81)
constexpr int DENS_WARPS = 4, DENS_UNROLL = 4;
// k_knn_t33 runs 32 warps per SM at 64 registers, in blocks of 1 warp with the
// default leaf size and of 2 or 4 with others (the batched form's autotuner
// picks).
constexpr unsigned FULL = 0xffffffffu;

// A lane's queue holds up to KNN_SLOTS candidates; a flush merges the KNN_QUEUE
// newest.  With room for twice as many values as a flush takes, the queues are
// checked once per 16 candidates instead of once per 2, and a flush finds 8.4
// values per lane instead of 6.3 (a CPU model on the 256^3 cube's clustering:
// 12.6 flushes per bundle for 106 queued values per lane, against 14.0 for 89
// with 16 slots and a check every 2).
constexpr int KNN_SLOTS = 32;
constexpr int KNN_CHUNK = 16;  // candidates between two checks
static_assert(KNN_SLOTS >= KNN_QUEUE + KNN_CHUNK, "a chunk must fit behind a full flush");
static_assert(KNN_SLOTS == K_NN - 1 && KNN_SLOTS % KNN_QUEUE == 0 && 3 * KNN_CHUNK >= 32, "a list handed over");

// A warp's shared memory in k_knn_t33, addressed with 32-bit shared addresses: a
// lane's words lie at `column` (4 x lane into the struct) plus a constant.
struct KnnWarp {
    float queue[KNN_SLOTS][32];          // [slot][lane], +inf where unused
    float cand[3][KNN_CHUNK];            // x, y, z of the candidates of a chunk
    unsigned keys[TREE_LEVELS - 1][32];  // [level - 1][lane], pending children of the upper levels
    TreeBox box;                         // the bundle's box
};
constexpr unsigned QUEUE_ROW = 32 * sizeof(float);

template <unsigned OFF>
__device__ __forceinline__ float lds_f32(unsigned a)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1 + %2];" : "=f"(v) : "r"(a), "n"(OFF) : "memory");
    return v;
}
template <unsigned OFF>
__device__ __forceinline__ void sts_f32(unsigned a, float v)
{
    asm volatile("st.shared.f32 [%0 + %1], %2;" : : "r"(a), "n"(OFF), "f"(v) : "memory");
}
template <unsigned OFF>
__device__ __forceinline__ void lds_x2(unsigned a, f32x2& u, f32x2& v)
{
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2 + %3];" : "=l"(u), "=l"(v) : "r"(a), "n"(OFF) : "memory");
}
// queues d when d <= limit: three predicated instructions, no branch
__device__ __forceinline__ void knn_push(unsigned& slot, float d, float limit)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.le.f32 p, %1, %2;\n\t"
        "@p st.shared.f32 [%0], %1;\n\t"
        "@p add.u32 %0, %0, %3;\n\t}"
        : "+r"(slot) : "f"(d), "f"(limit), "n"(QUEUE_ROW) : "memory");
}

template <int I>
__device__ __forceinline__ void knn_take(float (&v)[KNN_QUEUE], unsigned q0)
{
    if constexpr (I < KNN_QUEUE) {
        v[I] = lds_f32<I * QUEUE_ROW>(q0);
        sts_f32<I * QUEUE_ROW>(q0, INFINITY);
        knn_take<I + 1>(v, q0);
    }
}

// Merges KNN_QUEUE ascending values into the ascending top-33 a[].  tie_out ("a
// particle outside a[] has d2 == a[32]") stays exact: the values dropped by the
// merge are all >= the 34th smallest t34, so one of them ties the new a[32] exactly
// when t34 == a[32]; an earlier tie survives only while a[32] is unchanged.
__device__ __forceinline__ void knn_take_sorted(float (&a)[K_NN], float (&v)[KNN_QUEUE], bool& tie_out)
{
    const float old = a[K_NN - 1];
    const float t34 = knn_merge33(a, v);
    const float top = a[K_NN - 1];
    tie_out = (top == old && tie_out) || t34 == top;
}

// Merges the up to KNN_QUEUE newest candidates of a lane's queue (at `column`;
// `slot`: its next free slot) into its ascending top-33 a[] and refills their
// slots with +inf.
__device__ __forceinline__ void knn_flush(float (&a)[K_NN], unsigned column, unsigned& slot,
                                          bool& tie_out)
{
    slot = max(slot, column + QUEUE_ROW * KNN_QUEUE) - QUEUE_ROW * KNN_QUEUE;
    float v[KNN_QUEUE];
    knn_take<0>(v, slot);
    knn_sort16(v);
    knn_take_sorted(a, v, tie_out);
}

// the largest of SPLIT warps' shared values of a lane, 128 bytes apart
template <int SPLIT>
__device__ __forceinline__ float knn_shared_bound(unsigned at)
{
    float r = lds_f32<0>(at);
    if constexpr (SPLIT >= 2) r = fmaxf(r, lds_f32<128>(at));
    if constexpr (SPLIT >= 4) r = fmaxf(r, fmaxf(lds_f32<256>(at), lds_f32<384>(at)));
    return r;
}

// four candidates against the lane's query: the distances two at a time in
// packed f32x2 operations (equal values queue too: the merge tracks ties)
template <int J>
__device__ __forceinline__ void knn_scan(unsigned warp_base, f32x2 qx, f32x2 qy, f32x2 qz,
                                         float limit, unsigned& slot)
{
    if constexpr (J < KNN_CHUNK) {
        constexpr unsigned C = (unsigned)offsetof(KnnWarp, cand) + 4u * J, ROW = 4u * KNN_CHUNK;
        f32x2 x0, x1, y0, y1, z0, z1;
        lds_x2<C>(warp_base, x0, x1);
        lds_x2<C + ROW>(warp_base, y0, y1);
        lds_x2<C + 2 * ROW>(warp_base, z0, z1);
        const f32x2 d01 = norm2_rn_x2(qx, qy, qz, x0, y0, z0);
        const f32x2 d23 = norm2_rn_x2(qx, qy, qz, x1, y1, z1);
        knn_push(slot, lo2(d01), limit);
        knn_push(slot, hi2(d01), limit);
        knn_push(slot, lo2(d23), limit);
        knn_push(slot, hi2(d23), limit);
        knn_scan<J + 4>(warp_base, qx, qy, qz, limit, slot);
    }
}

// t33 = the 33rd smallest d2 (with multiplicity), rk = sqrtf(t33), and a tie
// flag: idx33 = -1 when exactly one particle sits at d2 == t33 (then the
// 32-set is {d2 < t33} and needs no index), -2 when ties must be resolved.
// Each lane keeps its 33 smallest d2 sorted in registers; a candidate with
// d2 <= a[32] goes to the lane's queue in shared memory, and when any lane's
// queue holds more than KNN_QUEUE values after a chunk of 16 candidates the
// warp merges the newest of every queue with two comparator networks (sort,
// odd-even merge with a[]), about a quarter of the min/max work of inserting
// each candidate as it comes.  Thresholds are the merged a[32], an upper bound
// of the true one while values wait in the queue.  The leaves scanned go to
// blist for k_dens_scatter.
//
// Bound by instruction issue: 74% of issue slots busy, 17.4 K warp instructions
// per bundle of 2.5 M particles in NFW halos (a fifth of them the networks' min/max on
// the ALU pipe, 54% busy), DRAM below 1%.  16.7 -> 10.3 ms on the 256^3 step (18.3 M
// particles) against the binary radix tree; 0.43 -> 0.26 ms at 377 k particles.
//
// The walk goes up from the bundle's own leaf: the siblings of its leaves
// first, then at every level the siblings of its ancestor.  A node is opened by
// all lanes together, a child per lane: the distance of the child's box to the
// bundle's box, as an integer key with the lane in its low bits, so one warp
// minimum gives the nearest child left, and a node is done when that one lies
// beyond the largest radius of the bundle.  Keys of the levels above wait in
// shared memory.  A node is opened and a leaf scanned if some lane's own radius reaches
// its box: at the edge of a clump a bundle's box holds all of it, and without the test
// at the nodes its warp looked at every leaf (3 M particles in one Gaussian clump 14.0
// -> 1.9 ms, 16.8 M in NFW halos 10.0 -> 9.5).
// LEAF16: leaves of 16 particles (the default), one chunk each.
//
// SPLIT > 1 (few bundles): the block's SPLIT warps search for the same bundle, each
// in the leaves of its own (leaf number mod SPLIT), and merge their lists at the
// end, since one warp's search is a serial chain of some 50 us.  Any SPLIT lists
// whose SHARE-th values lie within r hold 33 particles within r, so the largest of
// these values bounds t33 from above: it goes with a[32] into the pruning radius
// (read without synchronisation: values only shrink, an old one is a looser bound).
// Particles that it shuts out lie beyond t33, so ties stay exact.  4099 particles
// 56 -> 28 us, 13,840 in Plummer spheres 75 -> 42.
template <int T33_WARPS, bool LEAF16, int SPLIT>
__global__ void __launch_bounds__(T33_WARPS * 32, (SPLIT > 1 ? 16 : 32) / T33_WARPS)
k_knn_t33(const float4* __restrict__ pos, const __grid_constant__ TreeView t,
          float* __restrict__ t33, float* __restrict__ rk, int* __restrict__ idx33,
          int* __restrict__ blist, int* err)
{
    grid_begin();
    static_assert(SPLIT == 1 || (SPLIT == T33_WARPS && LEAF16), "one bundle per block");
    constexpr int SHARE = (K_NN + SPLIT - 1) / SPLIT;
    __shared__ __align__(16) KnnWarp smem[T33_WARPS];
    __shared__ float shares[SPLIT > 1 ? SPLIT : 1][32];  // each warp's a[SHARE - 1]
    __shared__ int listed;                               // leaves in the bundle's list
    const int lane = threadIdx.x & 31, part = SPLIT > 1 ? threadIdx.x >> 5 : 0;
    const int n = t.n;
    const int base = SPLIT > 1 ? blockIdx.x * 32 : (blockIdx.x * T33_WARPS + (threadIdx.x >> 5)) * 32;
    if (base >= n) return;
    if constexpr (SPLIT > 1) {
        shares[part][lane] = INFINITY;
        if (threadIdx.x == 0) listed = 0;
        __syncthreads();
    }
    const unsigned share_at = (unsigned)__cvta_generic_to_shared(&shares[0][lane]);
    KnnWarp& S = smem[threadIdx.x >> 5];
    const unsigned warp_base = (unsigned)__cvta_generic_to_shared(&S);
    const unsigned column = warp_base + 4u * (unsigned)lane;
    const int leaf = LEAF16 ? 16 : t.leaf;
#pragma unroll
    for (int i = 0; i < KNN_SLOTS; ++i) S.queue[i][lane] = INFINITY;
    f32x2 qx, qy, qz;
    {
        const float4 p = pos[min(base + lane, n - 1)];
        qx = pack2(p.x, p.x);
        qy = pack2(p.y, p.y);
        qz = pack2(p.z, p.z);
    }
    float a[K_NN];
#pragma unroll
    for (int k = 0; k < K_NN; ++k) a[k] = INFINITY;
    bool tie_out = false;  // a particle outside a[] has d2 == a[32]
    unsigned slot = column;
    int nlist = 0, entry = 0;  // leaves scanned; entry 32 k + lane of the list not yet written

    // keys up to `bound` are within the bundle's largest radius.  The bundle's
    // own leaves have keys below 32, all others at least 32, so they come first;
    // a node at distance 0 (a key below 64) always passes.
    unsigned bound = 0x7fffffffu;
    int g;  // the open group of leaves, 32 g ... 32 g + 31
    auto child_key = [&](int level, int id) {
        return max(__float_as_uint(boxes_dist2_fast(S.box, tree_box(t, level, id))) & ~31u, 32u) |
               (unsigned)lane;
    };
    unsigned key = ~0u;  // the lane's leaf of the group, ~0: none or visited
    {
        const int own0 = base / leaf, own1 = (min(base + 32, n) - 1) / leaf;
        const TreeBox b = bundle_box(t, own0, own1);
        if (lane == 0) S.box = b;
        __syncwarp();
        g = own0 >> 5;
        const int id = g * 32 + lane;
        if (id < t.cnt[0]) key = id >= own0 && id <= own1 ? (unsigned)lane : child_key(0, id);
        if (id % SPLIT != part) key = ~0u;
    }
    // the newest `cnt` entries into the bundle's list
    auto write_list = [&](int cnt) {
        int at = nlist - cnt;
        if constexpr (SPLIT > 1) {
            if (lane == 0) at = atomicAdd(&listed, cnt);
            at = __shfl_sync(FULL, at, 0);
        }
        if (lane < cnt && at + cnt <= KNN_LIST)
            blist[(size_t)(base >> 5) * (KNN_LIST + 1) + 1 + at + lane] = entry;
    };
    // a lane's t33 is at most this
    float limit = INFINITY;
    auto shrink = [&]() {
        limit = a[K_NN - 1];
        if constexpr (SPLIT > 1) limit = fminf(limit, knn_shared_bound<SPLIT>(share_at));
        bound = max(__reduce_max_sync(FULL, __float_as_uint(prune_bound(limit))) | 31u, 63u);
    };
    int top = 0;  // the highest level opened so far
    for (;;) {
        // ---- the leaves of group g, nearest first ----
        for (;;) {
            const unsigned m = __reduce_min_sync(FULL, key);
            if (m > bound) break;
            if (key == m) key = ~0u;
            const int id = g * 32 + (int)(m & 31u);
            const float4* bp = t.box + 2 * (size_t)id;
            const TreeBox c = {bp[0], bp[1]};
            if (!__any_sync(FULL, point_box_fast(qx, qy, qz, c) <=
                                      prune_bound(SPLIT > 1 ? limit : a[K_NN - 1])))
                continue;
            if (lane == (nlist & 31)) entry = id;
            ++nlist;
            if (blist && (nlist & 31) == 0) write_list(32);
            const int cnt = LEAF16 ? 16 : leaf_count(t, id);
            for (int c0 = 0; c0 < cnt; c0 += KNN_CHUNK) {
                __syncwarp();  // every lane is done with the chunk before it
                if (lane < KNN_CHUNK) {
                    // missing candidates are NaN points, whose distances queue nowhere
                    const int i = id * leaf + c0 + lane;
                    const bool have = LEAF16 ? i < n : c0 + lane < cnt;
                    const float4 p = pos[have ? i : 0];
                    constexpr unsigned C = (unsigned)offsetof(KnnWarp, cand), ROW = 4u * KNN_CHUNK;
                    sts_f32<C>(column, have ? p.x : __int_as_float(0x7fc00000));
                    sts_f32<C + ROW>(column, p.y);
                    sts_f32<C + 2 * ROW>(column, p.z);
                }
                __syncwarp();
                knn_scan<0>(warp_base, qx, qy, qz, SPLIT > 1 ? limit : a[K_NN - 1], slot);
                if (__any_sync(FULL, slot > column + QUEUE_ROW * KNN_QUEUE)) {
                    knn_flush(a, column, slot, tie_out);
                    if constexpr (SPLIT > 1) sts_f32<0>(share_at + 128u * part, a[SHARE - 1]);
                    else shrink();
                }
                if constexpr (SPLIT > 1) shrink();
                if (LEAF16) break;
            }
        }
        // ---- the next group: down the nearest pending child of the lowest level
        // that has one, else the siblings of the bundle's ancestor ----
        int L = 0, id = g;  // `id`: the group just done is node `id` of level L + 1
        bool found = false;
        for (;;) {
            ++L;
            int own = -1;
            unsigned k;
            if (L <= top) {
                k = S.keys[L - 1][lane];
            } else {
                if (top == t.nlev - 1) break;
                top = L;
                own = id;
                k = ~0u;
            }
            id >>= 5;  // the group of level L that node `id` was in
            if (own >= 0) {
                const int c = id * 32 + lane;
                if (c < t.cnt[L] && c != own) k = child_key(L, c);
            }
            // descend as long as a child within reach is left
            for (;;) {
                const unsigned m = __reduce_min_sync(FULL, k);
                if (m > bound) break;
                k = k == m ? ~0u : k;
                if (!__any_sync(FULL, point_box_fast(qx, qy, qz, tree_box(t, L, id * 32 + (int)(m & 31u))) <=
                                          prune_bound(SPLIT > 1 ? limit : a[K_NN - 1])))
                    continue;
                S.keys[L - 1][lane] = k;
                id = id * 32 + (int)(m & 31u);
                --L;
                const int c = id * 32 + lane;
                k = c < t.cnt[L] ? child_key(L, c) : ~0u;
                if (L == 0) {
                    g = id;
                    key = c % SPLIT == part ? k : ~0u;
                    found = true;
                    break;
                }
            }
            if (found) break;
            S.keys[L - 1][lane] = ~0u;  // nothing left here, now or later (radii only shrink)
        }
        if (!found) break;
    }
    if (__any_sync(FULL, slot > column)) knn_flush(a, column, slot, tie_out);
    // every leaf any lane's final radius reaches was scanned, so the list is
    // complete for k_dens_scatter unless it overflowed
    if (blist && (nlist & 31)) write_list(nlist & 31);
    if constexpr (SPLIT > 1) {
        __syncthreads();  // nobody prunes by the shared values any more
        // pairs of warps, pairs of pairs ...: the upper one hands its list over in its
        // queue's memory, and in `shares` the value of a particle that it left out
#pragma unroll
        for (int step = 1; step < SPLIT; step *= 2) {
            if (part % (2 * step) == step) {
#pragma unroll
                for (int k = 0; k < K_NN - 1; ++k) S.queue[k][lane] = a[k];
                (&S.cand[0][0])[lane] = a[K_NN - 1];
                shares[part][lane] = tie_out ? a[K_NN - 1] : -1.0f;
            }
            __syncthreads();
            if (part % (2 * step) == 0) {
                KnnWarp& G = smem[part + step];
                for (int k0 = 0; k0 < K_NN; k0 += KNN_QUEUE) {
                    const float first = k0 < KNN_SLOTS ? G.queue[k0][lane] : (&G.cand[0][0])[lane];
                    if (!__any_sync(FULL, first <= a[K_NN - 1])) break;
                    float v[KNN_QUEUE];
                    v[0] = first;
#pragma unroll
                    for (int k = 1; k < KNN_QUEUE; ++k)
                        v[k] = k0 < KNN_SLOTS ? G.queue[k0 + k][lane] : INFINITY;
                    knn_take_sorted(a, v, tie_out);
                }
                tie_out |= shares[part + step][lane] == a[K_NN - 1];
            }
            __syncthreads();
        }
        nlist = listed;
        if (part) return;
    }
    if (blist && lane == 0) blist[(size_t)(base >> 5) * (KNN_LIST + 1)] = nlist > KNN_LIST ? -1 : nlist;
    if (base + lane < n) {
        const float v = a[K_NN - 1];
        t33[base + lane] = v;
        rk[base + lane] = __fsqrt_rn(v);
        idx33[base + lane] = (tie_out || a[K_NN - 2] == v) ? -2 : -1;
        if (!(v < INFINITY)) atomicOr(err, ERR_FEW);
        else if (!(v > 0.0f)) atomicOr(err, ERR_ZERO_RK);
    }
}

// dens is summed as 64-bit fixed point per receiver j: a weight w counts as
// w * 2^(FIX_BITS - e_j), where 2^e_j bounds hinv_j^3.  A query q that has j in
// its 32-set has rk_j <= 2 rk_q (its 33 nearest lie within 2 rk_q of j), so
// w <= hinv_q^3 <= 8 hinv_j^3 and every term stays below 2^(FIX_BITS + 3 + a
// rounding margin).  A lane adds the terms it takes in one leaf (at most 32, in
// query order) as a double-float and converts the sum to an integer once; the
// integer atomics make the total independent of the order of the leaves.
constexpr int FIX_BITS = 40;

// e_j with hinv_j^3 <= 2^e_j up to rounding: minus the exponent of rk^3
__device__ __forceinline__ int dens_exponent(float rk)
{
    const float h3 = __fmul_rn(__fmul_rn(rk, rk), rk);
    const int e = 127 - ((__float_as_int(h3) >> 23) & 0xff);
    return max(-86, min(86, e));
}

// The 33rd key of flagged queries: with the exact radius T = t33 each lane
// counts L = #(d2 < T) and collects the tied indices (d2 == T); the 33rd key is
// the (33 - L)-th smallest tied index.  A pass keeps the TIE_MAX smallest tied
// indices above a floor (registers, an insertion network); a lane that needs a
// deeper one runs another pass with the floor at its last kept index, so any
// number of ties resolves in at most TIE_PASSES = ceil(33 / TIE_MAX) passes.
constexpr int TIE_PASSES = (K_NN + TIE_MAX - 1) / TIE_MAX;
// Mostly a bundle has one such query, if any, and the kernel lasts as long as one
// bundle: 24 -> 10 us at 377 k particles, 40 -> 18 with a zip decode's rounded
// positions.
constexpr int TIE_FEW = 8;  // queries of a bundle up to which each is resolved by itself

__global__ void __launch_bounds__(KNN_WARPS * 32)
k_knn_ties(const float4* __restrict__ pos, const __grid_constant__ TreeView t, const float* __restrict__ t33,
           int* __restrict__ idx33, int all, const int* __restrict__ blist, const float* __restrict__ rk,
           int* __restrict__ dexp, unsigned long long* __restrict__ acc, int* err)
{
    grid_begin();
    __shared__ float4 cand[KNN_WARPS][LEAF_MAX];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = t.n;
    const int base = (blockIdx.x * KNN_WARPS + warp) * 32;
    if (base >= n) return;
    const int q = min(base + lane, n - 1);
    if (dexp && base + lane < n) {  // ready for k_dens_scatter
        dexp[q] = dens_exponent(rk[q]);
        acc[q] = 0ull;
    }
    // unless every index is wanted, only queries flagged by k_knn_t33 (-2) need it
    const bool want = (base + lane < n) && (all || idx33[q] == -2);
    if (!__any_sync(FULL, want)) return;
    const float4 xq = pos[q];
    const float T = t33[q], bound = prune_bound(T);
    // few queries, and the leaves that k_knn_t33 scanned: one query at a time, a leaf's
    // box or a particle per lane; the k-th smallest tied index in lane k
    unsigned few = __ballot_sync(FULL, want);
    const int* bl = blist ? blist + (size_t)(base >> 5) * (KNN_LIST + 1) : nullptr;
    const int nlist = bl && t.leaf <= 16 ? bl[0] : -1;
    if (nlist >= 0 && __popc(few) <= TIE_FEW) {
        for (; few; few &= few - 1) {
            const int l = __ffs(few) - 1;
            const float x = __shfl_sync(FULL, xq.x, l), y = __shfl_sync(FULL, xq.y, l), z = __shfl_sync(FULL, xq.z, l);
            const float Tl = __shfl_sync(FULL, T, l), bl_ = prune_bound(Tl);
            int less = 0, eq = 0, tie = INT_MAX;
            for (int i0 = 0; i0 < nlist; i0 += 32) {
                const int e = i0 + lane < nlist ? bl[1 + i0 + lane] : 0;
                unsigned m = __ballot_sync(FULL, i0 + lane < nlist &&
                                                     point_box_fast(make_float4(x, y, z, 0.f), tree_box(t, 0, e)) <= bl_);
                while (m) {  // two leaves, a half-warp each
                    const int l0 = __ffs(m) - 1;
                    m &= m - 1;
                    const int l1 = m ? __ffs(m) - 1 : -1;
                    m &= m - 1;
                    const int mine = lane < 16 ? l0 : l1;
                    const int id = __shfl_sync(FULL, e, mine < 0 ? 0 : mine);
                    const bool have = mine >= 0 && (lane & 15) < leaf_count(t, id);
                    const float4 c = pos[have ? id * t.leaf + (lane & 15) : 0];
                    const float d2 = norm2_rn(x, y, z, c.x, c.y, c.z);
                    less += __popc(__ballot_sync(FULL, have && d2 < Tl));
                    unsigned ties = __ballot_sync(FULL, have && d2 == Tl);
                    eq += __popc(ties);
                    for (; ties; ties &= ties - 1) {
                        const int v = __shfl_sync(FULL, __float_as_int(c.w), __ffs(ties) - 1);
                        const int up = __shfl_up_sync(FULL, tie, 1);
                        const int at = __popc(__ballot_sync(FULL, tie < v));
                        tie = lane < at ? tie : lane == at ? v : up;
                    }
                }
            }
            // position of the 33rd key among all the ties: at most 32, as the query itself is
            // nearer than any T > 0 (T = 0 is reported as ERR_ZERO_RK, whatever the index)
            const int rank = K_NN - less;
            const int found = __shfl_sync(FULL, tie, (rank - 1) & 31);
            if (rank < 1 || rank > eq) {
                if (lane == l) {
                    atomicOr(err, ERR_FEW);
                    idx33[q] = -1;
                }
            } else if (lane == l) {
                idx33[q] = found;
            }
        }
        return;
    }
    int nless = 0, neq = 0;
    int need = 0;          // rank of the wanted index among the ties above floor
    int floor_idx = -1;    // this pass keeps tied indices > floor_idx
    bool open = want;      // this lane still looks for its index
    int result = -1;
    int tie[TIE_MAX];

    for (int pass = 0; pass < TIE_PASSES; ++pass) {
        if (!__any_sync(FULL, open)) break;
#pragma unroll
        for (int k = 0; k < TIE_MAX; ++k) tie[k] = INT_MAX;
        // the box of the queries still open and their largest radius
        TreeBox box;
        box.a = open ? make_float4(xq.x, xq.x, xq.y, xq.y)
                     : make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY);
        box.b = open ? make_float4(xq.z, xq.z, 0.f, 0.f) : make_float4(INFINITY, -INFINITY, 0.f, 0.f);
        float reach = open ? bound : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            TreeBox v;
            v.a = make_float4(__shfl_xor_sync(FULL, box.a.x, o), __shfl_xor_sync(FULL, box.a.y, o),
                              __shfl_xor_sync(FULL, box.a.z, o), __shfl_xor_sync(FULL, box.a.w, o));
            v.b = make_float4(__shfl_xor_sync(FULL, box.b.x, o), __shfl_xor_sync(FULL, box.b.y, o),
                              0.f, 0.f);
            box_grow(box, v);
            reach = fmaxf(reach, __shfl_xor_sync(FULL, reach, o));
        }
        tree_walk(t,
            [&](const TreeBox& c, int, int) { return boxes_dist2_fast(box, c) <= reach; },
            [&](int level, int id) {
                return __any_sync(FULL, open && point_box_fast(xq, tree_box(t, level, id)) <= bound) != 0;
            },
            [&](int id) {
                if (!__any_sync(FULL, open && point_box_fast(xq, tree_box(t, 0, id)) <= bound))
                    return true;
                const int first = id * t.leaf, cnt = leaf_count(t, id);
                __syncwarp();
                if (lane < cnt) cand[warp][lane] = pos[first + lane];
                __syncwarp();
                for (int j = 0; j < cnt; ++j) {
                    const float4 c = cand[warp][j];
                    const float d2 = norm2_rn(xq.x, xq.y, xq.z, c.x, c.y, c.z);
                    if (pass == 0) nless += d2 < T ? 1 : 0;
                    const int ci = __float_as_int(c.w);
                    const bool eq = open && d2 == T && ci > floor_idx;
                    if (__any_sync(FULL, eq)) {
                        if (pass == 0) neq += eq ? 1 : 0;
                        int v = eq ? ci : INT_MAX;
#pragma unroll
                        for (int k = 0; k < TIE_MAX; ++k) {
                            const int lo = min(tie[k], v);
                            v = max(tie[k], v);
                            tie[k] = lo;
                        }
                    }
                }
                return true;
            });
        if (open) {
            if (pass == 0) {
                need = K_NN - nless;  // position of the 33rd key among all the ties
                if (need < 1 || need > neq) {
                    atomicOr(err, ERR_FEW);
                    open = false;
                }
            }
            if (open && need <= TIE_MAX) {
#pragma unroll
                for (int k = 0; k < TIE_MAX; ++k)
                    if (k == need - 1) result = tie[k];
                open = false;
            } else if (open) {
                // the wanted index lies above the TIE_MAX kept ones
                need -= TIE_MAX;
                floor_idx = tie[TIE_MAX - 1];
            }
        }
    }
    if (open) atomicOr(err, ERR_TIES);  // unreachable: need <= 33 <= TIE_PASSES * TIE_MAX
    if (want) idx33[base + lane] = result;
}

// The warp serves the 32 queries (sources) q of a bundle with their exact radii
// and visits the leaves k_knn_t33 recorded for the bundle (each re-tested), or
// walks the tree when the list overflowed or is absent.  In a leaf each lane
// holds one candidate receiver j.  The queries whose radius reaches the leaf's
// box (a ballot; about 10 of 32) put themselves into a list in shared memory,
// and the warp loops over that list: for each such q every lane tests whether
// its j is in q's 32-set ((d2, index) below q's 33rd key) and adds ker(q, j) as 64-bit fixed point to a register; one integer
// atomic per receiver and leaf adds the sum to acc[j].  The sums are exact
// integers, so the order of the additions and atomics does not matter.
// HALVES (leaves of at most 16 particles): both half-warps hold the leaf's
// receivers and take every second query, so no lane idles; their integer sums
// are added by a shuffle before the atomic.
// PARTS: nparts warps share a bundle's leaves where bundles are few.
// Bound by instruction issue (79% of slots busy, 10.7 K warp instructions per
// bundle, of which the distances and weights are half): 7.10 -> 6.09 ms on the
// 256^3 step against radix-tree buckets of 22 particles on average.
template <bool HALVES, bool PARTS>
__global__ void __launch_bounds__(DENS_WARPS * 32)
k_dens_scatter(const float4* __restrict__ pos, const __grid_constant__ TreeView t, const float* __restrict__ t33,
               const int* __restrict__ idx33, const int* __restrict__ blist,
               const float* __restrict__ rk, const int* __restrict__ dexp,
               unsigned long long* __restrict__ acc, int nparts)
{
    grid_begin();
    // the queries that reach the leaf at hand: x, y, z, t33 and hinv, hinv^3,
    // idx33 (int bits), then entries that take nothing
    __shared__ float4 qlist[DENS_WARPS][2][32 + 3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = t.n;
    const int parts = PARTS ? nparts : 1;
    const int unit = blockIdx.x * DENS_WARPS + warp, part = unit % parts;
    const int base = unit / parts * 32;
    if (base >= n) return;
    const bool valid = base + lane < n;
    const int q = min(base + lane, n - 1);
    const float4 xq = pos[q];
    const float T = valid ? t33[q] : -1.0f;  // a padding lane takes nothing
    const float hinv = __fdiv_rn(1.0f, rk[q]);
    const float bound = prune_bound(T);
    const float4 qpos = make_float4(xq.x, xq.y, xq.z, T);
    const float4 qaux = make_float4(hinv, __fmul_rn(__fmul_rn(hinv, hinv), hinv),
                                    __int_as_float(idx33[q]), 0.0f);
    // the index rule of the 33rd key only matters in a bundle with a tied query
    const bool any_tie = __any_sync(FULL, valid && __float_as_int(qaux.z) >= 0);
    constexpr int STEP = HALVES ? 2 : 1;  // queries taken at a time
    const bool upper = HALVES && lane >= 16;
    // leaf `id` against the queries of mask M
    auto scan = [&](int id, unsigned M, auto ties) {
        const int first = id * t.leaf, cnt = leaf_count(t, id);
        const int r = HALVES ? lane & 15 : lane;
        const bool have = r < cnt;
        const int j = first + (have ? r : 0);
        const float4 c = pos[j];
        const float sc = __int_as_float((127 + FIX_BITS - dexp[j]) << 23);  // 2^(FIX_BITS - e_j)
        // the reaching queries, in lane order, padded to a multiple of the step
        const int nq = __popc(M);
        __syncwarp();  // the previous leaf's list is no longer read
        if (M >> lane & 1u) {
            const int k = __popc(M & lanemask_lt());
            qlist[warp][0][k] = qpos;
            qlist[warp][1][k] = qaux;
        }
        if (HALVES && lane == 0) qlist[warp][0][nq] = make_float4(0.f, 0.f, 0.f, -1.0f);
        __syncwarp();
        const int cj = __float_as_int(c.w);
        const f32x2 cxy = pack2(c.x, c.y);
        float sh = 0.0f, sl = 0.0f;  // sum of the scaled weights, double-float
        const float4* qp = &qlist[warp][0][upper ? 1 : 0];
#pragma unroll DENS_UNROLL
        for (int k = 0; k < nq; k += STEP) {
            const float4 Q = qp[k];
            const float4 A = qp[k + 35];
            // norm2 (nbr_search.cpp:20-25) and ker (:27-37) of (q, j), query first;
            // x and y as one packed pair (the same roundings)
            const f32x2 dxy = sub2_rn(pack2(Q.x, Q.y), cxy);
            const float dx = lo2(dxy), dy = hi2(dxy), dz = __fsub_rn(Q.z, c.z);
            const f32x2 sxy = sq2_rn(dxy);
            const float d2 = __fadd_rn(__fadd_rn(lo2(sxy), hi2(sxy)), __fmul_rn(dz, dz));
            bool member = d2 < Q.w;
            if constexpr (decltype(ties)::value) member = member || (d2 == Q.w && cj < __float_as_int(A.z));
            float w = A.y;
            w = __fmul_rn(w, __fsub_rn(1.0f, __fmul_rn(fabsf(dx), A.x)));
            w = __fmul_rn(w, __fsub_rn(1.0f, __fmul_rn(fabsf(dy), A.x)));
            w = __fmul_rn(w, __fsub_rn(1.0f, __fmul_rn(fabsf(dz), A.x)));
            // w * 2^(FIX_BITS - e_j) is exact (a power-of-two scale)
            if (member) two_sum_acc_nonneg(sh, sl, __fmul_rn(w, sc));
        }
        // one conversion per receiver and leaf: hi and lo rounded to integers
        // (lo may be negative; the sum is not)
        long long sum = __float2ll_rn(sh) + __float2ll_rn(sl);
        if constexpr (HALVES) sum += __shfl_down_sync(FULL, sum, 16);
        if (have && !upper && sum) atomicAdd(&acc[j], (unsigned long long)sum);
    };
    auto visit = [&](int id) {
        // the queries whose radius reaches the leaf's box
        const float4* bp = t.box + 2 * (size_t)id;
        const unsigned M = __ballot_sync(FULL, point_box_fast(xq, TreeBox{bp[0], bp[1]}) <= bound);
        if (!M) return;
        if (any_tie) scan(id, M, std::true_type{});
        else scan(id, M, std::false_type{});
    };

    const int* bl = blist ? blist + (size_t)(base >> 5) * (KNN_LIST + 1) : nullptr;
    const int nlist = bl ? bl[0] : -1;
    if (nlist >= 0) {
        for (int i0 = 0; i0 < nlist; i0 += 32) {
            const int cnt = min(32, nlist - i0);
            const int e = lane < cnt ? bl[1 + i0 + lane] : 0;
            for (int i = part; i < cnt; i += parts) visit(__shfl_sync(FULL, e, i));
        }
        return;
    }
    const TreeBox box = bundle_box(t, base / t.leaf, (min(base + 32, n) - 1) / t.leaf);
    float reach = bound;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) reach = fmaxf(reach, __shfl_xor_sync(FULL, reach, o));
    tree_walk(t, [&](const TreeBox& c, int, int) { return boxes_dist2_fast(box, c) <= reach; },
              // (70,000 particles in one Gaussian clump 573 -> 137 us)
              [&](int level, int id) {
                  return __any_sync(FULL, point_box_fast(xq, tree_box(t, level, id)) <= bound) != 0;
              },
              [&](int id) {
                  if (id % parts == part) visit(id);
                  return true;
              });
}

// dens_j += acc_j * 2^(e_j - FIX_BITS), one rounding to float
__global__ void k_dens_finish(const unsigned long long* __restrict__ acc,
                              const int* __restrict__ dexp, int n, float4* __restrict__ vel)
{
    grid_begin();
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const double scale = __longlong_as_double((long long)(1023 + dexp[j] - FIX_BITS) << 52);
    const float d = __double2float_rn(__dmul_rn(__ull2double_rn(acc[j]), scale));
    float4 v = vel[j];
    v.w = __fadd_rn(v.w, d);  // dens accumulates onto the incoming value, as q->dens += ... does
    vel[j] = v;
}

// Bundles up to which k_knn_t33 puts 4 and 2 warps on each: a search of 20,000 uniform
// particles takes 60 us with 1, 41 with 2, 40 with 4; 65,000 80, 72, 96; 90,000 87, 89,
// 120; in Plummer spheres 20,000 87, 61, 52; 65,000 99, 79, 98; 130,000 139, 125, 169.
// (8 warps: never better than 4.)
constexpr int KNN_SPLIT4 = 5 * 152, KNN_SPLIT2 = 18 * 152;
// and k_dens_scatter 8, 4 and 2 (4099 uniform particles 45, 29, 20 and 14 us with 1, 2,
// 4 and 8; 13,840 33, 25, 16 with 2, 4, 8 (in NFW halos 74, 61, 55); 30,000 49, 33, 25,
// 23; 50,000 35, 33, 31; 130,000 71, 66 with 1, 2, 200,000 100, 101)
constexpr int DENS_SPLIT8 = 10 * 152, DENS_SPLIT4 = 18 * 152, DENS_SPLIT2 = 32 * 152;

static int knn_blocks(int n) { return (n + KNN_WARPS * 32 - 1) / (KNN_WARPS * 32); }

void launch_knn_t33(const float4* pos, const TreeView& t, float* t33, float* rk, int* idx33,
                    int* blist, int* err, cudaStream_t s, int warps)
{
    if (t.n <= 0) return;
    auto run = [&](auto kern, int w) {
        launch(kern, (unsigned)(((long long)t.n + 32 * w - 1) / (32 * w)), 32 * w, 0, s, 
            pos, t, t33, rk, idx33, blist, err);
    };
    // Leaves of 16 run one warp per block, so that every warp that ends makes
    // room at once: 11.02 against 11.44 ms in blocks of 2 on the 256^3 step
    // (persistent warps that take bundles by ticket: 11.53).
    if (t.leaf == 16) {
        const int bundles = (t.n + 31) / 32;
        auto split = [&](auto kern, int w) {
            launch(kern, bundles, 32 * w, 0, s, pos, t, t33, rk, idx33, blist, err);
        };
        if (bundles <= KNN_SPLIT4) split(k_knn_t33<4, true, 4>, 4);
        else if (bundles <= KNN_SPLIT2) split(k_knn_t33<2, true, 2>, 2);
        else run(k_knn_t33<1, true, 1>, 1);
    } else if (warps == 4) run(k_knn_t33<4, false, 1>, 4);
    else run(k_knn_t33<2, false, 1>, 2);
    count_launches(1);
}

void launch_knn_ties(const float4* pos, const TreeView& t, const float* t33, int* idx33,
                     int all, const int* blist, const float* rk, int* dexp, unsigned long long* acc,
                     int* err, cudaStream_t s)
{
    if (t.n <= 0) return;
    launch(k_knn_ties, knn_blocks(t.n), KNN_WARPS * 32, 0, s, pos, t, t33, idx33, all, blist, rk, dexp, acc, err);
    count_launches(1);
}

void launch_dens(const float4* pos, const TreeView& t, const float* t33, const int* idx33,
                 const int* blist, const float* rk, const int* dexp, unsigned long long* acc,
                 float4* vel, cudaStream_t s)
{
    if (t.n <= 0) return;
    const int nb = (t.n + 255) / 256, bundles = (t.n + 31) / 32;
    const int parts = bundles <= DENS_SPLIT8 ? 8 : bundles <= DENS_SPLIT4 ? 4 : bundles <= DENS_SPLIT2 ? 2 : 1;
    const unsigned nw = (unsigned)(((long long)bundles * parts + DENS_WARPS - 1) / DENS_WARPS);
    auto kern = parts > 1 ? (t.leaf <= 16 ? k_dens_scatter<true, true> : k_dens_scatter<false, true>)
                          : (t.leaf <= 16 ? k_dens_scatter<true, false> : k_dens_scatter<false, false>);
    launch(kern, nw, DENS_WARPS * 32, 0, s, pos, t, t33, idx33, blist, rk, dexp, acc, parts);
    launch(k_dens_finish, nb, 256, 0, s, acc, dexp, t.n, vel);
    count_launches(2);
}

// every kernel of the search and density with leaves of 16 particles
bool load_search_kernels()
{
    return kernel_loaded(k_knn_t33<4, true, 4>) && kernel_loaded(k_knn_t33<2, true, 2>) &&
           kernel_loaded(k_knn_t33<1, true, 1>) && kernel_loaded(k_knn_ties) &&
           kernel_loaded(k_dens_scatter<true, true>) && kernel_loaded(k_dens_scatter<true, false>) &&
           kernel_loaded(k_dens_finish);
}

}  // namespace asg
