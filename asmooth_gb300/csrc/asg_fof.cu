// asg_fof.cu -- friends-of-friends groups and SO-halo marking.
//
// FOF (group_fof / link_friends_recursive1, fof.cpp:34-102; remove_small_groups,
// fof.cpp:104-166): two particles are friends when norm2 <= ll*ll in float
// (the reference's predicate, fof.cpp:85-91); groups are the connected
// components.  GPU form: a warp-bundle range search over the box tree links
// every friend pair (i < j) in a lock-free union-find whose parent pointers
// only ever decrease, so each component's root is its smallest sorted position
// whatever the order of the unions.  Labels 1..ngroup are then assigned in
// order of each group's smallest INPUT index by a scan over input indices
// (membership is bit-exact; the reference numbers groups in kd-tree order).
//
// SO halos (mark_halo_particles, nbr_search.cpp:140-165, driven by the loop at
// clumping_tree_main.cpp:474-485): a halo's warps walk the tree with its sphere;
// lanes test bucket particles with d2 < r*r and set igrp = -1.
#include <climits>

#include "asg_common.cuh"
#include "asg_internal.h"
#include "asg_tree.cuh"

namespace asg {

constexpr int FOF_WARPS = 4;
constexpr unsigned FM = 0xffffffffu;
constexpr int UF_LIMIT = 1 << 20;
constexpr int FOF_MANY = 8;  // leaves of a group

__device__ __forceinline__ int uf_find(int* P, int x)
{
    for (;;) {
        const int p = __ldcg(P + x);
        if (p == x) return x;
        const int g = __ldcg(P + p);
        if (g == p) return p;
        // path halving: g is an ancestor of x.  A plain store could put it over the root
        // that k_fof_root wrote meanwhile
        atomicCAS(P + x, p, g);
        x = g;
    }
}

// links the components of a and b; their common root, or -1 past the retry limit
__device__ __forceinline__ int uf_union(int* P, int a, int b)
{
    for (int it = 0; it < UF_LIMIT; ++it) {
        int ra = uf_find(P, a), rb = uf_find(P, b);
        if (ra == rb) return ra;
        if (ra < rb) { const int t = ra; ra = rb; rb = t; }
        // link the larger root under the smaller one
        if (atomicCAS(P + ra, ra, rb) == ra) return rb;
        a = ra;
        b = rb;
    }
    return -1;
}

// A friend pair inside one component needs no link, and in a halo nearly every
// pair is one: a leaf is staged with each particle's root, a lane keeps its
// query's root, and a pair is tested only while the two differ (being in one
// component is never undone, so an old root is good evidence).  A leaf whose
// particles and the bundle's queries all share one root is passed over.  Before,
// every friend pair searched both roots: 3.02 -> 1.14 ms on a 128^3 NFW cube (2.5 M
// particles) at a fifth of the mean separation, 0.80 with the leaves of a group in a
// mask; bound by the L2 round trips of the root searches.
__global__ void __launch_bounds__(FOF_WARPS * 32)
k_fof_link(const float4* __restrict__ pos, const __grid_constant__ TreeView t, float ll2, int* P, int* err)
{
    grid_begin();
    __shared__ float4 cand[FOF_WARPS][LEAF_MAX];  // x, y, z, root
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = t.n;
    const int base = (blockIdx.x * FOF_WARPS + warp) * 32;
    if (base >= n) return;
    const int q = min(base + lane, n - 1);
    const bool active = base + lane < n;
    const float4 xq = pos[q];
    const float bound = prune_bound(ll2);
    bool bad = false;
    int rq = q;  // a root, now or earlier, of the query's component
    const TreeBox box = bundle_box(t, base / t.leaf, (min(base + 32, n) - 1) / t.leaf);
    auto pass = [&](const TreeBox& c, int level, int id) {
        // only partners with a larger sorted position are linked from q
        const long long last = (((long long)id + 1) << (5 * level)) * t.leaf - 1;
        return last > base && boxes_dist2_fast(box, c) <= bound;
    };
    auto link = [&](int id) {
        const int first = id * t.leaf, cnt = leaf_count(t, id);
        if (!__any_sync(FM, active && first + cnt - 1 > q &&
                                point_box_fast(xq, tree_box(t, 0, id)) <= bound))
            return;
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        int rc = -1;
        if (lane < cnt) {
            p = pos[first + lane];
            rc = uf_find(P, first + lane);
        }
        rq = uf_find(P, rq);
        const int r0 = __shfl_sync(FM, rq, 0);
        if (__all_sync(FM, rq == r0 && (rc < 0 || rc == r0))) return;
        __syncwarp();
        if (lane < cnt) cand[warp][lane] = make_float4(p.x, p.y, p.z, __int_as_float(rc));
        __syncwarp();
        for (int j = 0; j < cnt; ++j) {
            const int s = first + j;
            const float4 c = cand[warp][j];
            if (active && s > q && __float_as_int(c.w) != rq &&
                norm2_rn(xq.x, xq.y, xq.z, c.x, c.y, c.z) <= ll2) {
                const int r = uf_union(P, rq, __float_as_int(c.w));
                bad |= r < 0;
                rq = r < 0 ? rq : r;
            }
        }
    };
    // A bundle's box that reaches much of a group may hold far more than its queries do (around
    // a clump, or where the curve leaves the set and comes back elsewhere), so such a group
    // is tested for each query: at 8 of 32 leaves 3,000,000 particles in a sheet across the
    // box 1000 -> 623 us, 300,000 along a line 959 -> 284, 262,144 in one Gaussian clump
    // 348 -> 134 (at 16 leaves 627, 290, 148, at 32 1000, 959, 179).  The same test of every
    // group or node, or once some leaves were in vain, costs other sets 1 to 4%.
    tree_walk_groups(t, pass, [](int, int) { return true; }, [&](int g) {
        unsigned m = group_leaves(t, g, pass);
        if (__popc(m) >= FOF_MANY && t.nlev > 1 &&
            !__any_sync(FM, active && point_box_fast(xq, tree_box(t, 1, g)) <= bound))
            return true;
        for (; m; m &= m - 1) link(g * 32 + __ffs(m) - 1);
        return true;
    });
    if (bad) atomicOr(err, ERR_UF);
}

void launch_fof_link(const float4* pos, const TreeView& t, float ll, int* parent, int* err,
                     cudaStream_t s)
{
    if (t.n <= 0) return;
    const float ll2 = ll * ll;  // host float multiply: fl(ll*ll) as in fof.cpp:86
    launch(k_fof_link, (t.n + FOF_WARPS * 32 - 1) / (FOF_WARPS * 32), FOF_WARPS * 32, 0, s, 
        pos, t, ll2, parent, err);
    count_launches(1);
}

// P[i] <- root (while others still search: any ancestor is right), and
// minin[root] <- min input index: one atomic per root and warp, as the members of
// a group lie close together; then mark[minin[root]] = 1
__global__ void k_fof_root(const float4* __restrict__ pos, int n, int* P, int* minin)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = i < n ? uf_find(P, i) : -1;
    const int w = i < n ? __float_as_int(pos[i].w) : 0;
    if (i < n) P[i] = r;
    const unsigned peers = __match_any_sync(FM, r);
    const int m = __reduce_min_sync(peers, w);
    if (i < n && (peers & lanemask_lt()) == 0u) atomicMin(minin + r, m);
}
__global__ void k_fof_mark(int n, const int* P, const int* minin, int* mark)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (P[i] == i) mark[minin[i]] = 1;
}

void launch_fof_finish(const float4* pos, int n, int* parent, int* minin, int* mark,
                       cudaStream_t s)
{
    if (n <= 0) return;
    const int nb = (n + 255) / 256;
    launch(k_fof_root, nb, 256, 0, s, pos, n, parent, minin);
    launch(k_fof_mark, nb, 256, 0, s, n, parent, minin, mark);
    count_launches(2);
}

__global__ void k_fof_label(int n, const int* __restrict__ P, const int* __restrict__ minin,
                            const uint32_t* __restrict__ scan, int* __restrict__ igrp)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    igrp[i] = (int)scan[minin[P[i]]] + 1;
}

void launch_fof_label(int n, const int* parent, const int* minin, const uint32_t* scan,
                      int* igrp_sorted, cudaStream_t s)
{
    if (n <= 0) return;
    launch(k_fof_label, (n + 255) / 256, 256, 0, s, n, parent, minin, scan, igrp_sorted);
    count_launches(1);
}

// remove_small_groups: count members per label, keep labels with >= threshold,
// relabel kept groups 1..nhalo in label order, all others 0
// Members of a group lie close together in the sorted order, so a warp adds one
// count per label it holds: one atomic per member made the largest groups'
// counters a queue (345 us on a 128^3 cube).
__global__ void k_count_labels(const int* __restrict__ igrp, int n, uint32_t* counts)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int g = i < n ? igrp[i] : -1;
    const unsigned peers = __match_any_sync(FM, g);
    if (i < n && (peers & lanemask_lt()) == 0u) atomicAdd(counts + g, (uint32_t)__popc(peers));
}
void launch_count_labels(const int* igrp, int n, uint32_t* counts, cudaStream_t s)
{
    if (n <= 0) return;
    launch(k_count_labels, (n + 255) / 256, 256, 0, s, igrp, n, counts);
    count_launches(1);
}
__global__ void k_keep_mask(uint32_t* counts, int ngrp, int threshold)
{
    grid_begin();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g > ngrp) return;
    counts[g] = (g > 0 && counts[g] >= (uint32_t)threshold) ? 1u : 0u;
}
void launch_keep_mask(uint32_t* counts, int ngrp, int threshold, cudaStream_t s)
{
    launch(k_keep_mask, (ngrp + 1 + 255) / 256, 256, 0, s, counts, ngrp, threshold);
    count_launches(1);
}
__global__ void k_relabel(int* igrp, int n, const uint32_t* __restrict__ scan,
                          const uint32_t* __restrict__ keep)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int g = igrp[i];
    igrp[i] = keep[g] ? (int)scan[g] + 1 : 0;
}
void launch_relabel(int* igrp, int n, const uint32_t* scan, const uint32_t* keep, cudaStream_t s)
{
    if (n <= 0) return;
    launch(k_relabel, (n + 255) / 256, 256, 0, s, igrp, n, scan, keep);
    count_launches(1);
}

// ---------------------------------------------------------------------------
// SO halos
// ---------------------------------------------------------------------------
// A halo's warps walk the upper levels together and take the groups of 32 leaves in
// turn; within a group they load 32 particles at a time, all loads independent. A
// leaf at a time on one warp was a chain of dependent loads, as long as the largest
// halo: 299 us for 102 halos of a 377,000-particle set, so 20.
constexpr int MH_WARPS = 8;
// warps per halo: 8 while few halos leave the chip idle (64 halos 18 us, 53 with one
// warp each), else 1, a walk of the upper levels costing more than most halos' leaves:
// 4864 halos 54 against 62 us, 20,000 halos 173 against 131.
constexpr int MH_MANY = 32 * 152;
static int mark_split(int nh) { return nh <= MH_MANY ? MH_WARPS : 1; }

__global__ void __launch_bounds__(MH_WARPS * 32)
k_mark_halos(const float4* __restrict__ pos, const __grid_constant__ TreeView t, const float* __restrict__ halos, int nh,
             int split, float left, float right, int* __restrict__ igrp, long long* __restrict__ counts,
             double* __restrict__ mass8)
{
    grid_begin();
    __shared__ int found[MH_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = (blockIdx.x * MH_WARPS + warp) / split, share = warp % split;
    int cnt = 0;
    bool inside = false;
    if (h < nh) {
        const float cx = halos[5 * (size_t)h], cy = halos[5 * (size_t)h + 1],
                    cz = halos[5 * (size_t)h + 2], r = halos[5 * (size_t)h + 3];
        inside = left < cx && cx < right && left < cy && cy < right && left < cz && cz < right;
        const float r2 = __fmul_rn(r, r);
        const float bound = prune_bound(r2);
        const float4 c4 = make_float4(cx, cy, cz, 0.f);
        auto pass = [&](const TreeBox& c, int, int) { return point_box_fast(c4, c) <= bound; };
        const int per = t.leaf <= 16 ? 2 : 1, width = 32 / per;
        int turn = 0;
        if (inside)
            tree_walk_groups(t, pass, [](int, int) { return true; }, [&](int g) {
                if (turn++ % split != share) return true;
                const unsigned m = group_leaves(t, g, pass);
                // a warp's load covers `per` leaves; four loads in flight
                for (int l0 = 0; l0 < 32; l0 += 4 * per) {
                    if (!(m >> l0 & (unsigned)((1ull << 4 * per) - 1))) continue;
                    float4 p[4];
                    int at[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int l = l0 + per * u + lane / width;
                        const int i = (g * 32 + l) * t.leaf + lane % width;
                        const bool on = l < 32 && (m >> l & 1u) && lane % width < t.leaf && i < t.n;
                        at[u] = on ? i : -1;
                        p[u] = on ? pos[i] : make_float4(INFINITY, INFINITY, INFINITY, 0.f);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        // norm2(x, particle[i].x) with x the halo centre (nbr_search.cpp:149)
                        const bool hit = at[u] >= 0 && norm2_rn(cx, cy, cz, p[u].x, p[u].y, p[u].z) < r2;
                        if (hit) igrp[at[u]] = -1;
                        cnt += hit ? 1 : 0;
                    }
                }
                return true;
            });
    }
    cnt = (int)__reduce_add_sync(FM, (unsigned)cnt);
    if (lane == 0) found[warp] = cnt;
    __syncthreads();
    if (h < nh && share == 0 && lane == 0) {
        long long sum = 0;
        for (int w = 0; w < split; ++w) sum += found[warp + w];
        counts[h] = sum;
        mass8[h] = inside ? (double)__fdiv_rn(halos[5 * (size_t)h + 4], 8.0f) : 0.0;  // h[i].mass/8.0f (:483)
    }
}

void launch_mark_halos(const float4* pos, const TreeView& t, const float* halos, int nh,
                       float left, float right, int* igrp, long long* counts, double* mass8,
                       cudaStream_t s)
{
    if (nh <= 0 || t.n <= 0) return;
    const int split = mark_split(nh);
    launch(k_mark_halos, (unsigned)(((long long)nh * split + MH_WARPS - 1) / MH_WARPS), MH_WARPS * 32, 0, s, 
        pos, t, halos, nh, split, left, right, igrp, counts, mass8);
    count_launches(1);
}

}  // namespace asg
