// asg_tree.cuh -- traversal of the blocked box tree (TreeView, asg_internal.h).
//
// Level 0 holds the boxes of `leaf` consecutive particles of the space-filling
// curve, every level above the boxes of 32 consecutive boxes below, up to a top
// level of at most 32 boxes.  The shape is implied by n and leaf, so a node is
// its number and its children are 32 * number + lane: a warp opens a node with
// one coalesced load, a child per lane.
//
// Why 32 children and a box test against the whole bundle: a binary radix tree
// walked with one test per query and child took about 115 dependent visits of
// some 60 instructions per 32-query bundle on the 256^3 cube; here a bundle
// opens about 17 nodes of some 40 instructions, and only the nodes and leaves whose box
// reaches the bundle's largest radius (about 110 leaves, of which 49 hold work) get a
// test per query.
#pragma once

#include "asg_common.cuh"
#include "asg_internal.h"

namespace asg {

// a box of the tree: two float4, lo.x hi.x lo.y hi.y | lo.z hi.z - -
struct TreeBox {
    float4 a, b;
};
__device__ __forceinline__ TreeBox tree_box(const TreeView& t, int level, int id)
{
    const float4* p = t.box + 2 * ((size_t)t.off[level] + (size_t)id);
    return {p[0], p[1]};
}

// Pruning-only squared distance between two boxes, compared against
// prune_bound: per axis fl(lo - hi') is at most |fl(p - q)| for every p of one
// box and q of the other (rounding is monotone), so point_box_fast's bound
// holds for every pair of points.
__device__ __forceinline__ float boxes_dist2_fast(const TreeBox& q, const TreeBox& c)
{
    const float dx = max3f(c.a.x - q.a.y, q.a.x - c.a.y, 0.0f);
    const float dy = max3f(c.a.z - q.a.w, q.a.z - c.a.w, 0.0f);
    const float dz = max3f(c.b.x - q.b.y, q.b.x - c.b.y, 0.0f);
    return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}
// Squared distance from a point to an AABB in the cheaper FMA form, for
// pruning only: compare it against prune_bound(t), never against t itself.
// Per axis d = fl(lo - q) (or fl(q - hi)) is at most |fl(p - q)| for every
// point p of the box (rounding is monotone); the FMA sum is at most
// (dx^2 + dy^2 + dz^2)(1 + u)^3 and norm2_rn(q, p) is at least
// (px^2 + py^2 + pz^2)(1 - u)^3 (u = 2^-24), so the result is at most
// norm2_rn(q, p)(1 + 6.1u) for every p in the box.
// The point's coordinates are given twice each: lo - q and hi - q of an axis are one
// packed subtraction, which is why a box holds its bounds in pairs (the kNN of the
// 256^3 step 11.07 -> 10.99 ms, dens 6.08 -> 6.04).
__device__ __forceinline__ float point_box_fast(f32x2 qx, f32x2 qy, f32x2 qz, const TreeBox& c)
{
    const f32x2 sx = sub2_rn(pack2(c.a.x, c.a.y), qx);
    const f32x2 sy = sub2_rn(pack2(c.a.z, c.a.w), qy);
    const f32x2 sz = sub2_rn(pack2(c.b.x, c.b.y), qz);
    const float dx = max3f(lo2(sx), -hi2(sx), 0.0f);
    const float dy = max3f(lo2(sy), -hi2(sy), 0.0f);
    const float dz = max3f(lo2(sz), -hi2(sz), 0.0f);
    return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}
__device__ __forceinline__ float point_box_fast(float4 q, const TreeBox& c)
{
    return point_box_fast(pack2(q.x, q.x), pack2(q.y, q.y), pack2(q.z, q.z), c);
}
__device__ __forceinline__ void box_grow(TreeBox& q, const TreeBox& c)
{
    q.a = make_float4(fminf(q.a.x, c.a.x), fmaxf(q.a.y, c.a.y), fminf(q.a.z, c.a.z), fmaxf(q.a.w, c.a.w));
    q.b = make_float4(fminf(q.b.x, c.b.x), fmaxf(q.b.y, c.b.y), 0.0f, 0.0f);
}
// the box of the leaves that hold particles [base, base + 31] (all of a bundle)
__device__ __forceinline__ TreeBox bundle_box(const TreeView& t, int leaf0, int leaf1)
{
    TreeBox q = tree_box(t, 0, leaf0);
    for (int i = leaf0 + 1; i <= leaf1; ++i) box_grow(q, tree_box(t, 0, i));
    return q;
}
__device__ __forceinline__ int leaf_count(const TreeView& t, int id)
{
    return min(t.leaf, t.n - id * t.leaf);
}

// Visits, in a fixed order, every group of 32 leaves (32 g ... 32 g + 31) all of whose
// ancestors pass: pass(box, level, id) is asked by each lane for its own child, then
// reach(level, id) by the whole warp for a child that passed, group(g) is called by the whole
// warp (and may end the walk by returning false).
// Lane l keeps the pending children of the node open at level l.
template <class Pass, class Reach, class Group>
__device__ __forceinline__ void tree_walk_groups(const TreeView& t, Pass pass, Reach reach, Group group)
{
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, top = t.nlev - 1;
    if (top == 0) {
        group(0);
        return;
    }
    int L = top, g = 0;
    unsigned pending = 0;
    auto open = [&]() {
        const unsigned id = (unsigned)g * 32u + (unsigned)lane;
        bool ok = id < (unsigned)t.cnt[L];
        if (ok) ok = pass(tree_box(t, L, (int)id), L, (int)id);
        const unsigned m = __ballot_sync(ALL, ok);
        if (lane == L) pending = m;
    };
    open();
    for (;;) {
        const unsigned m = __shfl_sync(ALL, pending, L);
        if (!m) {
            if (L == top) return;
            ++L;
            g >>= 5;
            continue;
        }
        if (lane == L) pending = m & (m - 1);
        const int id = g * 32 + __ffs(m) - 1;
        if (!reach(L, id)) continue;
        if (L == 1) {
            if (!group(id)) return;
        } else {
            --L;
            g = id;
            open();
        }
    }
}

// the leaves of group g that pass, as a mask
template <class Pass>
__device__ __forceinline__ unsigned group_leaves(const TreeView& t, int g, Pass pass)
{
    const unsigned id = (unsigned)g * 32u + (threadIdx.x & 31);
    bool ok = id < (unsigned)t.cnt[0];
    if (ok) ok = pass(tree_box(t, 0, (int)id), 0, (int)id);
    return __ballot_sync(0xffffffffu, ok);
}

// Visits, in a fixed order, every leaf all of whose ancestors pass and are reached;
// leaf(id) is called by the whole warp and may end the walk by returning false.
template <class Pass, class Reach, class Leaf>
__device__ __forceinline__ void tree_walk(const TreeView& t, Pass pass, Reach reach, Leaf leaf)
{
    tree_walk_groups(t, pass, reach, [&](int g) {
        for (unsigned m = group_leaves(t, g, pass); m; m &= m - 1)
            if (!leaf(g * 32 + __ffs(m) - 1)) return false;
        return true;
    });
}

}  // namespace asg
