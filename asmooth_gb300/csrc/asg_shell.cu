// asg_shell.cu -- the periodic buffer shell of a single-cube run, built on the
// device: what exchange_buffer (exchange_buffer.cpp:13-168) does when one rank
// owns the whole box (every direction a self-exchange), followed by the
// filter of remove_extra_particles (clumping_tree_main.cpp:550-576).
//
// Same particles, same float positions as the reference:
//   bin per axis = (x >= bf*L) + (x > (1-bf)*L)          (exchange_buffer.cpp:6-11)
//   a particle of bin b (b != 13) is copied once per direction d != 13 with
//   d_a == 1 or d_a == b_a on every axis, shifted x -= (d_a - 1)*L   (:120-144)
//   kept when -bf*L < x < L + bf*L on every axis          (clumping_tree_main.cpp:556-566)
// Order of the result: the interior particles as given, then the copies
// grouped by (source bin, direction) in the reference's loop order, each group
// in input order.  (The reference orders a bin by an in-place swap sort, so its
// order within a group differs; no output depends on it except index
// tie-breaks.)
#include "asg_common.cuh"
#include "asg_internal.h"
#include "asg_keys.cuh"

namespace asg {

__global__ void k_shell_bins(const float4* __restrict__ rec, int n, float lt, float rt,
                             uint32_t* __restrict__ keys)
{
    grid_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = rec[2 * (size_t)i];
    const int bx = (p.x >= lt) + (p.x > rt);
    const int by = (p.y >= lt) + (p.y > rt);
    const int bz = (p.z >= lt) + (p.z > rt);
    keys[i] = (uint32_t)(bx + 3 * by + 9 * bz);
}

// (none when the sort gave up: its output is not all written then)
__global__ void k_shell_bounds(const uint32_t* __restrict__ keys, int n, uint32_t* __restrict__ start,
                               uint32_t* __restrict__ end, const int* __restrict__ err)
{
    grid_begin();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n || (*err & ERR_SORT)) return;
    const uint32_t b = keys[m];
    if (m == 0 || keys[m - 1] != b) start[b] = (uint32_t)m;
    if (m == n - 1 || keys[m + 1] != b) end[b] = (uint32_t)m + 1;
}

// interior particles first, unchanged
__global__ void k_shell_interior(const float4* __restrict__ rec, const float* __restrict__ rk, int n,
                                 float4* __restrict__ arec, float* __restrict__ ark)
{
    grid_begin();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2LL * n) return;
    arec[i] = rec[i];
    if (rk && i < n) ark[i] = rk[i];
}

// every copy of the bin-sorted particle m, at its group's offset + rank in the bin
__global__ void k_shell_emit(const float4* __restrict__ rec, const float* __restrict__ rk,
                             const uint32_t* __restrict__ keys, const int* __restrict__ order,
                             const uint32_t* __restrict__ start, int n, ShellPlan plan, float L,
                             float4* __restrict__ arec, float* __restrict__ ark)
{
    grid_begin();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
    const int b = (int)keys[m];
    if (b == 13) return;
    const int i = order[m];
    const uint32_t r = (uint32_t)m - start[b];
    const float4 p = rec[2 * (size_t)i];
    const float4 v = rec[2 * (size_t)i + 1];
    const float h = rk ? rk[i] : 0.0f;
    for (int d = 0; d < 27; ++d) {
        const int base = plan.base[b][d];
        if (base < 0) continue;
        const size_t dst = (size_t)base + r;
        const float sx = __fmul_rn((float)(d % 3 - 1), L);
        const float sy = __fmul_rn((float)((d / 3) % 3 - 1), L);
        const float sz = __fmul_rn((float)(d / 9 - 1), L);
        arec[2 * dst] = make_float4(__fsub_rn(p.x, sx), __fsub_rn(p.y, sy), __fsub_rn(p.z, sz), p.w);
        arec[2 * dst + 1] = v;
        if (rk) ark[dst] = h;
    }
}

__global__ void k_shell_keep(const float4* __restrict__ arec, int n, float lo, float hi,
                             uint32_t* __restrict__ flags)
{
    grid_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float4 p = arec[2 * (size_t)k];
    flags[k] = (lo < p.x && p.x < hi && lo < p.y && p.y < hi && lo < p.z && p.z < hi) ? 1u : 0u;
}

// stable compaction, with the keys of the kept particles
__global__ void k_shell_compact(const float4* __restrict__ arec, const float* __restrict__ ark, int n,
                                const uint32_t* __restrict__ scan, float4* __restrict__ rec,
                                float* __restrict__ rk, KeyGrid grid, uint64_t* __restrict__ keys)
{
    grid_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || scan[k + 1] == scan[k]) return;
    const uint32_t o = scan[k];
    const float4 p = arec[2 * (size_t)k];
    rec[2 * (size_t)o] = p;
    rec[2 * (size_t)o + 1] = arec[2 * (size_t)k + 1];
    if (rk) rk[o] = ark[k];
    keys[o] = space_key(grid, p.x, p.y, p.z);
}

void launch_shell_bins(const float4* rec, int n, float lt, float rt, uint32_t* keys0, int* vals0,
                       uint32_t* keys1, int* vals1, void* sort_tmp, uint32_t* start, uint32_t* end,
                       const uint32_t** keys, const int** order, int* err, cudaStream_t s)
{
    cudaMemsetAsync(start, 0, 27 * sizeof(uint32_t), s);
    cudaMemsetAsync(end, 0, 27 * sizeof(uint32_t), s);
    launch(k_shell_bins, (n + 255) / 256, 256, 0, s, rec, n, lt, rt, keys0);
    const int cur = radix_sort32(keys0, vals0, keys1, vals1, n, 5, true, sort_tmp, err, s);
    *keys = cur ? keys1 : keys0;
    *order = cur ? vals1 : vals0;
    launch(k_shell_bounds, (n + 255) / 256, 256, 0, s, *keys, n, start, end, err);
    count_launches(2);
}

void launch_shell_emit(const float4* rec, const float* rk, const uint32_t* keys, const int* order,
                       const uint32_t* start, int n, const ShellPlan& plan, float L, float4* arec,
                       float* ark, cudaStream_t s)
{
    launch(k_shell_interior, (unsigned)((2LL * n + 255) / 256), 256, 0, s, rec, rk, n, arec, ark);
    launch(k_shell_emit, (n + 255) / 256, 256, 0, s, rec, rk, keys, order, start, n, plan, L, arec, ark);
    count_launches(2);
}

void launch_shell_filter(const float4* arec, const float* ark, int n_all, float lo, float hi,
                         uint32_t* flags, void* scan_tmp, float4* rec, float* rk, const KeyGrid& grid,
                         uint64_t* out_keys, cudaStream_t s)
{
    cudaMemsetAsync(flags + n_all, 0, sizeof(uint32_t), s);
    launch(k_shell_keep, (n_all + 255) / 256, 256, 0, s, arec, n_all, lo, hi, flags);
    exclusive_scan_u32(flags, (size_t)n_all + 1, scan_tmp, s);
    launch(k_shell_compact, (n_all + 255) / 256, 256, 0, s, arec, ark, n_all, flags, rec, rk, grid, out_keys);
    count_launches(2);
}

}  // namespace asg
