// asg_output.cu -- the outputs of the path: the FOF halo catalogue
// (write_fof_halos, fof.cpp:169-219) computed on the device, and the byte
// formats of the mesh and catalogue files (write_mesh, coarse_mesh.cpp:128-143;
// write_mesh_separate, coarse_mesh.cpp:147-208; write_fof_halos).
//
// Catalogue: per label 1..nhalo, the float sums of x and v over the members in
// the caller's array order (one lane per component adds them sequentially, as
// the reference's loop does, so the sums are the reference's bits), divided by
// the member count; halos whose centre is strictly inside (0, boxsize)^3 are
// kept in label order.  The members are grouped by a stable radix sort of the
// labels laid out in the caller's array order.
#include <cstdio>
#include <string>

#include "../../include/asmooth_gb300.h"
#include "asg_common.cuh"
#include "asg_internal.h"

namespace asg {

constexpr int REC_WORDS = 7;  // struct FofHalo (fof.cpp:22-25): float x[3], v[3]; int nfof

static size_t al256(size_t v) { return (v + 255) & ~size_t(255); }

struct CatLayout {
    size_t keys0, keys1, vals0, vals1, sort_tmp, start, end, rec, flags, scan_tmp, total;
};

static CatLayout cat_layout(int n, int nhalo)
{
    CatLayout L{};
    const size_t N = (size_t)n, H = (size_t)nhalo + 1;
    size_t o = 0;
    auto take = [&](size_t b) {
        const size_t at = o;
        o = al256(o + b);
        return at;
    };
    L.keys0 = take(4 * N);
    L.keys1 = take(4 * N);
    L.vals0 = take(4 * N);
    L.vals1 = take(4 * N);
    L.sort_tmp = take(radix_sort_temp_bytes(n));
    L.start = take(4 * H);
    L.end = take(4 * H);
    L.rec = take(4 * REC_WORDS * H);
    L.flags = take(4 * H);
    L.scan_tmp = take(scan_temp_bytes(H));
    L.total = o;
    return L;
}

size_t fof_catalogue_bytes(int n, int nhalo) { return cat_layout(n, nhalo).total; }

// the label of the particle at position i of the caller's array, and its place j
// in pos/vel (label 0: in no halo).  igrp: sorted arrays, pos.w the position;
// null: staged records, the label in pos.w
__global__ void k_cat_keys(const float4* __restrict__ pos, const int* __restrict__ igrp, int n,
                           int nhalo, uint32_t* __restrict__ keys, int* __restrict__ vals)
{
    grid_begin();
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int w = __float_as_int(pos[igrp ? (size_t)j : 2 * (size_t)j].w);
    const int lab = igrp ? igrp[j] : w, i = igrp ? w : j;
    keys[i] = (lab >= 1 && lab <= nhalo) ? (uint32_t)lab : 0u;
    vals[i] = j;
}

// (no members when the sort gave up)
__global__ void k_cat_bounds(const uint32_t* __restrict__ keys, int n, uint32_t* __restrict__ start,
                             uint32_t* __restrict__ end, const int* __restrict__ err)
{
    grid_begin();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n || (*err & ERR_SORT)) return;
    const uint32_t lab = keys[m];
    if (lab == 0) return;
    if (m == 0 || keys[m - 1] != lab) start[lab] = (uint32_t)m;
    if (m == n - 1 || keys[m + 1] != lab) end[lab] = (uint32_t)m + 1;
}

// The sums of a halo are six chains of dependent adds (four cycles each), so
// the work around them is kept off the chains: T threads (a warp, or a block
// for halos of more than CAT_BIG members) gather the next T members while
// lanes 0-5 of the first warp add the previous T, one component each, from
// shared memory.  On a 128^3 cube's catalogue (987 halos, the largest of 20,277
// members) 7.5 -> 0.15 ms against one thread per halo, gathering as it added.
// The blocks of large halos come first: they take longest.
constexpr int CAT_THREADS = 256, CAT_BIG = 512;

template <int T>
struct CatRows {
    float c[2][6][T + 4];  // [buffer][component][member of the chunk]
};

template <int T, class Sync>
__device__ __forceinline__ float cat_sum(CatRows<T>& R, int tid, uint32_t s, uint32_t e,
                                         const float4* __restrict__ pos,
                                         const float4* __restrict__ vel, int stride,
                                         const int* __restrict__ order, Sync sync)
{
    float sum = 0.f;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), v = p;
    // the member numbers are read one chunk before the members
    int j = s + tid < e ? order[s + tid] : 0;
    auto fetch = [&](uint32_t m) {
        if (m + tid < e) {
            p = pos[(size_t)j * stride];
            v = vel[(size_t)j * stride];
        }
        if (m + T + tid < e) j = order[m + T + tid];
    };
    fetch(s);
    int b = 0;
    for (uint32_t m = s; m < e; m += T, b ^= 1) {
        R.c[b][0][tid] = p.x;
        R.c[b][1][tid] = p.y;
        R.c[b][2][tid] = p.z;
        R.c[b][3][tid] = v.x;
        R.c[b][4][tid] = v.y;
        R.c[b][5][tid] = v.z;
        sync();  // the other buffer's chunk has been added by now, too
        fetch(m + T);
        if (tid < 6) {
            const float* row = R.c[b][tid];
            const int cnt = (int)min((uint32_t)T, e - m);
            int i = 0;
#pragma unroll 8
            for (; i + 4 <= cnt; i += 4) {
                const float4 x = *reinterpret_cast<const float4*>(row + i);
                sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, x.x), x.y), x.z), x.w);
            }
            for (; i < cnt; ++i) sum = __fadd_rn(sum, row[i]);
        }
    }
    sync();  // the rows may be used again
    return sum;
}

// lanes 0-5: the record's component sums divided by the member count
__device__ __forceinline__ void cat_record(int lane, float sum, uint32_t members, float boxsize,
                                           float* __restrict__ o, uint32_t* __restrict__ flag)
{
    const float r = __fdiv_rn(sum, __int2float_rn((int)members));
    if (lane < 6) o[lane] = r;
    if (lane == 6) o[6] = __int_as_float((int)members);
    const bool in = lane >= 3 || (0.0f < r && r < boxsize);
    const bool keep = __all_sync(0xffffffffu, in);
    if (lane == 0) *flag = keep ? 1u : 0u;
}

__global__ void __launch_bounds__(CAT_THREADS)
k_cat_sums(const float4* __restrict__ pos, const float4* __restrict__ vel, int stride,
           const int* __restrict__ order, const uint32_t* __restrict__ start,
           const uint32_t* __restrict__ end, int nhalo, int nbig, float boxsize,
           float* __restrict__ rec, uint32_t* __restrict__ flags)
{
    grid_begin();
    constexpr int W = CAT_THREADS / 32;
    __shared__ __align__(16) union Rows {
        CatRows<CAT_THREADS> block;
        CatRows<32> warp[W];
    } R;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if ((int)blockIdx.x < nbig) {  // the large halos of every nbig-th label
        for (int h = blockIdx.x; h < nhalo; h += nbig) {
            const uint32_t s = start[h + 1], e = end[h + 1];
            if (e - s <= CAT_BIG) continue;
            const float sum = cat_sum<CAT_THREADS>(R.block, tid, s, e, pos, vel, stride, order,
                                                   [] { __syncthreads(); });
            if (w == 0) cat_record(lane, sum, e - s, boxsize, rec + (size_t)REC_WORDS * h, flags + h);
        }
        return;
    }
    const int h = ((int)blockIdx.x - nbig) * W + w;  // a warp per halo
    const uint32_t s = h < nhalo ? start[h + 1] : 0u, e = h < nhalo ? end[h + 1] : 0u;
    if (h >= nhalo || e - s > CAT_BIG) return;
    const float sum = cat_sum<32>(R.warp[w], lane, s, e, pos, vel, stride, order, [] { __syncwarp(); });
    cat_record(lane, sum, e - s, boxsize, rec + (size_t)REC_WORDS * h, flags + h);
}

// scan: exclusive scan of the keep flags over nhalo + 1 entries (the last flag
// is 0), so halo h is kept when scan[h + 1] > scan[h] and scan[nhalo] is the count
__global__ void k_cat_compact(const float* __restrict__ rec, const uint32_t* __restrict__ scan,
                              int nhalo, float* __restrict__ out, uint32_t* __restrict__ nlocal)
{
    grid_begin();
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h == 0) *nlocal = scan[nhalo];
    if (h >= nhalo || scan[h + 1] == scan[h]) return;
    const float* a = rec + (size_t)REC_WORDS * h;
    float* b = out + (size_t)REC_WORDS * scan[h];
#pragma unroll
    for (int k = 0; k < REC_WORDS; ++k) b[k] = a[k];
}

void launch_fof_catalogue(const float4* pos, const float4* vel, const int* igrp, int n,
                          int nhalo, float boxsize, void* scratch, float* out, uint32_t* nlocal,
                          int* err, cudaStream_t s)
{
    const CatLayout L = cat_layout(n, nhalo);
    unsigned char* b = static_cast<unsigned char*>(scratch);
    auto I = [&](size_t o) { return reinterpret_cast<int*>(b + o); };
    auto U = [&](size_t o) { return reinterpret_cast<uint32_t*>(b + o); };
    const size_t H = (size_t)nhalo + 1;
    cudaMemsetAsync(b + L.start, 0, 4 * H, s);
    cudaMemsetAsync(b + L.end, 0, 4 * H, s);
    cudaMemsetAsync(b + L.flags, 0, 4 * H, s);
    if (n > 0) {
        launch(k_cat_keys, (n + 255) / 256, 256, 0, s, pos, igrp, n, nhalo, U(L.keys0),
                                                    I(L.vals0));
        int bits = 0;
        while (bits < 31 && (nhalo >> bits) != 0) ++bits;
        const int cur = radix_sort32(U(L.keys0), I(L.vals0), U(L.keys1), I(L.vals1), n, bits,
                                     false, b + L.sort_tmp, err, s);
        const uint32_t* keys = U(cur ? L.keys1 : L.keys0);
        const int* order = I(cur ? L.vals1 : L.vals0);
        launch(k_cat_bounds, (n + 255) / 256, 256, 0, s, keys, n, U(L.start), U(L.end), err);
        count_launches(2);
        if (nhalo > 0) {
            const int nbig = nhalo < 8192 ? nhalo : 8192, per = CAT_THREADS / 32;
            launch(k_cat_sums, nbig + (nhalo + per - 1) / per, CAT_THREADS, 0, s, 
                pos, vel, igrp ? 1 : 2, order, U(L.start), U(L.end), nhalo, nbig, boxsize,
                reinterpret_cast<float*>(b + L.rec), U(L.flags));
            count_launches(1);
        }
    }
    exclusive_scan_u32(U(L.flags), H, b + L.scan_tmp, s);  // in place: flags -> offsets
    launch(k_cat_compact, (unsigned)((H + 255) / 256), 256, 0, s, 
        reinterpret_cast<const float*>(b + L.rec), U(L.flags), nhalo, out, nlocal);
    count_launches(1);
}

// ---- file formats (host) ----------------------------------------------------------

// int nc, then the floats (one file of write_mesh_separate, coarse_mesh.cpp:180-206)
static int write_block(const std::string& name, int nc, const float* data, size_t count)
{
    FILE* fp = std::fopen(name.c_str(), "wb");
    if (!fp) return ASG_ERR_IO;
    bool ok = std::fwrite(&nc, sizeof(int), 1, fp) == 1;
    ok = ok && std::fwrite(data, sizeof(float), count, fp) == count;
    ok = (std::fclose(fp) == 0) && ok;
    return ok ? ASG_OK : ASG_ERR_IO;
}

// <base>{n,h,c,vel}<inode>.dat of an already normalised mesh [n | halo | c | v xyz]
int write_mesh_files(const char* base, int inode, const float* mesh, int nc)
{
    const size_t nm = (size_t)nc * nc * nc;
    const std::string b(base), i = std::to_string(inode) + ".dat";
    if (int r = write_block(b + "n" + i, nc, mesh, nm)) return r;
    if (int r = write_block(b + "h" + i, nc, mesh + nm, nm)) return r;
    if (int r = write_block(b + "c" + i, nc, mesh + 2 * nm, nm)) return r;
    return write_block(b + "vel" + i, nc, mesh + 3 * nm, 3 * nm);
}

// int nlocal, int sizeof(FofHalo) = 28, the records, int nlocal (fof.cpp:210-217)
int write_fof_file(const char* filename, const float* rec, int nlocal)
{
    FILE* fp = std::fopen(filename, "wb");
    if (!fp) return ASG_ERR_IO;
    const int size_halo = 4 * REC_WORDS;
    bool ok = std::fwrite(&nlocal, sizeof(int), 1, fp) == 1;
    ok = ok && std::fwrite(&size_halo, sizeof(int), 1, fp) == 1;
    ok = ok && std::fwrite(rec, 4 * REC_WORDS, (size_t)nlocal, fp) == (size_t)nlocal;
    ok = ok && std::fwrite(&nlocal, sizeof(int), 1, fp) == 1;
    ok = (std::fclose(fp) == 0) && ok;
    return ok ? ASG_OK : ASG_ERR_IO;
}

}  // namespace asg

// write_mesh (coarse_mesh.cpp:128-143): int nc, int dof = 6, float boxsize, 6*nc^3 floats
extern "C" int asg_write_mesh(const char* filename, const float* mesh, int nc, float boxsize)
{
    if (!filename || !mesh || nc <= 0 || nc > 1290) return ASG_ERR_ARG;
    FILE* fp = std::fopen(filename, "wb");
    if (!fp) return ASG_ERR_IO;
    const int dof = 6;
    const size_t count = (size_t)dof * nc * nc * nc;
    bool ok = std::fwrite(&nc, sizeof(int), 1, fp) == 1;
    ok = ok && std::fwrite(&dof, sizeof(int), 1, fp) == 1;
    ok = ok && std::fwrite(&boxsize, sizeof(float), 1, fp) == 1;
    ok = ok && std::fwrite(mesh, sizeof(float), count, fp) == count;
    ok = (std::fclose(fp) == 0) && ok;
    return ok ? ASG_OK : ASG_ERR_IO;
}
