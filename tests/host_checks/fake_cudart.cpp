// A CUDA runtime without a GPU: the library's object files are linked against it,
// so that a CPU test sees what the host code asks of the device.  Device memory is
// host memory, kernels do not run, and every call that matters to a test leaves a
// line in the log:
//   launch <kernel> <grid> <block> <dynamic shared bytes>
//   attr <kernel> <attribute> <value>          (cudaFuncSetAttribute)
//   load <kernel>                              (cudaFuncGetAttributes)
//   malloc <bytes>
//   boxes <bytes the tree takes> <bytes from its start to the end of its block>
//   tree <kernel> <particles per leaf>         (the tree that a kernel builds or walks)
// k_report (the words that a call brings to the host) is carried out, and so are
// the two counts of k_dep_prep, with the numbers that fake_counts() was given.
#include <sys/mman.h>

#include <climits>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

#include <cuda_runtime.h>

#include "asg_internal.h"

using namespace asg;

namespace {
std::string g_log;
std::map<const void*, std::string> g_kernels;
std::map<const void*, size_t> g_vars;
std::map<const void*, void*> g_var_at;
std::map<char*, size_t> g_blocks;
uint32_t g_entries = 0;
unsigned long long g_pairs[3] = {};
int g_timed = 0, g_fastest = INT_MAX;
bool g_spin = false;              // the device flags allow the host to poll
cudaError_t g_last = cudaSuccess;  // what cudaGetLastError returns next
size_t g_largest = SIZE_MAX;       // device blocks of more bytes are refused
std::map<cudaEvent_t, bool> g_done;  // events, done when something waited for them

void line(const std::string& s) { g_log += s + "\n"; }
std::string num(unsigned long long v) { return std::to_string(v); }
const std::string& name(const void* f) { return g_kernels[f]; }
bool is(const std::string& mangled, const char* kernel)
{
    return mangled.find(std::to_string(std::strlen(kernel)) + kernel) != std::string::npos;
}

// the members of asg_capi.cu's types that k_report touches
struct Words {
    const void* p;
    int n;
};
struct HostWords {
    uint32_t number, pad[31];
    int err;
    uint32_t word[64];
};

void launched(const std::string& k, dim3 grid, dim3 block, size_t smem, void** a)
{
    line("launch " + k + " " + num((unsigned long long)grid.x * grid.y * grid.z) + " " + num(block.x) + " " +
         num(smem));
    const int tree = is(k, "k_gather") ? 8 : is(k, "k_fof_link") || is(k, "k_mark_halos") || is(k, "k_knn_ties") ? 1 : -1;
    if (tree >= 0) line("tree " + k + " " + num(static_cast<TreeView*>(a[tree])->leaf));
    if (is(k, "k_report")) {
        HostWords* out = *static_cast<HostWords**>(a[4]);
        int at = 0;
        for (int i = 0; i < 3; ++i) {
            const Words& w = *static_cast<Words*>(a[i]);
            std::memcpy(out->word + at, w.p, 4 * (size_t)w.n);
            at += w.n;
        }
        out->err = **static_cast<const int**>(a[3]);
        out->number = *static_cast<uint32_t*>(a[5]);
    } else if (is(k, "k_dep_prep")) {
        const int n = *static_cast<int*>(a[4]);
        const DepositParams& p = *static_cast<DepositParams*>(a[5]);
        (*static_cast<uint32_t**>(a[7]))[(n + 31) / 32 << p.log_parts] = g_entries;
        **static_cast<unsigned long long**>(a[8]) = g_pairs[p.shift[1] < 3 ? 0 : p.shift[2] < 3 ? 1 : 2];
    } else if (is(k, "k_gather")) {
        const TreeView& t = *static_cast<TreeView*>(a[8]);
        char* at = (char*)t.box;
        auto it = g_blocks.upper_bound(at);
        const size_t have = it == g_blocks.begin() || (--it)->first + it->second < at
                                ? 0
                                : (size_t)(it->first + it->second - at);
        line("boxes " + num(32 * (unsigned long long)(t.off[t.nlev - 1] + t.cnt[t.nlev - 1])) + " " + num(have));
    }
}

void* block(size_t bytes)
{
    void* p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (p == MAP_FAILED) return nullptr;
    g_blocks[static_cast<char*>(p)] = bytes;
    return p;
}

template <class T>
cudaError_t handle(T* out)
{
    static uintptr_t next = 0x1000;
    *out = reinterpret_cast<T>(next += 16);
    return cudaSuccess;
}
}  // namespace

extern "C" {

const char* fake_log() { return g_log.c_str(); }
void fake_clear() { g_log.clear(); }
// entries, and the pairs with tiles of 8 x 4 x 4, 8 x 8 x 4 and 8 x 8 x 8 cells
void fake_counts(uint32_t entries, unsigned long long pairs844, unsigned long long pairs884,
                 unsigned long long pairs888)
{
    g_entries = entries;
    g_pairs[0] = pairs844;
    g_pairs[1] = pairs884;
    g_pairs[2] = pairs888;
}

// contexts created from now on may poll for their results instead of waiting
void fake_spin(int on) { g_spin = on != 0; }

// device memory has no room for a block of more bytes than this
void fake_largest(size_t bytes) { g_largest = bytes; }

// of the times that are asked for, the n-th from now on is the shortest
void fake_fastest(int n)
{
    g_timed = 0;
    g_fastest = n;
}

void** __cudaRegisterFatBinary(void*)
{
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* mangled, int, uint3*, uint3*, dim3*, dim3*,
                            int*)
{
    g_kernels[host] = mangled;
}
void __cudaRegisterVar(void**, char* host, char*, const char*, int, size_t size, int, int) { g_vars[host] = size; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f)
{
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void** a, size_t s, cudaStream_t)
{
    launched(name(k), g, b, s, a);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a)
{
    launched(name(f), c->gridDim, c->blockDim, c->dynamicSmemBytes, a);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute attr, int v)
{
    line("attr " + name(f) + " " + num(attr) + " " + std::to_string(v));
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* f)
{
    std::memset(a, 0, sizeof(*a));
    line("load " + name(f));
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*)
{
    *n = 1;
    return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t bytes)
{
    line("malloc " + num(bytes));
    *p = bytes > g_largest ? nullptr : block(bytes);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p)
{
    auto it = g_blocks.find(static_cast<char*>(p));
    if (it != g_blocks.end()) {
        munmap(p, it->second);
        g_blocks.erase(it);
    }
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned)
{
    *p = std::calloc(1, bytes);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t bytes) { return cudaHostAlloc(p, bytes, 0); }
cudaError_t cudaFreeHost(void* p)
{
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned)
{
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaHostRegister(void*, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol)
{
    void*& at = g_var_at[symbol];
    if (!at) at = block(g_vars[symbol]);
    *p = at;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t)
{
    std::memset(d, v, n);
    return cudaSuccess;
}

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceFlags(unsigned* f)
{
    *f = g_spin ? cudaDeviceScheduleAuto : cudaDeviceScheduleBlockingSync;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int)
{
    *v = 152;
    return cudaSuccess;
}
cudaError_t cudaGetLastError()
{
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return g_last; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    for (auto& e : g_done) e.second = true;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    line("capture");
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g)
{
    line("captured");
    return handle(g);
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t)
{
    g_done[e] = false;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t last)
{
    for (auto& e : g_done) e.second |= e.first <= last;  // those recorded before it, too
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b)
{
    if (!g_done[a] || !g_done[b]) return g_last = cudaErrorNotReady;
    *ms = (float)std::abs((long long)++g_timed - g_fastest);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { return handle(x); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

}  // extern "C"
