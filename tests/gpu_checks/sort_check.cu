// The radix sort with 64-bit tile states, which counts of 2^30 and more elements need,
// on sizes that fit a test: same order as std::stable_sort, for every key and digit
// width.  Prints one line per check.
#include <algorithm>
#include <cstdio>
#include <numeric>
#include <vector>

#include "../../asmooth_gb300/csrc/asg_index.cu"

namespace asg {
void count_launches(int) {}
}  // namespace asg

using namespace asg;

template <class K, int BITS, class S>
static int check(const char* name, int n, int passes, K mask)
{
    std::vector<K> key(n);
    unsigned long long r = 88172645463325252ull + n;
    for (int i = 0; i < n; ++i) {
        r ^= r << 13;
        r ^= r >> 7;
        r ^= r << 17;
        key[i] = (K)(i % 3 ? r : r & 0xff00ff) & mask;  // a third with many equal digits
    }
    std::vector<int> want(n), got(n);
    std::iota(want.begin(), want.end(), 0);
    std::stable_sort(want.begin(), want.end(), [&](int a, int b) { return key[a] < key[b]; });
    K* k[2];
    int *v[2], *err;
    void* tmp;
    const size_t tiles = (size_t)n / RS_TILE<K> + 1;
    cudaMalloc(&k[0], sizeof(K) * n);
    cudaMalloc(&k[1], sizeof(K) * n);
    cudaMalloc(&v[0], 4 * (size_t)n);
    cudaMalloc(&v[1], 4 * (size_t)n);
    cudaMalloc(&err, 4);
    cudaMalloc(&tmp, 4 * (RS_HEAD + RS_HIST) + sizeof(S) * tiles * (1 << BITS) * passes + 256);
    cudaMemset(err, 0, 4);
    cudaMemcpy(k[0], key.data(), sizeof(K) * n, cudaMemcpyHostToDevice);
    const int cur = radix_sort_t<K, BITS, S>(k[0], v[0], k[1], v[1], n, passes, true, tmp, err, 0);
    int bits = -1;
    cudaMemcpy(got.data(), v[cur], 4 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaMemcpy(&bits, err, 4, cudaMemcpyDeviceToHost);
    const cudaError_t e = cudaDeviceSynchronize();
    int bad = 0;
    for (int i = 0; i < n; ++i) bad += got[i] != want[i];
    std::printf("%s n=%d mismatches %d error word %d %s\n", name, n, bad, bits, cudaGetErrorString(e));
    for (int b = 0; b < 2; ++b) {
        cudaFree(k[b]);
        cudaFree(v[b]);
    }
    cudaFree(err);
    cudaFree(tmp);
    return bad != 0 || bits != 0 || e != cudaSuccess;
}

int main()
{
    int bad = 0;
    for (int n : {1, 3071, 3072, 3073, 4097, 70001, 3000001}) {
        bad |= check<uint64_t, 8, uint64_t>("64-bit keys, 48 bits, 64-bit states", n, 6, (1ull << 48) - 1);
        bad |= check<uint32_t, 8, uint64_t>("32-bit keys, 32 bits, 64-bit states", n, 4, 0xffffffffu);
        bad |= check<uint32_t, 9, uint64_t>("32-bit keys, 27 bits, 64-bit states", n, 3, (1u << 27) - 1);
    }
    return bad;
}
