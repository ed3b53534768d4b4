// Kernels and launchers for 32-bit populations.
#include <algorithm>
#define TL_COMMON_KERNELS
#include "tl_kernels.cuh"
#include "tl_call.cuh"
#define TL_POP int
#include "tl_kernels_pop.inc"
#undef TL_POP

namespace tl {

cudaError_t launch_plain_tally(const SimParams& p, cudaStream_t st) {
    k_plain_tally<<<152, 256, 0, st>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_stats_wide(const void* samp, long long R, int PK, int S, void* acc, double* mean, double* sd,
                              int sms, cudaStream_t st) {
    const size_t cols = (size_t)S * PK;
    cudaError_t e = cudaMemsetAsync(acc, 0, cols * 24, st);
    if (e != cudaSuccess) return e;
    // about eight CTAs an SM over the rows, 32 rows a CTA at least
    const int tiles = (PK + 31) / 32;
    const long long want = (8LL * sms + (long long)tiles * S - 1) / ((long long)tiles * S);
    const int split = (int)std::max<long long>(1, std::min<long long>(std::min<long long>(want, (R + 31) / 32), 65535));
    k_stats_wide<<<dim3((unsigned)tiles, (unsigned)split, (unsigned)S), 256, 0, st>>>(
        reinterpret_cast<const int*>(samp), R, PK, reinterpret_cast<unsigned long long*>(acc));
    k_stats_wide_finish<<<(unsigned)((cols + 127) / 128), 128, 0, st>>>(reinterpret_cast<const int*>(samp), R, PK,
                                                                       (int)cols,
                                                                       reinterpret_cast<unsigned long long*>(acc), mean, sd);
    return cudaGetLastError();
}

cudaError_t launch_philox(const void* ctr, const void* key, int n, void* out, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_philox<<<(n + 255) / 256, 256, 0, st>>>(reinterpret_cast<const uint4*>(ctr), reinterpret_cast<const uint2*>(key),
                                              n, reinterpret_cast<uint4*>(out));
    return cudaGetLastError();
}

cudaError_t launch_poisson(const float* mean, int n, unsigned k0, unsigned k1, unsigned step, int compat, int* out,
                           cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_poisson<<<(n + 255) / 256, 256, 0, st>>>(mean, n, k0, k1, step, compat, out);
    return cudaGetLastError();
}

}  // namespace tl
