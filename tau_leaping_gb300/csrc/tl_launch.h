// tl_launch.h - host launchers of the kernels, one set per population type
// (Pop = int for 32-bit, long long for 64-bit populations).
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace tl {

struct SimParams;

// kind: 1 = thread, 32 = warp, 0 = CTA, 2/4/8/16 = lanes per realization,
// kKindCtaGlobal = CTA with its propensities (or whole slot) in global memory;
// in the fast and scores builds a thread group is one lane (GThin) or, for
// small models, 4, 8 or 16 lanes (tl_tiny.cuh).
constexpr int kKindCtaGlobal = 64;
constexpr int kKindTeam = 132;  // four warps for one realization of a warp group
constexpr int kKindThin1 = 101, kKindTiny4 = 104, kKindTiny8 = 108, kKindTiny16 = 116;

// Table of a small model (N, M <= 16): per channel {s0, s1, order, 0}, then per
// species its 16 stoichiometries, then per species the g kind.
struct TinyTable {
    uint32_t chan[16];
    int8_t v[16][16];
    uint8_t gkind[16];
};
// mode: the kernel build a run needs.  Fast: no likelihood-ratio scores and
// no reference-compatibility switches; Scores: with scores; General: both.
// The sub-warp and global-slot kinds come in Fast and General only, two lanes in
// General only.
constexpr int kModeFast = 0, kModeScores = 1, kModeGeneral = 2;
// Thread, sub-warp and warp groups launch at most 256 threads per CTA and
// ask the compiler for a number of resident CTAs per SM, which sets the
// register budget 65536 / (256 * n) per thread: TL_THREAD_MINB for thread
// groups, TL_WARP_MINB for the others.  CTA groups use up to 1024 threads.
// Sweeps on GB300: warp and sub-warp groups of the fast builds run best at 4
// (64 registers, no spills to speak of: toy network 67.6 ms against 75.7 at 5
// and 74.4 at 3, the 45 x 83 network 90.9 against 102.2 and 98.1), thread
// groups at 3 (dimer 3.49 ms against 3.67 at 4).
#ifndef TL_WARP_MINB
#define TL_WARP_MINB 4
#endif
#ifndef TL_THREAD_MINB
#define TL_THREAD_MINB 3
#endif
// the general build's warp and sub-warp groups
#ifndef TL_GENERAL_MINB
#define TL_GENERAL_MINB 5
#endif
// The batch kernel's CTAs per SM: batch_minb() chooses.
#ifndef TL_BATCH_MINB
#define TL_BATCH_MINB 2
#endif
#ifndef TL_BATCH_MANY_MINB
#define TL_BATCH_MANY_MINB 3
#endif
#ifndef TL_BATCH_THIN_MINB
#define TL_BATCH_THIN_MINB 4
#endif
// staged: the tables are staged in shared memory.
template <class Pop>
cudaError_t launch_fused(const SimParams& p, int kind, int mode, bool staged, int block, int grid, size_t smem,
                         cudaStream_t st);
template <class Pop>
cudaError_t fused_occupancy(int kind, int mode, bool staged, int block, size_t smem, int* blocks_per_sm);
// parts of the two above, compiled in units of their own: a launch, or the
// occupancy where bps is not null
struct FusedCall {
    const SimParams* p;
    int kind, mode;
    bool staged;
    int block, grid;
    size_t smem;
    cudaStream_t st;
    int* bps;
};
template <class Pop>
cudaError_t call_general_sub(const FusedCall& c);
template <class Pop>
cudaError_t call_fast(const FusedCall& c);  // thread and warp groups
template <class Pop>
cudaError_t call_fast_cta(const FusedCall& c);
template <class Pop>
cudaError_t call_fast_sub(const FusedCall& c);
struct BatchParams;
template <class Pop>
cudaError_t launch_batch(const BatchParams& bp, int mode, int minb, int thin, int block, int grid, size_t smem,
                         cudaStream_t st);
template <class Pop>
cudaError_t batch_occupancy(int mode, bool staged, int minb, int thin, int block, size_t smem, int* blocks_per_sm);
// the same with four-warp teams in place of the warp units (staged tables only)
template <class Pop>
cudaError_t launch_batch_team(const BatchParams& bp, int mode, int thin, int grid, size_t smem, cudaStream_t st,
                              int* blocks_per_sm);
template <class Pop>
cudaError_t launch_plain_init(const SimParams& p, cudaStream_t st);
template <class Pop>
cudaError_t launch_plain_step(const SimParams& p, float* a_all, cudaStream_t st);
cudaError_t launch_plain_tally(const SimParams& p, cudaStream_t st);
template <class Pop>
cudaError_t launch_stats(const void* samp, long long R, int P, int K, int S, double* mean, double* sd,
                         cudaStream_t st);
// the same for many columns of 32-bit populations; acc: 24 bytes a column
cudaError_t launch_stats_wide(const void* samp, long long R, int PK, int S, void* acc, double* mean, double* sd,
                              int sms, cudaStream_t st);
template <class Pop>
cudaError_t launch_grad(const void* samp, const float* scores, long long R, int P, int K, int M, int S,
                        double* grad, double* se, double* meanf, cudaStream_t st);
template <class Pop>
cudaError_t launch_eval(const SimParams& p, const long long* x, int n, float* a, unsigned char* crit, float* mu,
                        float* s2, float* tau, double* a0, size_t smem, cudaStream_t st);
template <class Pop>
cudaError_t launch_replay(const SimParams& p, const long long* x0, const int* k, int n_leaps, long long* x_out,
                          int* status, size_t smem, cudaStream_t st);
cudaError_t launch_philox(const void* ctr, const void* key, int n, void* out, cudaStream_t st);
cudaError_t launch_poisson(const float* mean, int n, unsigned k0, unsigned k1, unsigned step, int compat,
                           int* out, cudaStream_t st);

}  // namespace tl
