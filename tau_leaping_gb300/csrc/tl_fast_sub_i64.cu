// Fast and scores builds, 64-bit populations: sub-warp groups.
#include "tl_kernels.cuh"
#include "tl_call.cuh"
#define TL_POP long long
#define TL_FAST_PART 3
#include "tl_fast.inc"
