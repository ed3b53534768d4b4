// The general build's sub-warp and global-slot kernels, 64-bit populations.
#include "tl_kernels.cuh"
#include "tl_call.cuh"
#define TL_POP long long
#include "tl_kernels_sub.inc"
#undef TL_POP
