// Fast and scores builds, 32-bit populations: the batch kernel.
#include "tl_kernels.cuh"
#include "tl_call.cuh"
#define TL_POP int
#define TL_FAST_PART 4
#include "tl_fast.inc"
