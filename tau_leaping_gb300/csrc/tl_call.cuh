// tl_call.cuh - one launch (or occupancy query) of a kernel over SimParams.
#pragma once

#include "tl_launch.h"

namespace tl {

template <class Kernel>
static cudaError_t call_kernel(Kernel k, const FusedCall& c) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.smem);
    if (e != cudaSuccess) return e;
    if (c.bps) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(c.bps, k, c.block, c.smem);
    k<<<c.grid, c.block, c.smem, c.st>>>(*c.p);
    return cudaGetLastError();
}

}  // namespace tl
