// tl_shared.h - what kernels, launch code and host tests compute alike.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define TL_SHARED __host__ __device__ __forceinline__
#else
#define TL_SHARED inline
#endif

namespace tl {

// Turns of four channels a lane that a queue group may mark before its queue is
// drained: four bits each in a lane's 32-bit masks, and a warp's marks counted in ten bits.
constexpr int kMaxRounds = 7;
static_assert(4 * kMaxRounds <= 32 && 4 * 32 * kMaxRounds < 1 << 10, "masks and counts of the firing pass");

// The Philox step counter wraps at 2^32; epochs counts that once a leap or block
// of direct-method steps, so that caps and counts of steps hold past it.  (The
// counter's words repeat from there on.)  Whether the counter wrapped since it stood at
// `from`, or in its last `steps` steps:
TL_SHARED uint32_t wrapped_past(uint32_t step, uint32_t from) { return step < from ? 1u : 0u; }
TL_SHARED uint32_t wrapped(uint32_t step, int steps) { return step < (uint32_t)steps ? 1u : 0u; }
// Accepted steps: attempts and direct-method steps less the rejected attempts.
TL_SHARED long long accepted(uint32_t epochs, uint32_t step, uint32_t rej) {
    return (long long)((unsigned long long)epochs << 32 | step) - (long long)rej;
}

}  // namespace tl
