// lla_ring.h -- which copies of a shared-memory ring may still be in flight.  Host and
// device code: a host test plays the ring.
#pragma once

#include <stdint.h>

#ifndef __CUDACC__  // host-only compilers: the qualifiers vanish
#ifndef __host__
#define __host__
#endif
#ifndef __device__
#define __device__
#endif
#ifndef __forceinline__
#define __forceinline__ inline
#endif
#endif

namespace lla {

// Copy g of a ring goes to stage g % stages and completes phase g / stages of the stage's
// barrier.  After `issued` copies: whether the stage has had one, and the parity of
// its last one's phase.  The earlier ones have landed: a stage is refilled only after
// its reader has waited for it.
__host__ __device__ __forceinline__ bool ring_last_phase(uint64_t issued, uint32_t stages, uint32_t stage, uint32_t &parity) {
    if (issued <= stage) return false;
    parity = (uint32_t)((issued - 1 - stage) / stages) & 1u;
    return true;
}

}  // namespace lla
