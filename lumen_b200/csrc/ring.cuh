// Which use of a ring's stage came last: plain arithmetic, for the kernels and for programs of the host.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define LUMEN_HD __host__ __device__ __forceinline__
#else
#define LUMEN_HD inline
#endif

namespace lumen {

// Uses of stage `stage` by the first `steps` steps, which take the `stages` stages in turn.
LUMEN_HD constexpr int ring_uses(int steps, int stage, int stages) { return steps > stage ? (steps - 1 - stage) / stages + 1 : 0; }

// Parity whose test says that the last of `uses` uses of an mbarrier is complete (uses > 0).  A test of the other parity
// says that the use before it is, which is so while the last one is still on its way: either-parity is always true.
LUMEN_HD constexpr uint32_t ring_last_parity(int uses) { return (uint32_t)(uses - 1) & 1u; }

}  // namespace lumen
