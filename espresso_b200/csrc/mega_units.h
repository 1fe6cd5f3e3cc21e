// Which K units of a chunk a load batch of the persistent kernels' products reads (mega_kernel.cuh).  Plain C++, so that the rule
// can be checked on the host.
#pragma once

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace esp {

// A warp owns the units first, first + step, ... of a chunk's `nu` and loads several of them at once: unit `x` of the batch that
// begins with unit i0 < nu.  A batch that runs past the chunk reads its own first unit again (and multiplies it by zeros): the
// operand and the block scale of every other unit belong to another warp, and nothing orders this warp behind their
// staging.  (A scale read too early can hold any bits, and zero times Inf or NaN would reach the sum.)
__host__ __device__ __forceinline__ constexpr int mega_batch_unit(int i0, int x, int step, int nu) { return i0 + x * step < nu ? i0 + x * step : i0; }

}  // namespace esp
