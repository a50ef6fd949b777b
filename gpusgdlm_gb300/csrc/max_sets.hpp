// Bookkeeping of block-wide maxima that take one barrier each (block_max,
// forecast_kernels.cu).  Kept free of device intrinsics so that the host can run
// the same rules in a model of the warps (tests/max_sets_check.cpp).
//
// Reduction c (counted from 0) of a block: every warp adds its maximum to the set
// set_of(c), the block meets at a barrier, every thread reads set_of(c), and one warp
// clears set_to_clear(c).  Nothing else need lie between two reductions, so a warp may
// be one barrier ahead of another, no more:
//  * the set that reduction c clears is filled by reduction c + 2, after the barrier of
//    c + 1, which the clearing warp passes only once it has cleared;
//  * it was read last by reduction c - 1, and every thread has done so before it
//    arrives at the barrier of c.
// With two sets (clear the next reduction's) a fast warp's maximum of c + 1 and the
// clearing of its set have no barrier between them, and the maximum can be lost.
#pragma once

#if defined(__CUDACC__)
#define SGDLM_MAX_HD __host__ __device__ __forceinline__
#else
#define SGDLM_MAX_HD inline
#endif

namespace sgdlm {

constexpr int kMaxSets = 3;

SGDLM_MAX_HD int set_after(int set) { return set + 1 == kMaxSets ? 0 : set + 1; }
// of a reduction that fills `set`: the one to clear, filled by the next but one
SGDLM_MAX_HD int set_to_clear(int set) { return set_after(set_after(set)); }

}  // namespace sgdlm
