/* Index arithmetic of the kernels in which several lanes share a target.  No
 * CUDA types: host code checks it with a plain C++ compiler. */
#pragma once

#if defined(__CUDACC__)
#define LQ_LANES_HD __host__ __device__ __forceinline__
#else
#define LQ_LANES_HD inline
#endif

namespace lqb {

/* The target of thread `thread` of block `block` (of `threads` threads) when
 * `lanes` consecutive threads share one.  block * threads, the thread's place
 * in the whole grid, is not formed: it wraps at 32 bits from 2^32 / lanes
 * targets on, which with eight lanes fit the card. */
LQ_LANES_HD int lane_target(unsigned block, unsigned thread, unsigned threads, unsigned lanes)
{
    return (int)(block * (threads / lanes) + thread / lanes);
}

}  // namespace lqb
