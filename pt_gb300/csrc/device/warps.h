// warps.h — work dealt out a warp to an item.  Plain C++, so that the index can
// be checked on the host.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define PT_WARPS_FN __host__ __device__ __forceinline__
#else
#define PT_WARPS_FN inline
#endif

namespace pt {

// The item of a thread's warp.  The thread's own number needs not fit 32 bits:
// 2^28 instances are 2^33 threads.
PT_WARPS_FN uint32_t warp_item(uint32_t block, uint32_t block_threads, uint32_t thread)
{
    return block * (block_threads / 32u) + thread / 32u;
}

} // namespace pt
