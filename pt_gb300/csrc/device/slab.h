// slab.h — which plane of a box's slab a ray meets first, for box tests that
// take one distance per plane (device/scene.cuh).  Plain C++, so that the rule
// can be checked on the host.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define PT_SLAB_FN __host__ __device__ __forceinline__
#else
#define PT_SLAB_FN inline
#endif

namespace pt {

// True when the upper plane comes first: a negative direction component.  The
// argument is the bit pattern of 1 / d.  An infinite 1 / d (a zero component)
// gets the other order: its distances fma(plane, 1/d, -o/d) are infinities and
// NaNs, and in this order the entry and exit taken one plane each are what the
// minimum and maximum of the two distances give, a NaN being ignored.  Adding
// one exponent step turns +inf into a negative and -inf into a positive
// integer and leaves every finite number's sign.
PT_SLAB_FN bool slab_hi_first(uint32_t inv_bits) { return (int32_t)(inv_bits + 0x00800000u) < 0; }

} // namespace pt
