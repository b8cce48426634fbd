// slab.h — one axis of the box test: the inverse direction it multiplies by, and
// which plane of a box's slab a ray meets first, for tests that take one
// distance per plane (device/scene.cuh).  Plain C++, so that the rules can be
// checked on the host.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define PT_SLAB_FN __host__ __device__ __forceinline__
#else
#define PT_SLAB_FN inline
#endif

namespace pt {

// Makes 1 / d and o / d of the distances fma(plane, 1/d, -o/d) finite.  For a
// zero component they are infinities, and of a slab that holds the origin and
// has its planes on both sides of coordinate 0 one distance is then the infinity
// of the wrong side and the other a NaN: the box is missed.  Such a component,
// or one so small that o / d overflows, is taken as a power of two instead, the
// largest that o times it stays finite with: o / d is then exact, a distance has
// the sign of plane - o, and one that is not zero is at least 2^102 for |o| >= 1
// (below, in proportion to |o|): past the end of any ray.
PT_SLAB_FN void slab_finite(float o, float& inv, float& o_inv)
{
    if (o_inv - o_inv == 0.0f || inv != inv) // finite, or a ray that is not a number
        return;
    uint32_t o_bits, bits;
    memcpy(&o_bits, &o, sizeof(bits));
    memcpy(&bits, &inv, sizeof(bits));
    const uint32_t exponent = (o_bits >> 23) & 255u;
    bits = (bits & 0x80000000u) | ((exponent > 127u ? 380u - exponent : 253u) << 23);
    memcpy(&inv, &bits, sizeof(bits));
    o_inv = o * inv;
}

// True when the upper plane comes first: a negative direction component.  The
// argument is the bit pattern of 1 / d.  An infinite 1 / d (a zero component,
// where slab_finite is not used) gets the other order: its distances are
// infinities and NaNs, and in this order the entry and exit taken one plane each
// are what the minimum and maximum of the two distances give, a NaN being
// ignored.  That form misses a slab that holds the origin and has its planes on
// both sides of coordinate 0.  Adding one exponent step turns +inf into a
// negative and -inf into a positive integer and leaves every finite number's
// sign.
PT_SLAB_FN bool slab_hi_first(uint32_t inv_bits) { return (int32_t)(inv_bits + 0x00800000u) < 0; }

} // namespace pt
