// order.h — the order of a wave's paths: which pixel and sample a path id
// stands for.  Plain C++, so that it can be checked on the host.
//
// Groups of SAMPLE_GROUP samples, in a group the samples of a pixel side by
// side, and the pixels through 8 x 4 tiles in Morton order: a warp's 32 rays
// leave from as few, as close pixels as the wave's samples allow, so its
// camera rays take nearly the same way through the tree and its secondary rays
// start from nearly the same place (queues keep the order).  Against one
// sample of 32 pixels of a row to a warp, on the mid scene at 1024 x 1024,
// 128 spp: extend 58.7 -> 52.8 ms, shadow 25.2 -> 24.0; heavy scene at
// 1920 x 1080, 4 spp: extend 24.5 -> 22.6.  Groups of 4 / 16 / all samples:
// extend 53.3 / 52.7 / 52.3 ms, but the accumulation, which reads a pixel's
// samples one after the other, takes 0.60 / 0.88 / 1.34 ms against 0.62 with 8
// (one 128-byte line per pixel and group).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define PT_ORDER_FN __host__ __device__ __forceinline__
#else
#define PT_ORDER_FN inline
#endif

namespace pt {

constexpr uint32_t SAMPLE_GROUP = 8;

PT_ORDER_FN uint32_t order_min(uint32_t a, uint32_t b) { return a < b ? a : b; }

// Path lp of `pixels` pixels x k samples: place q in the pixel order, sample j.
PT_ORDER_FN void path_place(uint32_t lp, uint32_t pixels, uint32_t k, uint32_t& q, uint32_t& j)
{
    if (k < SAMPLE_GROUP) { // one group (and SAMPLE_GROUP * pixels may not fit 32 bits)
        q = lp / k;
        j = lp - q * k;
        return;
    }
    const uint32_t group = lp / (SAMPLE_GROUP * pixels);
    const uint32_t in = lp - group * SAMPLE_GROUP * pixels;
    const uint32_t size = order_min(SAMPLE_GROUP, k - group * SAMPLE_GROUP);
    q = size == SAMPLE_GROUP ? in / SAMPLE_GROUP : in / size;
    j = group * SAMPLE_GROUP + (in - q * size);
}

// The path of place q, sample j (the inverse).
PT_ORDER_FN uint64_t path_at(uint32_t q, uint32_t j, uint32_t pixels, uint32_t k)
{
    const uint32_t first = j / SAMPLE_GROUP * SAMPLE_GROUP;
    return (uint64_t)first * pixels + (uint64_t)q * order_min(SAMPLE_GROUP, k - first) + (j - first);
}

// The pixel at place q of a w x h image: bands of four rows, blocks of eight
// columns inside a band, Morton order inside a whole block and row order in
// the ragged ones at the right and bottom edges.
PT_ORDER_FN void ordered_pixel(uint32_t q, uint32_t w, uint32_t h, uint32_t& px, uint32_t& py)
{
    const uint32_t whole = order_min(4u, h) * w; // pixels of a whole band
    const uint32_t band = q / whole;
    const uint32_t in_band = q - band * whole;
    const uint32_t rows = order_min(4u, h - 4u * band);
    const uint32_t block = in_band / (8u * rows);
    const uint32_t i = in_band - block * 8u * rows;
    const uint32_t cols = order_min(8u, w - 8u * block);
    uint32_t x, y;
    if (rows == 4u && cols == 8u) {
        x = (i & 1u) | ((i >> 1) & 2u) | ((i >> 2) & 4u);
        y = ((i >> 1) & 1u) | ((i >> 2) & 2u);
    } else {
        y = i / cols;
        x = i - y * cols;
    }
    px = 8u * block + x;
    py = 4u * band + y;
}

} // namespace pt
