// ops.cu — memory-bound kernels of the denoiser: 2x2 average pooling and
// nearest upsampling with their backward passes (ReLU masks fused), bias
// gradients, weight packing for the tensor-core layouts and Adam.  A thread of
// the pooling and upsampling kernels moves 16 channels (32-byte accesses) of
// one low-resolution pixel and its four high-resolution ones.
#include <cuda_bf16.h>

#include <algorithm>

#include "../device/chain.cuh"
#include "nn.h"
#include "tc.cuh"

namespace pt {
namespace nn {

namespace {

__device__ __forceinline__ uint32_t pack2(float a, float b)
{
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ size_t pixel(const Act& a, int img, int y, int x)
{
    return ((size_t)img * a.h + y) * a.w + x;
}

// 16 channels from c of a pixel, as floats or as they are.
struct Vec16 {
    uint32_t w[8];
    __device__ __forceinline__ float lo(int k) const { return __uint_as_float(w[k] << 16); }
    __device__ __forceinline__ float hi(int k) const { return __uint_as_float(w[k] & 0xFFFF0000u); }
};

__device__ __forceinline__ Vec16 ld16(const Act& a, size_t pix, int c)
{
    Vec16 v;
    load32(a.p + pix * a.pitch + c, v.w);
    return v;
}

__device__ __forceinline__ void st16(const Act& a, size_t pix, int c, const Vec16& v) { store32(a.p + pix * a.pitch + c, v.w); }

__device__ __forceinline__ Vec16 pack16(const float (&v)[16])
{
    Vec16 r;
#pragma unroll
    for (int k = 0; k < 8; k++)
        r.w[k] = pack2(v[2 * k], v[2 * k + 1]);
    return r;
}

__device__ __forceinline__ void add16(float (&acc)[16], const Vec16& v)
{
#pragma unroll
    for (int k = 0; k < 8; k++) {
        acc[2 * k] += v.lo(k);
        acc[2 * k + 1] += v.hi(k);
    }
}

// Zeroes the channels whose activation z is not positive.
__device__ __forceinline__ void relu_mask(float (&v)[16], const Vec16& z)
{
#pragma unroll
    for (int k = 0; k < 8; k++) {
        if (!(z.lo(k) > 0.0f))
            v[2 * k] = 0.0f;
        if (!(z.hi(k) > 0.0f))
            v[2 * k + 1] = 0.0f;
    }
}

// f(img, y, x, u): every pixel of `low` and unit u of `units` units of 16
// channels.  Rows over blockIdx.y, so that one 32-bit division finds the pixel.
// With 64-bit divisions of a flat index and 16-byte accesses upsampling was bound
// by its integer arithmetic (64 channels to 1080 x 1920, 331 MB: 81 us, 50 now;
// backward at 16 x 256 x 256: 39 us, 25 now).  Pooling is bound by DRAM before
// and after (42 us at 6.6 TB/s): the skip connection is 64 bytes of a pixel's 192
// and DRAM delivers 128.
template <class F>
__device__ __forceinline__ void for_low_pixels(const Act& low, int units, F f)
{
    const uint32_t rows = (uint32_t)low.n * (uint32_t)low.h, row_units = (uint32_t)low.w * (uint32_t)units;
    for (uint32_t row = blockIdx.y; row < rows; row += gridDim.y) {
        const uint32_t img = row / (uint32_t)low.h, y = row - img * (uint32_t)low.h;
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < row_units; i += gridDim.x * blockDim.x) {
            const uint32_t x = i / (uint32_t)units;
            f((int)img, (int)y, (int)x, (int)(i - x * (uint32_t)units));
        }
    }
}

constexpr int POOL_THREADS = 128;

__global__ void __launch_bounds__(POOL_THREADS) k_pool2(Act in, int in_c0, int units, Act out, int out_c0)
{
    chain_begin();
    for_low_pixels(out, units, [&](int img, int y, int x, int u) {
        float acc[16] = {};
        const size_t p = pixel(in, img, 2 * y, 2 * x);
        const Vec16 v00 = ld16(in, p, in_c0 + 16 * u), v01 = ld16(in, p + 1, in_c0 + 16 * u);
        const Vec16 v10 = ld16(in, p + in.w, in_c0 + 16 * u), v11 = ld16(in, p + in.w + 1, in_c0 + 16 * u);
        add16(acc, v00);
        add16(acc, v01);
        add16(acc, v10);
        add16(acc, v11);
#pragma unroll
        for (int k = 0; k < 16; k++)
            acc[k] *= 0.25f;
        st16(out, pixel(out, img, y, x), out_c0 + 16 * u, pack16(acc));
    });
}

__global__ void __launch_bounds__(POOL_THREADS) k_upsample2(Act in, int in_c0, int units, Act out, int out_c0)
{
    chain_begin();
    for_low_pixels(in, units, [&](int img, int y, int x, int u) {
        const Vec16 v = ld16(in, pixel(in, img, y, x), in_c0 + 16 * u);
        const size_t p = pixel(out, img, 2 * y, 2 * x);
        const int c = out_c0 + 16 * u;
        st16(out, p, c, v);
        st16(out, p + 1, c, v);
        st16(out, p + out.w, c, v);
        st16(out, p + out.w + 1, c, v);
    });
}

__global__ void __launch_bounds__(POOL_THREADS) k_upsample2_backward(Act gh, int g_c0, int units, Act z, int z_c0, Act gl)
{
    chain_begin();
    for_low_pixels(gl, units, [&](int img, int y, int x, int u) {
        float acc[16] = {};
        const size_t p = pixel(gh, img, 2 * y, 2 * x), pl = pixel(gl, img, y, x);
        const int c = g_c0 + 16 * u;
        const Vec16 v00 = ld16(gh, p, c), v01 = ld16(gh, p + 1, c), v10 = ld16(gh, p + gh.w, c), v11 = ld16(gh, p + gh.w + 1, c);
        const Vec16 zv = ld16(z, pl, z_c0 + 16 * u);
        add16(acc, v00);
        add16(acc, v01);
        add16(acc, v10);
        add16(acc, v11);
        relu_mask(acc, zv);
        st16(gl, pl, 16 * u, pack16(acc));
    });
}

__global__ void __launch_bounds__(POOL_THREADS) k_pool2_backward(Act gs, int s_c0, Act gp, int units, Act z, int z_c0, Act g_out)
{
    chain_begin();
    for_low_pixels(gp, units, [&](int img, int y, int x, int u) {
        const Vec16 b = ld16(gp, pixel(gp, img, y, x), 16 * u);
        const size_t p0 = pixel(g_out, img, 2 * y, 2 * x);
        // a pixel at a time: all eight loads first is slower (21 -> 23 us a level
        // below), for the registers cost more warps than the loads ahead give
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const size_t p = p0 + (size_t)(d >> 1) * g_out.w + (d & 1);
            const Vec16 s = ld16(gs, p, s_c0 + 16 * u), zv = ld16(z, p, z_c0 + 16 * u);
            float a[16];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                a[2 * k] = s.lo(k) + 0.25f * b.lo(k);
                a[2 * k + 1] = s.hi(k) + 0.25f * b.hi(k);
            }
            relu_mask(a, zv);
            st16(g_out, p, 16 * u, pack16(a));
        }
    });
}

// One block reduces a pixel range for all channels: thread t owns the 16-channel
// unit t % units and strides over pixels by the block's rows, four 32-byte loads
// ahead of the sums: 32 channels of 16 x 256 x 256 (67 MB) take 14 us, 19 with one
// 16-byte load at a time.
constexpr int BIAS_THREADS = 256;

__global__ void __launch_bounds__(BIAS_THREADS) k_bias_grad(Act g, int c0, int units, float* db, uint32_t pixels_per_block)
{
    chain_begin();
    __shared__ float red[BIAS_THREADS * 17];
    const int rows = BIAS_THREADS / units;
    const int u = threadIdx.x % units, row = threadIdx.x / units;
    float acc[16] = {};
    const size_t p0 = blockIdx.x * (size_t)pixels_per_block;
    const size_t left = g.pixels() - p0;
    const int n = (int)(left < pixels_per_block ? left : pixels_per_block);
    if (row < rows) {
        const uint16_t* q = g.p + p0 * g.pitch + c0 + 16 * u;
        int p = row;
        for (; p + 3 * rows < n; p += 4 * rows) {
            Vec16 v[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
                load32(q + (size_t)(p + k * rows) * g.pitch, v[k].w);
#pragma unroll
            for (int k = 0; k < 4; k++)
                add16(acc, v[k]);
        }
        for (; p < n; p += rows) {
            Vec16 v;
            load32(q + (size_t)p * g.pitch, v.w);
            add16(acc, v);
        }
    }
#pragma unroll
    for (int k = 0; k < 16; k++)
        red[threadIdx.x * 17 + k] = acc[k];
    __syncthreads();
    if ((int)threadIdx.x < units * 16) {
        const int uu = threadIdx.x / 16, k = threadIdx.x % 16;
        float s = 0.0f;
        for (int r = 0; r < rows; r++)
            s += red[(r * units + uu) * 17 + k];
        atomicAdd(db + 16 * uu + k, s);
    }
}

__global__ void k_pack_weights(const float* w, int cin, int cout, uint16_t* fwd, uint16_t* bwd)
{
    const size_t n = (size_t)9 * cin * cout;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        // i enumerates w[tap][ci][co]
        const int co = (int)(i % cout);
        const int ci = (int)((i / cout) % cin);
        const int tap = (int)(i / ((size_t)cout * cin));
        __nv_bfloat16 b = __float2bfloat16_rn(w[i]);
        const uint16_t bits = *reinterpret_cast<uint16_t*>(&b);
        // forward: [tap][ci/8][co][ci%8]
        fwd[(((size_t)tap * (cin / 8) + ci / 8) * cout + co) * 8 + ci % 8] = bits;
        // data gradient: tap' = 8 - tap, [tap'][co/8][ci][co%8]
        bwd[(((size_t)(8 - tap) * (cout / 8) + co / 8) * cin + ci) * 8 + co % 8] = bits;
    }
}

__global__ void k_adam(float* p, const float* g, float* m, float* v, size_t n, float lr, float b1, float b2, float eps, float bc1,
                       float bc2)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    }
}

unsigned grid_for(size_t n, int threads)
{
    size_t b = (n + threads - 1) / threads;
    if (b > 152 * 32)
        b = 152 * 32;
    return (unsigned)(b ? b : 1);
}

bool shape_ok(const Act& a, int c0, int c)
{
    return a.p && c > 0 && c % 8 == 0 && c0 % 8 == 0 && c0 + c <= a.pitch && a.pitch % 8 == 0;
}

// ... and for the kernels with 32-byte accesses.
bool shape_ok16(const Act& a, int c0, int c)
{
    return shape_ok(a, c0, c) && c % 16 == 0 && c0 % 16 == 0 && a.pitch % 16 == 0 && ((uintptr_t)a.p & 31) == 0;
}

dim3 low_grid(const Act& low, int units)
{
    const unsigned x = (unsigned)(((uint64_t)low.w * units + POOL_THREADS - 1) / POOL_THREADS);
    return dim3(x, (unsigned)std::min<uint64_t>((uint64_t)low.n * low.h, 65535));
}

} // namespace

cudaError_t pool2(const Act& in, int in_c0, int c, const Act& out, int out_c0, cudaStream_t st)
{
    if (!shape_ok16(in, in_c0, c) || !shape_ok16(out, out_c0, c) || in.h != 2 * out.h || in.w != 2 * out.w || in.n != out.n)
        return cudaErrorInvalidValue;
    k_pool2<<<low_grid(out, c / 16), POOL_THREADS, 0, st>>>(in, in_c0, c / 16, out, out_c0);
    return cudaGetLastError();
}

cudaError_t upsample2(const Act& in, int in_c0, int c, const Act& out, int out_c0, cudaStream_t st)
{
    if (!shape_ok16(in, in_c0, c) || !shape_ok16(out, out_c0, c) || out.h != 2 * in.h || out.w != 2 * in.w || in.n != out.n)
        return cudaErrorInvalidValue;
    k_upsample2<<<low_grid(in, c / 16), POOL_THREADS, 0, st>>>(in, in_c0, c / 16, out, out_c0);
    return cudaGetLastError();
}

cudaError_t upsample2_backward(const Act& g_high, int g_c0, int c, const Act& z, int z_c0, const Act& g_low, cudaStream_t st)
{
    if (!shape_ok16(g_high, g_c0, c) || !shape_ok16(z, z_c0, c) || !shape_ok16(g_low, 0, c) || g_high.h != 2 * g_low.h ||
        g_high.w != 2 * g_low.w || z.h != g_low.h || z.w != g_low.w)
        return cudaErrorInvalidValue;
    k_upsample2_backward<<<low_grid(g_low, c / 16), POOL_THREADS, 0, st>>>(g_high, g_c0, c / 16, z, z_c0, g_low);
    return cudaGetLastError();
}

cudaError_t pool2_backward(const Act& g_skip, int s_c0, const Act& g_pool, int c, const Act& z, int z_c0, const Act& g,
                           cudaStream_t st)
{
    if (!shape_ok16(g_skip, s_c0, c) || !shape_ok16(g_pool, 0, c) || !shape_ok16(z, z_c0, c) || !shape_ok16(g, 0, c) ||
        g.h != 2 * g_pool.h || g.w != 2 * g_pool.w || g_skip.h != g.h || z.h != g.h)
        return cudaErrorInvalidValue;
    k_pool2_backward<<<low_grid(g_pool, c / 16), POOL_THREADS, 0, st>>>(g_skip, s_c0, g_pool, c / 16, z, z_c0, g);
    return cudaGetLastError();
}

cudaError_t bias_grad(const Act& g, int c0, int c, float* db, cudaStream_t st)
{
    if (!shape_ok16(g, c0, c) || c > BIAS_THREADS)
        return cudaErrorInvalidValue;
    // four blocks per SM, and no block below 128 pixels: its reduction costs as much
    const size_t blocks = 152 * 4;
    size_t per = (g.pixels() + blocks - 1) / blocks;
    per = std::max<size_t>(per, 128);
    const size_t nb = (g.pixels() + per - 1) / per;
    if (nb == 0)
        return cudaSuccess;
    launch_chained(k_bias_grad, (unsigned)nb, BIAS_THREADS, 0, st, g, c0, c / 16, db, (uint32_t)per);
    return cudaGetLastError();
}

cudaError_t pack_weights(const float* w, int cin, int cout, uint16_t* fwd, uint16_t* bwd, cudaStream_t st)
{
    if (cin % 8 || cout % 8)
        return cudaErrorInvalidValue;
    k_pack_weights<<<grid_for((size_t)9 * cin * cout, 256), 256, 0, st>>>(w, cin, cout, fwd, bwd);
    return cudaGetLastError();
}

cudaError_t adam_step(float* p, const float* g, float* m, float* v, size_t n, float lr, float beta1, float beta2, float eps,
                      float bc1, float bc2, cudaStream_t st)
{
    k_adam<<<grid_for(n, 256), 256, 0, st>>>(p, g, m, v, n, lr, beta1, beta2, eps, bc1, bc2);
    return cudaGetLastError();
}

} // namespace nn
} // namespace pt
