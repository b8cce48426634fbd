// scene.cuh — device-side scene layout and two-level BVH traversal.
//
// HBM layout (one allocation per array, all 16-byte aligned):
//   vertices   float4 x 2 per vertex: the reference's 32-B Vertex (mesh.h:10-18)
//   indices    u32, mesh-local, 3 per triangle
//   instances  pt_instance_data, 128 B (scenebuffer.h:13-24)
//   materials  pt_material, 96 B (material.h:24-29)
//   light      u32 light-sampler stream (lightsample.cpp:89-221)
//   nodes      BvhNode, 64 B: both child boxes of a BVH2 node (one array for
//              every BLAS and the TLAS)
//   nodes4     Bvh4Node, 64 B (half-precision planes rounded outwards; two
//              nodes per cache line), same indices as `nodes`: node i's
//              grandchildren (a child that is a leaf stands for itself), so
//              the traversal descends two BVH2 levels per dependent fetch
//   tris       TriRec, 48 B: the three object-space vertices of a triangle in
//              BVH leaf order plus its mesh-local primitive index
//   dinst      DevInstance, 64 B: world-to-object rows + BLAS root reference
// Traversal reads nodes4 with 32-byte and nodes/tris/dinst with 16-byte vector
// loads through the read-only path.
#pragma once
#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "ptmath.cuh"
#include "slab.h"

namespace pt {

// Child / root reference: >= 0 interior node index; < 0 a leaf holding the
// primitives (first, count) encoded as ~((first << 2) | (count - 1)), with
// first < 2^28.  Three sentinels below the leaf range drive the traversal loop.
constexpr int REF_DONE = (int)0x80000000;
constexpr int REF_EXIT_BLAS = (int)0x80000001;
constexpr int REF_EMPTY = (int)0x80000002;
__host__ __device__ __forceinline__ bool ref_is_leaf(int r) { return r < 0 && r > (int)0x8000000F; }
__host__ __device__ __forceinline__ int make_leaf(uint32_t first, uint32_t count) { return ~(int)((first << 2) | (count - 1)); }
__host__ __device__ __forceinline__ uint32_t leaf_first(int r) { return ((uint32_t)~r) >> 2; }
__host__ __device__ __forceinline__ uint32_t leaf_count(int r) { return (((uint32_t)~r) & 3u) + 1u; }

struct __align__(16) BvhNode {
    float4 c0xy; // c0.lo.x, c0.hi.x, c0.lo.y, c0.hi.y
    float4 c1xy; // c1.lo.x, c1.hi.x, c1.lo.y, c1.hi.y
    float4 c01z; // c0.lo.z, c0.hi.z, c1.lo.z, c1.hi.z
    int4 link;   // child0, child1, -, -
};

// Four child boxes as x/y/z planes across the children (lane k = child k)
// and their references; REF_EMPTY marks an unused slot.
// Half-precision planes, rounded outwards from the BVH2's boxes (lower planes
// toward -inf, upper planes toward +inf), so each box contains the box it
// stands for; two nodes share a 128-byte line.  Per axis a uint4 holds
// (lo0, lo1), (lo2, lo3), (hi0, hi1), (hi2, hi3) as half2 pairs.
struct __align__(64) Bvh4Node {
    uint4 x, y, z;
    int4 link;
};

struct __align__(16) TriRec {
    float4 v0; // xyz, w = primitive index (bits)
    float4 v1;
    float4 v2;
};

struct __align__(16) DevInstance {
    float4 w2o[3];   // rows of the world-to-object 3x4 transform
    int blas_root;   // reference into nodes/tris (REF_EMPTY for an empty mesh)
    uint32_t flags;  // bit 0: opaque
    uint32_t mesh;
    uint32_t pad;
};

struct DevMaterial {
    float4 base_colour, emission, rmn, specular, sheen, cc;
};

struct DevInstanceData {
    uint32_t vertex_index, index_index, emitter_index, material_index;
    float4 t0, t1, t2, t3; // transform rows
    float4 n0, n1, n2;     // normal matrix rows
};

// pt_texture (include/pt_gpu.h): 8-bit texels, 1 / 2 / 4 channels.
struct DevTexture {
    unsigned long long offset;
    uint32_t width, height, channels, srgb;
};

struct DevScene {
    const float4* vertices;
    const uint32_t* indices;
    const DevInstanceData* inst_data;
    const DevMaterial* materials;
    const float* material_ior; // null, or per material: > 0 = smooth dielectric of that index
    const uint32_t* light;
    uint32_t light_words;
    uint32_t light_count;
    uint32_t instance_count;
    uint32_t vertex_count;
    uint32_t max_iterations; // traversal watchdog: loop iterations per ray
    const uint8_t* texels;   // textures (may be empty)
    const DevTexture* textures;
    uint32_t texture_count;
    const BvhNode* nodes;
    const Bvh4Node* nodes4; // null: traverse the BVH2 `nodes`
    const TriRec* tris;
    uint32_t node_count;  // entries of nodes (and nodes4)
    uint32_t tri_count;   // entries of tris
    uint32_t index_count; // entries of indices
    const DevInstance* dinst;
    int tlas_root;
    f3 env;
    uint32_t* error_word; // bit 0: traversal stack overflow
    uint32_t plain;       // 1: no material has a map bit, none refracts
};

constexpr uint32_t ERR_STACK_OVERFLOW = 1u;
constexpr uint32_t ERR_BAD_INDEX = 2u;
constexpr uint32_t ERR_WATCHDOG = 4u;

// Checked builds (-DPT_CHECKED, libptgpu_checked.so): every node, triangle,
// instance, vertex-index and queue index is compared with its array's length
// before it is used; a bad one sets ERR_BAD_INDEX and ends that ray or entry
// instead of reading outside the array (the stand-in for a memory checker).
#ifdef PT_CHECKED
#define PT_CHECK_INDEX(cond, s, on_fail)          \
    if (!(cond)) {                                \
        atomicOr((s).error_word, ERR_BAD_INDEX); \
        on_fail;                                  \
    }
#else
#define PT_CHECK_INDEX(cond, s, on_fail)
#endif

__device__ __forceinline__ float4 ldg4(const float4* p) { return __ldg(p); }
__device__ __forceinline__ int4 ldg4i(const int4* p) { return __ldg(p); }

// Material map bits (constants.h of the reference; include/pt_gpu.h).
constexpr uint32_t MAP_BASE_COLOUR = 1u << 0;
constexpr uint32_t MAP_EMISSION = 1u << 1;
constexpr uint32_t MAP_ROUGHNESS = 1u << 2;
constexpr uint32_t MAP_METALNESS = 1u << 3;
constexpr uint32_t MAP_ROUGHNESS_METALNESS = 1u << 4;
constexpr uint32_t MAP_SPECULAR = 1u << 5;
constexpr uint32_t MAP_SHEEN = 1u << 7;
constexpr uint32_t MAP_CLEARCOAT = 1u << 9;
constexpr uint32_t MAP_NORMAL = 1u << 12;

// sRGB-to-linear decode of 8-bit values (the _SRGB texture formats), filled
// from the host's FP64 evaluation of the sRGB curve (one copy per translation
// unit, uploaded by that unit's table initialiser).
static __constant__ float c_srgb[256];

__device__ __forceinline__ float4 texel(const DevScene& s, const DevTexture& t, uint32_t x, uint32_t y)
{
    const uint8_t* p = s.texels + t.offset + ((unsigned long long)y * t.width + x) * t.channels;
    if (t.channels == 4) {
        const uint8_t r = p[0], g = p[1], b = p[2], a = p[3]; // byte loads: texture offsets need no alignment
        if (t.srgb)
            return make_float4(c_srgb[r], c_srgb[g], c_srgb[b], (float)a / 255.0f);
        return make_float4((float)r / 255.0f, (float)g / 255.0f, (float)b / 255.0f, (float)a / 255.0f);
    }
    if (t.channels == 2)
        return make_float4((float)p[0] / 255.0f, (float)p[1] / 255.0f, 0.0f, 1.0f);
    return make_float4((float)p[0] / 255.0f, 0.0f, 0.0f, 1.0f);
}

// SampleLevel(uv, 0) with the reference's sampler (linear filtering, REPEAT,
// level 0; src/graphics/sampler.cpp:8-22): uv is wrapped to [0, 1), texel
// centres sit at (i + 0.5) / size, the four neighbours wrap, and the weights
// combine as (1-a)(1-b) t00 + a(1-b) t10 + (1-a)b t01 + ab t11 in that order.
// Out-of-range texture indices read zero.
__device__ __forceinline__ float4 sample_texture(const DevScene& s, uint32_t index, f2 uv)
{
    if (index >= s.texture_count)
        return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const DevTexture t = s.textures[index];
    float u = uv.x - floorf(uv.x), v = uv.y - floorf(uv.y);
    if (!(u >= 0.0f && u < 1.0f))
        u = 0.0f;
    if (!(v >= 0.0f && v < 1.0f))
        v = 0.0f;
    const float x = u * (float)t.width - 0.5f, y = v * (float)t.height - 0.5f;
    const float fx = floorf(x), fy = floorf(y);
    const float a = x - fx, b = y - fy;
    int x0 = (int)fx, y0 = (int)fy;
    if (x0 < 0)
        x0 += (int)t.width;
    if (y0 < 0)
        y0 += (int)t.height;
    if (x0 >= (int)t.width)
        x0 = (int)t.width - 1;
    if (y0 >= (int)t.height)
        y0 = (int)t.height - 1;
    const uint32_t x1 = (uint32_t)x0 + 1 == t.width ? 0u : (uint32_t)x0 + 1;
    const uint32_t y1 = (uint32_t)y0 + 1 == t.height ? 0u : (uint32_t)y0 + 1;
    const float4 t00 = texel(s, t, x0, y0), t10 = texel(s, t, x1, y0), t01 = texel(s, t, x0, y1), t11 = texel(s, t, x1, y1);
    const float w00 = (1.0f - a) * (1.0f - b), w10 = a * (1.0f - b), w01 = (1.0f - a) * b, w11 = a * b;
    return make_float4(((w00 * t00.x + w10 * t10.x) + w01 * t01.x) + w11 * t11.x,
                       ((w00 * t00.y + w10 * t10.y) + w01 * t01.y) + w11 * t11.y,
                       ((w00 * t00.z + w10 * t10.z) + w01 * t01.z) + w11 * t11.z,
                       ((w00 * t00.w + w10 * t10.w) + w01 * t01.w) + w11 * t11.w);
}

// Texture coordinate of a point of a triangle (get_vertex_attributes,
// geometry.hlsli:38-47); indices outside the vertex array read zero.
__device__ __forceinline__ f2 vertex_uv(const DevScene& s, unsigned long long i)
{
    if (i >= (unsigned long long)s.vertex_count)
        return f2{0.0f, 0.0f};
    const float4 b = __ldg(s.vertices + 2 * (size_t)i + 1);
    return f2{b.z, b.w};
}

__device__ __forceinline__ f2 hit_uv(const DevScene& s, uint32_t inst, uint32_t prim, float b1, float b2)
{
    const DevInstanceData* id = s.inst_data + inst;
    const uint32_t vbase = __ldg(&id->vertex_index), ibase = __ldg(&id->index_index);
    const f2 ua = vertex_uv(s, (unsigned long long)vbase + __ldg(s.indices + ibase + prim * 3 + 0));
    const f2 ub = vertex_uv(s, (unsigned long long)vbase + __ldg(s.indices + ibase + prim * 3 + 1));
    const f2 uc = vertex_uv(s, (unsigned long long)vbase + __ldg(s.indices + ibase + prim * 3 + 2));
    const float ba = (1.0f - b1) - b2;
    return f2{(ba * ua.x + b1 * ub.x) + b2 * uc.x, (ba * ua.y + b1 * ub.y) + b2 * uc.y};
}

// Light-stream word with robust-buffer-access semantics (out of range reads 0).
__device__ __forceinline__ uint32_t lw(const DevScene& s, uint32_t i) { return i < s.light_words ? __ldg(s.light + i) : 0u; }

struct Ray {
    f3 o, d;
};

struct ObjRay {
    f3 o, d;
    f3 inv_d, o_inv; // 1/d and o/d for the slab test
    uint32_t axes;   // SLAB_HI_*: the planes met first; AXIS_*: the permutation of the watertight test
    float sx, sy, sz;
};

// ObjRay::axes.  SLAB_HI_*: the upper plane of that slab is met first (slab.h).
constexpr uint32_t SLAB_HI_X = 1u, SLAB_HI_Y = 2u, SLAB_HI_Z = 4u;
constexpr uint32_t AXIS_X_IS_1 = 8u, AXIS_X_IS_2 = 16u, AXIS_Y_IS_1 = 32u, AXIS_Y_IS_2 = 64u, AXIS_Z_IS_1 = 128u, AXIS_Z_IS_2 = 256u;

// Shadow rays without an end lead to directional lights, and one along an axis
// makes every one of them a ray with zero components: they take the finite
// inverses (slab.h), without which they lost every node across a coordinate
// plane.  Any other ray has a component of exactly zero by chance only, about
// once in 10^8, and keeps 1 / d: of the mid scene at 1024 x 1024, 128 spp, two
// pixels would differ (they miss a hit that the oracle finds) and every ray and
// instance entry would pay for it (83.3 -> 84.6 ms).
__device__ __forceinline__ void setup_slab(ObjRay& r, bool endless)
{
    r.inv_d = mk3(1.0f / r.d.x, 1.0f / r.d.y, 1.0f / r.d.z);
    r.o_inv = mk3(r.o.x * r.inv_d.x, r.o.y * r.inv_d.y, r.o.z * r.inv_d.z);
    if (endless) {
        slab_finite(r.o.x, r.inv_d.x, r.o_inv.x);
        slab_finite(r.o.y, r.inv_d.y, r.o_inv.y);
        slab_finite(r.o.z, r.inv_d.z, r.o_inv.z);
    }
    r.axes = (slab_hi_first(__float_as_uint(r.inv_d.x)) ? SLAB_HI_X : 0u) | (slab_hi_first(__float_as_uint(r.inv_d.y)) ? SLAB_HI_Y : 0u) |
             (slab_hi_first(__float_as_uint(r.inv_d.z)) ? SLAB_HI_Z : 0u);
}

// Component of v along a permuted axis of the ray (is1, is2: its AXIS_ bits).
__device__ __forceinline__ float along(f3 v, uint32_t axes, uint32_t is1, uint32_t is2)
{
    return (axes & is2) ? v.z : (axes & is1) ? v.y : v.x;
}

__device__ __forceinline__ void setup_watertight(ObjRay& r)
{
    float ax = fabsf(r.d.x), ay = fabsf(r.d.y), az = fabsf(r.d.z);
    int kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    int kx = kz + 1;
    if (kx == 3)
        kx = 0;
    int ky = kx + 1;
    if (ky == 3)
        ky = 0;
    float dz = comp(r.d, kz);
    if (dz < 0.0f) {
        int t = kx;
        kx = ky;
        ky = t;
    }
    r.axes |= (kx == 1 ? AXIS_X_IS_1 : 0u) | (kx == 2 ? AXIS_X_IS_2 : 0u) | (ky == 1 ? AXIS_Y_IS_1 : 0u) |
              (ky == 2 ? AXIS_Y_IS_2 : 0u) | (kz == 1 ? AXIS_Z_IS_1 : 0u) | (kz == 2 ? AXIS_Z_IS_2 : 0u);
    r.sx = comp(r.d, kx) / dz;
    r.sy = comp(r.d, ky) / dz;
    r.sz = 1.0f / dz;
}

// Robust slab test (Ize 2013): far distances are scaled by 1 + 2*gamma(3).
// NaN distances (an infinite inverse of a zero direction component) are ignored
// by fminf / fmaxf; what that misses is said at setup_slab.
constexpr float SLAB_SCALE = 1.0f + 2.0f * (3.0f * 0x1p-24f) / (1.0f - 3.0f * 0x1p-24f);

__device__ __forceinline__ float slab_enter(float lo, float hi, float inv, float oinv, float& tfar)
{
    float t0 = fmaf(lo, inv, -oinv);
    float t1 = fmaf(hi, inv, -oinv);
    tfar = fmaxf(t0, t1) * SLAB_SCALE;
    return fminf(t0, t1);
}

// Intersect both children of a node; returns a bitmask (1 = c0, 2 = c1) and
// the entry distances.
__device__ __forceinline__ int node_children(const BvhNode* node, const ObjRay& r, float tmin, float tmax, float& e0, float& e1,
                                             int& c0, int& c1)
{
    float4 a = ldg4(&node->c0xy);
    float4 b = ldg4(&node->c1xy);
    float4 z = ldg4(&node->c01z);
    int4 l = ldg4i(&node->link);
    float f0x, f0y, f0z, f1x, f1y, f1z;
    float n0x = slab_enter(a.x, a.y, r.inv_d.x, r.o_inv.x, f0x);
    float n0y = slab_enter(a.z, a.w, r.inv_d.y, r.o_inv.y, f0y);
    float n0z = slab_enter(z.x, z.y, r.inv_d.z, r.o_inv.z, f0z);
    float n1x = slab_enter(b.x, b.y, r.inv_d.x, r.o_inv.x, f1x);
    float n1y = slab_enter(b.z, b.w, r.inv_d.y, r.o_inv.y, f1y);
    float n1z = slab_enter(z.z, z.w, r.inv_d.z, r.o_inv.z, f1z);
    e0 = fmaxf(fmaxf(fmaxf(n0x, n0y), n0z), tmin);
    float x0 = fminf(fminf(fminf(f0x, f0y), f0z), tmax);
    e1 = fmaxf(fmaxf(fmaxf(n1x, n1y), n1z), tmin);
    float x1 = fminf(fminf(fminf(f1x, f1y), f1z), tmax);
    c0 = l.x;
    c1 = l.y;
    return (e0 <= x0 ? 1 : 0) | (e1 <= x1 ? 2 : 0);
}

// Three-input minimum / maximum (PTX min/max.f32 with three operands on
// sm_100 and later): the same value as two nested fminf / fmaxf, NaN operands
// ignored likewise.
__device__ __forceinline__ float fmin3f(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmax3f(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// One axis of a half-precision 4-wide node: the planes of the four children
// that the ray meets first and last, as floats (exact: every half is a float).
__device__ __forceinline__ void unpack_planes(const uint4& q, bool hi_first, float4& first, float4& last)
{
    const uint32_t f0 = hi_first ? q.z : q.x, f1 = hi_first ? q.w : q.y, l0 = hi_first ? q.x : q.z, l1 = hi_first ? q.y : q.w;
    const float2 f01 = __half22float2(*reinterpret_cast<const __half2*>(&f0));
    const float2 f23 = __half22float2(*reinterpret_cast<const __half2*>(&f1));
    const float2 l01 = __half22float2(*reinterpret_cast<const __half2*>(&l0));
    const float2 l23 = __half22float2(*reinterpret_cast<const __half2*>(&l1));
    first = make_float4(f01.x, f01.y, f23.x, f23.y);
    last = make_float4(l01.x, l01.y, l23.x, l23.y);
}

// A 4-wide node by two 32-byte loads (sm_100 and later).  ptxas of CUDA 13.0
// crashes on them in the megakernel's out-of-line traversal, whose translation
// unit defines PT_NARROW_NODE_LOADS.  Heavy scene: 28.9 -> 28.4 ms of extend,
// the mid scene unchanged.
__device__ __forceinline__ void load_node4(const Bvh4Node* node, uint4& qx, uint4& qy, uint4& qz, int4& l)
{
#ifdef PT_NARROW_NODE_LOADS
    qx = __ldg(&node->x);
    qy = __ldg(&node->y);
    qz = __ldg(&node->z);
    l = ldg4i(&node->link);
#else
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(qx.x), "=r"(qx.y), "=r"(qx.z), "=r"(qx.w), "=r"(qy.x), "=r"(qy.y), "=r"(qy.z), "=r"(qy.w)
        : "l"(&node->x));
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(qz.x), "=r"(qz.y), "=r"(qz.z), "=r"(qz.w), "=r"(l.x), "=r"(l.y), "=r"(l.z), "=r"(l.w)
        : "l"(&node->z));
#endif
}

// Intersect the four child boxes of a 4-wide node; bit k of the result is
// set when child k is hit, e[k] its entry distance.  The boxes contain the
// BVH2's (outward rounding), so a child the BVH2 would enter is entered here
// too and the closest hit is the same.  The ray's direction signs say which
// plane of a slab is met first, so that entry and exit take one distance each
// (a select per packed pair of planes) instead of the minimum and maximum of
// both: the kernel is bound by its issue slots (70 % busy, the pipe that
// selects and compares 50 %), and with this and the unused slots below the
// extend stage of the mid scene at 1024 x 1024, 128 spp went from 69.7 to
// 58.7 ms, on the heavy scene at 1920 x 1080, 4 spp from 28.9 to 24.5.  The
// multiply-adds as packed pairs (fma.rn.f32x2) gained nothing (59.3 ms).  The exit distance is
// scaled once after the minimum over the axes instead of once per axis:
// rounding is monotonic, so min(a s, b s, c s) = min(a, b, c) s for s > 0.
// An unused slot (REF_EMPTY) has planes that no finite ray meets
// (k_make_bvh4); a ray that enters it all the same finds nothing there.
__device__ __forceinline__ int node4_children(const Bvh4Node* node, const ObjRay& r, float tmin, float tmax, float (&e)[4], int (&c)[4])
{
    uint4 qx, qy, qz;
    int4 l;
    load_node4(node, qx, qy, qz, l);
    float4 nx, fx, ny, fy, nz, fz;
    unpack_planes(qx, (r.axes & SLAB_HI_X) != 0, nx, fx);
    unpack_planes(qy, (r.axes & SLAB_HI_Y) != 0, ny, fy);
    unpack_planes(qz, (r.axes & SLAB_HI_Z) != 0, nz, fz);
    c[0] = l.x;
    c[1] = l.y;
    c[2] = l.z;
    c[3] = l.w;
    int m = 0;
#define PT_NODE4_CHILD(k, q)                                                                                                  \
    {                                                                                                                         \
        const float x0 = fmaf(nx.q, r.inv_d.x, -r.o_inv.x), x1 = fmaf(fx.q, r.inv_d.x, -r.o_inv.x);                           \
        const float y0 = fmaf(ny.q, r.inv_d.y, -r.o_inv.y), y1 = fmaf(fy.q, r.inv_d.y, -r.o_inv.y);                           \
        const float z0 = fmaf(nz.q, r.inv_d.z, -r.o_inv.z), z1 = fmaf(fz.q, r.inv_d.z, -r.o_inv.z);                           \
        e[k] = fmaxf(fmax3f(x0, y0, z0), tmin);                                                                               \
        const float far = fmin3f(x1, y1, z1) * SLAB_SCALE;                                                                    \
        m |= e[k] <= fminf(far, tmax) ? (1 << k) : 0;                                                                         \
    }
    PT_NODE4_CHILD(0, x)
    PT_NODE4_CHILD(1, y)
    PT_NODE4_CHILD(2, z)
    PT_NODE4_CHILD(3, w)
#undef PT_NODE4_CHILD
    return m;
}

constexpr int STACK_SIZE = 96;

// One interior step of a 4-wide traversal: the nearest hit child becomes
// `ref`, the others are pushed far to near (SORT; else in slot order, for
// any-hit queries whose result does not depend on the order).  Returns false
// when no child was hit (the caller pops).  A push that would overflow sets
// ERR_STACK_OVERFLOW and drops those children.
// All lanes with a hit go the same way, whatever their number of hits: a way of
// its own for one hit, and a loop over the other hits of an any-hit step, cost a
// warp both ways on nearly every step (mid scene at 1024 x 1024, 128 spp, extend
// 48.4 -> 47.5 ms, shadow rays 16.6 -> 15.1; heavy scene at 1920 x 1080, 4 spp
// 18.9 -> 18.4 and 8.9 -> 8.1).
template <bool SORT, class Stack>
__device__ __forceinline__ bool step4(const DevScene& s, const ObjRay& r, float tmin, float tmax, int& ref, Stack& stack, int& sp)
{
    float e[4];
    int c[4];
    const int m = node4_children(s.nodes4 + ref, r, tmin, tmax, e, c);
    const int cnt = __popc(m);
    if (!SORT) {
        ref = (m & 1) ? c[0] : (m & 2) ? c[1] : (m & 4) ? c[2] : c[3];
        if (sp + cnt - 1 > STACK_SIZE) {
            atomicOr(s.error_word, ERR_STACK_OVERFLOW);
            return true;
        }
        if ((m & 2) && (m & 1))
            stack.set(sp++, c[1]);
        if ((m & 4) && (m & 3))
            stack.set(sp++, c[2]);
        if ((m & 8) && (m & 7))
            stack.set(sp++, c[3]);
        return cnt != 0;
    }
    if (cnt == 0)
        return false;
    // sort (entry, child) ascending with misses keyed +inf: a five-exchange network
    const float inf = __int_as_float(0x7f800000);
    float k0 = (m & 1) ? e[0] : inf, k1 = (m & 2) ? e[1] : inf, k2 = (m & 4) ? e[2] : inf, k3 = (m & 8) ? e[3] : inf;
    int r0 = c[0], r1 = c[1], r2 = c[2], r3 = c[3];
#define PT_CSWAP(ka, ra, kb, rb)  \
    if (kb < ka) {                \
        const float tk = ka;      \
        ka = kb;                  \
        kb = tk;                  \
        const int tr = ra;        \
        ra = rb;                  \
        rb = tr;                  \
    }
    PT_CSWAP(k0, r0, k1, r1)
    PT_CSWAP(k2, r2, k3, r3)
    PT_CSWAP(k0, r0, k2, r2)
    PT_CSWAP(k1, r1, k3, r3)
    PT_CSWAP(k1, r1, k2, r2)
#undef PT_CSWAP
    if (sp + cnt - 1 > STACK_SIZE) {
        atomicOr(s.error_word, ERR_STACK_OVERFLOW);
    } else {
        if (cnt == 4)
            stack.set(sp++, r3);
        if (cnt >= 3)
            stack.set(sp++, r2);
        if (cnt >= 2)
            stack.set(sp++, r1);
    }
    ref = r0;
    return true;
}

// Watertight ray/triangle test (Woop, Benthin & Wald 2013) without culling.
__device__ __forceinline__ bool watertight(const ObjRay& r, f3 p0, f3 p1, f3 p2, float& t, float& b1, float& b2)
{
    f3 A = p0 - r.o, B = p1 - r.o, C = p2 - r.o;
    float Akx = along(A, r.axes, AXIS_X_IS_1, AXIS_X_IS_2), Aky = along(A, r.axes, AXIS_Y_IS_1, AXIS_Y_IS_2);
    float Akz = along(A, r.axes, AXIS_Z_IS_1, AXIS_Z_IS_2);
    float Bkx = along(B, r.axes, AXIS_X_IS_1, AXIS_X_IS_2), Bky = along(B, r.axes, AXIS_Y_IS_1, AXIS_Y_IS_2);
    float Bkz = along(B, r.axes, AXIS_Z_IS_1, AXIS_Z_IS_2);
    float Ckx = along(C, r.axes, AXIS_X_IS_1, AXIS_X_IS_2), Cky = along(C, r.axes, AXIS_Y_IS_1, AXIS_Y_IS_2);
    float Ckz = along(C, r.axes, AXIS_Z_IS_1, AXIS_Z_IS_2);
    float Ax = Akx - r.sx * Akz, Ay = Aky - r.sy * Akz;
    float Bx = Bkx - r.sx * Bkz, By = Bky - r.sy * Bkz;
    float Cx = Ckx - r.sx * Ckz, Cy = Cky - r.sy * Ckz;
    float U = Cx * By - Cy * Bx;
    float V = Ax * Cy - Ay * Cx;
    float W = Bx * Ay - By * Ax;
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
        V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
        W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f))
        return false;
    float det = (U + V) + W;
    if (det == 0.0f)
        return false;
    float Az = r.sz * Akz, Bz = r.sz * Bkz, Cz = r.sz * Ckz;
    float T = (U * Az + V * Bz) + W * Cz;
    float inv = 1.0f / det;
    t = T * inv;
    b1 = V * inv;
    b2 = W * inv;
    return true;
}

__device__ __forceinline__ void to_object(const DevInstance* di, f3 o, f3 d, ObjRay& r, bool endless)
{
    float4 w0 = ldg4(&di->w2o[0]), w1 = ldg4(&di->w2o[1]), w2 = ldg4(&di->w2o[2]);
    r.o = mk3(((w0.x * o.x + w0.y * o.y) + w0.z * o.z) + w0.w, ((w1.x * o.x + w1.y * o.y) + w1.z * o.z) + w1.w,
              ((w2.x * o.x + w2.y * o.y) + w2.z * o.z) + w2.w);
    r.d = mk3((w0.x * d.x + w0.y * d.y) + w0.z * d.z, (w1.x * d.x + w1.y * d.y) + w1.z * d.z, (w2.x * d.x + w2.y * d.y) + w2.z * d.z);
    setup_slab(r, endless);
    setup_watertight(r);
}

struct Hit {
    float t, b1, b2;
    uint32_t inst, prim;
};

// Traversal work of one ray: interior nodes whose child boxes were tested and
// ray/triangle tests.
struct TraceCounters {
    uint32_t nodes, tris;
};

__device__ __forceinline__ bool better(float t, uint32_t inst, uint32_t prim, const Hit& h)
{
    if (t < h.t)
        return true;
    if (t > h.t)
        return false;
    return inst < h.inst || (inst == h.inst && prim < h.prim);
}


// BVH2 interior step: the nearer hit child becomes `ref`, the farther is
// pushed; false when nothing is hit (the caller pops).
template <class Stack>
__device__ __forceinline__ bool step2(const DevScene& s, const ObjRay& r, float tmin, float tmax, int& ref, Stack& stack, int& sp)
{
    float e0, e1;
    int c0, c1;
    const int m = node_children(s.nodes + ref, r, tmin, tmax, e0, e1, c0, c1);
    if (m == 0)
        return false;
    if (m == 3) {
        const bool swap = e1 < e0;
        if (sp < STACK_SIZE)
            stack.set(sp++, swap ? c0 : c1);
        else
            atomicOr(s.error_word, ERR_STACK_OVERFLOW);
        ref = swap ? c1 : c0;
    } else {
        ref = m == 1 ? c0 : c1;
    }
    return true;
}

// Closest-hit traversal of one ray as a resumable state: closest_begin sets
// it up and each closest_step advances it by one node visit, leaf or
// instance entry, returning true when the ray is finished.  The hit is
// the (t, instance, primitive) minimum of the oracle whatever the BVH.  The
// stack lives in local memory (L1-resident).  W4 walks the 4-wide nodes
// (s.nodes4, which must be present), else the BVH2.
struct ClosestTrace {
    ObjRay world, r;
    Hit h;
    float tmin;
    int ref, sp;
    uint32_t cur_inst, iter;
    bool in_blas, found;
};
// The traversal stack is kept apart from the state: inside the state it
// would pull every field of the state into local memory with it.  Measured
// against it on the mid scene: its top staged in shared memory (extend 72.0 ->
// 77.9 ms with 8 entries, 78.6 with 16: the per-access branch and the smaller
// L1 cost more than the bank-parallel accesses save), and entries that carry
// the child's entry distance, so that a pop can drop what lies beyond the best
// hit (9 % fewer node visits, but every access twice as wide: extend 69.7 ->
// 71.9 ms, on the heavy scene 28.9 -> 32.8).
struct TraceStack {
    int loc[STACK_SIZE];
    __device__ __forceinline__ int get(int i) const { return loc[i]; }
    __device__ __forceinline__ void set(int i, int v) { loc[i] = v; }
};

__device__ __forceinline__ void closest_begin(const DevScene& s, f3 o, f3 d, float tmin, float tmax, ClosestTrace& t, TraceStack& stack)
{
    t.h.t = tmax;
    t.h.inst = 0xFFFFFFFFu;
    t.h.prim = 0xFFFFFFFFu;
    t.h.b1 = t.h.b2 = 0.0f;
    t.found = false;
    t.world.o = o;
    t.world.d = d;
    setup_slab(t.world, false);
    t.r = t.world;
    t.tmin = tmin;
    t.sp = 0;
    stack.set(t.sp++, REF_DONE);
    t.ref = s.tlas_root == REF_EMPTY ? REF_DONE : s.tlas_root;
    t.in_blas = false;
    t.cur_inst = 0;
    t.iter = 0;
}

// Ends a traversal at the next pop (the bottom of the stack is REF_DONE).
__device__ __forceinline__ bool end_trace(int& sp)
{
    sp = 1;
    return true;
}

// Pops the next reference of a ray; leaving an instance restores the world
// ray on the way.  True when the stack is exhausted.
template <class Trace>
__device__ __forceinline__ bool pop_ref(Trace& t, const TraceStack& stack)
{
    t.ref = stack.get(--t.sp);
    if (t.ref == REF_EXIT_BLAS) { // never two in a row: instances are entered from the TLAS only
        t.r = t.world;
        t.in_blas = false;
        t.ref = stack.get(--t.sp);
    }
    return t.ref == REF_DONE;
}

// The node step of closest_step (t.ref >= 0); true when the ray must pop.
template <bool W4>
__device__ __forceinline__ bool closest_node(const DevScene& s, ClosestTrace& t, TraceStack& stack, TraceCounters& tc)
{
    PT_CHECK_INDEX((uint32_t)t.ref < s.node_count, s, return end_trace(t.sp))
    tc.nodes++;
    return !(W4 ? step4<true>(s, t.r, t.tmin, t.h.t, t.ref, stack, t.sp) : step2(s, t.r, t.tmin, t.h.t, t.ref, stack, t.sp));
}

// The leaf step of closest_step (t.ref < 0), an instance entry or triangles;
// true when the ray must pop.
__device__ __forceinline__ bool closest_leaf(const DevScene& s, ClosestTrace& t, TraceStack& stack, TraceCounters& tc)
{
    const int ref = t.ref;
    if (ref == REF_DONE) // an empty scene
        return end_trace(t.sp);
    if (ref == REF_EMPTY) // an unused slot of a 4-wide node, met by a NaN ray
        return true;
    const uint32_t first = leaf_first(ref), count = leaf_count(ref);
    if (!t.in_blas) {
        // TLAS leaf: instances [first, first + count); one per leaf here.
        PT_CHECK_INDEX(first < s.instance_count, s, return end_trace(t.sp))
        t.cur_inst = first;
        const DevInstance* di = s.dinst + first;
        const int root = __ldg(&di->blas_root);
        if (root == REF_EMPTY || count != 1)
            return true;
        if (t.sp >= STACK_SIZE) {
            atomicOr(s.error_word, ERR_STACK_OVERFLOW);
            return true;
        }
        to_object(di, t.world.o, t.world.d, t.r, false);
        stack.set(t.sp++, REF_EXIT_BLAS);
        t.in_blas = true;
        t.ref = root;
        return false;
    }
    PT_CHECK_INDEX((uint64_t)first + count <= s.tri_count, s, return end_trace(t.sp))
    tc.tris += count;
    for (uint32_t k = 0; k < count; k++) {
        const TriRec* tr = s.tris + first + k;
        const float4 a = ldg4(&tr->v0), b = ldg4(&tr->v1), c = ldg4(&tr->v2);
        float tt, b1, b2;
        const uint32_t prim = __float_as_uint(a.w);
        if (watertight(t.r, mk3(a.x, a.y, a.z), mk3(b.x, b.y, b.z), mk3(c.x, c.y, c.z), tt, b1, b2) && tt >= t.tmin &&
            tt <= t.h.t && better(tt, t.cur_inst, prim, t.h)) {
            t.h.t = tt;
            t.h.b1 = b1;
            t.h.b2 = b2;
            t.h.inst = t.cur_inst;
            t.h.prim = prim;
            t.found = true;
        }
    }
    return true;
}

// The watchdog of a traversal step: a well-formed BVH never gets there; a
// malformed one must not hang the GPU.
__device__ __forceinline__ bool out_of_steps(const DevScene& s, uint32_t& iter)
{
    if (iter >= s.max_iterations) {
        atomicOr(s.error_word, ERR_WATCHDOG);
        return true;
    }
    iter++;
    return false;
}

template <bool W4>
__device__ __forceinline__ bool closest_step(const DevScene& s, ClosestTrace& t, TraceStack& stack, TraceCounters& tc)
{
    if (out_of_steps(s, t.iter))
        return true;
    const bool pop = t.ref >= 0 ? closest_node<W4>(s, t, stack, tc) : closest_leaf(s, t, stack, tc);
    return pop && pop_ref(t, stack); // one copy of the pop: node and leaf lanes pop together
}

// A closest-hit traversal paused after a step budget (its "parking"): what a
// later pass needs to continue it exactly where it stopped.  The world ray is
// rebuilt from the path state and the object-space ray from the instance, so
// a slot holds the node reference, the stack, the instance, the step count and
// the best hit so far; slots are SoA arrays of `cap` entries, the stack
// word-major (stack[k * cap + slot]) so a warp's loads and stores coalesce.
constexpr int PARK_STACK = 32; // deeper stacks finish in the first pass

struct TraceParking {
    uint32_t* path;  // the path of each slot
    int4* state;     // ref, sp | in_blas << 16 | found << 17, cur_inst, iter
    float4* hit;     // t, b1, b2, bits(inst)
    uint32_t* prim;  // primitive of the best hit
    int* stack;      // PARK_STACK words per slot, word-major
    uint32_t cap;    // slots
};

__device__ __forceinline__ void park_closest(const TraceParking& pk, uint32_t slot, uint32_t path, const ClosestTrace& t,
                                             const TraceStack& stack)
{
    pk.path[slot] = path;
    pk.state[slot] = make_int4(t.ref, t.sp | (t.in_blas ? 1 << 16 : 0) | (t.found ? 1 << 17 : 0), (int)t.cur_inst, (int)t.iter);
    pk.hit[slot] = make_float4(t.h.t, t.h.b1, t.h.b2, __uint_as_float(t.h.inst));
    pk.prim[slot] = t.h.prim;
    for (int k = 0; k < t.sp; k++)
        pk.stack[(size_t)k * pk.cap + slot] = stack.get(k);
}

// Restores a parked traversal of the ray (o, d, tmin): the same state the
// first pass left, so closest_step continues the same sequence of steps.
__device__ __forceinline__ void resume_closest(const DevScene& s, const TraceParking& pk, uint32_t slot, f3 o, f3 d, float tmin,
                                               ClosestTrace& t, TraceStack& stack)
{
    const int4 st = pk.state[slot];
    const float4 h = pk.hit[slot];
    t.world.o = o;
    t.world.d = d;
    setup_slab(t.world, false);
    t.tmin = tmin;
    t.ref = st.x;
    t.sp = st.y & 0xFFFF;
    t.in_blas = (st.y >> 16) & 1;
    t.found = (st.y >> 17) & 1;
    t.cur_inst = (uint32_t)st.z;
    t.iter = (uint32_t)st.w;
    t.h.t = h.x;
    t.h.b1 = h.y;
    t.h.b2 = h.z;
    t.h.inst = __float_as_uint(h.w);
    t.h.prim = pk.prim[slot];
    if (t.in_blas)
        to_object(s.dinst + t.cur_inst, t.world.o, t.world.d, t.r, false);
    else
        t.r = t.world;
    for (int k = 0; k < t.sp; k++)
        stack.set(k, pk.stack[(size_t)k * pk.cap + slot]);
}

// Closest hit of one ray, traversed to the end.  Returns true on a hit.
template <bool W4>
static __device__ __forceinline__ bool trace_closest_inl(const DevScene& s, f3 o, f3 d, float tmin, float tmax, Hit& h, TraceCounters& tc)
{
    ClosestTrace t;
    TraceStack stack;
    closest_begin(s, o, d, tmin, tmax, t, stack);
    while (!closest_step<W4>(s, t, stack, tc)) {
    }
    h = t.h;
    return t.found;
}

// Closest hit as trace_closest_inl, traversed "while-while" with speculative
// leaves (Aila & Laine 2009): a lane that reaches a BLAS leaf parks it and
// keeps descending interior nodes until every converged lane of the warp holds
// a parked leaf (or has none left), then the warp tests triangles together.
// Instance entry and exit happen in the node phase, but only with no leaf
// parked (a parked leaf belongs to the current instance's object-space ray).
// The hit is the same (t, instance, primitive) minimum: triangles are only
// tested later, never skipped, and culling compares against the best t so far.
static __device__ __forceinline__ bool trace_closest_ww(const DevScene& s, f3 o, f3 d, float tmin, float tmax, Hit& h,
                                                        TraceCounters& tc)
{
    uint32_t n_nodes = 0, n_tris = 0;
    h.t = tmax;
    h.inst = 0xFFFFFFFFu;
    h.prim = 0xFFFFFFFFu;
    h.b1 = h.b2 = 0.0f;
    bool found = false;
    ObjRay world;
    world.o = o;
    world.d = d;
    setup_slab(world, false);
    ObjRay r = world;
    int stack[STACK_SIZE];
    int sp = 0;
    stack[sp++] = REF_DONE;
    int ref = s.tlas_root;
    bool in_blas = false;
    uint32_t cur_inst = 0;
    if (ref == REF_EMPTY)
        return false;
    int leaf = REF_EMPTY; // parked BLAS leaf (REF_EMPTY: none)
    uint32_t iter = 0;
    for (;;) {
        // node phase
        while (ref != REF_DONE) {
            if (++iter >= s.max_iterations)
                break;
            if (ref >= 0) {
                float e0, e1;
                int c0, c1;
                n_nodes++;
                int m = node_children(s.nodes + ref, r, tmin, h.t, e0, e1, c0, c1);
                if (m == 3) {
                    int near = c0, far = c1;
                    if (e1 < e0) {
                        near = c1;
                        far = c0;
                    }
                    if (sp < STACK_SIZE)
                        stack[sp++] = far;
                    else
                        atomicOr(s.error_word, ERR_STACK_OVERFLOW);
                    ref = near;
                } else if (m == 1) {
                    ref = c0;
                } else if (m == 2) {
                    ref = c1;
                } else {
                    ref = stack[--sp];
                }
            } else if (ref == REF_EXIT_BLAS) {
                if (leaf != REF_EMPTY)
                    break;
                r = world;
                in_blas = false;
                ref = stack[--sp];
            } else if (!in_blas) {
                // TLAS leaf: instances [first, first + count); one per leaf here.
                const uint32_t first = leaf_first(ref), count = leaf_count(ref);
                const DevInstance* di = s.dinst + first;
                const int root = __ldg(&di->blas_root);
                if (root == REF_EMPTY || count != 1 || sp >= STACK_SIZE) {
                    if (sp >= STACK_SIZE)
                        atomicOr(s.error_word, ERR_STACK_OVERFLOW);
                    ref = stack[--sp];
                } else {
                    cur_inst = first;
                    to_object(di, o, d, r, false);
                    stack[sp++] = REF_EXIT_BLAS;
                    in_blas = true;
                    ref = root;
                }
            } else {
                if (leaf != REF_EMPTY)
                    break;
                leaf = ref;
                ref = stack[--sp];
            }
            if (!__any_sync(__activemask(), leaf == REF_EMPTY))
                break;
        }
        if (iter >= s.max_iterations) {
            // A well-formed BVH never gets here; a malformed one must not hang the GPU.
            atomicOr(s.error_word, ERR_WATCHDOG);
            break;
        }
        // leaf phase
        if (leaf != REF_EMPTY) {
            const uint32_t first = leaf_first(leaf), count = leaf_count(leaf);
            n_tris += count;
            for (uint32_t k = 0; k < count; k++) {
                const TriRec* tr = s.tris + first + k;
                float4 a = ldg4(&tr->v0), b = ldg4(&tr->v1), c = ldg4(&tr->v2);
                float t, b1, b2;
                uint32_t prim = __float_as_uint(a.w);
                if (watertight(r, mk3(a.x, a.y, a.z), mk3(b.x, b.y, b.z), mk3(c.x, c.y, c.z), t, b1, b2) && t >= tmin && t <= h.t &&
                    better(t, cur_inst, prim, h)) {
                    h.t = t;
                    h.b1 = b1;
                    h.b2 = b2;
                    h.inst = cur_inst;
                    h.prim = prim;
                    found = true;
                }
            }
            leaf = REF_EMPTY;
        } else if (ref == REF_DONE) {
            break;
        }
    }
    tc.nodes += n_nodes;
    tc.tris += n_tris;
    return found;
}

// Shadow ray of shadowray.ah.hlsl / shadowray.ms.hlsl: the first opaque hit in
// [tmin, tmax] occludes; transparent instances attenuate by (1 - alpha).
// Returns the visibility throughput (0 = occluded).
// Any-hit shadow traversal of one ray as a resumable state (shadowray.ah.hlsl:
// 12-40): opaque hits end it with visibility 0, transparent instances scale
// the throughput by 1 - alpha and it ends occluded below 1e-5.
struct ShadowTrace {
    ObjRay world, r;
    float tmin, tmax, throughput, alpha_pass;
    int ref, sp;
    uint32_t iter, alpha_tex, alpha_inst, inst;
    bool in_blas, opaque, alpha_map; // alpha_map: the transparent instance's alpha comes from a base colour map
};

// A shadow ray to a directional light (setup_slab).
__device__ __forceinline__ bool endless(float tmax) { return tmax > 3.402823466e38f; }

__device__ __forceinline__ void shadow_begin(const DevScene& s, f3 o, f3 d, float tmin, float tmax, ShadowTrace& t, TraceStack& stack)
{
    t.world.o = o;
    t.world.d = d;
    setup_slab(t.world, endless(tmax));
    t.r = t.world;
    t.tmin = tmin;
    t.tmax = tmax;
    t.sp = 0;
    stack.set(t.sp++, REF_DONE);
    t.ref = s.tlas_root == REF_EMPTY ? REF_DONE : s.tlas_root;
    t.in_blas = false;
    t.opaque = true;
    t.alpha_map = false;
    t.alpha_tex = t.alpha_inst = t.inst = 0;
    t.alpha_pass = 1.0f;
    t.throughput = 1.0f;
    t.iter = 0;
}

// Visibility of a finished shadow ray.
__device__ __forceinline__ float shadow_result(const ShadowTrace& t) { return t.throughput < 1e-5f ? 0.0f : t.throughput; }

// The node step of shadow_step (t.ref >= 0).
template <bool W4>
__device__ __forceinline__ bool shadow_node(const DevScene& s, ShadowTrace& t, TraceStack& stack, TraceCounters& tc)
{
    PT_CHECK_INDEX((uint32_t)t.ref < s.node_count, s, return end_trace(t.sp))
    tc.nodes++;
    return !(W4 ? step4<false>(s, t.r, t.tmin, t.tmax, t.ref, stack, t.sp) : step2(s, t.r, t.tmin, t.tmax, t.ref, stack, t.sp));
}

// The leaf step of shadow_step (t.ref < 0): an instance entry or triangles.
__device__ __forceinline__ bool shadow_leaf(const DevScene& s, ShadowTrace& t, TraceStack& stack, TraceCounters& tc)
{
    const int ref = t.ref;
    if (ref == REF_DONE) // an empty scene
        return end_trace(t.sp);
    if (ref == REF_EMPTY) // an unused slot of a 4-wide node, met by a NaN ray
        return true;
    const uint32_t first = leaf_first(ref), count = leaf_count(ref);
    if (!t.in_blas) {
        PT_CHECK_INDEX(first < s.instance_count, s, return end_trace(t.sp))
        const DevInstance* di = s.dinst + first;
        const int root = __ldg(&di->blas_root);
        if (root == REF_EMPTY || count != 1)
            return true;
        const uint32_t flags = __ldg(&di->flags);
        t.inst = first;
        t.opaque = (flags & 1u) != 0;
        if (!t.opaque) {
            const uint32_t mi = __ldg(&s.inst_data[first].material_index);
            t.alpha_map = (__float_as_uint(__ldg(&s.materials[mi].rmn.w)) & MAP_BASE_COLOUR) != 0;
            t.alpha_tex = __float_as_uint(__ldg(&s.materials[mi].base_colour.x));
            t.alpha_inst = first;
            t.alpha_pass = 1.0f - __ldg(&s.materials[mi].base_colour.w);
        }
        if (t.sp >= STACK_SIZE) {
            atomicOr(s.error_word, ERR_STACK_OVERFLOW);
            return true;
        }
        to_object(di, t.world.o, t.world.d, t.r, endless(t.tmax));
        stack.set(t.sp++, REF_EXIT_BLAS);
        t.in_blas = true;
        t.ref = root;
        return false;
    }
    PT_CHECK_INDEX((uint64_t)first + count <= s.tri_count, s, return end_trace(t.sp))
    tc.tris += count;
    for (uint32_t k = 0; k < count; k++) {
        const TriRec* tr = s.tris + first + k;
        const float4 a = ldg4(&tr->v0), b = ldg4(&tr->v1), c = ldg4(&tr->v2);
        float tt, b1, b2;
        if (watertight(t.r, mk3(a.x, a.y, a.z), mk3(b.x, b.y, b.z), mk3(c.x, c.y, c.z), tt, b1, b2) && tt >= t.tmin &&
            tt <= t.tmax) {
            if (t.opaque) {
                t.throughput = 0.0f;
                break;
            }
            // shadowray.ah.hlsl:29-34: throughput *= 1 - base colour alpha at the hit
            if (t.alpha_map)
                t.alpha_pass = 1.0f - sample_texture(s, t.alpha_tex, hit_uv(s, t.alpha_inst, __float_as_uint(a.w), b1, b2)).w;
            t.throughput *= t.alpha_pass;
            if (t.throughput < 1e-5f)
                break;
        }
    }
    if (t.throughput < 1e-5f)
        t.sp = 1; // occluded: the next pop ends the ray
    return true;
}

template <bool W4>
__device__ __forceinline__ bool shadow_step(const DevScene& s, ShadowTrace& t, TraceStack& stack, TraceCounters& tc)
{
    if (out_of_steps(s, t.iter))
        return true;
    const bool pop = t.ref >= 0 ? shadow_node<W4>(s, t, stack, tc) : shadow_leaf(s, t, stack, tc);
    return pop && pop_ref(t, stack);
}

// One step of a whole warp's traversals: the lanes whose ray is at a node and
// those at a leaf wait for one another, and the larger group steps.  Stepping
// both groups in turn costs a warp the instructions of both on nearly every
// iteration (a ray has about six node steps to each leaf step, so some lane is
// nearly always at a leaf): on the mid scene at 1024 x 1024, 128 spp extend
// went from 79.1 to 69.7 ms and on the heavy scene at 1920 x 1080, 4 spp from
// 32.4 to 28.9; letting the leaves go at half or only at twice as many lanes
// was 2-7 % slower.  Each
// ray goes through the same steps as alone.  Called by all lanes of a warp
// (`live`: the lane has an unfinished ray); true for a lane whose ray ends.
__device__ __forceinline__ bool leaves_step(bool live, int ref)
{
    const unsigned nodes = __ballot_sync(0xffffffffu, live && ref >= 0), leaves = __ballot_sync(0xffffffffu, live && ref < 0);
    return __popc(leaves) >= __popc(nodes);
}

template <bool W4>
__device__ __forceinline__ bool closest_step_warp(const DevScene& s, bool live, ClosestTrace& t, TraceStack& stack, TraceCounters& tc)
{
    bool pop = false;
    if (leaves_step(live, t.ref)) {
        if (live && t.ref < 0)
            pop = out_of_steps(s, t.iter) ? end_trace(t.sp) : closest_leaf(s, t, stack, tc);
    } else if (live && t.ref >= 0) {
        pop = out_of_steps(s, t.iter) ? end_trace(t.sp) : closest_node<W4>(s, t, stack, tc);
    }
    return pop && pop_ref(t, stack);
}

template <bool W4>
__device__ __forceinline__ bool shadow_step_warp(const DevScene& s, bool live, ShadowTrace& t, TraceStack& stack, TraceCounters& tc)
{
    bool pop = false;
    if (leaves_step(live, t.ref)) {
        if (live && t.ref < 0)
            pop = out_of_steps(s, t.iter) ? end_trace(t.sp) : shadow_leaf(s, t, stack, tc);
    } else if (live && t.ref >= 0) {
        pop = out_of_steps(s, t.iter) ? end_trace(t.sp) : shadow_node<W4>(s, t, stack, tc);
    }
    return pop && pop_ref(t, stack);
}

// Parking of an any-hit (shadow) traversal in the slots of TraceParking:
// state = ref, sp | in_blas << 16 | opaque << 17 | alpha_map << 18, the
// instance being traversed, iter; hit = throughput, alpha_pass,
// bits(alpha_tex), unused.  The instance's object-space ray is rebuilt on
// resume from the world ray, as on entry.
__device__ __forceinline__ void park_shadow(const TraceParking& pk, uint32_t slot, uint32_t path, const ShadowTrace& t,
                                            const TraceStack& stack)
{
    pk.path[slot] = path;
    pk.state[slot] = make_int4(t.ref,
                               t.sp | (t.in_blas ? 1 << 16 : 0) | (t.opaque ? 1 << 17 : 0) | (t.alpha_map ? 1 << 18 : 0),
                               (int)t.inst, (int)t.iter);
    pk.hit[slot] = make_float4(t.throughput, t.alpha_pass, __uint_as_float(t.alpha_tex), 0.0f);
    for (int k = 0; k < t.sp; k++)
        pk.stack[(size_t)k * pk.cap + slot] = stack.get(k);
}

__device__ __forceinline__ void resume_shadow(const DevScene& s, const TraceParking& pk, uint32_t slot, f3 o, f3 d, float tmin,
                                              float tmax, ShadowTrace& t, TraceStack& stack)
{
    const int4 st = pk.state[slot];
    const float4 h = pk.hit[slot];
    t.world.o = o;
    t.world.d = d;
    setup_slab(t.world, endless(tmax));
    t.tmin = tmin;
    t.tmax = tmax;
    t.ref = st.x;
    t.sp = st.y & 0xFFFF;
    t.in_blas = (st.y >> 16) & 1;
    t.opaque = (st.y >> 17) & 1;
    t.alpha_map = (st.y >> 18) & 1;
    t.inst = (uint32_t)st.z;
    t.alpha_inst = t.inst;
    t.iter = (uint32_t)st.w;
    t.throughput = h.x;
    t.alpha_pass = h.y;
    t.alpha_tex = __float_as_uint(h.z);
    if (t.in_blas)
        to_object(s.dinst + t.inst, t.world.o, t.world.d, t.r, endless(t.tmax));
    else
        t.r = t.world;
    for (int k = 0; k < t.sp; k++)
        stack.set(k, pk.stack[(size_t)k * pk.cap + slot]);
}

template <bool W4>
static __device__ __forceinline__ float trace_shadow_inl(const DevScene& s, f3 o, f3 d, float tmin, float tmax, TraceCounters& tc)
{
    ShadowTrace t;
    TraceStack stack;
    shadow_begin(s, o, d, tmin, tmax, t, stack);
    while (!shadow_step<W4>(s, t, stack, tc)) {
    }
    return shadow_result(t);
}

// Out-of-line copies for the megakernel (keeps its code size down); the
// wavefront traversal kernels inline the traversal instead.  The node width
// follows the scene (4-wide when s.nodes4 is present).
template <bool W4>
static __device__ __noinline__ bool trace_closest_out(const DevScene& s, f3 o, f3 d, float tmin, float tmax, Hit& h, TraceCounters& tc)
{
    return trace_closest_inl<W4>(s, o, d, tmin, tmax, h, tc);
}
template <bool W4>
static __device__ __noinline__ float trace_shadow_out(const DevScene& s, f3 o, f3 d, float tmin, float tmax, TraceCounters& tc)
{
    return trace_shadow_inl<W4>(s, o, d, tmin, tmax, tc);
}
static __device__ __forceinline__ bool trace_closest(const DevScene& s, f3 o, f3 d, float tmin, float tmax, Hit& h, TraceCounters& tc)
{
    return s.nodes4 ? trace_closest_out<true>(s, o, d, tmin, tmax, h, tc) : trace_closest_out<false>(s, o, d, tmin, tmax, h, tc);
}
static __device__ __forceinline__ float trace_shadow(const DevScene& s, f3 o, f3 d, float tmin, float tmax, TraceCounters& tc)
{
    return s.nodes4 ? trace_shadow_out<true>(s, o, d, tmin, tmax, tc) : trace_shadow_out<false>(s, o, d, tmin, tmax, tc);
}

} // namespace pt
