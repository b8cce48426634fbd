// bvh_build.cu — two-level BVH construction on the device.
//
// Replaces the driver's acceleration-structure build of the reference
// (vkCmdBuildAccelerationStructuresKHR, src/pathtrace/accstruct.cpp:57-61,
// 69-164 for the per-mesh BLAS, 186-286 for the TLAS).
//
// Method: linear BVH (Karras 2012, "Maximizing parallelism in the
// construction of BVHs, octrees, and k-d trees").  All meshes are built in a
// single pass: each primitive's 64-bit key is (segment << 48 | 48-bit Morton
// code of its centroid within the segment's centroid bounds), so after one
// radix sort every mesh is a contiguous key range and the binary radix tree
// over all keys contains, for every mesh, a node whose range is exactly that
// mesh (the mesh's BLAS root).  Nodes that straddle two meshes are never
// referenced.  Boxes are reduced bottom-up with one atomic counter per node,
// then every node is written with both child boxes padded outward (relative
// 1e-5 of the largest coordinate) so the traversal's box tests stay
// conservative.  The TLAS is the same construction over instance world boxes
// with one segment.
//
// Default topology: PLOC (Meister & Bittner 2018, "Parallel locally-ordered
// clustering for bounding volume hierarchy construction") on the same sorted
// keys: every primitive starts as a cluster; each round, every cluster finds
// the neighbour within a window of positions (same segment) whose merged box
// has the smallest surface area (ties broken by the lower index pair, so the
// globally closest pair in each segment is always mutual), mutual nearest
// neighbours merge into a new node, and the survivors are compacted in
// order, until each segment is one cluster.  Rounds over all segments at once
// run until every segment is small; then a block or a cluster of blocks per
// segment finishes it in shared memory.  Nodes are numbered in merge order by
// prefix sums (deterministic).  PT_BVH=lbvh selects the radix tree instead (kept
// for A/B).
#include <cooperative_groups.h>
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "device/scene.cuh"
#include "device/warps.h"
#include "kernels.h"

namespace pt {

namespace cg = cooperative_groups;

namespace {

constexpr int MORTON_BITS = 16;           // per axis
constexpr int KEY_SEG_SHIFT = 3 * MORTON_BITS;

__device__ __forceinline__ int f2ord(float f)
{
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float ord2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }

// Spread the 16 bits of v to every third bit (bit b -> bit 3b), 48 bits wide.
__host__ __device__ __forceinline__ uint64_t expand_bits16(uint32_t v)
{
    uint64_t x = v & 0xFFFFu;
    x = (x | (x << 16)) & 0x0000FF0000FFull;
    x = (x | (x << 8)) & 0x00F00F00F00Full;
    x = (x | (x << 4)) & 0x0C30C30C30C3ull;
    x = (x | (x << 2)) & 0x249249249249ull;
    return x;
}

__device__ __forceinline__ uint32_t upper_segment(const uint32_t* base, uint32_t nseg, uint32_t g)
{
    // largest m with base[m] <= g (base has nseg + 1 entries, base[0] = 0)
    uint32_t lo = 0, hi = nseg;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (base[mid] <= g)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

struct Scratch {
    float4* lo;      // primitive boxes
    float4* hi;
    uint32_t* seg;   // segment of each primitive
    uint64_t* keys_in;
    uint64_t* keys_out;
    uint32_t* vals_in;
    uint32_t* vals_out;
    int* parent;       // internal nodes (n - 1)
    int* leaf_parent;  // leaves (n)
    int* child0;
    int* child1;
    uint32_t* flags;
    float4* nlo;     // internal node boxes (unpadded)
    float4* nhi;
    int* seg_cb;     // 6 ints per segment: centroid bounds (ordered ints)
    int* seg_box;    // 6 ints per segment: primitive bounds
    uint32_t* seg_base; // segment begin (nseg + 1)
    int* seg_root;
    void* cub_temp;
    size_t cub_bytes;
    // PLOC clusters (double-buffered) and per-round flags / prefix sums
    int* c_ref[2];
    float4* c_lo[2];
    float4* c_hi[2];
    uint32_t* c_seg[2];
    int* nn;
    uint64_t* scan;     // exclusive sums of (merge flag << 32 | survivor flag)
    uint32_t* counters; // rounds alternate between two pairs: [2p] nodes emitted, [2p + 1] live clusters at the
                        // start of rounds of parity p; [4] the most live clusters of a segment, [5] segments that
                        // have any, [6] segments with more than PLOC_SMALL_CAP
    uint32_t* seg_live; // live clusters of each segment when its block takes over,
    uint32_t* seg_first; // and the first of them
    void* scan_temp;
    size_t scan_bytes;
    // leaf collapse of the BLAS trees
    uint32_t* cnt;      // triangles under a node
    float* sah;         // SAH cost of a node's best form
    uint32_t* collapse; // 1: the node is cheaper as one leaf
    uint32_t* newpos;   // depth-first position of each triangle (sorted position -> TriRec slot)
    uint32_t* node_off; // depth-first position of a node's first triangle
    uint32_t* visits;   // bottom-up arrival counters
    uint32_t blas_nodes; // host: BLAS nodes emitted by PLOC
};

template <typename T>
T* carve(char*& p, size_t count)
{
    uintptr_t a = ((uintptr_t)p + 255) & ~(uintptr_t)255;
    T* r = (T*)a;
    p = (char*)(a + count * sizeof(T));
    return r;
}

size_t cub_sort_bytes(uint32_t n)
{
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, (uint64_t*)nullptr, (uint64_t*)nullptr, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (int)n, 0, 64);
    return bytes;
}

// Merge and survivor flags of cluster i, (merge << 32) | survivor: mutual
// nearest neighbours merge and the lower index of a pair keeps the merged
// cluster; zero past the live count.
struct PlocFlags {
    const int* nn;
    const uint32_t* live;
    __host__ __device__ uint64_t operator()(int i) const
    {
#ifdef __CUDA_ARCH__
        if (i >= (int)*live)
            return 0;
        const int j = nn[i];
        const bool mutual = j >= 0 && nn[j] == i;
        return (mutual && i < j ? 1ull << 32 : 0ull) | (mutual && i > j ? 0ull : 1ull);
#else
        return 0;
#endif
    }
};
using PlocFlagIter = thrust::transform_iterator<PlocFlags, thrust::counting_iterator<int>, uint64_t>;

PlocFlagIter ploc_flags(const int* nn, const uint32_t* live)
{
    return PlocFlagIter(thrust::counting_iterator<int>(0), PlocFlags{nn, live});
}

size_t cub_scan_bytes(uint32_t n)
{
    size_t bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, bytes, ploc_flags(nullptr, nullptr), (uint64_t*)nullptr, (int)n);
    return bytes;
}

Scratch carve_scratch(void* base, uint32_t n, uint32_t nseg)
{
    char* p = (char*)base;
    Scratch s;
    uint32_t nn = n > 0 ? n : 1;
    s.lo = carve<float4>(p, nn);
    s.hi = carve<float4>(p, nn);
    s.seg = carve<uint32_t>(p, nn);
    s.keys_in = carve<uint64_t>(p, nn);
    s.keys_out = carve<uint64_t>(p, nn);
    s.vals_in = carve<uint32_t>(p, nn);
    s.vals_out = carve<uint32_t>(p, nn);
    s.parent = carve<int>(p, nn);
    s.leaf_parent = carve<int>(p, nn);
    s.child0 = carve<int>(p, nn);
    s.child1 = carve<int>(p, nn);
    s.flags = carve<uint32_t>(p, nn);
    s.nlo = carve<float4>(p, nn);
    s.nhi = carve<float4>(p, nn);
    s.seg_cb = carve<int>(p, 6 * (size_t)(nseg + 1));
    s.seg_box = carve<int>(p, 6 * (size_t)(nseg + 1));
    s.seg_base = carve<uint32_t>(p, nseg + 2);
    s.seg_root = carve<int>(p, nseg + 1);
    for (int b = 0; b < 2; b++) {
        s.c_ref[b] = carve<int>(p, nn);
        s.c_lo[b] = carve<float4>(p, nn);
        s.c_hi[b] = carve<float4>(p, nn);
        s.c_seg[b] = carve<uint32_t>(p, nn);
    }
    s.nn = carve<int>(p, nn);
    s.scan = carve<uint64_t>(p, nn);
    s.seg_live = carve<uint32_t>(p, nseg + 1);
    s.seg_first = carve<uint32_t>(p, nseg + 1);
    s.counters = carve<uint32_t>(p, 8);
    s.cnt = carve<uint32_t>(p, nn);
    s.sah = carve<float>(p, nn);
    s.collapse = carve<uint32_t>(p, nn);
    s.newpos = carve<uint32_t>(p, nn);
    s.node_off = carve<uint32_t>(p, nn);
    s.visits = carve<uint32_t>(p, nn);
    s.blas_nodes = 0;
    s.scan_bytes = cub_scan_bytes(nn);
    s.scan_temp = carve<char>(p, s.scan_bytes);
    s.cub_bytes = cub_sort_bytes(nn);
    s.cub_temp = carve<char>(p, s.cub_bytes);
    return s;
}

size_t scratch_bytes_for(uint32_t n, uint32_t nseg)
{
    Scratch s = carve_scratch((void*)0, n, nseg);
    return (size_t)((char*)s.cub_temp - (char*)0) + s.cub_bytes + 256;
}

__global__ void k_init_bounds(int* cb, int* box, int* roots, uint32_t nseg)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nseg)
        return;
    roots[i] = REF_EMPTY;
    for (int k = 0; k < 3; k++) {
        cb[6 * i + k] = f2ord(__int_as_float(0x7f800000));
        cb[6 * i + 3 + k] = f2ord(-__int_as_float(0x7f800000));
        box[6 * i + k] = f2ord(__int_as_float(0x7f800000));
        box[6 * i + 3 + k] = f2ord(-__int_as_float(0x7f800000));
    }
}

__device__ __forceinline__ void atomic_bounds(int* b, float4 lo, float4 hi)
{
    atomicMin(b + 0, f2ord(lo.x));
    atomicMin(b + 1, f2ord(lo.y));
    atomicMin(b + 2, f2ord(lo.z));
    atomicMax(b + 3, f2ord(hi.x));
    atomicMax(b + 4, f2ord(hi.y));
    atomicMax(b + 5, f2ord(hi.z));
}

// Bounds of the centroids (cb) and boxes (box, may be null) of a block's
// primitives, all threads of the block calling.  When they are of one segment,
// one thread's atomics for the whole block: with a thread each, 12 atomics per
// triangle queued on a few addresses, and k_tri_boxes took 6,300 us for two
// million triangles in 64 meshes, 33 us with this.
constexpr int BOUNDS_THREADS = 256;

__device__ __forceinline__ void segment_bounds(bool valid, uint32_t m, int* cb, int* box, float4 cen, float4 lo, float4 hi)
{
    __shared__ int s_b[12][BOUNDS_THREADS / 32];
    __shared__ uint32_t s_m;
    if (threadIdx.x == 0) // valid in every block that is launched
        s_m = m;
    __syncthreads();
    if (!__syncthreads_and(!valid || m == s_m)) {
        if (valid) {
            atomic_bounds(cb + 6 * m, cen, cen);
            if (box)
                atomic_bounds(box + 6 * m, lo, hi);
        }
        return;
    }
    const int none_lo = 0x7FFFFFFF, none_hi = (int)0x80000000;
    const int v[12] = {valid ? f2ord(cen.x) : none_lo, valid ? f2ord(cen.y) : none_lo, valid ? f2ord(cen.z) : none_lo,
                       valid ? f2ord(cen.x) : none_hi, valid ? f2ord(cen.y) : none_hi, valid ? f2ord(cen.z) : none_hi,
                       valid ? f2ord(lo.x) : none_lo,  valid ? f2ord(lo.y) : none_lo,  valid ? f2ord(lo.z) : none_lo,
                       valid ? f2ord(hi.x) : none_hi,  valid ? f2ord(hi.y) : none_hi,  valid ? f2ord(hi.z) : none_hi};
    const int warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 12; k++) {
        const int w = k % 6 < 3 ? __reduce_min_sync(0xffffffffu, v[k]) : __reduce_max_sync(0xffffffffu, v[k]);
        if ((threadIdx.x & 31) == 0)
            s_b[k][warp] = w;
    }
    __syncthreads();
    if (threadIdx.x < (box ? 12 : 6)) {
        const int k = threadIdx.x;
        int w = s_b[k][0];
        for (int i = 1; i < (int)(blockDim.x / 32); i++)
            w = k % 6 < 3 ? min(w, s_b[k][i]) : max(w, s_b[k][i]);
        int* to = (k < 6 ? cb : box) + 6 * s_m + k % 6;
        if (k % 6 < 3)
            atomicMin(to, w);
        else
            atomicMax(to, w);
    }
}

__global__ void __launch_bounds__(BOUNDS_THREADS) k_tri_boxes(BvhBuildInput in, Scratch s)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = g < in.tri_count;
    uint32_t m = 0;
    float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
    if (valid) {
        m = upper_segment(in.mesh_tri_base, in.mesh_count, g);
        uint32_t local = g - in.mesh_tri_base[m];
        uint32_t ib = in.mesh_index_offset[m] + 3 * local;
        uint32_t vb = in.mesh_vertex_offset[m];
        float4 a = in.vertices[2 * (size_t)(vb + in.indices[ib + 0])];
        float4 b = in.vertices[2 * (size_t)(vb + in.indices[ib + 1])];
        float4 c = in.vertices[2 * (size_t)(vb + in.indices[ib + 2])];
        lo = make_float4(fminf(fminf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y), fminf(fminf(a.z, b.z), c.z), 0.0f);
        hi = make_float4(fmaxf(fmaxf(a.x, b.x), c.x), fmaxf(fmaxf(a.y, b.y), c.y), fmaxf(fmaxf(a.z, b.z), c.z), 0.0f);
        s.lo[g] = lo;
        s.hi[g] = hi;
        s.seg[g] = m;
    }
    float4 cen = make_float4(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z), 0.0f);
    segment_bounds(valid, m, s.seg_cb, s.seg_box, cen, lo, hi);
}

// World boxes of the instances, one warp each: the box around the transformed
// boxes of the mesh's tree eight levels down (up to 256), cut to the box of the
// mesh box's eight transformed corners.  A rotated mesh fills little of the
// latter (a sphere a third of its surface), and every ray that meets it enters
// the instance.  Each lane follows the five bits of its number down the tree
// and then takes the eight boxes three levels below.  Heavy scene (10,000
// rotated grids and spheres) at 1920 x 1080, 4 spp: extend 22.3 -> 21.1 ms, shadow
// 12.4 -> 11.6; mid scene (196 rotated boxes) at 1024 x 1024, 128 spp: 51.9 -> 50.7
// and 24.0 -> 22.2.
constexpr int BOX_LANE_LEVELS = 5, BOX_MORE_LEVELS = 3;

// Box of node `ref`'s child on side `bit`, and the child.
__device__ __forceinline__ int child_box(const BvhNode* nodes, int ref, uint32_t bit, float4& lo, float4& hi)
{
    const BvhNode nd = nodes[ref];
    const float4 xy = bit ? nd.c1xy : nd.c0xy;
    lo = make_float4(xy.x, xy.z, bit ? nd.c01z.z : nd.c01z.x, 0.0f);
    hi = make_float4(xy.y, xy.w, bit ? nd.c01z.w : nd.c01z.y, 0.0f);
    return bit ? nd.link.y : nd.link.x;
}

// Bounds of row . p + row.w over a box of centre c and half size h, widened by
// `err` for the rounding of the single-precision sums.
__device__ __forceinline__ void widen_by_row(float4 row, float4 c, float4 h, float err, float& lo, float& hi)
{
    const float mid = ((row.x * c.x + row.y * c.y) + row.z * c.z) + row.w;
    const float ext = ((fabsf(row.x) * h.x + fabsf(row.y) * h.y) + fabsf(row.z) * h.z) + err;
    lo = fminf(lo, mid - ext);
    hi = fmaxf(hi, mid + ext);
}

__global__ void __launch_bounds__(BOUNDS_THREADS) k_inst_boxes(BvhBuildInput in, const int* mesh_box, const int* mesh_root,
                                                               const BvhNode* nodes, Scratch s)
{
    const uint32_t i = warp_item(blockIdx.x, BOUNDS_THREADS, threadIdx.x), lane = threadIdx.x & 31;
    const bool valid = i < in.instance_count && lane == 0;
    const float inf = __int_as_float(0x7f800000);
    float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
    if (i < in.instance_count) { // the whole warp
        const uint32_t m = in.inst_mesh[i];
        const int* mb = mesh_box + 6 * m;
        const float blo[3] = {ord2f(mb[0]), ord2f(mb[1]), ord2f(mb[2])};
        const float bhi[3] = {ord2f(mb[3]), ord2f(mb[4]), ord2f(mb[5])};
        const DevInstanceData& d = in.inst_data[i];
        const float4 rows[3] = {d.t0, d.t1, d.t2};
        if (!(blo[0] <= bhi[0])) {
            // empty mesh: a point at the instance origin (its BLAS root is empty)
            lo = make_float4(rows[0].w, rows[1].w, rows[2].w, 0.0f);
            hi = lo;
        } else {
            float clo[3], chi[3], tlo[3] = {inf, inf, inf}, thi[3] = {-inf, -inf, -inf}, err[3];
            const double p[3] = {(lane & 1) ? bhi[0] : blo[0], (lane & 2) ? bhi[1] : blo[1], (lane & 4) ? bhi[2] : blo[2]};
            const float mag[3] = {fmaxf(fabsf(blo[0]), fabsf(bhi[0])), fmaxf(fabsf(blo[1]), fabsf(bhi[1])),
                                  fmaxf(fabsf(blo[2]), fabsf(bhi[2]))};
#pragma unroll
            for (int r = 0; r < 3; r++) {
                clo[r] = chi[r] =
                    (float)((double)rows[r].x * p[0] + (double)rows[r].y * p[1] + (double)rows[r].z * p[2] + (double)rows[r].w);
                // at most 8 roundings of terms no larger than this sum (boxes are padded by 1e-5)
                err[r] = 8.0f * 0x1p-24f * 1.001f *
                         (((fabsf(rows[r].x) * mag[0] + fabsf(rows[r].y) * mag[1]) + fabsf(rows[r].z) * mag[2]) + fabsf(rows[r].w));
            }
            auto add = [&](float4 a, float4 b) {
                const float4 c = make_float4(0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z), 0.0f);
                const float4 h = make_float4(0.5f * (b.x - a.x), 0.5f * (b.y - a.y), 0.5f * (b.z - a.z), 0.0f);
#pragma unroll
                for (int r = 0; r < 3; r++)
                    widen_by_row(rows[r], c, h, err[r], tlo[r], thi[r]);
            };
            int ref = mesh_root[m];
            const bool single = ref < 0; // one leaf: no tree to follow
            float4 a, b;
            for (int l = 0; l < BOX_LANE_LEVELS && ref >= 0; l++)
                ref = child_box(nodes, ref, (lane >> l) & 1u, a, b);
            if (!single && ref < 0)
                add(a, b);
            for (uint32_t k = 0; ref >= 0 && k < (1u << BOX_MORE_LEVELS); k++) {
                int c = ref;
                for (int l = 0; l < BOX_MORE_LEVELS && c >= 0; l++)
                    c = child_box(nodes, c, (k >> l) & 1u, a, b);
                add(a, b);
            }
            float out[6];
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const float c0 = ord2f(__reduce_min_sync(0xffffffffu, f2ord(clo[r]))), c1 = ord2f(__reduce_max_sync(0xffffffffu, f2ord(chi[r])));
                const float t0 = ord2f(__reduce_min_sync(0xffffffffu, f2ord(tlo[r]))), t1 = ord2f(__reduce_max_sync(0xffffffffu, f2ord(thi[r])));
                const bool use = !single && t0 <= t1; // false for sums that are not numbers
                out[r] = use ? fmaxf(c0, t0) : c0;
                out[3 + r] = use ? fminf(c1, t1) : c1;
                if (!(out[r] <= out[3 + r])) { // rounding pushed the two apart
                    out[r] = c0;
                    out[3 + r] = c1;
                }
            }
            lo = make_float4(out[0], out[1], out[2], 0.0f);
            hi = make_float4(out[3], out[4], out[5], 0.0f);
        }
        if (lane == 0) {
            s.lo[i] = lo;
            s.hi[i] = hi;
            s.seg[i] = 0;
        }
    }
    float4 cen = make_float4(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z), 0.0f);
    segment_bounds(valid, 0, s.seg_cb, nullptr, cen, lo, hi);
}

__global__ void k_morton(Scratch s, uint32_t n)
{
    uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n)
        return;
    uint32_t m = s.seg[g];
    const int* cb = s.seg_cb + 6 * m;
    float4 lo = s.lo[g], hi = s.hi[g];
    float c[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
    uint32_t q[3];
    for (int k = 0; k < 3; k++) {
        float a = ord2f(cb[k]), b = ord2f(cb[3 + k]);
        float x = (b > a) ? (c[k] - a) / (b - a) : 0.0f;
        x = fminf(fmaxf(x, 0.0f), 1.0f);
        q[k] = (uint32_t)(x * 65535.0f);
    }
    uint64_t code = (expand_bits16(q[0]) << 2) | (expand_bits16(q[1]) << 1) | expand_bits16(q[2]);
    s.keys_in[g] = ((uint64_t)m << KEY_SEG_SHIFT) | code;
    s.vals_in[g] = g;
}

__device__ __forceinline__ int delta(const uint64_t* keys, int n, int i, int j)
{
    if (j < 0 || j >= n)
        return -1;
    uint64_t a = keys[i], b = keys[j];
    if (a != b)
        return __clzll((long long)(a ^ b));
    return 64 + __clz(i ^ j);
}

// Karras 2012, Algorithm 1 (node ranges and splits of the binary radix tree).
__global__ void k_karras(Scratch s, int n, int node_base, int mode_tlas)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1)
        return;
    const uint64_t* keys = s.keys_out;
    int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin)
        lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(keys, n, i, i + (l + t) * d) > dmin)
            l += t;
    int j = i + l * d;
    int dnode = delta(keys, n, i, j);
    int sp = 0;
    for (int div = 2;; div <<= 1) {
        int t = (l + div - 1) / div;
        if (delta(keys, n, i, i + (sp + t) * d) > dnode)
            sp += t;
        if (t <= 1)
            break;
    }
    int gamma = i + sp * d + min(d, 0);
    int lo = min(i, j), hi = max(i, j);
    int c0 = (lo == gamma) ? ~gamma : gamma;
    int c1 = (hi == gamma + 1) ? ~(gamma + 1) : gamma + 1;
    s.child0[i] = c0;
    s.child1[i] = c1;
    if (c0 >= 0)
        s.parent[c0] = i;
    else
        s.leaf_parent[~c0] = i;
    if (c1 >= 0)
        s.parent[c1] = i;
    else
        s.leaf_parent[~c1] = i;
    uint32_t seg_lo = (uint32_t)(keys[lo] >> KEY_SEG_SHIFT), seg_hi = (uint32_t)(keys[hi] >> KEY_SEG_SHIFT);
    // flags: bit 31 marks a node that straddles two segments
    s.flags[i] = (seg_lo != seg_hi) ? 0x80000000u : 0u;
    if (seg_lo == seg_hi && (uint32_t)lo == s.seg_base[seg_lo] && (uint32_t)hi + 1 == s.seg_base[seg_lo + 1])
        s.seg_root[seg_lo] = node_base + i;
    (void)mode_tlas;
}

// Segments with zero or one primitive have no internal root.
__global__ void k_small_roots(Scratch s, uint32_t nseg, int mode_tlas)
{
    uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nseg)
        return;
    uint32_t b = s.seg_base[m], e = s.seg_base[m + 1];
    if (e == b)
        s.seg_root[m] = REF_EMPTY;
    else if (e - b == 1)
        s.seg_root[m] = mode_tlas ? make_leaf(s.vals_out[b], 1) : make_leaf(b, 1);
}

__global__ void k_bottom_up(Scratch s, int n)
{
    int pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= n || n < 2)
        return;
    int node = s.leaf_parent[pos];
    while (node >= 0) {
        if (s.flags[node] & 0x80000000u)
            return; // straddling node: above every mesh root
        __threadfence();
        uint32_t old = atomicAdd(&s.flags[node], 1u);
        if ((old & 0xFFu) == 0)
            return; // first arrival; the sibling finishes this node
        float4 lo = make_float4(__int_as_float(0x7f800000), __int_as_float(0x7f800000), __int_as_float(0x7f800000), 0.0f);
        float4 hi = make_float4(-lo.x, -lo.y, -lo.z, 0.0f);
        int cs[2] = {s.child0[node], s.child1[node]};
        for (int k = 0; k < 2; k++) {
            float4 a, b;
            if (cs[k] < 0) {
                uint32_t p = s.vals_out[~cs[k]];
                a = s.lo[p];
                b = s.hi[p];
            } else {
                a = __ldcg(s.nlo + cs[k]);
                b = __ldcg(s.nhi + cs[k]);
            }
            lo.x = fminf(lo.x, a.x);
            lo.y = fminf(lo.y, a.y);
            lo.z = fminf(lo.z, a.z);
            hi.x = fmaxf(hi.x, b.x);
            hi.y = fmaxf(hi.y, b.y);
            hi.z = fmaxf(hi.z, b.z);
        }
        __stcg(s.nlo + node, lo);
        __stcg(s.nhi + node, hi);
        __threadfence();
        node = s.parent[node];
    }
}

__device__ __forceinline__ void padded(float4 lo, float4 hi, float4& plo, float4& phi)
{
    float mag = fmaxf(fmaxf(fmaxf(fabsf(lo.x), fabsf(hi.x)), fmaxf(fabsf(lo.y), fabsf(hi.y))), fmaxf(fabsf(lo.z), fabsf(hi.z)));
    float eps = mag * 1e-5f + 1e-30f;
    plo = make_float4(lo.x - eps, lo.y - eps, lo.z - eps, 0.0f);
    phi = make_float4(hi.x + eps, hi.y + eps, hi.z + eps, 0.0f);
}

__global__ void k_emit_nodes(Scratch s, int n, BvhNode* nodes, int node_base, int mode_tlas)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1)
        return;
    if (s.flags[i] & 0x80000000u)
        return;
    int cs[2] = {s.child0[i], s.child1[i]};
    float4 blo[2], bhi[2];
    int ref[2];
    for (int k = 0; k < 2; k++) {
        float4 a, b;
        if (cs[k] < 0) {
            int pos = ~cs[k];
            uint32_t p = s.vals_out[pos];
            a = s.lo[p];
            b = s.hi[p];
            ref[k] = mode_tlas ? make_leaf(p, 1) : make_leaf((uint32_t)pos, 1);
        } else {
            a = s.nlo[cs[k]];
            b = s.nhi[cs[k]];
            ref[k] = node_base + cs[k];
        }
        padded(a, b, blo[k], bhi[k]);
    }
    BvhNode nd;
    nd.c0xy = make_float4(blo[0].x, bhi[0].x, blo[0].y, bhi[0].y);
    nd.c1xy = make_float4(blo[1].x, bhi[1].x, blo[1].y, bhi[1].y);
    nd.c01z = make_float4(blo[0].z, bhi[0].z, blo[1].z, bhi[1].z);
    nd.link = make_int4(ref[0], ref[1], 0, 0);
    nodes[node_base + i] = nd;
}

// ---- PLOC
// Neighbour windows of the BLAS and TLAS passes: PT_PLOC_RADIUS and
// PT_PLOC_RADIUS_TLAS (1..256), default 64 for both (measured on the mid and
// heavy scenes against 8..256; wider windows did not lower node visits).
int env_radius(const char* name, int dflt)
{
    const char* e = std::getenv(name);
    const int r = e ? std::atoi(e) : dflt;
    return r < 1 ? 1 : (r > 256 ? 256 : r);
}

int ploc_radius(int mode_tlas)
{
    static const int blas = env_radius("PT_PLOC_RADIUS", 64);
    static const int tlas = env_radius("PT_PLOC_RADIUS_TLAS", 64);
    return mode_tlas ? tlas : blas;
}

__device__ __forceinline__ float half_area(float4 lo, float4 hi)
{
    const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return dx * dy + dy * dz + dz * dx;
}

__device__ __forceinline__ float4 box_min(float4 a, float4 b) { return make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.0f); }
__device__ __forceinline__ float4 box_max(float4 a, float4 b) { return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), 0.0f); }

// Initial clusters: one per primitive, in sorted order.
__global__ void k_ploc_init(Scratch s, uint32_t n, int mode_tlas)
{
    uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= n)
        return;
    const uint32_t p = s.vals_out[pos];
    s.c_ref[0][pos] = mode_tlas ? make_leaf(p, 1) : make_leaf(pos, 1);
    s.c_lo[0][pos] = s.lo[p];
    s.c_hi[0][pos] = s.hi[p];
    s.c_seg[0][pos] = (uint32_t)(s.keys_out[pos] >> KEY_SEG_SHIFT);
}

// Nearest neighbours of clusters `own` and own + 1 (own even) among the
// clusters k0 .. k1 + 1 (k0, k1 even) staged in shared memory, `stride` floats
// each of lo.x, lo.y, lo.z, hi.x, hi.y, hi.z: of those at most `radius` away (and
// of the own segment, SEG; below n otherwise) the one whose box merges with the
// smallest surface, of equal ones the first (the lower index pair).
//
// Inside the window (all but its ends and the pair itself) nothing needs testing
// when both of its ends belong to the pair's segment: clusters are in their
// segments' order.  There four clusters are read at a time and only the smallest
// of their four distances is compared; which of the four it was is found at the
// end.  The kernels that call it are bound by the ALU pipe (minima, maxima,
// compares, selects; 80 % busy with a test of each distance): two million
// clusters 229 us with the tests, 182 without.
template <bool SEG>
__device__ __forceinline__ void nn_pair(const float* box, int stride, const uint32_t* seg, int own, int k0, int k1, int n, int radius,
                                        int& j0, int& j1)
{
    auto pair_at = [&](int row, int k) { return *reinterpret_cast<const float2*>(box + row * stride + k); };
    const float2 ax = pair_at(0, own), ay = pair_at(1, own), az = pair_at(2, own);
    const float2 bx = pair_at(3, own), by = pair_at(4, own), bz = pair_at(5, own);
    uint2 as = make_uint2(0u, 0u);
    if (SEG)
        as = *reinterpret_cast<const uint2*>(seg + own);
    float best0 = __int_as_float(0x7F800000), best1 = best0; // infinity
    int quad0 = -1, quad1 = -1;                              // the four clusters that hold the best, if it is inside the window
    j0 = j1 = -1;
    // half the surface of the merged box of own + q and k + r
#define PT_NN_DIST(q, r)                                                                                             \
    half_area(make_float4(fminf(ax.q, cx.r), fminf(ay.q, cy.r), fminf(az.q, cz.r), 0.0f),                            \
              make_float4(fmaxf(bx.q, dx.r), fmaxf(by.q, dy.r), fmaxf(bz.q, dz.r), 0.0f))
#define PT_NN_LOAD(k)                                                                                                \
    const float2 cx = pair_at(0, k), cy = pair_at(1, k), cz = pair_at(2, k), dx = pair_at(3, k), dy = pair_at(4, k), \
                 dz = pair_at(5, k);
#define PT_NN_TRY(q, r, i, j, best, jbest, quad)                                                                     \
    {                                                                                                                \
        const float d = PT_NN_DIST(q, r);                                                                            \
        const int off = (j) - (i);                                                                                   \
        if (cs.r == as.q && off != 0 && off >= -radius && off <= radius && ((jbest < 0 && quad < 0) || d < best)) {  \
            best = d;                                                                                                \
            jbest = (j);                                                                                             \
            quad = -1;                                                                                               \
        }                                                                                                            \
    }
    auto tested = [&](int k) {
        PT_NN_LOAD(k)
        uint2 cs = make_uint2(0u, k + 1 < n ? 0u : 1u);
        if (SEG)
            cs = *reinterpret_cast<const uint2*>(seg + k);
        PT_NN_TRY(x, x, own, k, best0, j0, quad0)
        PT_NN_TRY(x, y, own, k + 1, best0, j0, quad0)
        PT_NN_TRY(y, x, own + 1, k, best1, j1, quad1)
        PT_NN_TRY(y, y, own + 1, k + 1, best1, j1, quad1)
    };
    const int inner = (radius - 1) & ~1; // both clusters of every pair this far away are in both windows
    int ka = max(k0, own - inner), kb = min(k1, own + inner);
    if (SEG) {
        if (as.x != as.y || seg[k0] != as.x || seg[k1 + 1] != as.x)
            kb = ka - 2; // another segment's clusters, or none, in the window
    } else if (kb + 1 >= n)
        kb -= 2;
    int k = k0;
    for (; k < min(ka, k1 + 2); k += 2)
        tested(k);
    for (int side = 0; side < 2; side++) {
        const int end = side == 0 ? min(own - 2, kb) : kb;
#pragma unroll (SEG ? 2 : 1) // the block kernel has no registers to spare
        for (; k + 2 <= end; k += 4) {
            float m0, m1;
            {
                PT_NN_LOAD(k)
                m0 = fminf(PT_NN_DIST(x, x), PT_NN_DIST(x, y));
                m1 = fminf(PT_NN_DIST(y, x), PT_NN_DIST(y, y));
            }
            {
                PT_NN_LOAD(k + 2)
                m0 = fminf(m0, fminf(PT_NN_DIST(x, x), PT_NN_DIST(x, y)));
                m1 = fminf(m1, fminf(PT_NN_DIST(y, x), PT_NN_DIST(y, y)));
            }
            if (m0 < best0) {
                best0 = m0;
                quad0 = k;
            }
            if (m1 < best1) {
                best1 = m1;
                quad1 = k;
            }
        }
        // what is left of this side, and the pair itself or the rest
        const int stop = side == 0 ? min(own, k1) : k1;
        for (; k <= stop; k += 2)
            tested(k);
    }
    // the first of the four that is as near as the best
    for (int h = 2; h >= 0; h -= 2) {
        if (quad0 >= 0) {
            PT_NN_LOAD(quad0 + h)
            if (!(PT_NN_DIST(x, y) > best0))
                j0 = quad0 + h + 1;
            if (!(PT_NN_DIST(x, x) > best0))
                j0 = quad0 + h;
        }
        if (quad1 >= 0) {
            PT_NN_LOAD(quad1 + h)
            if (!(PT_NN_DIST(y, y) > best1))
                j1 = quad1 + h + 1;
            if (!(PT_NN_DIST(y, x) > best1))
                j1 = quad1 + h;
        }
    }
    // no distance in range (boxes that overflow): the first in the window, as with a test of each
    if ((j0 < 0 && own < n) || (j1 < 0 && own + 1 < n)) {
        const bool first0 = j0 < 0, first1 = j1 < 0;
        quad0 = quad1 = -1;
        for (k = k0; k <= k1; k += 2) {
            PT_NN_LOAD(k)
            uint2 cs = make_uint2(0u, k + 1 < n ? 0u : 1u);
            if (SEG)
                cs = *reinterpret_cast<const uint2*>(seg + k);
            if (first0) {
                PT_NN_TRY(x, x, own, k, best0, j0, quad0)
                PT_NN_TRY(x, y, own, k + 1, best0, j0, quad0)
            }
            if (first1) {
                PT_NN_TRY(y, x, own + 1, k, best1, j1, quad1)
                PT_NN_TRY(y, y, own + 1, k + 1, best1, j1, quad1)
            }
        }
    }
#undef PT_NN_TRY
#undef PT_NN_LOAD
#undef PT_NN_DIST
}

// Nearest neighbours of all live clusters: a block stages its NN_CLUSTERS
// clusters and the window on either side.  Bound by the arithmetic of the
// n (2 radius + 1) distances: two million clusters 182 us (381 with a thread
// to a cluster reading the boxes through L1), 10,000 10 us (29).
constexpr int NN_THREADS = 128, NN_CLUSTERS = 2 * NN_THREADS;

__global__ void __launch_bounds__(NN_THREADS) k_ploc_nn(const float4* lo, const float4* hi, const uint32_t* seg, const uint32_t* live,
                                                        int radius, int* nn)
{
    extern __shared__ __align__(16) float s_box[]; // lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, segment: `span` of each
    const int n = (int)*live;
    const int base = blockIdx.x * NN_CLUSTERS;
    if (base >= n)
        return;
    const int pad = (radius + 1) & ~1, span = NN_CLUSTERS + 2 * pad;
    uint32_t* s_seg = reinterpret_cast<uint32_t*>(s_box + 6 * span);
    for (int k = threadIdx.x; k < span; k += NN_THREADS) {
        const int j = base - pad + k;
        const bool in = j >= 0 && j < n;
        const float4 a = in ? lo[j] : make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = in ? hi[j] : a;
        s_box[k] = a.x;
        s_box[span + k] = a.y;
        s_box[2 * span + k] = a.z;
        s_box[3 * span + k] = b.x;
        s_box[4 * span + k] = b.y;
        s_box[5 * span + k] = b.z;
        s_seg[k] = in ? seg[j] : 0xFFFFFFFFu; // no segment has this number
    }
    __syncthreads();
    const int i0 = base + 2 * threadIdx.x;
    if (i0 >= n)
        return;
    const int own = pad + 2 * threadIdx.x;
    int j0, j1;
    nn_pair<true>(s_box, span, s_seg, own, own - pad, own + pad, span, radius, j0, j1);
    nn[i0] = j0 < 0 ? -1 : base - pad + j0;
    if (i0 + 1 < n)
        nn[i0 + 1] = j1 < 0 ? -1 : base - pad + j1;
}

__device__ __forceinline__ BvhNode merged_node(float4 lo0, float4 hi0, int ref0, float4 lo1, float4 hi1, int ref1)
{
    float4 blo[2], bhi[2];
    padded(lo0, hi0, blo[0], bhi[0]);
    padded(lo1, hi1, blo[1], bhi[1]);
    BvhNode nd;
    nd.c0xy = make_float4(blo[0].x, bhi[0].x, blo[0].y, bhi[0].y);
    nd.c1xy = make_float4(blo[1].x, bhi[1].x, blo[1].y, bhi[1].y);
    nd.c01z = make_float4(blo[0].z, bhi[0].z, blo[1].z, bhi[1].z);
    nd.link = make_int4(ref0, ref1, 0, 0);
    return nd;
}

// Merges the pairs of round `parity` and compacts the survivors into the other
// cluster buffer; the last cluster's thread writes the next round's counters.
__global__ void k_ploc_merge(Scratch s, int parity, BvhNode* nodes, int node_base)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = (int)s.counters[2 * parity + 1];
    if (i >= n)
        return;
    const uint64_t flags = PlocFlags{s.nn, &s.counters[2 * parity + 1]}(i);
    const uint64_t before = s.scan[i];
    const uint32_t nodes_before = s.counters[2 * parity];
    const int nxt = parity ^ 1;
    if (i == n - 1) {
        const uint64_t total = before + flags;
        s.counters[2 * nxt] = nodes_before + (uint32_t)(total >> 32);
        s.counters[2 * nxt + 1] = (uint32_t)total;
    }
    if (!(uint32_t)flags)
        return;
    const uint32_t o = (uint32_t)before;
    float4 lo = s.c_lo[parity][i], hi = s.c_hi[parity][i];
    int ref = s.c_ref[parity][i];
    if (flags >> 32) {
        const int j = s.nn[i];
        const float4 lo_j = s.c_lo[parity][j], hi_j = s.c_hi[parity][j];
        const int node = node_base + (int)(nodes_before + (uint32_t)(before >> 32));
        nodes[node] = merged_node(lo, hi, ref, lo_j, hi_j, s.c_ref[parity][j]);
        ref = node;
        lo = box_min(lo, lo_j);
        hi = box_max(hi, hi_j);
    }
    s.c_ref[nxt][o] = ref;
    s.c_lo[nxt][o] = lo;
    s.c_hi[nxt][o] = hi;
    s.c_seg[nxt][o] = s.c_seg[parity][i];
}

// First live cluster and live count of each segment (clusters keep their
// segments' order), the most of any, and how many have more than PLOC_SMALL_CAP.
constexpr uint32_t PLOC_SMALL_CAP = 512, PLOC_BLOCK_CAP = 4096;

__global__ void k_ploc_segments(Scratch s, int parity, uint32_t nseg)
{
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nseg)
        return;
    const uint32_t n = s.counters[2 * parity + 1];
    const uint32_t* seg = s.c_seg[parity];
    auto first_at_least = [&](uint32_t v) {
        uint32_t a = 0, b = n;
        while (a < b) {
            const uint32_t mid = (a + b) >> 1;
            if (seg[mid] < v)
                a = mid + 1;
            else
                b = mid;
        }
        return a;
    };
    const uint32_t first = first_at_least(m), live = first_at_least(m + 1) - first;
    s.seg_first[m] = first;
    s.seg_live[m] = live;
    atomicMax(&s.counters[4], live);
    if (live)
        atomicAdd(&s.counters[5], 1u);
    if (live > PLOC_SMALL_CAP)
        atomicAdd(&s.counters[6], 1u);
}

// Finishes the segments with lo_count < live clusters <= CAP, a cluster of
// blocks (or one block) each: the same rounds as above on the segment's clusters
// in shared memory.  A segment's merges do not depend on the others', so the tree
// is the one that rounds over all segments would give (only the nodes' numbers
// differ).  The rounds' launches and scans, at 25 us a round however few clusters
// were left, took most of the build: 36,000 triangles in 56 meshes and 232
// instances 3.2 ms, two million in 64 meshes and 10,256 instances 13.4 ms.
//
// The search, all but the last few rounds of a segment's time, is shared by the
// cluster's blocks: each searches for its part of the clusters and writes what it
// found to every block, and all of them then merge and compact their own copies
// alike: 10,256 instances, from 4,096 clusters on, 415 us with one block and 179
// with eight; 44 meshes of 36,000 triangles 323 and 154.  While there are fewer
// clusters than threads, several lanes share a window; at SOLO_CLUSTERS and below
// the first block goes on alone.  What is left is the latency of some 50 rounds;
// more threads or blocks for the small segments changed nothing.
constexpr uint32_t SOLO_CLUSTERS = 64;

template <int THREADS, int CAP, bool MULTI>
__global__ void __launch_bounds__(THREADS) k_ploc_block(Scratch s, int parity, BvhNode* nodes, int node_base, uint32_t lo_count,
                                                        uint32_t multi_count, int radius)
{
    constexpr int PER = CAP / THREADS;
    extern __shared__ __align__(16) float s_box[]; // CAP each of lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, reference, neighbour (two)
    int* s_ref = reinterpret_cast<int*>(s_box + 6 * CAP);
    __shared__ uint32_t s_warp[THREADS / 32], s_rank;
    cg::cluster_group cluster = cg::this_cluster();
    uint32_t nblocks = MULTI ? cluster.num_blocks() : 1u;
    const uint32_t rank = MULTI ? cluster.block_rank() : 0u;
    const uint32_t m = blockIdx.x / nblocks;
    uint32_t n = s.seg_live[m];
    if (n == 0 || n <= lo_count || n > (uint32_t)CAP)
        return;
    if (n <= multi_count)
        nblocks = 1;
    if (rank >= nblocks)
        return;
    const uint32_t first = s.seg_first[m], tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (n == 1) {
        if (tid == 0 && rank == 0)
            s.seg_root[m] = s.c_ref[parity][first];
        return;
    }
    // this segment's nodes come after those of the segments before it: one per cluster less one per segment
    if (tid == 0)
        s_rank = 0;
    __syncthreads();
    uint32_t filled = 0;
    for (uint32_t k = tid; k < m; k += THREADS)
        filled += s.seg_live[k] != 0 ? 1u : 0u;
    if (filled)
        atomicAdd(&s_rank, filled);
    for (uint32_t k = tid; k < n; k += THREADS) {
        const float4 a = s.c_lo[parity][first + k], b = s.c_hi[parity][first + k];
        s_box[k] = a.x;
        s_box[CAP + k] = a.y;
        s_box[2 * CAP + k] = a.z;
        s_box[3 * CAP + k] = b.x;
        s_box[4 * CAP + k] = b.y;
        s_box[5 * CAP + k] = b.z;
        s_ref[k] = s.c_ref[parity][first + k];
    }
    if (MULTI && nblocks > 1)
        cluster.sync(); // every block of the cluster is up before its memory is written
    else
        __syncthreads();
    int node = node_base + (int)(s.counters[2 * parity] + first - s_rank);
    auto box_lo = [&](int k) { return make_float4(s_box[k], s_box[CAP + k], s_box[2 * CAP + k], 0.0f); };
    auto box_hi = [&](int k) { return make_float4(s_box[3 * CAP + k], s_box[4 * CAP + k], s_box[5 * CAP + k], 0.0f); };
    const int pad = (radius + 1) & ~1;
    // Two lists of neighbours: a block may be a round ahead of another that still reads the last round's.
    for (uint32_t round = 0; n > 1; round++) { // every round merges at least one pair
        int* s_nn = s_ref + CAP + (round & 1) * CAP;
        auto found = [&](int i, int j) {
            if (MULTI && nblocks > 1) {
                for (uint32_t b = 0; b < nblocks; b++)
                    cluster.map_shared_rank(s_nn, b)[i] = j;
            } else
                s_nn[i] = j;
        };
        const uint32_t threads = THREADS * nblocks, me = rank * THREADS + tid;
        if ((n + 1) / 2 > threads / 2) {
            for (int own = 2 * (int)me; own < (int)n; own += 2 * (int)threads) {
                int j0, j1;
                nn_pair<false>(s_box, CAP, nullptr, own, max(0, own - pad), min(own + pad, ((int)n - 1) & ~1), (int)n, radius, j0, j1);
                found(own, j0);
                if (own + 1 < (int)n)
                    found(own + 1, j1);
            }
        } else {
            // lanes per cluster: as many as the blocks have to spare (a power of two)
            uint32_t share = 1;
            while (share < 32 && 2 * share * n <= threads)
                share *= 2;
            const uint32_t k = me;
            if (k < (n * share + 31) / 32 * 32) { // whole warps: the shuffles below
                const int i = (int)(k / share), sub = (int)(k % share);
                float best = 0.0f;
                int bj = -1;
                if (i < (int)n) {
                    const float4 li = box_lo(i), hi_i = box_hi(i);
                    const int j_end = min((int)n - 1, i + radius);
#pragma unroll 4
                    for (int j = max(0, i - radius) + sub; j <= j_end; j += (int)share) {
                        const float d = half_area(box_min(li, box_lo(j)), box_max(hi_i, box_hi(j)));
                        if (j != i && (bj < 0 || d < best)) {
                            best = d;
                            bj = j;
                        }
                    }
                }
                for (uint32_t o = 1; o < share; o <<= 1) {
                    const float od = __shfl_xor_sync(0xffffffffu, best, o);
                    const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
                    if (oj >= 0 && (bj < 0 || od < best || (od == best && oj < bj))) {
                        best = od;
                        bj = oj;
                    }
                }
                if (sub == 0 && i < (int)n)
                    found(i, bj);
            }
        }
        if (MULTI && nblocks > 1) {
            cluster.sync();
            if (n <= SOLO_CLUSTERS) {
                nblocks = 1; // nothing of another block's memory is touched from here on
                if (rank != 0)
                    return;
            }
        } else
            __syncthreads();
        // each thread's own run of clusters
        const uint32_t per = (n + THREADS - 1) / THREADS;
        uint32_t flags = 0, mine = 0; // flags: 2 bits each (survives, merges); mine: merges << 16 | survivors
#pragma unroll
        for (int c = 0; c < PER; c++) {
            const int i = (int)(tid * per) + c;
            if (c >= (int)per || i >= (int)n)
                continue;
            const int j = s_nn[i];
            const bool mutual = s_nn[j] == i;
            if (mutual && i > j)
                continue;
            flags |= (mutual ? 3u : 1u) << (2 * c);
            mine += mutual ? (1u << 16) + 1u : 1u;
        }
        // exclusive sums over the block
        uint32_t sum = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= (uint32_t)o)
                sum += v;
        }
        if (lane == 31)
            s_warp[warp] = sum;
        __syncthreads();
        const uint32_t of_warp = lane < THREADS / 32 ? s_warp[lane] : 0u;
        const uint32_t total = __reduce_add_sync(0xffffffffu, of_warp);
        // the survivors are read before any is overwritten
        const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? of_warp : 0u) + sum - mine;
        float4 lo[PER], hi[PER];
        int ref[PER];
        int id = node + (int)(before >> 16);
#pragma unroll
        for (int c = 0; c < PER; c++) {
            const uint32_t fl = (flags >> (2 * c)) & 3u;
            if (!fl)
                continue;
            const int i = (int)(tid * per) + c;
            lo[c] = box_lo(i);
            hi[c] = box_hi(i);
            ref[c] = s_ref[i];
            if (fl & 2u) {
                const int j = s_nn[i];
                const float4 lo_j = box_lo(j), hi_j = box_hi(j);
                if (rank == 0)
                    nodes[id] = merged_node(lo[c], hi[c], ref[c], lo_j, hi_j, s_ref[j]);
                lo[c] = box_min(lo[c], lo_j);
                hi[c] = box_max(hi[c], hi_j);
                ref[c] = id++;
            }
        }
        __syncthreads();
        int o = (int)(before & 0xFFFFu);
#pragma unroll
        for (int c = 0; c < PER; c++) {
            if (!((flags >> (2 * c)) & 3u))
                continue;
            s_box[o] = lo[c].x;
            s_box[CAP + o] = lo[c].y;
            s_box[2 * CAP + o] = lo[c].z;
            s_box[3 * CAP + o] = hi[c].x;
            s_box[4 * CAP + o] = hi[c].y;
            s_box[5 * CAP + o] = hi[c].z;
            s_ref[o] = ref[c];
            o++;
        }
        node += (int)(total >> 16);
        n = total & 0xFFFFu;
        __syncthreads();
        if ((total >> 16) == 0)
            break; // only boxes that are not numbers get here: the root is then any of the clusters
    }
    if (tid == 0 && rank == 0)
        s.seg_root[m] = s_ref[0];
}

// ---- SAH leaf collapse of the BLAS trees (PLOC output, leaves of one triangle)
constexpr int TREE_DEPTH_CAP = 1 << 16; // walks of a valid tree end far earlier
// Cost model (unnormalised SAH): leaf of n triangles = CT * n * A, interior
// node = CI * A + cost(c0) + cost(c1), A the node's surface area.  A node
// whose best form is a leaf of at most LEAF_MAX triangles is collapsed; the
// triangles are then laid out depth-first so every leaf is a contiguous range.

__global__ void k_link_parents(Scratch s, const BvhNode* nodes, uint32_t nb)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb)
        return;
    const int4 l = nodes[i].link;
    const int cs[2] = {l.x, l.y};
    for (int k = 0; k < 2; k++) {
        if (cs[k] >= 0)
            s.parent[cs[k]] = (int)i;
        else
            s.leaf_parent[leaf_first(cs[k])] = (int)i;
    }
    s.visits[i] = 0;
}

__device__ __forceinline__ float child_area(const BvhNode& nd, int k)
{
    return k == 0 ? half_area(make_float4(nd.c0xy.x, nd.c0xy.z, nd.c01z.x, 0.0f), make_float4(nd.c0xy.y, nd.c0xy.w, nd.c01z.y, 0.0f))
                  : half_area(make_float4(nd.c1xy.x, nd.c1xy.z, nd.c01z.z, 0.0f), make_float4(nd.c1xy.y, nd.c1xy.w, nd.c01z.w, 0.0f));
}

__device__ __forceinline__ float node_area(const BvhNode& nd)
{
    const float4 lo = make_float4(fminf(nd.c0xy.x, nd.c1xy.x), fminf(nd.c0xy.z, nd.c1xy.z), fminf(nd.c01z.x, nd.c01z.z), 0.0f);
    const float4 hi = make_float4(fmaxf(nd.c0xy.y, nd.c1xy.y), fmaxf(nd.c0xy.w, nd.c1xy.w), fmaxf(nd.c01z.y, nd.c01z.w), 0.0f);
    return half_area(lo, hi);
}

// Bottom-up from every triangle: the second arrival at a node evaluates it.
__global__ void k_sah_up(Scratch s, const BvhNode* nodes, uint32_t n, float ci, float ct, uint32_t leaf_max)
{
    const uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= n)
        return;
    int node = s.leaf_parent[pos];
    for (int depth = 0; node >= 0 && depth < TREE_DEPTH_CAP; depth++) {
        __threadfence();
        if (atomicAdd(&s.visits[node], 1u) == 0)
            return; // the sibling subtree finishes this node
        const BvhNode nd = nodes[node];
        const int cs[2] = {nd.link.x, nd.link.y};
        uint32_t cnt = 0;
        float sub = 0.0f;
        for (int k = 0; k < 2; k++) {
            if (cs[k] < 0) {
                cnt += 1;
                sub += ct * child_area(nd, k);
            } else {
                cnt += __ldcg(&s.cnt[cs[k]]);
                sub += __ldcg(&s.sah[cs[k]]);
            }
        }
        const float a = node_area(nd);
        const float inner = ci * a + sub;
        const float leaf = ct * (float)cnt * a;
        const bool col = cnt <= leaf_max && leaf <= inner;
        __stcg(&s.cnt[node], cnt);
        __stcg(&s.sah[node], col ? leaf : inner);
        __stcg(&s.collapse[node], col ? 1u : 0u);
        __threadfence();
        node = s.parent[node];
    }
}

// Depth-first positions: a triangle's (or node's) offset inside its mesh is
// the sum of the left siblings' triangle counts along the path to the root.
__device__ __forceinline__ uint32_t dfs_offset(const Scratch& s, const BvhNode* nodes, int node, int from_ref, int& root)
{
    uint32_t off = 0;
    int child = from_ref;
    for (int depth = 0; node >= 0 && depth < TREE_DEPTH_CAP; depth++) {
        const int4 l = nodes[node].link;
        if (child == l.y)
            off += l.x < 0 ? 1u : s.cnt[l.x];
        root = node;
        child = node;
        node = s.parent[node];
    }
    return off;
}

__global__ void k_dfs_positions(Scratch s, const BvhNode* nodes, uint32_t n)
{
    const uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= n)
        return;
    const uint32_t seg = (uint32_t)(s.keys_out[pos] >> KEY_SEG_SHIFT);
    int root = -1;
    const uint32_t off = dfs_offset(s, nodes, s.leaf_parent[pos], make_leaf(pos, 1), root);
    s.newpos[pos] = s.seg_base[seg] + off;
}

// A subtree's first depth-first slot is its leftmost triangle's.
__global__ void k_node_offsets(Scratch s, const BvhNode* nodes, uint32_t nb)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb)
        return;
    int c = (int)i;
    for (int depth = 0; c >= 0 && depth < TREE_DEPTH_CAP; depth++)
        c = nodes[c].link.x;
    s.node_off[i] = c < 0 ? s.newpos[leaf_first(c)] : 0u;
}

__global__ void k_rewrite_links(Scratch s, BvhNode* nodes, uint32_t nb)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb)
        return;
    int4 l = nodes[i].link;
    int* cs[2] = {&l.x, &l.y};
    for (int k = 0; k < 2; k++) {
        const int c = *cs[k];
        if (c < 0)
            *cs[k] = make_leaf(s.newpos[leaf_first(c)], 1);
        else if (s.collapse[c])
            *cs[k] = make_leaf(s.node_off[c], s.cnt[c]);
    }
    nodes[i].link = l;
}

__global__ void k_rewrite_roots(Scratch s, uint32_t nseg)
{
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nseg)
        return;
    const int r = s.seg_root[m];
    if (r >= 0) {
        if (s.collapse[r])
            s.seg_root[m] = make_leaf(s.node_off[r], s.cnt[r]);
    } else if (ref_is_leaf(r)) {
        s.seg_root[m] = make_leaf(s.newpos[leaf_first(r)], 1);
    }
}

__global__ void k_identity_positions(Scratch s, uint32_t n)
{
    const uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos < n)
        s.newpos[pos] = pos;
}

__global__ void k_write_tris(BvhBuildInput in, Scratch s, TriRec* tris)
{
    uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= in.tri_count)
        return;
    uint32_t g = s.vals_out[pos];
    uint32_t m = s.seg[g];
    uint32_t local = g - in.mesh_tri_base[m];
    uint32_t ib = in.mesh_index_offset[m] + 3 * local;
    uint32_t vb = in.mesh_vertex_offset[m];
    float4 a = in.vertices[2 * (size_t)(vb + in.indices[ib + 0])];
    float4 b = in.vertices[2 * (size_t)(vb + in.indices[ib + 1])];
    float4 c = in.vertices[2 * (size_t)(vb + in.indices[ib + 2])];
    TriRec r;
    r.v0 = make_float4(a.x, a.y, a.z, __uint_as_float(local));
    r.v1 = make_float4(b.x, b.y, b.z, 0.0f);
    r.v2 = make_float4(c.x, c.y, c.z, 0.0f);
    tris[s.newpos[pos]] = r;
}

__global__ void k_set_roots(BvhBuildInput in, const int* mesh_root, DevInstance* dinst)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= in.instance_count)
        return;
    uint32_t m = in.inst_mesh[i];
    dinst[i].blas_root = m < in.mesh_count ? mesh_root[m] : REF_EMPTY;
    dinst[i].mesh = m;
}

inline unsigned blocks(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

int bits_for(uint32_t v)
{
    int b = 0;
    while ((1ull << b) < (uint64_t)v)
        b++;
    return b;
}

bool use_ploc()
{
    static const bool v = [] {
        const char* e = std::getenv("PT_BVH");
        return !(e && std::strcmp(e, "lbvh") == 0);
    }();
    return v;
}

// The TLAS builder may differ (PT_BVH_TLAS=lbvh|ploc; default: as PT_BVH).
bool use_ploc_tlas()
{
    static const bool v = [] {
        const char* e = std::getenv("PT_BVH_TLAS");
        if (e && std::strcmp(e, "lbvh") == 0)
            return false;
        if (e && std::strcmp(e, "ploc") == 0)
            return true;
        return use_ploc();
    }();
    return v;
}

// k_ploc_block, `cluster` blocks to a segment (MULTI).
template <int THREADS, int CAP, bool MULTI>
cudaError_t launch_ploc_block(const Scratch& s, int parity, uint32_t nseg, BvhNode* nodes, int node_base, uint32_t lo_count,
                              uint32_t multi_count, uint32_t cluster, int radius, cudaStream_t st)
{
    const int bytes = 9 * CAP * (int)sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(k_ploc_block<THREADS, CAP, MULTI>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess)
        return e;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = cluster;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = nseg * cluster;
    cfg.blockDim = THREADS;
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = MULTI ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_ploc_block<THREADS, CAP, MULTI>, s, parity, nodes, node_base, lo_count, multi_count, radius);
}

// After the rounds over all segments: blocks for the small segments and
// clusters of them for the others.  The clusters are as large as leaves a
// multiprocessor to each block, and take the small segments along (one block
// each) where all of them fit: one launch instead of two, one behind the other.
cudaError_t finish_segments(const Scratch& s, int parity, uint32_t nseg, uint32_t most, uint32_t large, BvhNode* nodes, int node_base,
                            int radius, cudaStream_t st)
{
    int dev = 0, sm_count = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess)
        return e;
    const uint32_t sms = (uint32_t)sm_count;
    if (most <= PLOC_SMALL_CAP || nseg > sms)
        e = launch_ploc_block<PLOC_SMALL_CAP / 2, PLOC_SMALL_CAP, false>(s, parity, nseg, nodes, node_base, 0u, 0u, 1u, radius, st);
    if (e != cudaSuccess || most <= PLOC_SMALL_CAP)
        return e;
    const uint32_t small = nseg > sms ? 0u : nseg - large;
    uint32_t cluster = 8;
    while (cluster > 1 && cluster * large + small > sms)
        cluster /= 2;
    return launch_ploc_block<1024, PLOC_BLOCK_CAP, true>(s, parity, nseg, nodes, node_base, nseg > sms ? PLOC_SMALL_CAP : 0u, PLOC_SMALL_CAP,
                                                         cluster, radius, st);
}

// PLOC over the sorted primitives: rounds over all segments until the largest
// has at most PLOC_BLOCK_CAP clusters, then finish_segments.  A round takes
// about 0.84 of the clusters to the next (0.56 the first), so the host
// estimates how many are needed and looks at the counters once or twice.
cudaError_t build_ploc(Scratch& s, uint32_t n, uint32_t nseg, BvhNode* nodes, int node_base, int mode_tlas, cudaStream_t st)
{
    const int radius = ploc_radius(mode_tlas);
    k_ploc_init<<<blocks(n, 256), 256, 0, st>>>(s, n, mode_tlas);
    const uint32_t init[4] = {0u, n, 0u, 0u};
    cudaError_t e = cudaMemcpyAsync(s.counters, init, sizeof(init), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess)
        return e;
    const size_t nn_bytes = 7 * sizeof(float) * (size_t)(NN_CLUSTERS + 2 * ((radius + 1) & ~1));
    int parity = 0;
    uint32_t cap = n, rounds = 0, most = 0, large = 0;
    for (;;) {
        if ((e = cudaMemsetAsync(&s.counters[4], 0, 3 * sizeof(uint32_t), st)) != cudaSuccess)
            return e;
        k_ploc_segments<<<blocks(nseg, 128), 128, 0, st>>>(s, parity, nseg);
        uint32_t c[7];
        e = cudaMemcpyAsync(c, s.counters, sizeof(c), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(st);
        if (e != cudaSuccess)
            return e;
        cap = c[2 * parity + 1];
        most = c[4];
        large = c[6];
        s.blas_nodes = n - c[5]; // a segment of k primitives gets k - 1 nodes
        if (most <= PLOC_BLOCK_CAP)
            break;
        if (rounds > n)
            return cudaErrorUnknown; // every round merges at least one pair while a segment has two clusters
        const double ratio = (double)most / PLOC_BLOCK_CAP;
        const uint32_t more = (uint32_t)std::ceil(std::log(rounds == 0 ? std::max(0.56 * ratio, 1.01) : ratio) / 0.174) + (rounds == 0 ? 1u : 0u);
        for (uint32_t k = 0; k < std::min(std::max(more, 1u), 32u); k++, rounds++) {
            const uint32_t* live = &s.counters[2 * parity + 1];
            k_ploc_nn<<<blocks(cap, NN_CLUSTERS), NN_THREADS, nn_bytes, st>>>(s.c_lo[parity], s.c_hi[parity], s.c_seg[parity], live, radius,
                                                                           s.nn);
            size_t bytes = s.scan_bytes;
            if ((e = cub::DeviceScan::ExclusiveSum(s.scan_temp, bytes, ploc_flags(s.nn, live), s.scan, (int)cap, st)) != cudaSuccess)
                return e;
            k_ploc_merge<<<blocks(cap, 128), 128, 0, st>>>(s, parity, nodes, node_base);
            parity ^= 1;
        }
    }
    return finish_segments(s, parity, nseg, most, large, nodes, node_base, radius, st);
}

float env_float(const char* name, float dflt)
{
    const char* e = std::getenv(name);
    return e ? (float)std::atof(e) : dflt;
}

// Collapses the BLAS trees of `nb` nodes over n triangles and fills newpos
// (identity when collapse is off: PT_LEAF_MAX=1 or the radix tree).
cudaError_t collapse_leaves(Scratch& s, uint32_t n, uint32_t nseg, BvhNode* nodes, uint32_t nb, cudaStream_t st)
{
    // Off by default (PT_LEAF_MAX=1): on the mid scene leaves of up to 2-4
    // triangles cut node visits per ray from 28.8 to 27.4 but raised triangle
    // tests from 2.5 to 2.9 and ran 1 % slower (11 % slower at PT_SAH_CT=0.5).
    static const uint32_t leaf_max = (uint32_t)std::min(4, std::max(1, (int)env_float("PT_LEAF_MAX", 1.0f)));
    static const float ct = env_float("PT_SAH_CT", 1.0f);
    if (n == 0)
        return cudaSuccess;
    if (!use_ploc() || leaf_max <= 1 || nb == 0) {
        k_identity_positions<<<blocks(n, 256), 256, 0, st>>>(s, n);
        return cudaGetLastError();
    }
    cudaMemsetAsync(s.parent, 0xFF, sizeof(int) * nb, st);
    cudaMemsetAsync(s.leaf_parent, 0xFF, sizeof(int) * n, st); // single-triangle meshes have no parent node
    k_link_parents<<<blocks(nb, 256), 256, 0, st>>>(s, nodes, nb);
    k_sah_up<<<blocks(n, 256), 256, 0, st>>>(s, nodes, n, 1.0f, ct, leaf_max);
    k_dfs_positions<<<blocks(n, 256), 256, 0, st>>>(s, nodes, n);
    k_node_offsets<<<blocks(nb, 256), 256, 0, st>>>(s, nodes, nb);
    k_rewrite_links<<<blocks(nb, 256), 256, 0, st>>>(s, nodes, nb);
    k_rewrite_roots<<<blocks(nseg, 128), 128, 0, st>>>(s, nseg);
    return cudaGetLastError();
}

// Sort + tree topology + node emission for one key set.
cudaError_t build_tree(Scratch& s, uint32_t n, uint32_t nseg, BvhNode* nodes, int node_base, int mode_tlas, cudaStream_t st)
{
    if (n == 0) {
        k_small_roots<<<blocks(nseg, 128), 128, 0, st>>>(s, nseg, mode_tlas);
        return cudaGetLastError();
    }
    k_morton<<<blocks(n, 256), 256, 0, st>>>(s, n);
    int end_bit = KEY_SEG_SHIFT + bits_for(nseg);
    if (end_bit > 64)
        return cudaErrorInvalidValue;
    size_t bytes = s.cub_bytes;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(s.cub_temp, bytes, s.keys_in, s.keys_out, s.vals_in, s.vals_out, (int)n, 0, end_bit, st);
    if (e != cudaSuccess)
        return e;
    if (mode_tlas ? use_ploc_tlas() : use_ploc()) {
        k_small_roots<<<blocks(nseg, 128), 128, 0, st>>>(s, nseg, mode_tlas);
        return build_ploc(s, n, nseg, nodes, node_base, mode_tlas, st);
    }
    cudaMemsetAsync(s.parent, 0xFF, sizeof(int) * n, st);
    if (n > 1)
        k_karras<<<blocks(n - 1, 256), 256, 0, st>>>(s, (int)n, node_base, mode_tlas);
    k_small_roots<<<blocks(nseg, 128), 128, 0, st>>>(s, nseg, mode_tlas);
    if (n > 1) {
        k_bottom_up<<<blocks(n, 256), 256, 0, st>>>(s, (int)n);
        k_emit_nodes<<<blocks(n - 1, 256), 256, 0, st>>>(s, (int)n, nodes, node_base, mode_tlas);
    }
    return cudaGetLastError();
}

} // namespace

size_t bvh_node_count(uint32_t tri_count, uint32_t instance_count)
{
    return (size_t)(tri_count > 1 ? tri_count - 1 : 0) + (instance_count > 1 ? instance_count - 1 : 0) + 1;
}

// 4-wide nodes from the finished BVH2, one per BVH2 node (same index): the
// children of node i's children in order (c00, c01, c10, c11), a child that
// is a leaf standing for itself.  (Filling the four slots greedily by box
// surface instead measured 1.3 % slower on the mid scene, and the order
// c00, c10, c01, c11 1.2 % slower: sibling boxes stay next to each other.)
// Boxes are the BVH2's rounded outwards to half precision (lower planes
// toward -inf, upper toward +inf), so every 4-wide box contains the one the
// BVH2 tests and no hit is lost; the node takes 64 bytes instead of 128 (mid
// scene 1,024x1,024 at 128 spp: 1,582 -> 1,609 Mpath-segs/s, heavy scene
// 470 -> 509, node visits per ray +3.7 %).  A plane beyond the half range
// (|x| > 65504) rounds to an infinity; the node stays conservative, but
// `*overflow` is set so that the caller traverses the BVH2 instead (an
// infinite plane times the infinite inverse direction of an axis-parallel ray
// gives NaN slab distances).  An unused child slot holds planes that no ray
// with a finite inverse direction meets (x planes at +inf, y planes at -inf: a
// ray that goes toward both has its z exit before the infinite entry), so the
// traversal need not compare the links.  Slots of the node array that no tree
// uses hold zeros (the caller clears the array before the build); the bounds check
// keeps their derivation inside the array.
__global__ void k_make_bvh4(const BvhNode* nodes, uint32_t n, Bvh4Node* out, uint32_t* overflow)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const BvhNode nd = nodes[i];
    float b[6][4];
    int ref[4];
    int k = 0;
    auto put = [&](float4 xy, float zlo, float zhi, int r) {
        b[0][k] = xy.x;
        b[1][k] = xy.y;
        b[2][k] = xy.z;
        b[3][k] = xy.w;
        b[4][k] = zlo;
        b[5][k] = zhi;
        ref[k] = r;
        k++;
    };
    for (int c = 0; c < 2; c++) {
        const int cr = c == 0 ? nd.link.x : nd.link.y;
        if (cr >= 0 && (uint32_t)cr < n) {
            const BvhNode g = nodes[cr];
            put(g.c0xy, g.c01z.x, g.c01z.y, g.link.x);
            put(g.c1xy, g.c01z.z, g.c01z.w, g.link.y);
        } else if (c == 0) {
            put(nd.c0xy, nd.c01z.x, nd.c01z.y, cr);
        } else {
            put(nd.c1xy, nd.c01z.z, nd.c01z.w, cr);
        }
    }
    for (; k < 4; k++) {
        for (int a = 0; a < 6; a++)
            b[a][k] = a < 2 ? __int_as_float(0x7f800000) : a < 4 ? __int_as_float(0xff800000) : 0.0f;
        ref[k] = REF_EMPTY;
    }
    Bvh4Node o;
    uint32_t q[6][2];
    for (int a = 0; a < 6; a++) {
        for (int j = 0; j < 2; j++) {
            // lower planes (even a) rounded toward -inf, upper toward +inf
            const __half h0 = (a & 1) ? __float2half_ru(b[a][2 * j]) : __float2half_rd(b[a][2 * j]);
            const __half h1 = (a & 1) ? __float2half_ru(b[a][2 * j + 1]) : __float2half_rd(b[a][2 * j + 1]);
            q[a][j] = (uint32_t)__half_as_ushort(h0) | ((uint32_t)__half_as_ushort(h1) << 16);
            if ((__hisinf(h0) && ref[2 * j] != REF_EMPTY) || (__hisinf(h1) && ref[2 * j + 1] != REF_EMPTY))
                *overflow = 1u;
        }
    }
    o.x = make_uint4(q[0][0], q[0][1], q[1][0], q[1][1]);
    o.y = make_uint4(q[2][0], q[2][1], q[3][0], q[3][1]);
    o.z = make_uint4(q[4][0], q[4][1], q[5][0], q[5][1]);
    o.link = make_int4(ref[0], ref[1], ref[2], ref[3]);
    out[i] = o;
}

cudaError_t build_bvh4(const BvhNode* nodes, uint32_t n, Bvh4Node* out, uint32_t* overflow, cudaStream_t st)
{
    if (n == 0)
        return cudaSuccess;
    k_make_bvh4<<<blocks(n, 128), 128, 0, st>>>(nodes, n, out, overflow);
    return cudaGetLastError();
}

bool use_bvh4()
{
    static const bool on = [] {
        const char* e = std::getenv("PT_BVH_WIDTH");
        return !(e && std::atoi(e) == 2);
    }();
    return on;
}

size_t bvh_scratch_bytes(uint32_t mesh_count, uint32_t tri_count, uint32_t instance_count)
{
    uint32_t n = tri_count > instance_count ? tri_count : instance_count;
    uint32_t nseg = mesh_count > 1 ? mesh_count : 1;
    return scratch_bytes_for(n, nseg) + 6 * sizeof(int) * (size_t)(nseg + 1) + 512;
}

cudaError_t bvh_build(const BvhBuildInput& in, BvhBuildOutput& out, void* scratch, size_t scratch_bytes, cudaStream_t st)
{
    if (scratch_bytes < bvh_scratch_bytes(in.mesh_count, in.tri_count, in.instance_count))
        return cudaErrorInvalidValue;
    uint32_t n_max = in.tri_count > in.instance_count ? in.tri_count : in.instance_count;
    uint32_t nseg_max = in.mesh_count > 1 ? in.mesh_count : 1;
    Scratch s = carve_scratch(scratch, n_max, nseg_max);
    // per-mesh primitive boxes survive the TLAS pass: keep them after the scratch
    size_t used = (size_t)((char*)s.cub_temp - (char*)scratch) + s.cub_bytes;
    int* mesh_box = (int*)(((uintptr_t)scratch + used + 255) & ~(uintptr_t)255);
    cudaError_t e;

    // ---- BLAS: every mesh in one key set
    if (in.mesh_count > 0) {
        k_init_bounds<<<blocks(in.mesh_count, 128), 128, 0, st>>>(s.seg_cb, mesh_box, s.seg_root, in.mesh_count);
        cudaMemcpyAsync(s.seg_base, in.mesh_tri_base, sizeof(uint32_t) * (in.mesh_count + 1), cudaMemcpyDeviceToDevice, st);
        if (in.tri_count > 0) {
            Scratch sb = s;
            sb.seg_box = mesh_box;
            k_tri_boxes<<<blocks(in.tri_count, BOUNDS_THREADS), BOUNDS_THREADS, 0, st>>>(in, sb);
        }
        s.blas_nodes = 0;
        e = build_tree(s, in.tri_count, in.mesh_count, out.nodes, 0, 0, st);
        if (e == cudaSuccess)
            e = collapse_leaves(s, in.tri_count, in.mesh_count, out.nodes, s.blas_nodes, st);
        if (e != cudaSuccess)
            return e;
        if (in.tri_count > 0)
            k_write_tris<<<blocks(in.tri_count, 256), 256, 0, st>>>(in, s, out.tris);
        cudaMemcpyAsync(out.mesh_root, s.seg_root, sizeof(int) * in.mesh_count, cudaMemcpyDeviceToDevice, st);
    }
    if (in.instance_count == 0) {
        out.tlas_root = REF_EMPTY;
        return cudaGetLastError();
    }
    k_set_roots<<<blocks(in.instance_count, 128), 128, 0, st>>>(in, out.mesh_root, out.dinst);

    // ---- TLAS over instance world boxes (one segment)
    int tlas_base = (int)(in.tri_count > 1 ? in.tri_count - 1 : 0);
    uint32_t tb[2] = {0, in.instance_count};
    k_init_bounds<<<1, 32, 0, st>>>(s.seg_cb, s.seg_box, s.seg_root, 1);
    cudaMemcpyAsync(s.seg_base, tb, sizeof(tb), cudaMemcpyHostToDevice, st);
    k_inst_boxes<<<blocks((uint64_t)in.instance_count * 32, BOUNDS_THREADS), BOUNDS_THREADS, 0, st>>>(in, mesh_box, out.mesh_root, out.nodes, s);
    e = build_tree(s, in.instance_count, 1, out.nodes, tlas_base, 1, st);
    if (e != cudaSuccess)
        return e;
    int root = REF_EMPTY;
    e = cudaMemcpyAsync(&root, s.seg_root, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess)
        return e;
    e = cudaStreamSynchronize(st);
    out.tlas_root = root;
    return e;
}

} // namespace pt
