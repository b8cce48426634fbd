// tc.cuh — sm_103a building blocks for the denoiser's tensor-core kernels:
// mbarriers, TMA (tiled tensor loads and 1-D bulk copies) and the fifth-
// generation tensor core (tcgen05: TMEM allocation, MMA from shared-memory
// matrix descriptors, commit to an mbarrier, TMEM loads).
//
// Every wait is bounded: a wait that runs out returns false, the caller
// records an error word and returns instead of hanging the GPU.
#pragma once
#include <cuda.h>
#include <cstdint>

namespace pt {
namespace nn {

// SM clock cycles a barrier wait may take before it gives up (about two
// seconds at 2 GHz; a healthy wait here lasts microseconds).
constexpr long long WAIT_CYCLES = 4000000000ll;

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

// Makes barrier initialisation visible to the async proxy (TMA, tcgen05).
__device__ __forceinline__ void mbar_init_fence()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Arrive once and add `bytes` to the transaction count of the current phase.
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}

// Waits for the phase with the given parity to complete; false on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity)
{
    if (mbar_try_wait(bar, parity))
        return true;
    const long long start = clock64();
    while (!mbar_try_wait(bar, parity))
        if (clock64() - start > WAIT_CYCLES)
            return false;
    return true;
}

// --------------------------------------------------------------------- TMA
// Tiled 4-D tensor load (box given by the tensor map); out-of-range
// elements are zero-filled and still count toward the transaction bytes.
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3)
{
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_addr(dst)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_addr(bar))
                 : "memory");
}

// Contiguous global -> shared copy by the TMA engine (16-byte aligned ends).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// ----------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(cols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Shared-memory matrix descriptor, no swizzle.  `lbo` and `sbo` are byte
// strides between 8x16-byte core matrices: without swizzling, lbo steps
// along K and sbo along M/N for K-major and MN-major operands alike.
// Bits 46-47 hold the descriptor version (1).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16 with BF16 inputs and FP32 accumulation.
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t m, uint32_t n, bool a_mn_major, bool b_mn_major)
{
    return (1u << 4)                           // D: f32
           | (1u << 7)                         // A: bf16
           | (1u << 10)                        // B: bf16
           | ((a_mn_major ? 1u : 0u) << 15)    // A major-ness
           | ((b_mn_major ? 1u : 0u) << 16)    // B major-ness
           | ((n >> 3) << 17)                  // N / 8
           | ((m >> 4) << 24);                 // M / 16
}

// D[tmem] (+)= A * B on the tensor core; issued by one thread.
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
                 : "memory");
}

// The same for a whole converged warp, of which one elected lane (the same
// every time) issues: the loop around it stays uniform, and a
// multiplication takes 25 cycles to issue instead of 45.  COLLECT says what
// happens to the A operand in the tensor core's collector buffer: kept for the
// next ones (FILL), taken from there (USE), taken for the last time (LAST_USE),
// or neither.  Reading A (128 rows, 32 cycles) is most of a multiplication by
// few columns: measured per multiplication with N = 16, 32, 64, 96: 39, 40, 48
// and 56 cycles, and 20, 25, 36 and 48 when three share A.
enum Collect { DISCARD, FILL, USE, LAST_USE };

template <Collect COLLECT>
__device__ __forceinline__ void mma_bf16_warp(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
#define PT_MMA_WARP(OP)                                                             \
    asm volatile("{\n\t.reg .pred p, q;\n\t"                                       \
                 "elect.sync _|q, 0xffffffff;\n\t"                                  \
                 "setp.ne.b32 p, %4, 0;\n\t"                                        \
                 "@q tcgen05.mma.cta_group::1.kind::f16.collector::a::" OP          \
                 " [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),                        \
                 "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)              \
                 : "memory")
    if (COLLECT == FILL)
        PT_MMA_WARP("fill");
    else if (COLLECT == USE)
        PT_MMA_WARP("use");
    else if (COLLECT == LAST_USE)
        PT_MMA_WARP("lastuse");
    else
        PT_MMA_WARP("discard");
#undef PT_MMA_WARP
}

// mma_commit for multiplications issued by mma_bf16_warp.
__device__ __forceinline__ void mma_commit_warp(uint64_t* bar)
{
    asm volatile("{\n\t.reg .pred q;\n\t"
                 "elect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_addr(bar))
                 : "memory");
}

// Arrives on `bar` once every tcgen05 operation this thread issued is done.
__device__ __forceinline__ void mma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

// 32 TMEM lanes x 16 columns of 32 bits: lane i of the warp receives TMEM lane
// (lane base + i), columns [col, col + 16).  Warp-collective; the values are
// there after tmem_ld_wait, which ties them so that none is used before.
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                   "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    tmem_ld16_issue(taddr, r);
    tmem_ld_wait(r);
}

// 32 bytes (32-byte aligned) by one access.
__device__ __forceinline__ void store32(void* p, const uint32_t (&v)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void load32(const void* p, uint32_t (&v)[8])
{
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p)
                 : "memory");
}

} // namespace nn
} // namespace pt
