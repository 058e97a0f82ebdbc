// rla_tc_ptx.cuh -- tcgen05 / TMA / mbarrier wrappers and the BF16 term split shared by the tensor-core
// kernels (rla_tc.cu, rla_tc_conv.cu).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "rla_internal.cuh"

namespace rla {

using bf16 = __nv_bfloat16;

template <int NT>
__device__ __forceinline__ void split_terms(float v, bf16 (&t)[NT]) {
    float rem = v;
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        t[q] = __float2bfloat16_rn(rem);
        rem -= __bfloat162float(t[q]);
    }
}

// Eight values at once, two per conversion instruction; o[q] holds term q (the same values as
// split_terms).
template <int NT>
__device__ __forceinline__ void split_terms8(const float (&v)[8], uint4 (&o)[NT]) {
    float r[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) r[i] = v[i];
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[i]) : "f"(r[2 * i + 1]), "f"(r[2 * i]));
            if (q + 1 < NT) {
                r[2 * i] -= __uint_as_float(w[i] << 16);
                r[2 * i + 1] -= __uint_as_float(w[i] & 0xffff0000u);
            }
        }
        o[q] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// ------------------------------------------------------------------------------------
// PTX wrappers (sm_100a)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Wait for the phase of parity `parity` to complete; gives up after limit_ns (and 2^26
// polls) or once another CTA has recorded a failure, records the failure in *status and
// returns false.
static __device__ __noinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int *status, uint64_t limit_ns) {
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t it = 0; it < (1u << 26) && limit_ns > 0; ++it) {
        if (mbar_try(bar, parity)) return true;
        if ((it & 63u) == 0u && (global_ns() - t0 > limit_ns || *(volatile int *)status != 0)) break;
    }
    atomicExch(status, 1);
    return false;
}

// Drain wait before a CTA releases its shared memory or tensor memory: waits for copies or
// MMAs already issued, whatever the pipeline limit, for at most 2 s (and 2^26 polls).
constexpr uint64_t TC_DRAIN_NS = 2000000000ull;
static __device__ __noinline__ bool mbar_drain(uint32_t bar, uint32_t parity, int *status) {
    const uint64_t t0 = global_ns();
    for (uint32_t it = 0; it < (1u << 26); ++it) {
        if (mbar_try(bar, parity)) return true;
        if ((it & 63u) == 0u && global_ns() - t0 > TC_DRAIN_NS) break;
    }
    atomicExch(status, 2);
    return false;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor, 64-byte swizzle (Blackwell descriptor version 1).
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

// Instruction descriptor of kind::f16 with BF16 inputs and an FP32 accumulator.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int a_mn_major, int b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn_major << 15) | ((uint32_t)b_mn_major << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

constexpr int TC_BM = 128, TC_BK = 32;
constexpr uint32_t TC_A_BYTES = TC_BM * TC_BK * 2;  // 8 KB per operand term

// 2-D BF16 map over a column-major array (rla_tc.cu).
int tc_make_map(rla_ctx *ctx, CUtensorMap *map, const bf16 *ptr, int64_t inner, int64_t outer, int64_t ld,
                uint32_t box_inner, uint32_t box_outer);

}  // namespace rla
