// khq_common.cuh -- shared constants and device helpers for the sm_100a KHQ kernels.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace khq {

constexpr int D = 256;          // head_dim
constexpr int NP = 64;          // 4-dim patches per row
constexpr int HKV = 4;          // kv heads
constexpr int NREP = 6;         // query heads per kv head
constexpr int HQ = HKV * NREP;  // 24
constexpr int K_PAY = 40;       // bytes per K payload row
constexpr int V_PAY = 104;      // bytes per V payload row
constexpr int MAX_OUT = 50;     // outliers kept per K row
constexpr int PART = D + 2;     // floats per partial: acc[D], max, sum_exp
constexpr float NEG_BIG = -1e20f;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- mbarrier + 1-D bulk asynchronous copy (global -> shared), no multicast ----------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up after ~2^22 polls, records it in *status and returns false.  The
// caller carries on (its result is then meaningless, and the host can see why) instead of
// spinning for ever.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int* status) {
    for (uint32_t it = 0; it < (1u << 22); ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if (it > 64) __nanosleep(32);
    }
    atomicExch(status, 1);
    return false;
}
// size must be a multiple of 16; both addresses 16-byte aligned.
__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes,
                                         uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst_smem)),
        "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// ---- programmatic dependent launch ------------------------------------------------------------
// A kernel launched with the attribute may start while the one before it in the stream still runs; wait() returns when
// that one has completed and its writes are visible.  trigger() lets the next kernel start.
//   * Late trigger, behind the kernel's own wait(): what starts then knows everything before its predecessor to be complete.  All
//     kernels but those of the next point.
//   * Early trigger, before the own wait(): the two pre-steps, the counter kernel, the ring fill, and the step's tail with a compressed region.  What
//     starts behind one of them may run beside the kernel before that one too.
// khq_ring_fill_kernel writes before its wait, behind kernels that trigger late or not at all, see there.
// So before its own wait() a kernel reads nothing but constants of the model (tables, their image: launch_khq_prepare_tables and
// the runtime order their writes) and writes nothing.  One exception: khq_window_step_kernel with a compressed region reads the step's
// inputs and rings and appends to the rings first.  decode_step_impl launches it directly behind the attention or its
// reduction, which trigger late, read no ring and write none of that.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- small math helpers ---------------------------------------------------------------------
__device__ __forceinline__ float hbits2f(uint16_t b) { return __half2float(__ushort_as_half(b)); }

// Packed pairs of fp32 (one instruction; each half is rounded like the scalar operation).
__device__ __forceinline__ void f32x2_addsub(float& s0, float& s1, float& d0, float& d1, float a0, float a1, float b0, float b1) {
    asm("{.reg .b64 a, b, s, d; mov.b64 a, {%4, %5}; mov.b64 b, {%6, %7}; add.rn.f32x2 s, a, b; sub.rn.f32x2 d, a, b;"
        " mov.b64 {%0, %1}, s; mov.b64 {%2, %3}, d;}"
        : "=f"(s0), "=f"(s1), "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
__device__ __forceinline__ void f32x2_fma(float& d0, float& d1, float a0, float a1, float b0, float b1, float c0, float c1) {
    asm("{.reg .b64 a, b, c, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mov.b64 c, {%6, %7};"
        " fma.rn.f32x2 d, a, b, c; mov.b64 {%0, %1}, d;}"
        : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}

// Unnormalised natural-order FWHT-256 when a lane holds the 8 consecutive elements 8*lane..8*lane+7: in-lane stages 1, 2, 4,
// then the cross-lane stages 8..128.  Each butterfly computes a+b and a-b exactly as a sequential implementation does: across
// lanes the lower one adds and the upper one subtracts its own value from the other's, which is one multiply-add by +1 or -1
// (exact products), two elements per instruction (12 instead of 32 instructions a stage).
__device__ __forceinline__ void fwht256_lane8(float (&v)[8], int lane) {
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        float a = v[j], b = v[j + 1];
        v[j] = a + b;
        v[j + 1] = a - b;
    }
#pragma unroll
    for (int b4 = 0; b4 < 8; b4 += 4) f32x2_addsub(v[b4], v[b4 + 1], v[b4 + 2], v[b4 + 3], v[b4], v[b4 + 1], v[b4 + 2], v[b4 + 3]);
#pragma unroll
    for (int j = 0; j < 4; j += 2) f32x2_addsub(v[j], v[j + 1], v[j + 4], v[j + 5], v[j], v[j + 1], v[j + 4], v[j + 5]);
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const float sign = (lane & m) == 0 ? 1.0f : -1.0f;
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const float o0 = __shfl_xor_sync(0xFFFFFFFFu, v[j], m), o1 = __shfl_xor_sync(0xFFFFFFFFu, v[j + 1], m);
            f32x2_fma(v[j], v[j + 1], v[j], v[j + 1], sign, sign, o0, o1);
        }
    }
}

}  // namespace khq
