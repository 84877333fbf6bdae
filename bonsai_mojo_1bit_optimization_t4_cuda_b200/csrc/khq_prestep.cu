// khq_prestep.cu -- the five launches that precede the KHQ decode step in the reference, as one:
//   per-head RMSNorm of q and k      (head_rmsnorm_sm75_gpu, src/kernels/elementwise_sm75.mojo:362-423;
//                                     called at src/models/qwen3_5/attention.mojo:329-336)
//   K un-RoPE'd -> ring_u[slot]      (khq_capture_unroped, src/khq/runtime.mojo:432-451)
//   half-split partial RoPE of q, k  (partial_rope_sm75_gpu, elementwise_sm75.mojo:1023-1061;
//                                     attention.mojo:348-353)
//   K RoPE'd, V -> ring_k/ring_v[slot] (khq_ring_dual_sm75_gpu, elementwise_sm75.mojo:293-312;
//                                     src/khq/runtime.mojo:486)
// One warp per head (24 query heads + 4 kv heads).  The arithmetic follows the reference kernels
// step by step (per-lane strided partial sums, shuffle-down tree, fp16 rounding between the norm
// and the rotation, fp32 angle pos*freq), so un-rotated dims are bit-identical to them.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "khq_common.cuh"
#include "khq_launch.cuh"

namespace khq_prestep {

__device__ __forceinline__ void norm_head(__half* x, const float* w, int dim, float eps, int lane) {
    float sum_sq = 0.0f;
    for (int d = lane; d < dim; d += 32) {
        const float v = __half2float(x[d]);
        sum_sq += v * v;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum_sq += __shfl_down_sync(0xFFFFFFFFu, sum_sq, off);
    float rms = 0.0f;
    if (lane == 0) rms = 1.0f / sqrtf(sum_sq / (float)dim + eps);
    rms = __shfl_sync(0xFFFFFFFFu, rms, 0);
    for (int d = lane; d < dim; d += 32) {
        float n = __half2float(x[d]) * rms;
        if (w) n *= w[d];
        x[d] = __float2half(n);
    }
    __syncwarp();
}

// cosine and sine of the lane's rotary pair
__device__ __forceinline__ float2 rope_turn(int rotary_dim, int pos, float theta, int lane) {
    const float ex = -(float)(2 * lane) / (float)rotary_dim;
    const float freq = expf(logf(theta) * ex);
    const float ang = (float)pos * freq;
    return make_float2(cosf(ang), sinf(ang));
}

__device__ __forceinline__ void rope_head(__half* x, int rotary_dim, float2 turn, int lane) {
    const int half_r = rotary_dim / 2;
    if (lane < half_r) {
        const float c = turn.x, s = turn.y;
        const float x0 = __half2float(x[lane]), x1 = __half2float(x[lane + half_r]);
        x[lane] = __float2half(x0 * c - x1 * s);
        x[lane + half_r] = __float2half(x0 * s + x1 * c);
    }
    __syncwarp();
}

__device__ __forceinline__ void copy_head(__half* dst, const __half* src, int dim, int lane) {
    for (int d = lane * 8; d < dim; d += 256)
        *reinterpret_cast<uint4*>(dst + d) = *reinterpret_cast<const uint4*>(src + d);
}

// d = 256 with 64 rotary dims: a head stays in registers (lane l holds dims l + 32 i, so both halves of its rotary pair), one load
// and one store instead of three passes over global memory that depend on each other.  turn(): cosine and sine, evaluated
// while the loads are in flight.  ring_u takes the head before the rotation, ring_r (K) behind it, ring_v copies v.
template <class Turn>
__device__ __forceinline__ void head_256(__half* x, const float* w, float eps, int lane, Turn turn, __half* ring_u, __half* ring_r,
                                         __half* ring_v, const __half* v) {
    __half h[8];
    float wv[8];
    uint4 vv = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = x[lane + 32 * i];
#pragma unroll
    for (int i = 0; i < 8; ++i) wv[i] = w ? w[lane + 32 * i] : 1.0f;
    if (ring_v) vv = *reinterpret_cast<const uint4*>(v + lane * 8);
    const float2 cs = turn();
    float sum_sq = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float f = __half2float(h[i]);
        sum_sq += f * f;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum_sq += __shfl_down_sync(0xFFFFFFFFu, sum_sq, off);
    float rms = 0.0f;
    if (lane == 0) rms = 1.0f / sqrtf(sum_sq / 256.0f + eps);
    rms = __shfl_sync(0xFFFFFFFFu, rms, 0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        h[i] = __float2half(__half2float(h[i]) * rms * wv[i]);
        if (ring_u) ring_u[lane + 32 * i] = h[i];
    }
    const float x0 = __half2float(h[0]), x1 = __half2float(h[1]);
    h[0] = __float2half(x0 * cs.x - x1 * cs.y);
    h[1] = __float2half(x0 * cs.y + x1 * cs.x);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        x[lane + 32 * i] = h[i];
        if (ring_r) ring_r[lane + 32 * i] = h[i];
    }
    if (ring_v) *reinterpret_cast<uint4*>(ring_v + lane * 8) = vv;
}

// grid = H_q + H_kv warps (one block of 32 threads each).  Latency-bound, and in the chain of every step: 3.7 us behind the kernel
// before it when cosine and sine were evaluated there and the head went through global memory between the passes, 1.9 so.
__global__ void __launch_bounds__(32)
khq_prestep_kernel(__half* __restrict__ q_gate, __half* __restrict__ k, const __half* __restrict__ v,
                   const float* __restrict__ q_norm_w, const float* __restrict__ k_norm_w, __half* __restrict__ ring_k,
                   __half* __restrict__ ring_v, __half* __restrict__ ring_u, int H_q, int d, int rotary_dim, int pos,
                   float theta, float eps, int has_norms) {
    const int h = blockIdx.x, lane = threadIdx.x;
    khq::pdl_trigger();  // the kernel behind reads nothing but constants before its own wait
    const float2 cs = rope_turn(rotary_dim, pos, theta, lane);
    khq::pdl_wait();
    const bool is_q = h < H_q;
    const size_t off = (size_t)(is_q ? h : h - H_q) * d;
    __half* x = is_q ? q_gate + 2 * off : k + off;
    const float* w = !has_norms ? nullptr : is_q ? q_norm_w : k_norm_w;
    __half* u = !is_q && ring_u ? ring_u + off : nullptr;
    __half* rk = !is_q && ring_k ? ring_k + off : nullptr;
    __half* rv = !is_q && ring_v ? ring_v + off : nullptr;
    if (d == 256 && rotary_dim == 64) {
        head_256(x, w, eps, lane, [&] { return cs; }, u, rk, rv, v + off);
        return;
    }
    norm_head(x, w, d, eps, lane);
    if (u) copy_head(u, x, d, lane);
    __syncwarp();
    rope_head(x, rotary_dim, cs, lane);
    if (rk) copy_head(rk, x, d, lane);
    if (rv) copy_head(rv, v + off, d, lane);
}

// The same work for B sequences in one launch: grid = B * (H_q + H_kv) warps.  Sequence b reads
// q_gate + b * 2 * H_q * d, k / v + b * H_kv * d, appends to ring slot slots[b] of its own rings
// (ring base + b * ring_seq_stride halfs) and rotates at position positions[b].
__global__ void __launch_bounds__(32)
khq_prestep_batched_kernel(__half* __restrict__ q_gate, __half* __restrict__ k, const __half* __restrict__ v,
                           const float* __restrict__ q_norm_w, const float* __restrict__ k_norm_w,
                           __half* __restrict__ ring_k, __half* __restrict__ ring_v, __half* __restrict__ ring_u,
                           long long ring_seq_stride, const int* __restrict__ slots, const int* __restrict__ positions,
                           int H_q, int H_kv, int d, int rotary_dim, float theta, float eps, int has_norms) {
    const int per = H_q + H_kv;
    const int b = blockIdx.x / per, h = blockIdx.x % per, lane = threadIdx.x;
    khq::pdl_trigger();
    khq::pdl_wait();
    const bool is_q = h < H_q;
    const size_t in = is_q ? 0 : ((size_t)b * H_kv + (h - H_q)) * d;
    const size_t slot_off = is_q ? 0 : (size_t)b * ring_seq_stride + ((size_t)slots[b] * H_kv + (h - H_q)) * d;
    __half* x = is_q ? q_gate + ((size_t)b * H_q + h) * 2 * d : k + in;
    const float* w = !has_norms ? nullptr : is_q ? q_norm_w : k_norm_w;
    __half* u = !is_q && ring_u ? ring_u + slot_off : nullptr;
    __half* rk = !is_q && ring_k ? ring_k + slot_off : nullptr;
    __half* rv = !is_q && ring_v ? ring_v + slot_off : nullptr;
    if (d == 256 && rotary_dim == 64) {
        head_256(x, w, eps, lane, [&] { return rope_turn(64, positions[b], theta, lane); }, u, rk, rv, v + in);
        return;
    }
    norm_head(x, w, d, eps, lane);
    if (u) copy_head(u, x, d, lane);
    __syncwarp();
    rope_head(x, rotary_dim, rope_turn(rotary_dim, positions[b], theta, lane), lane);
    if (rk) copy_head(rk, x, d, lane);
    if (rv) copy_head(rv, v + in, d, lane);
}

}  // namespace khq_prestep

extern "C" int launch_khq_prestep_fp16(void* q_gate, void* k, const void* v, const void* q_norm_w,
                                       const void* k_norm_w, void* ring_k_slot, void* ring_v_slot,
                                       void* ring_u_slot, int H_q, int H_kv, int d, int rotary_dim, int pos,
                                       float rope_theta, float rms_eps, int has_norms, cudaStream_t stream) {
    if (H_q <= 0 || H_kv <= 0 || d <= 0 || !q_gate || !k || !v) return -100;
    if (d % 8 != 0 || rotary_dim <= 0 || rotary_dim > 64 || rotary_dim > d || (rotary_dim & 1)) return -103;
    const void* ptrs[] = {q_gate, k, v, ring_k_slot, ring_v_slot, ring_u_slot};
    for (const void* p : ptrs)
        if ((reinterpret_cast<uintptr_t>(p) & 15) != 0) return -104;
    const cudaError_t err = khq::launch_pdl(
        khq_prestep::khq_prestep_kernel, (unsigned)(H_q + H_kv), 0, 0, stream, 32, static_cast<__half*>(q_gate), static_cast<__half*>(k), static_cast<const __half*>(v),
        static_cast<const float*>(q_norm_w), static_cast<const float*>(k_norm_w), static_cast<__half*>(ring_k_slot),
        static_cast<__half*>(ring_v_slot), static_cast<__half*>(ring_u_slot), H_q, d, rotary_dim, pos, rope_theta,
        rms_eps, has_norms);
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

// launch_khq_prestep_fp16 for `batch` sequences at once (no counterpart in the reference, which
// serves one sequence).  slots / positions: device int32 arrays of `batch` entries (ring slot of
// the new token, its absolute position); ring_seq_stride: halfs between two sequences' rings.
extern "C" int launch_khq_prestep_batched_fp16(void* q_gate, void* k, const void* v, const void* q_norm_w,
                                               const void* k_norm_w, void* ring_k, void* ring_v, void* ring_u,
                                               long long ring_seq_stride, const void* slots, const void* positions,
                                               int batch, int H_q, int H_kv, int d, int rotary_dim, float rope_theta,
                                               float rms_eps, int has_norms, cudaStream_t stream) {
    if (batch <= 0 || H_q <= 0 || H_kv <= 0 || d <= 0 || !q_gate || !k || !v || !slots || !positions) return -100;
    if (d % 8 != 0 || rotary_dim <= 0 || rotary_dim > 64 || rotary_dim > d || (rotary_dim & 1)) return -103;
    const void* ptrs[] = {q_gate, k, v, ring_k, ring_v, ring_u};
    for (const void* p : ptrs)
        if ((reinterpret_cast<uintptr_t>(p) & 15) != 0) return -104;
    if ((ring_seq_stride & 7) != 0) return -104;
    const cudaError_t err = khq::launch_pdl(
        khq_prestep::khq_prestep_batched_kernel, (unsigned)(batch * (H_q + H_kv)), 0, 0, stream, 32, static_cast<__half*>(q_gate), static_cast<__half*>(k), static_cast<const __half*>(v),
        static_cast<const float*>(q_norm_w), static_cast<const float*>(k_norm_w), static_cast<__half*>(ring_k),
        static_cast<__half*>(ring_v), static_cast<__half*>(ring_u), ring_seq_stride, static_cast<const int*>(slots),
        static_cast<const int*>(positions), H_q, H_kv, d, rotary_dim, rope_theta, rms_eps, has_norms);
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}
