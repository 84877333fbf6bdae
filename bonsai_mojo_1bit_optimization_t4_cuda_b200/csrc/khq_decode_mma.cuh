// khq_decode_mma.cuh -- second-generation compressed-region decode: the two contractions of
// attention (q.K^T and p.V), the inverse K rotor + block sum, and the 64-dim rotary dot product
// run on the tensor cores with the 16 tokens of a block as the M dimension and the GQA group's
// six query heads (padded to 8) as N.  Included by khq_decode.cu (shares its helpers).
//
// Algebra.  K^ = RoPE_s( dinv * H256 * R * y ), y = alpha_k*k_norm*(mult*c*t + rs*sign*code).
// Everything left of y is linear, so it moves to the query side once per (sequence, layer):
//   * non-rotary output dims (>= 64):  q.K^ = y . q~,  q~ = R^T H256 (q * dinv * [dim >= 64])
//     -> one GEMM  S_pass[token, head] = T[token, dim] Q1[dim, head] + C[token, dim] Q2[dim, head]
//        with T = ternary symbols, C = sign*code (both exact in fp16), Q1 = q~*c, Q2 = q~, each accumulated by itself
//        and scaled by its row's factor afterwards;
//   * rotary output dims (< 64): the first 64 outputs of H256 are H64 of the sum of the four
//     64-dim blocks, so u[token, 64] = T * (R c)-blocks + C * R-blocks is a second GEMM with the
//     same A operands; H64, /d, the rotation by the token's angle, and a 64-deep GEMM with the raw
//     query finish it.
// V is accumulated in the rotated domain exactly as the first-generation kernel does:
//   O^T[dim, head] += V^T[dim, token] P^T[token, head], V^T = raw fp16 codebook entries (exact),
//   the per-token scales (alpha_v*v_norm*energy etc.) folded into three variants of P (dim 3: see M2State).
//
// Thread mapping (mma.sync.m16n8k16 fragments): lane = 4*g + t.  K side: token rows g and g+8,
// thread t owns the 64-dim quarter [64t, 64t+64) of both rows (mask words 4t..4t+3), k-step s
// covers dims 64t'+4s..+3 of all four quarters, i.e. the four patches that the rotor block sum
// adds up.  V side: thread (g, t) owns patch group g (patches 8g..8g+7) of tokens 2t, 2t+1,
// 2t+8, 2t+9.
//
// Registers and warps.  Twelve warps (three per scheduler) of at most 168 registers: what a warp keeps for a
// whole work item or layer -- the query-side and rotor-side B fragments and the 64 O^T accumulators -- lives in
// tensor memory, used here as a per-lane scratch file (tcgen05.st / tcgen05.ld; no tcgen05.mma), see M2_TM_COLS.
#pragma once
#include "khq_kdecode3.cuh"

namespace khq {

constexpr int M2_WPK = 3;           // warps per kv-head (12 warps: three per scheduler, at most 168 registers each)
constexpr int M2_BT = 16;           // tokens per block: one warp's share of a stage
constexpr int M2_TT = M2_BT * M2_WPK;  // tokens that the CTA's three groups advance together
constexpr int M2_THREADS = 32 * HKV * M2_WPK;
constexpr int M2_GTHREADS = 32 * HKV;  // a group: the four warps (one per kv-head) that share a block
constexpr int M2_NSTAGE = 2;           // stages per group
constexpr int M2_ROWS = M2_BT * HKV;
constexpr int M2_OFF_MASK = 0;
constexpr int M2_OFF_KPAY = M2_OFF_MASK + M2_ROWS * 64;
constexpr int M2_OFF_VPAY = M2_OFF_KPAY + M2_ROWS * K_PAY;
constexpr int M2_OFF_KN = M2_OFF_VPAY + M2_ROWS * V_PAY;
constexpr int M2_OFF_KRN = M2_OFF_KN + M2_ROWS * 2;
constexpr int M2_OFF_VN = M2_OFF_KRN + M2_ROWS * 2;
constexpr int M2_OFF_VRN = M2_OFF_VN + M2_ROWS * 2;
constexpr int M2_OFF_VSM = M2_OFF_VRN + M2_ROWS * 2;
constexpr int M2_STAGE_BYTES = M2_OFF_VSM + M2_ROWS * 4;  // 14080
constexpr int M2_STAGES_BYTES = M2_WPK * M2_NSTAGE * M2_STAGE_BYTES;

constexpr int M2_SM_STAGES = 0;
// V codebook, one row per code: for every pair of patches the two (d0, d1) words, then the two d2 halfs
// (12 bytes), so that both look-ups of a (code, patch) share one address computation.  A row has one word of
// padding: the bank of a look-up then depends on the code as well as on the patch, which spreads the
// warp's 32 look-ups (8 patches x 4 tokens per instruction) over the banks.
constexpr int M2_VQ_ROW = (NP / 2) * 12 + 4;                         // 388 bytes per code
constexpr int M2_SM_VQ = M2_SM_STAGES + M2_STAGES_BYTES;
constexpr int M2_SM_ROPE = M2_SM_VQ + 256 * M2_VQ_ROW;               // per group two buffers of M2_BT tokens x 64 floats
constexpr int M2_SM_RSC = M2_SM_ROPE + 2 * M2_TT * 64 * 4;           // 16 rows x 2 float4 per warp: scalars of a block's rows
// small tables of a layer, in the order of the prepared image
constexpr int M2_SM_FREQ = M2_SM_RSC + M2_THREADS / 32 * 16 * 32;      // 32 floats: RoPE frequencies
constexpr int M2_SM_DINV = M2_SM_FREQ + 128;                         // 64 floats: 1 / (256 d) of the rotary dims
constexpr int M2_SM_C3 = M2_SM_DINV + 256;                           // 64 patches x float2: alpha_v x (mean, half the difference 0 - 1) of the two dim-3 centroids
constexpr int M2_SM_RSTEP = M2_SM_C3 + NP * 8;                       // 32 x float2: cos / sin of M2_TT positions of each rotary pair
constexpr int M2_SM_FLAGS = M2_SM_RSTEP + 32 * 8;                    // nonzero: rotor fragments have low-order parts
constexpr int M2_SMALL_BYTES = 128 + 256 + NP * 8 + 32 * 8 + 16;
constexpr int M2_SM_BARS = M2_SM_FREQ + M2_SMALL_BYTES;              // M2_WPK * M2_NSTAGE stages, then the image's small tables and codebook
constexpr int M2_BAR_SMALL = M2_WPK * M2_NSTAGE, M2_BAR_VQ = M2_BAR_SMALL + 1, M2_NBARS = M2_BAR_VQ + 1;
constexpr int M2_SM_TMSLOT = M2_SM_BARS + M2_NBARS * 8;
constexpr int M2_SM_QR = (M2_SM_TMSLOT + 4 + 15) / 16 * 16;   // raw rotary query fragments: 4 kv-heads x 4 k-steps x 32 lanes x 8 B
// Prepared image of a layer's tables (launch_khq_prepare_tables): the codebook's shared-memory rows, the small tables, the
// rotor fragments (two uint4 per k-step and lane), and the codebook once more as [code][patch] of 8 bytes (one load per look-up
// for kernels that leave it in L2).
constexpr int M2_IMG_VQ = 0, M2_IMG_SMALL = 256 * M2_VQ_ROW, M2_IMG_ROT = M2_IMG_SMALL + M2_SMALL_BYTES, M2_IMG_VQ8 = M2_IMG_ROT + 16 * 32 * 32,
              M2_IMG_BYTES = M2_IMG_VQ8 + 256 * NP * 8;
static_assert(M2_IMG_VQ8 % 16 == 0 && M2_IMG_SMALL % 16 == 0 && M2_IMG_ROT % 16 == 0 && M2_SM_FREQ % 16 == 0 && M2_SM_QR % 16 == 0 && M2_SM_BARS % 8 == 0, "alignment");
constexpr int M2_SM_TOTAL = M2_SM_QR + HKV * 4 * 32 * 8;
// Tensor memory as a second register file.  The B fragments of the K side are per-lane constants: the query
// side (ternary part q1 and residual part q2, fp16 hi and lo, eight registers per k-step) for a whole work
// item, the rotor side (rotor x centroid and rotor, hi and lo, eight registers per k-step) for a whole layer.
// Held in registers the hi query fragments alone took 64 of the 255 across the tile loop, and the rest came
// from shared memory with six loads per k-step.  They are written to tensor memory (tcgen05.st: the query side
// once per item, the rotor side once per layer) and fetched one k-step ahead of use with two tcgen05.ld.
// Warp w owns lanes 32 (w & 3) .. +31, which it shares with the other warps of its kv-head.  Columns: 0 .. 127 =
// the kv-head's query fragments (eight per k-step: q1.x, q1.y, q2.x, q2.y and their low-order halves; written by
// the kv-head's first warp), 128 .. 255 = the rotor fragments of the lane quadrant (eight per k-step: b1.x, b1.y,
// b2.x, b2.y and their low-order halves; the same values in all four quadrants), 256 + 80 (w >> 2) .. +79 = the
// warp's O^T accumulators, twenty per pair of patches, which are in registers only while the V side of that pair runs.
constexpr uint32_t M2_TM_COLS = 512, M2_TM_ROT = 128, M2_TM_ACC = 256, M2_TM_ACC_WARP = 80;
static_assert(M2_TM_ACC + M2_TM_ACC_WARP * M2_WPK <= M2_TM_COLS, "tensor-memory columns");
static_assert(M2_SM_TOTAL <= 227 * 1024 && M2_SM_C3 % 16 == 0 && M2_SM_ROPE % 16 == 0 && M2_SM_VQ % 16 == 0,
              "shared memory budget");
// Per-warp record: six heads of 256 floats, four floats of padding after every 32 (none after the last), then the maxima and
// sums.  A thread stores eight consecutive dims of two heads; with this padding the float4 stores of a quarter-warp hit
// distinct banks (unpadded, all 24 lanes of a store hit one bank and the records cost 7.5 us of a 25 us launch).
constexpr int M2_REC_HEAD = D + 28, M2_REC_FLOATS = NREP * M2_REC_HEAD + 2 * NREP;
static_assert(HKV * M2_WPK * M2_REC_FLOATS * 4 <= M2_STAGES_BYTES, "records alias the stages");
__device__ __forceinline__ HeadRec m2_head_of_record(const float* rec, int hh) {
    return {rec + hh * M2_REC_HEAD, rec + NREP * M2_REC_HEAD + hh, rec + NREP * M2_REC_HEAD + NREP + hh};
}
__device__ __forceinline__ void m2_store_record(const WarpState& st, float* rec, int lane) {
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
        float* p = rec + h * M2_REC_HEAD + lane * 8 + 4 * (lane >> 2);
        *reinterpret_cast<float4*>(p) = make_float4(st.acc[h][0], st.acc[h][1], st.acc[h][2], st.acc[h][3]);
        *reinterpret_cast<float4*>(p + 4) = make_float4(st.acc[h][4], st.acc[h][5], st.acc[h][6], st.acc[h][7]);
        if (lane == h) {  // static indices keep the state in registers
            rec[NREP * M2_REC_HEAD + h] = st.m[h];
            rec[NREP * M2_REC_HEAD + NREP + h] = st.l[h];
        }
    }
}
static_assert(HKV * NREP * D * 4 <= M2_SM_RSC - M2_SM_ROPE, "the query build's scratch aliases the RoPE buffers");
static_assert(M2_STAGE_BYTES % 16 == 0 && M2_OFF_KPAY % 16 == 0 && M2_OFF_VPAY % 16 == 0 && M2_OFF_KN % 16 == 0 &&
                  M2_OFF_VSM % 16 == 0, "bulk copy alignment");

__device__ __forceinline__ void m2_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t m2_movmatrix_t(uint32_t x) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}
// d = a b (nothing to add: no registers to clear)
__device__ __forceinline__ void m2_mma0(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
// low-order ("what fp16 lost") products go through the same instruction
#define m2_mma_lo(c, a, b0, b1) m2_mma(c, a, b0, b1)
__device__ __forceinline__ uint32_t m2_pack(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// Packed pairs of fp32 (one instruction for two neighbouring accumulator registers; each half is
// rounded like the scalar operation).
__device__ __forceinline__ void m2_add2(float& d0, float& d1, float a0, float a1, float b0, float b1) {
    asm("{.reg .b64 a, b, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; add.rn.f32x2 d, a, b; mov.b64 {%0, %1}, d;}"
        : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
__device__ __forceinline__ void m2_sub2(float& d0, float& d1, float a0, float a1, float b0, float b1) {
    asm("{.reg .b64 a, b, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; sub.rn.f32x2 d, a, b; mov.b64 {%0, %1}, d;}"
        : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
__device__ __forceinline__ void m2_mul2(float& d0, float& d1, float a0, float a1, float b0, float b1) {
    asm("{.reg .b64 a, b, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mul.rn.f32x2 d, a, b; mov.b64 {%0, %1}, d;}"
        : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
__device__ __forceinline__ void m2_fma2(float& d0, float& d1, float a0, float a1, float b0, float b1, float c0,
                                        float c1) {
    asm("{.reg .b64 a, b, c, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mov.b64 c, {%6, %7};"
        " fma.rn.f32x2 d, a, b, c; mov.b64 {%0, %1}, d;}"
        : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}

// fp16x2 of (a, b) and fp16x2 of what that rounding lost: hi + lo carries ~22 mantissa bits.
__device__ __forceinline__ void m2_pack_hilo(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    const float2 f = __half22float2(h);
    float ra, rb;
    m2_sub2(ra, rb, a, b, f.x, f.y);
    lo = m2_pack(ra, rb);
}
// The CTA's three groups (warps of the same warp >> 2) walk their own blocks at their own pace: a barrier of the whole CTA
// per tile made the twelve warps run through the same phase together, all of them on the same pipe, and wait for the slowest.
__device__ __forceinline__ void m2_group_sync(int sub) {
    asm volatile("bar.sync %0, %1;" ::"r"(2 + HKV + sub), "n"(M2_GTHREADS) : "memory");
}

// Stage `ntok` tokens starting at `tok0` for group `sub` (tid: thread inside the group).  Bulk path: one lane of each of the
// group's four warps issues two of the eight copies and posts their bytes (the stage's mbarrier counts four arrivals); issued
// by one lane they held up its warp, and at the next group barrier the other three.  Plain path (odd tail or unaligned
// arrays): all threads copy with 32-bit loads.
__device__ __forceinline__ void m2_stage_tile(const CompressedKV& P, unsigned char* stage, uint64_t* bar, int tok0,
                                              int ntok, int tid, int sub) {
    const size_t r0 = (size_t)tok0 * HKV;
    const int rows = ntok * HKV;
    const unsigned char* const k_mask = reinterpret_cast<const unsigned char*>(P.k_mask) + r0 * 64;
    const unsigned char* const k_pay = P.k_payload + r0 * K_PAY;
    const unsigned char* const v_pay = P.v_payload + r0 * V_PAY;
    const unsigned char* const kn = reinterpret_cast<const unsigned char*>(P.k_norms) + r0 * 2;
    const unsigned char* const krn = reinterpret_cast<const unsigned char*>(P.k_r_norms) + r0 * 2;
    const unsigned char* const vn = reinterpret_cast<const unsigned char*>(P.v_norms) + r0 * 2;
    const unsigned char* const vrn = reinterpret_cast<const unsigned char*>(P.v_r_norms) + r0 * 2;
    const unsigned char* const vsm = P.v_shared_meta + r0 * 4;
    if (P.bulk_ok && ((tok0 & 1) == 0) && ((ntok & 1) == 0)) {
        if ((tid & 31) == 0) {
            const auto two = [&](int dst_a, const unsigned char* a, int bytes_a, int dst_b, const unsigned char* b, int bytes_b) {
                mbar_arrive_expect_tx(bar, (uint32_t)(rows * (bytes_a + bytes_b)));
                bulk_g2s(stage + dst_a, a, (uint32_t)(rows * bytes_a), bar);
                bulk_g2s(stage + dst_b, b, (uint32_t)(rows * bytes_b), bar);
            };
            switch (tid >> 5) {
                case 0: two(M2_OFF_MASK, k_mask, 64, M2_OFF_KN, kn, 2); break;
                case 1: two(M2_OFF_KPAY, k_pay, K_PAY, M2_OFF_KRN, krn, 2); break;
                case 2: two(M2_OFF_VPAY, v_pay, V_PAY, M2_OFF_VN, vn, 2); break;
                default: two(M2_OFF_VSM, vsm, 4, M2_OFF_VRN, vrn, 2); break;
            }
        }
    } else {
        const auto copy = [&](int dst, const unsigned char* src, int bytes) {
            const unsigned int* s = reinterpret_cast<const unsigned int*>(src);
            unsigned int* d = reinterpret_cast<unsigned int*>(stage + dst);
            for (int i = tid; i < rows * bytes / 4; i += M2_GTHREADS) d[i] = s[i];
        };
        copy(M2_OFF_MASK, k_mask, 64);
        copy(M2_OFF_KPAY, k_pay, K_PAY);
        copy(M2_OFF_VPAY, v_pay, V_PAY);
        copy(M2_OFF_KN, kn, 2);
        copy(M2_OFF_KRN, krn, 2);
        copy(M2_OFF_VN, vn, 2);
        copy(M2_OFF_VRN, vrn, 2);
        copy(M2_OFF_VSM, vsm, 4);
        fence_proxy_async();
        m2_group_sync(sub);
        if ((tid & 31) == 0) mbar_arrive(bar);
    }
}

// RoPE table of a block: 64 floats per token; pairs 2i and 2i + 1 are the four floats cos, cos, sin, sin at 4i.
__device__ __forceinline__ void m2_fill_rope(float* tab, const float* freq, const CompressedKV& P, int tok0, int tid) {
    for (int e = tid; e < M2_BT * 32; e += M2_GTHREADS) {
        const int t = e >> 5, m = e & 31;
        double th = (double)token_pos(P, tok0 + t) * (double)freq[m];
        th -= rint(th * 0.15915494309189535) * 6.283185307179586;
        float s, c;
        __sincosf((float)th, &s, &c);
        float* o = tab + 64 * t + 4 * (m >> 1) + (m & 1);
        o[0] = c;
        o[2] = s;
    }
}

// A group's next RoPE table from its last: every entry turns by M2_TT positions of its pair (four FMAs
// instead of a range reduction and a sincos).  The caller re-seeds with m2_fill_rope every M2_ROPE_RESEED
// blocks, so that rounding never accumulates over more than that many turns (< 4e-6), and whenever the
// positions are not contiguous.
constexpr int M2_ROPE_RESEED = 64;
__device__ __forceinline__ void m2_step_rope(float* dst, const float* src, const float* step, int tid) {
#pragma unroll
    for (int e = tid; e < M2_BT * 16; e += M2_GTHREADS) {
        const float4 a = reinterpret_cast<const float4*>(src)[e], d = reinterpret_cast<const float4*>(step)[e & 15];
        reinterpret_cast<float4*>(dst)[e] =
            make_float4(a.x * d.x - a.z * d.z, a.y * d.y - a.w * d.w, a.z * d.x + a.x * d.z, a.w * d.y + a.y * d.w);
    }
}

// The layer's V codebook (entry (patch, code) starts at half 3 (256 patch + code)) into its shared-memory rows.  Two
// codes (three words) per thread and iteration, eleven iterations' loads in flight: bound by load latency.
__device__ __forceinline__ void m2_stage_codebook(unsigned char* dst, const __half* __restrict__ vq, int tid) {
    const unsigned int* src = reinterpret_cast<const unsigned int*>(vq);
#pragma unroll 11
    for (int u = tid; u < NP * 256 / 2; u += M2_THREADS) {
        const unsigned int w0 = __ldg(src + 3 * u), w1 = __ldg(src + 3 * u + 1), w2 = __ldg(src + 3 * u + 2);
        const int patch = u >> 7, code = 2 * (u & 127);  // the pair never straddles a patch (256 codes)
        unsigned char* e = dst + code * M2_VQ_ROW + (patch >> 1) * 12;
        *reinterpret_cast<unsigned int*>(e + 4 * (patch & 1)) = w0;
        *reinterpret_cast<unsigned short*>(e + 8 + 2 * (patch & 1)) = (unsigned short)(w1 & 0xFFFFu);
        e += M2_VQ_ROW;
        *reinterpret_cast<unsigned int*>(e + 4 * (patch & 1)) = (w1 >> 16) | (w2 << 16);
        *reinterpret_cast<unsigned short*>(e + 8 + 2 * (patch & 1)) = (unsigned short)(w2 >> 16);
    }
}

// A layer's small tables to `dst` (the order of M2_SM_FREQ ..), one entry per thread; without the flags.
__device__ __forceinline__ void m2_small_tables(unsigned char* dst, const CompressedKV& P, int tid) {
    constexpr int O_DINV = M2_SM_DINV - M2_SM_FREQ, O_C3 = M2_SM_C3 - M2_SM_FREQ, O_RSTEP = M2_SM_RSTEP - M2_SM_FREQ;
    if (tid < 32) reinterpret_cast<float*>(dst)[tid] = powf(P.rope_base, -2.0f * (float)tid / 64.0f);
    if (tid >= 128 && tid < 128 + NP) {
        const float c0 = __half2float(P.cents_v[0 * D + 4 * (tid - 128) + 3]), c1 = __half2float(P.cents_v[1 * D + 4 * (tid - 128) + 3]);
        reinterpret_cast<float2*>(dst + O_C3)[tid - 128] = make_float2(0.5f * (c0 + c1) * P.alpha_v, 0.5f * (c0 - c1) * P.alpha_v);
    }
    if (tid < 64) reinterpret_cast<float*>(dst + O_DINV)[tid] = (1.0f / 256.0f) / (__half2float(P.d_k[tid]) + 1e-8f);
    if (tid >= 192 && tid < 224) {
        const int m = tid - 192;
        // half turns of M2_TT positions: reduced in double, so the fp32 sine and cosine get an exact small argument
        double th = (double)M2_TT * (double)powf(P.rope_base, -2.0f * (float)m / 64.0f) * 0.3183098861837907;
        th -= 2.0 * rint(0.5 * th);
        float* o = reinterpret_cast<float*>(dst + O_RSTEP) + 4 * (m >> 1) + (m & 1);
        sincospif((float)th, &o[2], &o[0]);
    }
}

// Query-side operands of one (sequence, layer, kv-head): this warp's B fragments.
struct M2Query {
    uint32_t tm;   // tensor-memory address of this warp's query fragments
    uint32_t rot;  // ... and of its lane quadrant's rotor fragments
    bool low;      // the rotor fragments have low-order parts
};

__device__ __forceinline__ void m2_tm_st4f(uint32_t taddr, const float* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%0,%1,%2,%3};" ::"f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void m2_tm_ld4f(uint32_t taddr, float* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void m2_tm_st8(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f,
                                          uint32_t g, uint32_t h) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(a), "r"(b), "r"(c), "r"(d), "r"(e),
                 "r"(f), "r"(g), "r"(h), "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void m2_tm_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void m2_tm_ld4(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void m2_tm_st16f(uint32_t taddr, const float* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"f"(r[0]),
        "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "f"(r[8]), "f"(r[9]), "f"(r[10]), "f"(r[11]),
        "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void m2_tm_ld16f(uint32_t taddr, float* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]),
          "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void m2_tm_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void m2_tm_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Allocation by warp 0 of a CTA (one CTA per SM by shared memory, so the columns are always free); the address goes
// through `slot` in shared memory.  Followed by a CTA barrier by the caller.
__device__ __forceinline__ void m2_tm_alloc(uint32_t* slot, int warp) {
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "n"(M2_TM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
// After a CTA barrier behind the last use.
__device__ __forceinline__ void m2_tm_free(uint32_t tmem, int warp) {
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(M2_TM_COLS) : "memory");
    }
}

// A lane's rotor fragments of k-step s: rotor x centroid (ternary operand) and rotor (residual operand), fp16 and what fp16
// lost.  The three low index bits of the 64-point Hadamard transform are folded in: u[8j + n] is produced by step s = 2j + (n
// >> 2) as rotor output c = n & 3, and H64 = H8 (bits 0..2, inside a tile) x H8 (bits 3..5, across tiles), so column n' of the
// folded operand is sum_n H8[n][n'] * (column n of the plain one).
__device__ __forceinline__ void m2_rotor_fragment(const CompressedKV& P, int s, int lane, uint32_t (&r)[8]) {
    const int g = lane >> 2, t = lane & 3, patch = 16 * t + s;
    __half hr[16], hc[4];
    *reinterpret_cast<uint4*>(&hr[0]) = *reinterpret_cast<const uint4*>(P.k_rotor + patch * 16);
    *reinterpret_cast<uint4*>(&hr[8]) = *reinterpret_cast<const uint4*>(P.k_rotor + patch * 16 + 8);
    *reinterpret_cast<uint2*>(&hc[0]) = *reinterpret_cast<const uint2*>(P.cents_k + 2 * D + 64 * t + 4 * s);
    const int kk[4] = {0, 2, 1, 3};  // dims 64t+4s + {0, 2, 1, 3}
    float rc[4], r1[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float acc = 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int n = 4 * (s & 1) + c;
            const float v = __half2float(hr[c * 4 + kk[i]]);
            acc += (__popc(n & g) & 1) ? -v : v;
        }
        r1[i] = acc;
        rc[i] = acc * __half2float(hc[kk[i]]);
    }
    m2_pack_hilo(rc[0], rc[1], r[0], r[4]);
    m2_pack_hilo(rc[2], rc[3], r[1], r[5]);
    m2_pack_hilo(r1[0], r1[1], r[2], r[6]);
    m2_pack_hilo(r1[2], r1[3], r[3], r[7]);
}

// The layer's tables into shared memory and its rotor fragments into the tensor memory of every lane quadrant (the M2_WPK
// warps of a quadrant share the k-steps).  Without an image they are computed (a CTA barrier and a tcgen05 fence have to
// follow); with one they are fetched: bulk copies that m2_wait_tables waits for (`loads` counts them), a third of the
// instructions that a CTA with one or two blocks per warp executes.
__device__ __forceinline__ void m2_load_tables(unsigned char* smem, const CompressedKV& P, uint32_t tmem, int tid, int warp, int lane) {
    const uint32_t dst = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + M2_TM_ROT;
    if (P.image != nullptr) {
        uint64_t* bars = reinterpret_cast<uint64_t*>(smem + M2_SM_BARS);
        if (tid == 0) {
            mbar_arrive_expect_tx(&bars[M2_BAR_SMALL], M2_SMALL_BYTES);
            bulk_g2s(smem + M2_SM_FREQ, P.image + M2_IMG_SMALL, M2_SMALL_BYTES, &bars[M2_BAR_SMALL]);
            mbar_arrive_expect_tx(&bars[M2_BAR_VQ], 256 * M2_VQ_ROW);
            bulk_g2s(smem + M2_SM_VQ, P.image + M2_IMG_VQ, 256 * M2_VQ_ROW, &bars[M2_BAR_VQ]);
        }
        const uint4* src = reinterpret_cast<const uint4*>(P.image + M2_IMG_ROT) + 2 * lane;
#pragma unroll 2
        for (int s = warp >> 2; s < 16; s += M2_WPK) {
            const uint4 a = __ldg(src + 64 * s), b = __ldg(src + 64 * s + 1);
            m2_tm_st8(dst + 8 * s, a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w);
        }
    } else {
        m2_small_tables(smem + M2_SM_FREQ, P, tid);
        m2_stage_codebook(smem + M2_SM_VQ, P.vq, tid);
#pragma unroll 2
        for (int s = warp >> 2; s < 16; s += M2_WPK) {
            uint32_t r[8];
            m2_rotor_fragment(P, s, lane, r);
            m2_tm_st8(dst + 8 * s, r[0], r[1], r[2], r[3], r[4], r[5], r[6], r[7]);
        }
    }
    m2_tm_st_wait();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

// grid = 1: the image of one layer.
__global__ void __launch_bounds__(M2_THREADS) khq_prepare_tables_kernel(CompressedKV P, unsigned char* __restrict__ image) {
    uint32_t low = 0;
    m2_small_tables(image + M2_IMG_SMALL, P, threadIdx.x);
    m2_stage_codebook(image + M2_IMG_VQ, P.vq, threadIdx.x);
    for (int c = threadIdx.x; c < 256; c += M2_THREADS) *reinterpret_cast<uint32_t*>(image + M2_IMG_VQ + c * M2_VQ_ROW + M2_VQ_ROW - 4) = 0u;
#pragma unroll 8
    for (int e = threadIdx.x; e < 256 * NP; e += M2_THREADS) {  // e = patch * 256 + code
        const unsigned short* c = reinterpret_cast<const unsigned short*>(P.vq) + 3 * e;
        reinterpret_cast<uint2*>(image + M2_IMG_VQ8)[(e & 255) * NP + (e >> 8)] = make_uint2(c[0] | ((uint32_t)c[1] << 16), c[2]);
    }
    for (int e = threadIdx.x; e < 16 * 32; e += M2_THREADS) {
        uint32_t r[8];
        m2_rotor_fragment(P, e >> 5, e & 31, r);
        uint4* o = reinterpret_cast<uint4*>(image + M2_IMG_ROT) + 2 * e;
        o[0] = make_uint4(r[0], r[1], r[2], r[3]);
        o[1] = make_uint4(r[4], r[5], r[6], r[7]);
        low |= (r[4] | r[5] | r[6] | r[7]) & 0x7FFF7FFFu;
    }
    const int any = __syncthreads_or((int)low);
    if (threadIdx.x < 4) reinterpret_cast<uint32_t*>(image + M2_IMG_SMALL + (M2_SM_FLAGS - M2_SM_FREQ))[threadIdx.x] = any != 0 ? 1u : 0u;
}

// Where the query build's scratch keeps the four dims 4c .. 4c + 3 of head h: swizzled so that the eight lanes (two heads, four
// 64-dim quarters) of a float4 phase read distinct banks.
__device__ __forceinline__ int m2_q_chunk(int h, int c) { return 4 * (c ^ ((c >> 4) & 3) ^ ((h & 1) << 2)); }

// What the query build takes from the layer's tables: 1 / d and the rotor of the lane's 8 dims, and the centroids of the dims
// 64 t + 4 s + {0..3} of the warp's k-steps.
constexpr int M2_SPW = (16 + M2_WPK - 1) / M2_WPK;  // k-steps per warp (the last warps may have one less)
struct M2QueryTables {
    uint4 rotor[4], d;
    uint2 cents[M2_SPW];
    __device__ __forceinline__ void load(const CompressedKV& P, int sub, int lane) {
        const int g = lane >> 2, t = lane & 3;
        const uint4* rp = reinterpret_cast<const uint4*>(P.k_rotor + lane * 32);
#pragma unroll
        for (int i = 0; i < 4; ++i) rotor[i] = rp[i];
        d = *reinterpret_cast<const uint4*>(P.d_k + lane * 8);
#pragma unroll
        for (int i = 0; i < M2_SPW; ++i) {
            const int s = sub + M2_WPK * i;
            cents[i] = (g < NREP && s < 16) ? *reinterpret_cast<const uint2*>(P.cents_k + 2 * D + 64 * t + 4 * s) : make_uint2(0u, 0u);
        }
    }
};

// q: (H_q, ..) with `q_head_stride` halfs between heads.  scratch: this kv-head's NREP*D floats.
__device__ __forceinline__ void m2_build_query(M2Query& Q, const __half* __restrict__ q, size_t q_head_stride,
                                               const M2QueryTables& qt, int kvh, int sub, int lane, float* scratch,
                                               uint2* qr_s /* this kv-head's [4][32] raw rotary query fragments */) {
    // The M2_WPK warps of a kv-head share the work (it runs once per work item, on the critical path): warp `sub`
    // transforms query heads sub, sub + M2_WPK, ... into the kv-head's scratch, the warps meet at a named barrier,
    // then warp `sub` builds the B fragments of k-steps sub, sub + M2_WPK, ... .  Every global load is issued before
    // the first one is needed.
    const int g = lane >> 2, t = lane & 3;
    constexpr int HPW = NREP / M2_WPK;  // heads per warp
    static_assert(NREP % M2_WPK == 0, "query heads split evenly over the warps of a kv-head");
    float dv[8], rr[2][16];
    uint4 qraw[HPW];
#pragma unroll
    for (int i = 0; i < HPW; ++i)
        qraw[i] = *reinterpret_cast<const uint4*>(q + (size_t)(kvh * NREP + sub + M2_WPK * i) * q_head_stride + lane * 8);
    uint32_t qrw[4][2];  // the raw rotary query dims
    if (sub == 0) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const __half* qh = q + (size_t)(kvh * NREP + (g < NREP ? g : 0)) * q_head_stride + 16 * kk + 2 * t;
            qrw[kk][0] = (g < NREP) ? *reinterpret_cast<const uint32_t*>(qh) : 0u;
            qrw[kk][1] = (g < NREP) ? *reinterpret_cast<const uint32_t*>(qh + 8) : 0u;
        }
    }
    {
        const __half* hd = reinterpret_cast<const __half*>(&qt.d);
        const __half* hr = reinterpret_cast<const __half*>(qt.rotor);
#pragma unroll
        for (int j = 0; j < 8; ++j) dv[j] = (lane >= 8) ? __fdividef(1.0f / 256.0f, __half2float(hd[j]) + 1e-8f) : 0.0f;
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int i = 0; i < 16; ++i) rr[p][i] = __half2float(hr[p * 16 + i]);
    }
    // q~ in the lane-owns-8-dims layout: q~ = R^T H256 (q * dinv * [dim >= 64])
#pragma unroll
    for (int i = 0; i < HPW; ++i) {
        const int h = sub + M2_WPK * i;
        const __half* hq = reinterpret_cast<const __half*>(&qraw[i]);
        float x[8], y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = __half2float(hq[j]) * dv[j];
        fwht256_lane8(x, lane);
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float a = 0.0f;
#pragma unroll
                for (int c = 0; c < 4; ++c) a = fmaf(rr[p][c * 4 + k], x[p * 4 + c], a);
                y[p * 4 + k] = a;
            }
        *reinterpret_cast<float4*>(scratch + h * D + m2_q_chunk(h, 2 * lane)) = make_float4(y[0], y[1], y[2], y[3]);
        *reinterpret_cast<float4*>(scratch + h * D + m2_q_chunk(h, 2 * lane + 1)) = make_float4(y[4], y[5], y[6], y[7]);
    }
    asm volatile("bar.sync %0, %1;" ::"r"(2 + kvh), "n"(32 * M2_WPK) : "memory");  // the kv-head's warps: all six heads are in the scratch
#pragma unroll
    for (int i = 0; i < M2_SPW; ++i) {
        const int s = sub + M2_WPK * i;
        if (s < 16) {
            const int d0 = 64 * t + 4 * s;
            float v[4] = {0.0f, 0.0f, 0.0f, 0.0f}, c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (g < NREP) {
                const float4 qq = *reinterpret_cast<const float4*>(scratch + g * D + m2_q_chunk(g, d0 >> 2));
                const __half* hc = reinterpret_cast<const __half*>(&qt.cents[i]);
                v[0] = qq.x; v[1] = qq.z; v[2] = qq.y; v[3] = qq.w;  // dims d0 + {0, 2, 1, 3}
                c[0] = __half2float(hc[0]); c[1] = __half2float(hc[2]); c[2] = __half2float(hc[1]); c[3] = __half2float(hc[3]);
            }
            uint2 lo, hi;
            m2_pack_hilo(v[0] * c[0], v[1] * c[1], hi.x, lo.x);
            m2_pack_hilo(v[2] * c[2], v[3] * c[3], hi.y, lo.y);
            uint2 lo2, hi2;
            m2_pack_hilo(v[0], v[1], hi2.x, lo2.x);
            m2_pack_hilo(v[2], v[3], hi2.y, lo2.y);
            m2_tm_st8(Q.tm + 8 * s, hi.x, hi.y, hi2.x, hi2.y, lo.x, lo.y, lo2.x, lo2.y);
        }
    }
    m2_tm_st_wait();
    if (sub == 0) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) qr_s[kk * 32 + lane] = make_uint2(qrw[kk][0], qrw[kk][1]);
    }
    __syncwarp();
}

// Running attention state of a warp in fragment layout: thread (g, t) holds heads 2t, 2t+1.
//
// O^T lives in tensor memory, twenty columns per pair of patches (2pp, 2pp + 1) of the thread's patch group g: three
// accumulator tiles of the dims 0..2 (rows idx = 2 jj + r of the pair's six (patch, dim) rows), one of the dim-3 residual
// fields, one of the dim-3 centroid signs.  Dim 3 of a patch is centroid[bit] * alpha_v * s2 + (field - 8) * s3 per token
// with per-token scales s2, s3; the sums over tokens are
//     sum p s2 (1 - 2 bit)  and  sum p s3 (field - 8)   (exact fp16 operands made from the payload's bits),
// and half the centroids' difference and, with sum p s2, their mean enter once per item.  Both operands are signed, so that
// what an accumulator holds cancels as it goes, like the dims 0..2: sums of the raw non-negative fields with the -8 taken off at the
// end grow with the number of tokens while the wanted sum grows with its root, and the tensor core's additions lose on one side.
// Error of dim 3 relative to the spread of the sums, 131 072 tokens of equal weight through one split: 8.5e-3 with the raw
// fields, 4e-6 so (dims 0..2: 1.2e-5); an item of 8192 tokens: 8.6e-4 and 2e-6.  Time: 0.5 % of a full batch's step.
struct M2State {
    uint32_t tm_o;
    float m[2], l[2], p2[2];  // reference of the weights, sum of weights, sum of p s2 (per lane)
    float top[2];             // largest score (per lane)
    __device__ __forceinline__ void init() {  // whole warp
        float z[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) z[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < (int)M2_TM_ACC_WARP / 16; ++c) m2_tm_st16f(tm_o + 16 * c, z);
        m2_tm_st_wait();
        m[0] = m[1] = top[0] = top[1] = NEG_BIG;
#pragma unroll
        for (int e = 0; e < 2; ++e) l[e] = p2[e] = 0.0f;
    }
};
// How far a score may lie above the reference maximum before that follows: the weights stay below e^2.  Times a row's V
// scales they are fp16 operands, so a block with a scale from 8192 on (8192 e^2 < 65 504) allows none.
constexpr float M2_SLACK = 2.0f, M2_SLACK_SCALES = 8192.0f;
// Two tokens' dim-3 operands.  field - 8: a field in bits 0..3 under the bits of 1024 (unit 1), or in bits 4..7 under those of
// 64 (unit 1/16), minus the offset in one packed subtraction, exact.  1 - 2 bit: the bit as the sign of 1.
__device__ __forceinline__ uint32_t m2_field_lo(uint32_t w) {
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"((w & 0x000F000Fu) | 0x64006400u), "r"(0x64086408u));
    return r;
}
__device__ __forceinline__ uint32_t m2_field_hi(uint32_t w) {
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"((w & 0x00F000F0u) | 0x54005400u), "r"(0x54805480u));
    return r;
}
__device__ __forceinline__ uint32_t m2_sign(uint32_t w) { return (w & 0x80008000u) | 0x3C003C00u; }

// The two rows of a lane (g and g + 8 of the block), its 64-dim quarter of each.
struct M2KRows {
    const uint32_t* kp[2];      // payload words of the row
    uint4 mw[2];                // the quarter's mask words
    khq3::KQuarter kq[2];
    uint32_t wc[2], first[2];   // outliers of the four words, eight bits each; ordinal of the quarter's first one
};
// What the K side of a block leaves: pass-part scores (rows g (0, 1) and g + 8 (2, 3), heads 2t, 2t + 1) of the ternary and
// of the residual part, and the rotor block sums u[token, 8j + n].
struct M2KSums {
    float cs[4], cs2[4], cu[8][4];
};

// Returns whether a word of the lane needs another path than the common one.
__device__ __forceinline__ bool m2_open_rows(M2KRows& kr, const unsigned char* __restrict__ S, int kvh, int lane, int valid_hi) {
    const int g = lane >> 2, t = lane & 3;
    bool odd = false;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int row = (g + 8 * x) * HKV + kvh;
        kr.kp[x] = reinterpret_cast<const uint32_t*>(S + M2_OFF_KPAY + row * K_PAY);
        uint4 m = *reinterpret_cast<const uint4*>(S + M2_OFF_MASK + row * 64 + 16 * t);
        if (g + 8 * x >= valid_hi) m = make_uint4(0u, 0u, 0u, 0u);  // nothing may be staged there: leftovers would take the rare paths
        kr.mw[x] = m;
        // outliers of this thread's quarter, then the ordinal of its first one (scan over the quad)
        const uint32_t wc = khq3::k3_count(m.x) + (khq3::k3_count(m.y) << 8) + (khq3::k3_count(m.z) << 16) + (khq3::k3_count(m.w) << 24);
        const uint32_t cnt = (wc * 0x01010101u) >> 24;
        uint32_t incl = cnt;
        uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, 1);
        if (t >= 1) incl += up;
        up = __shfl_up_sync(0xFFFFFFFFu, incl, 2);
        if (t >= 2) incl += up;
        kr.wc[x] = wc;
        kr.first[x] = incl - cnt;
        khq3::kq_open(kr.kq[x], kr.kp[x], kr.first[x], cnt);
        odd = odd || cnt > khq3::KQ_MAX || ((wc + 0x07070707u) & 0x10101010u) != 0u;  // a word with 9 .. 16 outliers
    }
    return odd;
}

// Mask word wi of row x into operand words.  ANY: words with more than eight outliers and quarters with more than the
// window holds come up.
template <bool ANY>
__device__ __forceinline__ void m2_word(M2KRows& kr, int x, int wi, uint32_t (&t2)[8], uint32_t (&c2)[8]) {
    const uint32_t w = wi == 0 ? kr.mw[x].x : wi == 1 ? kr.mw[x].y : wi == 2 ? kr.mw[x].z : kr.mw[x].w;
    const uint32_t cnt = (kr.wc[x] >> (8 * wi)) & 0xFFu;
    if (!ANY) {
        khq3::kq_word(kr.kq[x], w, cnt, t2, c2);
    } else if (((kr.wc[x] * 0x01010101u) >> 24) > khq3::KQ_MAX) {
        khq3::kq_word_slow(w, kr.first[x] + (((wi ? kr.wc[x] << (32 - 8 * wi) : 0u) * 0x01010101u) >> 24), kr.kp[x], t2, c2);
    } else if (cnt > 8u) {
        khq3::kq_word_dense(kr.kq[x], w, t2, c2);
    } else {
        khq3::kq_word(kr.kq[x], w, cnt, t2, c2);
    }
}

// LOW: the rotor fragments have low-order parts.  The products of an identity rotor (centroids and +-1, what a calibration leaves for
// K) are exact in fp16, so 32 of a block's 176 products would add zeros.
template <bool ANY, bool LOW>
__device__ __forceinline__ void m2_k_gemm(M2KRows& kr, const M2Query& Q, const float (&ratio)[2], M2KSums& ks) {
    float (&cs)[4] = ks.cs, (&cs2)[4] = ks.cs2, (&cu)[8][4] = ks.cu;
    float cur[4];  // residual part of a rotor tile, before the row scale
    uint32_t qf[2][8], rf[2][8];  // this and the next k-step's query and rotor fragments
    m2_tm_ld8(Q.tm, qf[0]);
    const auto load_rot = [&](int s, uint32_t (&r)[8]) {
        if (LOW) m2_tm_ld8(Q.rot + 8 * s, r);
        else m2_tm_ld4(Q.rot + 8 * s, r);
    };
    load_rot(0, rf[0]);
#pragma unroll
    for (int wi = 0; wi < 4; ++wi) {
        // a whole mask word (16 dims = this thread's share of four k-steps) of each of the two rows at once
        uint32_t ta[8], xa[8], tb[8], xb[8];
        m2_word<ANY>(kr, 0, wi, ta, xa);
        m2_word<ANY>(kr, 1, wi, tb, xb);
        if (ANY) __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int s = wi * 4 + q;
            const uint32_t a1[4] = {ta[q], tb[q], ta[4 + q], tb[4 + q]};  // dims (4q, 4q + 2) and (4q + 1, 4q + 3) of rows g, g + 8
            const uint32_t ax[4] = {xa[q], xb[q], xa[4 + q], xb[4 + q]};  // sign * code
            m2_tm_ld_wait();
            if (s + 1 < 16) {
                m2_tm_ld8(Q.tm + 8 * (s + 1), qf[(s + 1) & 1]);
                load_rot(s + 1, rf[(s + 1) & 1]);
            }
            const uint32_t(&qq)[8] = qf[s & 1];  // q1.x, q1.y, q2.x, q2.y, then their low-order halves
            const uint32_t(&rr)[8] = rf[s & 1];  // b1.x, b1.y, b2.x, b2.y, then their low-order halves
            if (s == 0) {
                m2_mma0(cs, a1, qq[0], qq[1]);
                m2_mma0(cs2, ax, qq[2], qq[3]);
            } else {
                m2_mma(cs, a1, qq[0], qq[1]);
                m2_mma(cs2, ax, qq[2], qq[3]);
            }
            // residual part of the rotor sums: exact operand first, the row's scale in fp32 after the two k-steps that
            // feed this tile
            if ((s & 1) == 0) {
                m2_mma0(cu[s >> 1], a1, rr[0], rr[1]);
                m2_mma0(cur, ax, rr[2], rr[3]);
            } else {
                m2_mma(cu[s >> 1], a1, rr[0], rr[1]);
                m2_mma(cur, ax, rr[2], rr[3]);
            }
            m2_mma_lo(cs, a1, qq[4], qq[5]);  // low-order halves of the query operands: the code operands are exact
            m2_mma_lo(cs2, ax, qq[6], qq[7]);
            if (LOW) {
                m2_mma_lo(cu[s >> 1], a1, rr[4], rr[5]);
                m2_mma_lo(cur, ax, rr[6], rr[7]);
            }
            if (s & 1) {
                float* c = cu[s >> 1];
                m2_fma2(c[0], c[1], ratio[0], ratio[0], cur[0], cur[1], c[0], c[1]);
                m2_fma2(c[2], c[3], ratio[1], ratio[1], cur[2], cur[3], c[2], c[3]);
            }
        }
    }
}
// Blocks with a word off the common path (about one in 300 at 11 % outliers), out of line: as branches inside the common
// path the rare words cost copies of all operand registers (MOVs were 15 % of the instructions).
__device__ __noinline__ void m2_k_gemm_odd(const M2KRows& kr0, const M2Query& Q0, float ratio0, float ratio1, M2KSums& out) {
    M2KRows kr = kr0;
    const M2Query Q = Q0;
    M2KSums ks;
    const float ratio[2] = {ratio0, ratio1};
    m2_k_gemm<true, true>(kr, Q, ratio, ks);
    out = ks;
}

// One staged block of 16 tokens of kv-head `kvh`.
// valid_lo/valid_hi: block-relative range of tokens that belong to the caller's range.
__device__ __forceinline__ void m2_block(const unsigned char* __restrict__ S, const unsigned char* __restrict__ smem,
                                         const float* __restrict__ rope, int kvh, int lane, int valid_lo, int valid_hi,
                                         const M2Query& Q, const CompressedKV& P, float scale,
                                         M2State& st, bool& vq_ready, uint64_t* vq_bar, uint32_t vq_parity) {
    const int g = lane >> 2, t = lane & 3;
    const float* dinv_s = reinterpret_cast<const float*>(smem + M2_SM_DINV);
    const uint2* qr_s = reinterpret_cast<const uint2*>(smem + M2_SM_QR) + kvh * 4 * 32;
    float4* rsc = reinterpret_cast<float4*>(const_cast<unsigned char*>(smem) + M2_SM_RSC) + 32 * (threadIdx.x >> 5);

    // ---- the block's row scalars, one row per lane ---------------------------------------------
    // {score scale of the ternary part, of the residual part, residual / ternary scale of the rotor sums, -} and the three
    // V scales {dims 0..2, dim-3 centroid bit, dim-3 residual field, -}; the residual operand is in units of 2^-24
    bool large = false;
    if (lane < 16) {
        const int row = lane * HKV + kvh;
        float mult = (float)*reinterpret_cast<const uint32_t*>(S + M2_OFF_KPAY + row * K_PAY) / 1000.0f;
        if (mult < 0.1f || mult > 10.0f || isnan(mult)) mult = 1.0f;
        const float rs = 16777216.0f * hbits2f(reinterpret_cast<const uint16_t*>(S + M2_OFF_KRN)[row]);
        const float kn = P.alpha_k * scale * hbits2f(reinterpret_cast<const uint16_t*>(S + M2_OFF_KN)[row]);
        const float vn = hbits2f(reinterpret_cast<const uint16_t*>(S + M2_OFF_VN)[row]);
        const float en = hbits2f(reinterpret_cast<const uint16_t*>(S + M2_OFF_VRN)[row]);
        const float sm = reinterpret_cast<const float*>(S + M2_OFF_VSM)[row];
        const bool in = lane >= valid_lo && lane < valid_hi;
        const float s1 = P.alpha_v * vn * en, s3 = sm * vn * (1.0f / 7.0f);
        large = in && !(fmaxf(fmaxf(fabsf(s1), fabsf(s3)), vn) < M2_SLACK_SCALES);
        rsc[2 * lane] = make_float4(kn * mult, kn * rs, rs / mult, 0.0f);
        rsc[2 * lane + 1] = in ? make_float4(s1, vn, s3, 0.0f) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    // ================================ K side: scores ==========================================
    M2KRows kr;
    const bool odd = m2_open_rows(kr, S, kvh, lane, valid_hi);
    __syncwarp();
    const float ratio[2] = {rsc[2 * g].z, rsc[2 * (g + 8)].z};
    M2KSums ks;
    if (!__any_sync(0xFFFFFFFFu, odd)) {
        if (Q.low) m2_k_gemm<false, true>(kr, Q, ratio, ks);
        else m2_k_gemm<false, false>(kr, Q, ratio, ks);
    } else {  // only these have their address taken
        const M2KRows krm = kr;
        const M2Query Qm = Q;
        M2KSums ksm;
        m2_k_gemm_odd(krm, Qm, ratio[0], ratio[1], ksm);
        ks = ksm;
    }
    float (&cs)[4] = ks.cs, (&cs2)[4] = ks.cs2, (&cu)[8][4] = ks.cu;
    // ---- rotary part: rest of H64 over idx = 8j + 2t + e, /d, rotation, dot with the raw query ----
    float cr[4];
    {
        // index bits 0..2 were transformed inside the GEMM (folded into the rotor operand)
        // bits 3, 4, 5 (j)
#pragma unroll
        for (int m = 1; m <= 4; m <<= 1)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if ((j & m) == 0)
#pragma unroll
                    for (int e = 0; e < 4; e += 2) {
                        const float a0 = cu[j][e], a1 = cu[j][e + 1], b0 = cu[j | m][e], b1 = cu[j | m][e + 1];
                        m2_add2(cu[j][e], cu[j][e + 1], a0, a1, b0, b1);
                        m2_sub2(cu[j | m][e], cu[j | m][e + 1], a0, a1, b0, b1);
                    }
        // scale by dinv, rotate pairs (idx, idx + 32) = tiles (j, j + 4): two neighbouring pairs per packed operation
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 dlo = *reinterpret_cast<const float2*>(dinv_s + 8 * j + 2 * t);
            const float2 dhi = *reinterpret_cast<const float2*>(dinv_s + 32 + 8 * j + 2 * t);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const float4 rc = *reinterpret_cast<const float4*>(rope + (g + 8 * x) * 64 + 16 * j + 4 * t);  // cos, cos, sin, sin
                float *a = &cu[j][2 * x], *b = &cu[j + 4][2 * x];
                float z0, z1, w0, w1, u0, u1;
                m2_mul2(z0, z1, a[0], a[1], dlo.x, dlo.y);
                m2_mul2(w0, w1, b[0], b[1], dhi.x, dhi.y);
                m2_mul2(u0, u1, w0, w1, -rc.z, -rc.w);
                m2_fma2(a[0], a[1], z0, z1, rc.x, rc.y, u0, u1);
                m2_mul2(u0, u1, w0, w1, rc.x, rc.y);
                m2_fma2(b[0], b[1], z0, z1, rc.z, rc.w, u0, u1);
            }
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            uint32_t a[4], al[4];  // rotated K^ dims as fp16 hi + lo: the raw query operand is exact
            m2_pack_hilo(cu[2 * kk][0], cu[2 * kk][1], a[0], al[0]);
            m2_pack_hilo(cu[2 * kk][2], cu[2 * kk][3], a[1], al[1]);
            m2_pack_hilo(cu[2 * kk + 1][0], cu[2 * kk + 1][1], a[2], al[2]);
            m2_pack_hilo(cu[2 * kk + 1][2], cu[2 * kk + 1][3], a[3], al[3]);
            const uint2 qrk = qr_s[kk * 32 + lane];
            if (kk == 0) m2_mma0(cr, a, qrk.x, qrk.y);
            else m2_mma(cr, a, qrk.x, qrk.y);
            m2_mma_lo(cr, al, qrk.x, qrk.y);
        }
    }
    // ================================ softmax over the block ====================================
    float sc[2][2], pw[2][2];  // [row x: g, g+8][head e: 2t, 2t+1]
    bool valid[2];
    bool raise = false;
    const float slack = __any_sync(0xFFFFFFFFu, large) ? 0.0f : M2_SLACK;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        valid[x] = (g + 8 * x) >= valid_lo && (g + 8 * x) < valid_hi;
        const float2 sp = *reinterpret_cast<const float2*>(rsc + 2 * (g + 8 * x));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            sc[x][e] = valid[x] ? fmaf(sp.x, cs[2 * x + e] + cr[2 * x + e], sp.y * cs2[2 * x + e]) : -1e30f;
            st.top[e] = fmaxf(st.top[e], sc[x][e]);
            raise = raise || sc[x][e] > st.m[e] + slack;
        }
    }
    // The reference the weights are taken against follows the maximum only when a score is more than the slack above it: most
    // blocks need no reduction over the warp and no pass over the accumulators.
    float corr[2] = {1.0f, 1.0f};
    const bool rescale = __any_sync(0xFFFFFFFFu, raise);
    if (rescale) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float bm = fmaxf(sc[0][e], sc[1][e]);
            bm = fmaxf(bm, __shfl_xor_sync(0xFFFFFFFFu, bm, 4));
            bm = fmaxf(bm, __shfl_xor_sync(0xFFFFFFFFu, bm, 8));
            bm = fmaxf(bm, __shfl_xor_sync(0xFFFFFFFFu, bm, 16));
            const float mn = fmaxf(st.m[e], bm);
            corr[e] = __expf(st.m[e] - mn);
            st.m[e] = mn;
            st.l[e] *= corr[e];
            st.p2[e] *= corr[e];
        }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        pw[0][e] = valid[0] ? __expf(sc[0][e] - st.m[e]) : 0.0f;
        pw[1][e] = valid[1] ? __expf(sc[1][e] - st.m[e]) : 0.0f;
        st.l[e] += pw[0][e] + pw[1][e];
    }
    // three scaled variants of P, transposed into B fragments (tokens = k, heads = n)
    uint32_t pb[3][2], pl_[3][2];  // fp16 hi and the fp16 of what hi lost
    {
        float s1[2], s2[2], s3[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const float4 v = rsc[2 * (g + 8 * x) + 1];
            s1[x] = v.x;  // dims 0..2: codebook entry
            s2[x] = v.y;  // dim 3: centroid bit
            s3[x] = v.z;  // dim 3: residual field
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) st.p2[e] = fmaf(pw[1][e], s2[1], fmaf(pw[0][e], s2[0], st.p2[e]));
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            uint32_t hi, lo;
            m2_pack_hilo(pw[x][0] * s1[x], pw[x][1] * s1[x], hi, lo);
            pb[0][x] = m2_movmatrix_t(hi);
            pl_[0][x] = m2_movmatrix_t(lo);
            m2_pack_hilo(pw[x][0] * s2[x], pw[x][1] * s2[x], hi, lo);
            pb[1][x] = m2_movmatrix_t(hi);
            pl_[1][x] = m2_movmatrix_t(lo);
            m2_pack_hilo(pw[x][0] * s3[x], pw[x][1] * s3[x], hi, lo);
            pb[2][x] = m2_movmatrix_t(hi);
            pl_[2][x] = m2_movmatrix_t(lo);
        }
    }
    // ================================ V side: O^T += V^T P^T ====================================
    // thread (g, t): patch group g of tokens 2t, 2t+1, 2t+8, 2t+9; per pass two patches = 24 bits of each token's
    // fields, and the accumulators of that pair come out of tensor memory
    uint32_t vw[4][3], hb[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int tok = 2 * t + (i & 1) + 8 * (i >> 1);
        const uint32_t* row = reinterpret_cast<const uint32_t*>(S + M2_OFF_VPAY + (tok * HKV + kvh) * V_PAY);
#pragma unroll
        for (int w = 0; w < 3; ++w) vw[i][w] = row[3 * g + w];
        hb[i] = ((row[24 + (g >> 2)] >> (8 * (g & 3))) & 0xFFu) << 7;  // bit 7 + pl = high code bit of patch pl
    }
    const unsigned char* vq = smem + M2_SM_VQ + 48 * g;
    if (!vq_ready) {
        mbar_wait_bounded(vq_bar, vq_parity, &g_status);
        vq_ready = true;
    }
#pragma unroll
    for (int pp = 0; pp < 4; ++pp) {
        float o[5][4];
        m2_tm_ld16f(st.tm_o + 20 * pp, &o[0][0]);
        m2_tm_ld4f(st.tm_o + 20 * pp + 16, &o[4][0]);
        uint32_t f24[4];  // the pair's two 12-bit fields: code bits 0..6, centroid bit 7, residual 8..11
#pragma unroll
        for (int i = 0; i < 4; ++i)
            f24[i] = pp == 0 ? vw[i][0] : pp == 1 ? __funnelshift_r(vw[i][0], vw[i][1], 24)
                   : pp == 2 ? __funnelshift_r(vw[i][1], vw[i][2], 16) : vw[i][2] >> 8;
        uint32_t ex[2][4], ey[2][4];  // [patch of the pair][token i]: (d0,d1), (d2,-)
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t code = ((u ? f24[i] >> 12 : f24[i]) & 0x7Fu) | ((hb[i] >> (2 * pp + u)) & 0x80u);
                const unsigned char* e = vq + code * M2_VQ_ROW + 12 * pp;
                ex[u][i] = *reinterpret_cast<const uint32_t*>(e + 4 * u);
                ey[u][i] = *reinterpret_cast<const unsigned short*>(e + 8 + 2 * u);
            }
        // rows: idx = 2j + r -> (patch idx/3, dim idx%3); the pair's six (patch, dim) rows in order
        uint32_t lo[6], hi[6];  // token pairs (2t, 2t+1) and (2t+8, 2t+9)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            lo[3 * u + 0] = __byte_perm(ex[u][0], ex[u][1], 0x5410);
            lo[3 * u + 1] = __byte_perm(ex[u][0], ex[u][1], 0x7632);
            lo[3 * u + 2] = __byte_perm(ey[u][0], ey[u][1], 0x5410);
            hi[3 * u + 0] = __byte_perm(ex[u][2], ex[u][3], 0x5410);
            hi[3 * u + 1] = __byte_perm(ex[u][2], ex[u][3], 0x7632);
            hi[3 * u + 2] = __byte_perm(ey[u][2], ey[u][3], 0x5410);
        }
        // dim 3 of the two patches: byte 1 (even patch) or 2 (odd) of a token's 24 bits holds the residual field, and for
        // the odd patch the centroid bit too; the even patch's centroid bit is the top bit of byte 0.  The masks leave
        // nothing of the neighbouring bits.
        const uint32_t b01l = __byte_perm(f24[0], f24[1], 0x5410), b01h = __byte_perm(f24[2], f24[3], 0x5410);
        const uint32_t b2l = __byte_perm(f24[0], f24[1], 0x7632), b2h = __byte_perm(f24[2], f24[3], 0x7632);
        const uint32_t da[4] = {m2_field_lo(b01l >> 8), m2_field_hi(b2l), m2_field_lo(b01h >> 8), m2_field_hi(b2h)};
        const uint32_t ca[4] = {m2_sign(b01l << 8), m2_sign(b2l << 12), m2_sign(b01h << 8), m2_sign(b2h << 12)};
        m2_tm_ld_wait();
        if (rescale) {
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                o[i][0] *= corr[0];
                o[i][1] *= corr[1];
                o[i][2] *= corr[0];
                o[i][3] *= corr[1];
            }
        }
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) {
            const uint32_t a[4] = {lo[2 * jj], lo[2 * jj + 1], hi[2 * jj], hi[2 * jj + 1]};
            m2_mma(o[jj], a, pb[0][0], pb[0][1]);
            m2_mma_lo(o[jj], a, pl_[0][0], pl_[0][1]);
        }
        m2_mma(o[3], da, pb[2][0], pb[2][1]);
        m2_mma_lo(o[3], da, pl_[2][0], pl_[2][1]);
        m2_mma(o[4], ca, pb[1][0], pb[1][1]);
        m2_mma_lo(o[4], ca, pl_[1][0], pl_[1][1]);
        m2_tm_st16f(st.tm_o + 20 * pp, &o[0][0]);
        m2_tm_st4f(st.tm_o + 20 * pp + 16, &o[4][0]);
    }
    m2_tm_st_wait();
}

// Attention of all 24 query heads over compressed tokens [my_lo, my_hi) of P; the CTA's 12 warps
// are (kv-head = warp & 3) x (group = warp >> 2: every third 16-token block).  On return (behind a CTA barrier) the
// stages hold one record per warp (store_record's layout, rotated V domain).  The tables (see m2_load_tables, `table_loads` of them so
// far) may still be under way; all M2_THREADS threads call it.
__device__ __forceinline__ void m2_compressed_range(unsigned char* smem, const __half* __restrict__ q,
                                                    size_t q_head_stride, const CompressedKV& P, int my_lo, int my_hi,
                                                    float scale, unsigned& blocks_done, uint32_t tmem, const M2QueryTables& qt,
                                                    unsigned table_loads, VInverse& inv) {
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;  // uniform: tensor-memory addresses are
    const int kvh = warp & 3, sub = warp >> 2, g = lane >> 2, t = lane & 3;
    const float* freq_s = reinterpret_cast<const float*>(smem + M2_SM_FREQ);
    // group `sub` takes blocks sub, sub + M2_WPK, ... of M2_BT tokens; the first one is on its way during the query build
    const int base = (my_lo & ~1) + M2_BT * sub, gtid = 32 * kvh + lane;
    const int nblk = (my_hi > base) ? (my_hi - base + M2_TT - 1) / M2_TT : 0;
    const unsigned t0 = blocks_done;
    unsigned char* stages = smem + M2_SM_STAGES + sub * M2_NSTAGE * M2_STAGE_BYTES;
    float* rope_tab = reinterpret_cast<float*>(smem + M2_SM_ROPE) + sub * 2 * M2_BT * 64;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + M2_SM_BARS) + sub * M2_NSTAGE;
    if (nblk > 0)
        m2_stage_tile(P, stages + (t0 % M2_NSTAGE) * M2_STAGE_BYTES, &bars[t0 % M2_NSTAGE], base, min(M2_BT, P.c_len - base), gtid, sub);

    M2Query Q;
    Q.tm = tmem + ((uint32_t)(32 * kvh) << 16);
    Q.rot = tmem + ((uint32_t)(32 * kvh) << 16) + M2_TM_ROT;
    m2_build_query(Q, q, q_head_stride, qt, kvh, sub, lane, reinterpret_cast<float*>(smem + M2_SM_ROPE) + kvh * NREP * D,
                   reinterpret_cast<uint2*>(smem + M2_SM_QR) + kvh * 4 * 32);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // the query scratch aliases the RoPE buffers
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");  // the query and rotor fragments other warps stored
    // a layer's tables that come as an image: the small ones now, the codebook before the first V side
    uint64_t* table_bars = reinterpret_cast<uint64_t*>(smem + M2_SM_BARS) + M2_BAR_SMALL;
    const uint32_t table_parity = (table_loads + 1u) & 1u;
    if (P.image != nullptr) mbar_wait_bounded(&table_bars[0], table_parity, &g_status);
    bool vq_ready = P.image == nullptr;
    Q.low = P.image == nullptr || *reinterpret_cast<const uint32_t*>(smem + M2_SM_FLAGS) != 0u;
    if (nblk > 0) m2_fill_rope(rope_tab, freq_s, P, base, gtid);
    M2State st;
    st.tm_o = tmem + ((uint32_t)(32 * kvh) << 16) + M2_TM_ACC + M2_TM_ACC_WARP * (uint32_t)sub;
    st.init();
    m2_group_sync(sub);
#pragma unroll 1
    for (int i = 0; i < nblk; ++i) {
        const unsigned gi = t0 + i;
        const int stg = gi % M2_NSTAGE;
        if (i + 1 < nblk) {
            const int tok0 = base + (i + 1) * M2_TT;
            m2_stage_tile(P, stages + ((gi + 1) % M2_NSTAGE) * M2_STAGE_BYTES, &bars[(gi + 1) % M2_NSTAGE], tok0,
                          min(M2_BT, P.c_len - tok0), gtid, sub);
            float* next = rope_tab + ((i + 1) & 1) * M2_BT * 64;
            if (P.pos_chunk == 0 && ((i + 1) % M2_ROPE_RESEED) != 0)
                m2_step_rope(next, rope_tab + (i & 1) * M2_BT * 64, reinterpret_cast<const float*>(smem + M2_SM_RSTEP), gtid);
            else
                m2_fill_rope(next, freq_s, P, tok0, gtid);
        }
        mbar_wait_bounded(&bars[stg], (uint32_t)((gi / M2_NSTAGE) & 1), &g_status);
        const int blk0 = base + i * M2_TT;
        m2_block(stages + stg * M2_STAGE_BYTES, smem, rope_tab + (i & 1) * M2_BT * 64, kvh, lane, max(my_lo - blk0, 0), min(my_hi - blk0, M2_BT), Q,
                 P, scale, st, vq_ready, &table_bars[1], table_parity);
        m2_group_sync(sub);  // stage and rope buffer free for the block after next
    }
    blocks_done = t0 + (unsigned)nblk;
    if (!vq_ready) mbar_wait_bounded(&table_bars[1], table_parity, &g_status);  // a group without blocks: no copy outlives its phase
    __syncthreads();  // the records alias the stages
    inv.load(P, lane);  // for the caller, in flight behind the records

    // ---- per-warp record in the first generation's layout, then merge + inverse V transform --------
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int m = 4; m <= 16; m <<= 1) {
            st.l[e] += __shfl_xor_sync(0xFFFFFFFFu, st.l[e], m);
            st.p2[e] += __shfl_xor_sync(0xFFFFFFFFu, st.p2[e], m);
        }
    // the record is relative to the largest score itself
    float fin[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
        for (int m = 4; m <= 16; m <<= 1) st.top[e] = fmaxf(st.top[e], __shfl_xor_sync(0xFFFFFFFFu, st.top[e], m));
        fin[e] = __expf(st.m[e] - st.top[e]);
        st.l[e] *= fin[e];
    }
    float* rec = reinterpret_cast<float*>(smem + M2_SM_STAGES) + warp * M2_REC_FLOATS;
    const float2* c3s = reinterpret_cast<const float2*>(smem + M2_SM_C3) + 8 * g;
#pragma unroll
    for (int pp = 0; pp < 4; ++pp) {
        float o[5][4];
        m2_tm_ld16f(st.tm_o + 20 * pp, &o[0][0]);
        m2_tm_ld4f(st.tm_o + 20 * pp + 16, &o[4][0]);
        m2_tm_ld_wait();
        if (t < 3) {
            // heads 2t and 2t + 1, dims 32 g + 8 pp .. + 7
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float* rp = rec + (2 * t + e) * M2_REC_HEAD + 36 * g + 8 * pp;
                float v[8];
#pragma unroll
                for (int idx = 0; idx < 6; ++idx) v[4 * (idx / 3) + idx % 3] = fin[e] * o[idx >> 1][2 * (idx & 1) + e];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float2 c = c3s[2 * pp + u];
                    v[4 * u + 3] = fin[e] * fmaf(c.x, st.p2[e], fmaf(c.y, o[4][2 * u + e], o[3][2 * u + e]));
                }
                *reinterpret_cast<float4*>(rp) = make_float4(v[0], v[1], v[2], v[3]);
                *reinterpret_cast<float4*>(rp + 4) = make_float4(v[4], v[5], v[6], v[7]);
            }
        }
    }
    if (t < 3) {
        if (g == 0) {
            rec[NREP * M2_REC_HEAD + 2 * t] = st.top[0];
            rec[NREP * M2_REC_HEAD + 2 * t + 1] = st.top[1];
            rec[NREP * M2_REC_HEAD + NREP + 2 * t] = st.l[0];
            rec[NREP * M2_REC_HEAD + NREP + 2 * t + 1] = st.l[1];
        }
    }
    __syncthreads();
}

// Persistent batched kernel, second generation (same contract as khq_decode_batched_kernel, except that CTA b's first item is
// item b and the counter hands out the ones from gridDim.x on: a launch of one item per CTA needs no counter at all).
__global__ void __launch_bounds__(M2_THREADS, 1)
khq_decode_batched_mma_kernel(const KhqSeqDesc* __restrict__ descs, const KhqTablesDesc* __restrict__ tables,
                              const KhqWorkItem* __restrict__ items, int n_items, int* __restrict__ counter,
                              float* __restrict__ partials, float scale, float rope_base, int ring_cap,
                              const unsigned char* const* __restrict__ images) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_next;
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    const int kvh = warp & 3, sub = warp >> 2;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + M2_SM_BARS);
    uint32_t* tm_slot = reinterpret_cast<uint32_t*>(smem + M2_SM_TMSLOT);
    if (tid == 0) {
        for (int s = 0; s < M2_BAR_SMALL; ++s) mbar_init(&bars[s], HKV);
        for (int s = M2_BAR_SMALL; s < M2_NBARS; ++s) mbar_init(&bars[s], 1);
        fence_barrier_init();
    }
    m2_tm_alloc(tm_slot, warp);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tm_slot, 0);
    pdl_wait();
    pdl_trigger();
    int cur_table = -1;
    unsigned blocks_done = 0, table_loads = 0;
    const float* rec = reinterpret_cast<const float*>(smem + M2_SM_STAGES);
#pragma unroll 1
    for (int it = blockIdx.x; it < n_items;) {
        const KhqWorkItem w = items[it];
        const KhqSeqDesc d = descs[w.desc];
        const KhqTablesDesc tb = tables[d.table_id];
        CompressedKV P;
        P.k_payload = d.k_payload; P.v_payload = d.v_payload; P.v_shared_meta = d.v_shared_meta;
        P.k_mask = d.k_mask; P.k_norms = d.k_norms; P.k_r_norms = d.k_r_norms;
        P.v_norms = d.v_norms; P.v_r_norms = d.v_r_norms;
        P.cents_k = tb.cents_k; P.cents_v = tb.cents_v; P.vq = tb.vq; P.k_rotor = tb.k_rotor;
        P.v_rotor = tb.v_rotor; P.d_k = tb.d_k; P.d_v = tb.d_v;
        P.alpha_k = tb.alpha_k; P.alpha_v = tb.alpha_v; P.rope_base = rope_base;
        P.start_pos = d.start_pos; P.c_len = d.c_len; P.bulk_ok = 1;
        P.image = images != nullptr ? images[d.table_id] : nullptr;
        unpack_pos(d.pos_pack, P);
        VInverse inv;
        if (w.kind == 0) {
            M2QueryTables qt;
            qt.load(P, sub, lane);
            if (d.table_id != cur_table) {
                m2_load_tables(smem, P, tmem, tid, warp, lane);
                cur_table = d.table_id;
                ++table_loads;
            }
            m2_compressed_range(smem, d.q_gate, (size_t)2 * D, P, w.lo, w.hi, scale, blocks_done, tmem, qt, table_loads, inv);
        } else {
            WarpState ws;
            ws.init();
            window_range<4>(d.q_gate, d.ring_k, d.ring_v, d.win_start, w.lo + sub, M2_WPK, w.hi, ring_cap, scale, kvh, lane, ws);
            m2_store_record(ws, reinterpret_cast<float*>(smem + M2_SM_STAGES) + warp * M2_REC_FLOATS, lane);
            __syncthreads();
        }
        if (tid == 0) s_next = n_items > (int)gridDim.x ? (int)gridDim.x + atomicAdd(counter, 1) : n_items;
        // two query heads per warp: merge of the three groups' records, inverse V transform, store
#pragma unroll 1
        for (int h = warp; h < HQ; h += M2_THREADS / 32) {
            HeadAcc a = merge_head<true, M2_WPK>(M2_WPK, lane, [&](int i) { return m2_head_of_record(rec + (h / NREP + HKV * i) * M2_REC_FLOATS, h % NREP); });
            if (w.kind == 0) inv.apply(a.a, lane);
            store_head(a, partials + ((size_t)w.slot * HQ + h) * PART, lane);
        }
        fence_proxy_async();  // the next item's bulk copies land where the records were
        __syncthreads();      // the records and s_next
        it = s_next;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    m2_tm_free(tmem, warp);
}

// Drop-in (single sequence-layer) variant: grid = num_splits * cluster_size CTAs; the CTAs of a
// cluster share one of the caller's splits.  Their per-warp records stay in each CTA's shared memory; behind a cluster
// barrier the 24 heads are dealt to the cluster's warps, which merge them through distributed shared memory (one warp per
// kv-head of rank 0 merging the peers one after the other took 10 us of a 25 us launch).
__global__ void __launch_bounds__(M2_THREADS, 1)
khq_attn_compressed_mma_kernel(const __half* __restrict__ q, CompressedKV P, float* __restrict__ out_attn,
                               float* __restrict__ out_partial, int num_splits, int L_q, int l_idx, int s_limit,
                               float scale) {
    extern __shared__ __align__(128) unsigned char smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
    const int split_id = blockIdx.x / csize;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + M2_SM_BARS);
    int s_lo = 0, s_hi = s_limit;
    if (num_splits > 1) {
        const int per = (s_limit + num_splits - 1) / num_splits;
        s_lo = min(split_id * per, s_limit);
        s_hi = min(s_lo + per, s_limit);
    }
    const int len = s_hi - s_lo;
    const int chunk = (((len + csize - 1) / csize) + 1) & ~1;
    const int my_lo = min(s_lo + crank * chunk, s_hi);
    const int my_hi = min(my_lo + chunk, s_hi);
    uint32_t* tm_slot = reinterpret_cast<uint32_t*>(smem + M2_SM_TMSLOT);
    if (tid == 0) {
        for (int s = 0; s < M2_BAR_SMALL; ++s) mbar_init(&bars[s], HKV);
        for (int s = M2_BAR_SMALL; s < M2_NBARS; ++s) mbar_init(&bars[s], 1);
        fence_barrier_init();
    }
    m2_tm_alloc(tm_slot, warp);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tm_slot, 0);
    // Prepared tables are constants of the model, written long before the kernel in front of this one: fetched while that one
    // still runs.
    M2QueryTables qt;
    if (P.image == nullptr) pdl_wait();
    m2_load_tables(smem, P, tmem, tid, warp, lane);
    qt.load(P, warp >> 2, lane);
    if (P.image != nullptr) pdl_wait();
    pdl_trigger();
    unsigned blocks_done = 0;
    VInverse inv;
    m2_compressed_range(smem, q + (size_t)l_idx * 2 * D, (size_t)L_q * 2 * D, P, my_lo, my_hi, scale, blocks_done, tmem, qt, 1u, inv);
    // the query fragments are not needed any more; everything below is ordinary memory
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (csize > 1) cluster.sync();
    else __syncthreads();
    m2_tm_free(tmem, warp);
    const float* rec = reinterpret_cast<const float*>(smem + M2_SM_STAGES);
    const auto out_of = [&](int h) {
        const int total_id = h * L_q + l_idx;
        return (num_splits > 1) ? out_partial + ((size_t)total_id * num_splits + split_id) * PART : out_attn + (size_t)total_id * PART;
    };
    if (csize == 1) {  // two heads per warp, side by side
        static_assert(HQ == 2 * (M2_THREADS / 32), "two heads per warp");
        HeadAcc a[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int h = warp + k * (HQ / 2);
            a[k] = merge_head<true, M2_WPK>(M2_WPK, lane, [&](int i) { return m2_head_of_record(rec + (h / NREP + HKV * i) * M2_REC_FLOATS, h % NREP); });
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) inv.apply(a[k].a, lane);
#pragma unroll
        for (int k = 0; k < 2; ++k) store_head(a[k], out_of(warp + k * (HQ / 2)), lane);
        return;
    }
#pragma unroll 1
    for (int h = crank + csize * warp; h < HQ; h += csize * (M2_THREADS / 32)) {
        HeadAcc a = merge_head<true>(M2_WPK * csize, lane, [&](int i) {
            return m2_head_of_record(cluster.map_shared_rank(rec, i / M2_WPK) + (h / NREP + HKV * (i % M2_WPK)) * M2_REC_FLOATS, h % NREP);
        });
        inv.apply(a.a, lane);
        store_head(a, out_of(h), lane);
    }
    cluster.sync();  // peers must stay resident until their records have been read
}

}  // namespace khq
