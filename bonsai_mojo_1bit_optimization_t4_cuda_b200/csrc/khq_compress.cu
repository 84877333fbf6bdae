// khq_compress.cu -- KHQ compress for sm_100a: one warp per (token, kv-head) row, or per group of
// two (K) or four (V) rows in large launches.
//
// Code words must be bit-identical to the reference kernel's, which evaluates every row in one
// thread in a fixed fp32 order.  The work is therefore split in two kinds:
//   * order-insensitive steps run lane-parallel: the FWHT butterflies (each output of a stage is
//     the same a+b / a-b whatever thread computes it), the per-patch 4x4 rotor (the k-chain of a
//     patch stays inside one lane), the 64x256 VQ search (lexicographic (distance, index)
//     minimum == first strict minimum of an ascending scan), max reductions, bit packing;
//   * the few order-sensitive scalar sums (sum of squares over 256 dims, the two conditional
//     sums behind the K base multiplier, the two 64-term energy sums of V) are staged in shared
//     memory and accumulated strictly in index order; with a group of R rows lane l follows the
//     chain of row l % R, so one pass serves R rows.
// Arithmetic that feeds a threshold or a rounding is written with explicit __fmaf_rn where the
// reference's build (default -fmad=true) fuses a multiply into the following add/subtract.
#include "khq_common.cuh"
#include "khq_launch.cuh"

namespace khq {

constexpr int CMP_WARPS = 4;  // warps per block, each on its own row or group of rows
constexpr int CMP_KROWS = 4;  // K rows that a warp takes together (large launches)
constexpr int CMP_VROWS = 4;  // V rows of a CTA whose warps share the code search
// The rules count rows per SM; the figures are of 148 SMs.
// Below 64 rows an SM a K launch keeps one row per warp: groups of four give each of 16 warps per SM one group (9472 rows), and
// fewer rows than that leave warps without work (8192 rows: 26.4 us either way, 4096: 15.5 against 20.8, 16 384: 47.1 against
// 38.8).  Eight rows a warp cost more in occupancy than their shared sums save (129 024 rows: 259 against 227 us).
constexpr long long CMP_KROWS_MIN_PER_SM = 16 * CMP_KROWS;
// V launches.  Up to two CTAs of four rows per SM (1184 rows) the length of one CTA is what counts: 16 warps (512 rows:
// 9.2 us, 11.1 with 8 warps).  Above, 8 warps overlap more of the unshared work (8192 rows: 59 us, 66 with 16), 6.6 us per 1000
// rows (977 ns per row an SM).  The filtered search takes 64 rows per CTA, two CTAs per SM, and 50 us for each time that 64 rows
// an SM are begun (61 the first time), so it wins where that is less: from 8485 rows, except just behind a multiple of 9472 up
// to 29 500 rows.
constexpr long long CMP_V16_MAX_PER_SM = 2 * CMP_VROWS;
inline bool compress_v_filtered(long long n, long long sms) {
    const long long waves = (n + sms * 64 - 1) / (sms * 64);
    return (waves > 1 ? 50000 * waves : 61000) < 5000 + 4884 * n / (5 * sms);  // ns
}

// One run of rows of a batched launch: source rows (fp16, D per row, contiguous) and the first
// output row in the launch's output arrays (mirrored in include/khq_b200.h).
struct KhqCompressSeg {
    const __half* x;
    long long row0;
};
static_assert(sizeof(KhqCompressSeg) == 16, "ABI");

// Row strides of D + 4 (and NP + 4) floats: the in-order sums read R rows at once (lane l
// follows row l % R), and the odd multiple of 16 bytes keeps those 16-byte reads on different banks.
template <int R>
struct CompressScratchK {
    float q[R][D + 4];      // x as float, then the rotated projection
    unsigned char in[R][32 + (R > 1 ? 4 : 0)];  // per lane: which of its dims belong to the two conditional sums
    short incl[R][32];      // per lane: outlier candidates up to and including the lane's dims
    unsigned char oc[64];   // outlier 4-bit codes, by outlier ordinal
    unsigned char os[64];   // outlier sign flags, by outlier ordinal
};

struct CompressScratchV {
    float p[CMP_VROWS][D + 4];           // x as float, then the rotated projection
    float a[CMP_VROWS][NP + 4];          // per-patch true energies
    float b[CMP_VROWS][NP + 4];          // per-patch codebook energies
    unsigned short code[CMP_VROWS][NP];  // chosen code per (row, patch)
};

// One launch over one contiguous run of rows (segs == nullptr: input row = output row), or over
// many runs of rows_per_seg rows, each with its own source and first output row.
__device__ __forceinline__ const __half* compress_map_row(const __half* x, const KhqCompressSeg* segs,
                                                          int rows_per_seg, long long x_byte_offset,
                                                          long long lrow, long long& row) {
    row = lrow;
    if (segs == nullptr) return x + lrow * D;
    const KhqCompressSeg sg = segs[lrow / rows_per_seg];
    const long long rr = lrow % rows_per_seg;
    row = sg.row0 + rr;
    return reinterpret_cast<const __half*>(reinterpret_cast<const char*>(sg.x) + x_byte_offset) + rr * D;
}

// Normalisation, FWHT-256 and the 4x4 rotor of one row whose norm is known; lane owns dims
// 8*lane .. 8*lane+7 (xv).
__device__ __forceinline__ void compress_rotate(const float (&xv)[8], float norm,
                                                const __half* __restrict__ d_vec,
                                                const __half* __restrict__ rotor, float f_s, int lane,
                                                float (&proj)[8]) {
    const float den = norm + 1e-8f;

    const uint4 draw = *reinterpret_cast<const uint4*>(d_vec + lane * 8);
    const __half* hd = reinterpret_cast<const __half*>(&draw);
    float r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = __fdiv_rn(xv[j] * __half2float(hd[j]), den);
    fwht256_lane8(r, lane);

    // 4x4 rotor of the lane's two patches: rot[c] = sum_k r[k] * R[k][c], k ascending
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const uint4* rp = reinterpret_cast<const uint4*>(rotor + (lane * 2 + p) * 16);
        const uint4 r0 = rp[0], r1 = rp[1];
        __half hr[16];
        *reinterpret_cast<uint4*>(&hr[0]) = r0;
        *reinterpret_cast<uint4*>(&hr[8]) = r1;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                acc = __fmaf_rn(r[p * 4 + k], __half2float(hr[k * 4 + c]), acc);
            proj[p * 4 + c] = acc * f_s;
        }
    }
}

// ============ K rows: a warp takes a group of R rows; their in-order sums run side by side ============
// The three order-sensitive sums of a K row (256 squares, then the two conditional 256-term sums
// behind the base multiplier) are dependent chains that every lane of the warp would compute
// alike; with R rows per warp lane l follows row l % R, so one pass over shared memory serves R
// rows.  Between the passes a row's projection, which of its dims are in the sums (a bit each) and
// its outlier ordinals wait in shared memory: 1.2 KB a row, so that four rows a warp still leave
// 32 warps on an SM.  129 024 rows: 251 us with two rows a warp and the terms stored, 227 so.
template <int R>
__global__ void __launch_bounds__(CMP_WARPS * 32, 8)
khq_compress_k_kernel(const __half* __restrict__ x, const __half* __restrict__ d_vec,
                      const __half* __restrict__ rotor, const __half* __restrict__ cents,
                      unsigned int* __restrict__ out_mask, __half* __restrict__ out_norms,
                      __half* __restrict__ out_r_norms, unsigned char* __restrict__ out_payload,
                      unsigned char* __restrict__ out_shared_meta, int d_val, int n, float ts,
                      const KhqCompressSeg* __restrict__ segs, int rows_per_seg,
                      long long x_byte_offset) {
    __shared__ __align__(16) CompressScratchK<R> scratch[CMP_WARPS];
    __shared__ __align__(16) float cents2[D];  // the centroid row the base multiplier is fitted to
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    CompressScratchK<R>& S = scratch[warp];
    // The reference computes this factor at run time from the dimension argument.
    const float f_s = rsqrtf((float)d_val);
    const float th_out = 1.60f * f_s, th_lo = 0.47f * f_s;
    const long long n_groups = ((long long)n + R - 1) / R;
    const int cr = lane & (R - 1);
    float cb[8];  // the lane's 8 dims of the centroid row the base multiplier is fitted to
    {
        const uint4 craw = *reinterpret_cast<const uint4*>(cents + 2 * D + lane * 8);
        const __half* hc = reinterpret_cast<const __half*>(&craw);
#pragma unroll
        for (int j = 0; j < 8; ++j) cb[j] = __half2float(hc[j]);
        if (warp == 0) {
            *reinterpret_cast<float4*>(&cents2[lane * 8]) = make_float4(cb[0], cb[1], cb[2], cb[3]);
            *reinterpret_cast<float4*>(&cents2[lane * 8 + 4]) = make_float4(cb[4], cb[5], cb[6], cb[7]);
        }
        __syncthreads();
    }

    for (long long grp = (long long)blockIdx.x * CMP_WARPS + warp; grp < n_groups;
         grp += (long long)gridDim.x * CMP_WARPS) {
        const long long l0 = grp * R;
        const int nr = (n - l0 < R) ? (int)(n - l0) : R;
        // ---- the rows as fp32 in shared memory, then their sums of squares in dim order ----------
#pragma unroll 1
        for (int r = 0; r < nr; ++r) {
            long long row;
            const __half* xrow = compress_map_row(x, segs, rows_per_seg, x_byte_offset, l0 + r, row);
            const uint4 raw = *reinterpret_cast<const uint4*>(xrow + lane * 8);
            const __half2* hx = reinterpret_cast<const __half2*>(&raw);
            const float2 x0 = __half22float2(hx[0]), x1 = __half22float2(hx[1]), x2 = __half22float2(hx[2]),
                         x3 = __half22float2(hx[3]);
            *reinterpret_cast<float4*>(&S.q[r][lane * 8]) = make_float4(x0.x, x0.y, x1.x, x1.y);
            *reinterpret_cast<float4*>(&S.q[r][lane * 8 + 4]) = make_float4(x2.x, x2.y, x3.x, x3.y);
        }
        __syncwarp();
        float sum_sq = 0.0f;
#pragma unroll 8
        for (int i = 0; i < D; i += 4) {
            const float4 t = *reinterpret_cast<const float4*>(&S.q[cr][i]);
            sum_sq = __fmaf_rn(t.x, t.x, sum_sq);
            sum_sq = __fmaf_rn(t.y, t.y, sum_sq);
            sum_sq = __fmaf_rn(t.z, t.z, sum_sq);
            sum_sq = __fmaf_rn(t.w, t.w, sum_sq);
        }
        __syncwarp();
        // ---- per row: projection, symbols, mask words, the terms of the two conditional sums ------
#pragma unroll 1
        for (int r = 0; r < nr; ++r) {
            long long row;
            (void)compress_map_row(x, segs, rows_per_seg, x_byte_offset, l0 + r, row);
            const float norm = sqrtf(__shfl_sync(0xFFFFFFFFu, sum_sq, r) + 1e-8f);
            if (lane == 0) out_norms[row] = __float2half(norm);
            float xv[8], proj[8];
            *reinterpret_cast<float4*>(&xv[0]) = *reinterpret_cast<const float4*>(&S.q[r][lane * 8]);
            *reinterpret_cast<float4*>(&xv[4]) = *reinterpret_cast<const float4*>(&S.q[r][lane * 8 + 4]);
            compress_rotate(xv, norm, d_vec, rotor, f_s, lane, proj);
            *reinterpret_cast<float4*>(&S.q[r][lane * 8]) = make_float4(proj[0], proj[1], proj[2], proj[3]);
            *reinterpret_cast<float4*>(&S.q[r][lane * 8 + 4]) = make_float4(proj[4], proj[5], proj[6], proj[7]);

            unsigned cand = 0;  // dims whose |proj| is above the outlier threshold
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (fabsf(proj[j]) > th_out) cand |= 1u << j;
            // ordinal of the lane's first candidate among all candidates, in dim order
            const int cnt = __popc(cand);
            int incl = cnt;
#pragma unroll
            for (int dlt = 1; dlt < 32; dlt <<= 1) {
                const int t = __shfl_up_sync(0xFFFFFFFFu, incl, dlt);
                if (lane >= dlt) incl += t;
            }
            S.incl[r][lane] = (short)incl;
            int ord = incl - cnt;

            unsigned sym16 = 0;
            unsigned in = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float pj = proj[j];
                unsigned sym;
                if (cand & (1u << j)) {
                    // kept outlier, or overflow outlier (not part of the sums)
                    sym = (ord < MAX_OUT) ? 3u : ((pj > 0.0f) ? 2u : 1u);
                    ++ord;
                } else {
                    if (pj > th_lo) sym = 2;
                    else if (pj < -th_lo) sym = 1;
                    else sym = 0;
                    if (sym != 0) in |= 1u << j;
                }
                sym16 |= sym << (2 * j);
            }
            S.in[r][lane] = (unsigned char)in;
            // mask word w = dims 16w..16w+15 = lanes 2w (low half) and 2w+1 (high half)
            const unsigned hi16 = __shfl_down_sync(0xFFFFFFFFu, sym16, 1);
            if ((lane & 1) == 0) out_mask[row * 16 + (lane >> 1)] = sym16 | (hi16 << 16);
        }
        __syncwarp();
        // ---- the two conditional sums in dim order, R rows side by side ------------------------
        float sum_n = 0.0f, sum_c = 0.0f;
        // (a dim that is not in the sums adds nothing)
#pragma unroll (R == 1 ? 2 : 1)
        for (int w = 0; w < 8; ++w) {
            const unsigned in = *reinterpret_cast<const unsigned*>(&S.in[cr][w * 4]);
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 t = *reinterpret_cast<const float4*>(&S.q[cr][w * 32 + i]);
                const float4 c = *reinterpret_cast<const float4*>(&cents2[w * 32 + i]);
                if (in & (1u << i)) { sum_n += fabsf(t.x); sum_c += c.x; }
                if (in & (2u << i)) { sum_n += fabsf(t.y); sum_c += c.y; }
                if (in & (4u << i)) { sum_n += fabsf(t.z); sum_c += c.z; }
                if (in & (8u << i)) { sum_n += fabsf(t.w); sum_c += c.w; }
            }
        }
        float mult_own = (sum_c > 1e-5f) ? __fdiv_rn(sum_n, sum_c) : 1.0f;
        if (mult_own < 0.1f || mult_own > 10.0f || isnan(mult_own)) mult_own = 1.0f;
        // ---- per row: residuals of the kept outliers, their scale, the 40 payload bytes ----------
#pragma unroll 1
        for (int r = 0; r < nr; ++r) {
            long long row;
            (void)compress_map_row(x, segs, rows_per_seg, x_byte_offset, l0 + r, row);
            const float mult = __shfl_sync(0xFFFFFFFFu, mult_own, r);
            float proj[8];
            *reinterpret_cast<float4*>(&proj[0]) = *reinterpret_cast<const float4*>(&S.q[r][lane * 8]);
            *reinterpret_cast<float4*>(&proj[4]) = *reinterpret_cast<const float4*>(&S.q[r][lane * 8 + 4]);
            unsigned cand = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (fabsf(proj[j]) > th_out) cand |= 1u << j;
            int ord = S.incl[r][lane] - __popc(cand);
            const int total_cand = S.incl[r][31];
            const int n_out = total_cand < MAX_OUT ? total_cand : MAX_OUT;

            float res[8];
            int o_ord[8];
            float max_res = 0.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                res[j] = 0.0f;
                o_ord[j] = -1;
                if (cand & (1u << j)) {
                    if (ord < MAX_OUT) {
                        o_ord[j] = ord;
                        res[j] = fmaxf(0.0f, __fmaf_rn(-cb[j], mult, fabsf(proj[j] * ts)));
                        max_res = fmaxf(max_res, res[j]);
                    }
                    ++ord;
                }
            }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1)
                max_res = fmaxf(max_res, __shfl_xor_sync(0xFFFFFFFFu, max_res, m));
            const float rscale = (n_out > 0) ? __fdiv_rn(fmaxf(max_res, 1e-4f), 15.0f) : 0.0f;
            if (lane == 0) {
                out_r_norms[row] = __float2half(rscale);
                *reinterpret_cast<unsigned int*>(out_shared_meta + row * 4) = 0u;
            }
            // stage codes and signs by ordinal, then assemble the 40 payload bytes
            if (lane < 16) reinterpret_cast<unsigned int*>(S.oc)[lane] = 0u;
            else reinterpret_cast<unsigned int*>(S.os)[lane - 16] = 0u;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (o_ord[j] >= 0) {
                    unsigned char code = 0;
                    if (rscale > 0.0f) {
                        const float r4 = roundf(__fdiv_rn(res[j], rscale));
                        code = (unsigned char)fmaxf(0.0f, fminf(15.0f, r4));
                    }
                    S.oc[o_ord[j]] = code;
                    S.os[o_ord[j]] = (proj[j] > 0.0f) ? 1 : 0;
                }
            }
            __syncwarp();
            if (lane < 10) {
                unsigned int word = 0;
#pragma unroll
                for (int bb = 0; bb < 4; ++bb) {
                    const int byte = lane * 4 + bb;
                    unsigned int v = 0;
                    if (byte < 4) {
                        const unsigned int mu = (unsigned int)(mult * 1000.0f);
                        v = (mu >> (8 * byte)) & 0xFFu;
                    } else if (byte < 29) {
                        const int j0 = (byte - 4) * 2;
                        v = (unsigned)S.oc[j0] | ((unsigned)S.oc[j0 + 1] << 4);
                    } else if (byte < 36) {
                        const int j0 = (byte - 29) * 8;
#pragma unroll
                        for (int t = 0; t < 8; ++t)
                            if (j0 + t < MAX_OUT) v |= (unsigned)S.os[j0 + t] << t;
                    } else if (byte == 36) {
                        v = 0x02u;
                    }
                    word |= v << (8 * bb);
                }
                reinterpret_cast<unsigned int*>(out_payload + row * K_PAY)[lane] = word;
            }
            __syncwarp();
        }
    }
}

// packed pairs of fp32: one instruction, each half rounded like the scalar operation
__device__ __forceinline__ unsigned long long f2_pack(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b,
                                                     unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ float f_min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// The 8 codes of a patch that a lane scans, as fp32 (exact), paired by neighbouring codes: cc[k][i] = (code 2i, code 2i+1) of
// dim k.
__device__ __forceinline__ void v_load_codes(const __half* __restrict__ vq, int p, int lane, unsigned long long (&cc)[3][4]) {
    const uint4* cbp = reinterpret_cast<const uint4*>(vq + ((size_t)p * 256 + lane * 8) * 3);
    __half hcb[24];
    *reinterpret_cast<uint4*>(&hcb[0]) = __ldg(cbp);
    *reinterpret_cast<uint4*>(&hcb[8]) = __ldg(cbp + 1);
    *reinterpret_cast<uint4*>(&hcb[16]) = __ldg(cbp + 2);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            cc[k][i] = f2_pack(__half2float(hcb[6 * i + k]), __half2float(hcb[6 * i + 3 + k]));
}

// Code search of one (row, patch): every lane scans its 8 consecutive codes in ascending order, then
// the warp takes the lexicographic (distance, index) minimum.  cc[k][i] = (code 2i, code 2i+1) of
// dim k of the lane's 8 codes, as packed fp32 pairs.
__device__ __forceinline__ void v_search_row(const float* __restrict__ proj_row, unsigned short* __restrict__ code_row,
                                             int p, const unsigned long long (&cc)[3][4],
                                             unsigned long long nalpha2, int lane) {
    const float4 v = *reinterpret_cast<const float4*>(&proj_row[p * 4]);
    const unsigned long long v0 = f2_pack(v.x, v.x), v1 = f2_pack(v.y, v.y), v2 = f2_pack(v.z, v.z);
    float dist[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        // d = v - c * alpha with one rounding (c * -alpha is the exact negative of c * alpha),
        // dist = d2*d2 + (d0*d0 + d1*d1) in the reference's order
        const unsigned long long d0 = f2_fma(cc[0][i], nalpha2, v0);
        const unsigned long long d1 = f2_fma(cc[1][i], nalpha2, v1);
        const unsigned long long d2 = f2_fma(cc[2][i], nalpha2, v2);
        f2_unpack(f2_fma(d2, d2, f2_fma(d0, d0, f2_mul(d1, d1))), dist[2 * i], dist[2 * i + 1]);
    }
    // The reference's ascending scan from 1e20 with a strict '<' ends on the smallest distance
    // below 1e20 and on the first index that has it: the minimum first (three-input minima, which
    // pass over a NaN), then the first index equal to it.
    const float best = f_min3(f_min3(dist[0], dist[1], dist[2]), f_min3(dist[3], dist[4], dist[5]),
                              f_min3(dist[6], dist[7], 1e20f));
    unsigned bl = 7;  // index among the lane's 8 codes
#pragma unroll
    for (int i = 6; i >= 0; --i)
        if (dist[i] == best) bl = i;
    // warp minimum of (distance, index): a lane's best is a non-negative, non-NaN float (at most
    // 1e20), so its bit pattern orders like the value and two hardware warp reductions do the
    // work of five shuffle-and-compare steps
    const unsigned best_bits = __reduce_min_sync(0xFFFFFFFFu, __float_as_uint(best));
    unsigned bi = __reduce_min_sync(0xFFFFFFFFu, (__float_as_uint(best) == best_bits) ? (unsigned)(lane * 8) + bl : 0xFFFFFFFFu);
    // The reference starts from min=1e20 with a strict '<': if no distance is below 1e20
    // (NaN/inf input) it keeps code 0.
    if (!(__uint_as_float(best_bits) < 1e20f)) bi = 0;
    if (lane == 0) code_row[p] = (unsigned short)bi;
}

// What follows the code search of a V row: energies of its 64 patches (to a_row / b_row, for the in-order sums), dim-3
// centroid choice, residual, packing.  `codes`: the lane's two codes.
__device__ __forceinline__ void v_row_store(const float (&proj)[8], unsigned codes, long long row, const __half* __restrict__ vq,
                                            const __half* __restrict__ cents, float alpha, unsigned char* __restrict__ out_payload,
                                            unsigned char* __restrict__ out_shared_meta, float* a_row, float* b_row, int lane) {
    unsigned code[2];
    code[0] = codes & 0xFFFFu;
    code[1] = codes >> 16;
    // per-patch energies, dim-3 centroid choice and residual (in the owning lane)
    float e_true[2], e_vq[2], pres[2];
    unsigned sel[2];
    float max_res = 0.0f;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const int pid = lane * 2 + p;
        const float v0 = proj[p * 4 + 0], v1 = proj[p * 4 + 1], v2 = proj[p * 4 + 2];
        const __half* cbp = vq + ((size_t)pid * 256 + code[p]) * 3;
        const float b0 = __half2float(cbp[0]) * alpha;
        const float b1 = __half2float(cbp[1]) * alpha;
        const float b2 = __half2float(cbp[2]) * alpha;
        e_true[p] = __fmaf_rn(v2, v2, __fmaf_rn(v0, v0, v1 * v1));
        e_vq[p] = __fmaf_rn(b2, b2, __fmaf_rn(b0, b0, b1 * b1));
        const float v3 = proj[p * 4 + 3];
        const float c0 = __half2float(cents[0 * D + pid * 4 + 3]);
        const float c1 = __half2float(cents[1 * D + pid * 4 + 3]);
        const float dist0 = fabsf(__fmaf_rn(-c0, alpha, v3));
        const float dist1 = fabsf(__fmaf_rn(-c1, alpha, v3));
        // ascending scan from min=1e20 with strict '<': index 1 only when strictly closer
        unsigned s = 0;
        float bd = 1e20f;
        if (dist0 < bd) { bd = dist0; s = 0; }
        if (dist1 < bd) { bd = dist1; s = 1; }
        sel[p] = s;
        const float cbest = s ? c1 : c0;
        pres[p] = __fmaf_rn(-cbest, alpha, v3);
        max_res = fmaxf(max_res, fabsf(pres[p]));
        a_row[pid] = e_true[p];
        b_row[pid] = e_vq[p];
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1)
        max_res = fmaxf(max_res, __shfl_xor_sync(0xFFFFFFFFu, max_res, m));
    if (lane == 0) *reinterpret_cast<float*>(out_shared_meta + row * 4) = max_res;
    const float rs = fmaxf(max_res, 1e-4f);
    unsigned f24 = 0, hb = 0;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const float scaled = __fmaf_rn(__fdiv_rn(pres[p], rs), 7.0f, 8.0f);
        const unsigned dump = (unsigned)fmaxf(0.0f, fminf(15.0f, roundf(scaled)));
        const unsigned f = (code[p] & 0x7Fu) | ((sel[p] & 1u) << 7) | ((dump & 0xFu) << 8);
        f24 |= f << (12 * p);
        hb |= ((code[p] >> 7) & 1u) << p;
    }
    // 8 patches = 4 lanes = 96 bits = 3 words; lane k of the quad holds bits [24k, 24k+24)
    const unsigned nxt = __shfl_down_sync(0xFFFFFFFFu, f24, 1);
    unsigned int* prow = reinterpret_cast<unsigned int*>(out_payload + row * V_PAY);
    const int k4 = lane & 3, g = lane >> 2;
    if (k4 == 0) prow[g * 3 + 0] = f24 | (nxt << 24);
    else if (k4 == 1) prow[g * 3 + 1] = (f24 >> 8) | (nxt << 16);
    else if (k4 == 2) prow[g * 3 + 2] = (f24 >> 16) | (nxt << 8);
    const unsigned hv = hb << (2 * (lane & 15));
    const unsigned lo = __reduce_or_sync(0xFFFFFFFFu, lane < 16 ? hv : 0u);
    const unsigned hi = __reduce_or_sync(0xFFFFFFFFu, lane >= 16 ? hv : 0u);
    if (lane == 0) { prow[24] = lo; prow[25] = hi; }
}

// ============ V rows: the W warps of a CTA share the code search of 4 rows ============
// The search dominates a V row (64 patches x 256 codes).  Small launches are bound by its length, not by throughput, so the 64
// patches of four rows go to all warps of a CTA; a codebook slice is loaded once for the four rows, the first one while the
// first four warps prepare the rows.  512 rows: 23.5 us with a warp per row, 9.2 us; 8192 rows: 72 and 59 us.
template <int W>
__global__ void __launch_bounds__(W * 32, 32 / W)
khq_compress_v_kernel(const __half* __restrict__ x, const __half* __restrict__ d_vec,
                      const __half* __restrict__ rotor, const __half* __restrict__ cents,
                      const __half* __restrict__ vq, __half* __restrict__ out_norms,
                      __half* __restrict__ out_r_norms, unsigned char* __restrict__ out_payload,
                      unsigned char* __restrict__ out_shared_meta, int d_val, int n, float alpha,
                      const KhqCompressSeg* __restrict__ segs, int rows_per_seg,
                      long long x_byte_offset) {
    __shared__ __align__(16) CompressScratchV S;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float f_s = rsqrtf((float)d_val);
    const long long l0 = (long long)blockIdx.x * CMP_VROWS;
    const int nr = (n - l0 < CMP_VROWS) ? (int)(n - l0) : CMP_VROWS;
    unsigned long long cc[3][4];
    v_load_codes(vq, warp, lane, cc);
    long long row = 0;
    if (warp < nr) {
        const __half* xrow = compress_map_row(x, segs, rows_per_seg, x_byte_offset, l0 + warp, row);
        const uint4 raw = *reinterpret_cast<const uint4*>(xrow + lane * 8);
        const __half2* hx = reinterpret_cast<const __half2*>(&raw);
        float xv[8], proj[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = __half22float2(hx[j]);
            xv[2 * j] = f.x;
            xv[2 * j + 1] = f.y;
        }
        float* pr = S.p[warp];
        *reinterpret_cast<float4*>(&pr[lane * 8]) = make_float4(xv[0], xv[1], xv[2], xv[3]);
        *reinterpret_cast<float4*>(&pr[lane * 8 + 4]) = make_float4(xv[4], xv[5], xv[6], xv[7]);
        __syncwarp();
        // sum of squares strictly in dim order
        float sum_sq = 0.0f;
#pragma unroll 8
        for (int i = 0; i < D; i += 4) {
            const float4 t = *reinterpret_cast<const float4*>(&pr[i]);
            sum_sq = __fmaf_rn(t.x, t.x, sum_sq);
            sum_sq = __fmaf_rn(t.y, t.y, sum_sq);
            sum_sq = __fmaf_rn(t.z, t.z, sum_sq);
            sum_sq = __fmaf_rn(t.w, t.w, sum_sq);
        }
        __syncwarp();
        const float norm = sqrtf(sum_sq + 1e-8f);
        if (lane == 0) out_norms[row] = __float2half(norm);
        compress_rotate(xv, norm, d_vec, rotor, f_s, lane, proj);
        *reinterpret_cast<float4*>(&pr[lane * 8]) = make_float4(proj[0], proj[1], proj[2], proj[3]);
        *reinterpret_cast<float4*>(&pr[lane * 8 + 4]) = make_float4(proj[4], proj[5], proj[6], proj[7]);
    }
    __syncthreads();
    const unsigned long long nalpha2 = f2_pack(-alpha, -alpha);
#pragma unroll 1
    for (int p = warp; p < NP; p += W) {
        if (p != warp) v_load_codes(vq, p, lane, cc);
        if (nr == CMP_VROWS) {
#pragma unroll
            for (int r = 0; r < CMP_VROWS; ++r) v_search_row(S.p[r], S.code[r], p, cc, nalpha2, lane);
        } else {
            for (int r = 0; r < nr; ++r) v_search_row(S.p[r], S.code[r], p, cc, nalpha2, lane);
        }
    }
    __syncthreads();
    if (warp >= nr) return;
    // ---- per row: energies, dim-3 centroid choice, residual, packing ------------------------
    float proj[8];
    *reinterpret_cast<float4*>(&proj[0]) = *reinterpret_cast<const float4*>(&S.p[warp][lane * 8]);
    *reinterpret_cast<float4*>(&proj[4]) = *reinterpret_cast<const float4*>(&S.p[warp][lane * 8 + 4]);
    v_row_store(proj, *reinterpret_cast<const unsigned*>(&S.code[warp][lane * 2]), row, vq, cents, alpha, out_payload,
                out_shared_meta, S.a[warp], S.b[warp], lane);
    __syncwarp();
    // the two energy sums strictly in patch order
    float st = 0.0f, sv = 0.0f;
#pragma unroll 4
    for (int i = 0; i < NP; i += 4) {
        const float4 ta = *reinterpret_cast<const float4*>(&S.a[warp][i]);
        const float4 tb = *reinterpret_cast<const float4*>(&S.b[warp][i]);
        st += ta.x; sv += tb.x;
        st += ta.y; sv += tb.y;
        st += ta.z; sv += tb.z;
        st += ta.w; sv += tb.w;
    }
    if (lane == 0) out_r_norms[row] = __float2half(sqrtf(__fdiv_rn(st, sv + 1e-8f)));
}

// ============ V rows, large launches: the code search filtered on the tensor cores ============
// Of the 256 exact distances per (row, patch) only the smallest matters, and it is almost always smaller than the others by
// far more than an approximation is off.  The approximation is one m16n8k16 product per 16 rows x 8 codes:
//     64 (|a c|^2 - 2 a v.c)  =  (64 v, 64) . (-2 a c, |a c|^2)
// with v and a c as fp16 pieces that carry 22 bits (v = vh + vl, -2 a c = ch + cl, the norm in three pieces):
//     k   0..2 vh ch   3: 64 n1   4..6 vl ch   7: 64 n2   8..10 vh cl   11: 64 n3   12..15: 0.
// Both factors are first brought to a fixed range: per patch, v and a c are multiplied by the power of two that puts cm, the
// largest |a c_k| of the patch, into [8, 16).  That changes neither the order of the distances nor a rounding, and it keeps the
// pieces away from the ends of fp16: |2 a c| < 32, |a c|^2 < 768, 64 v < 32 000 (V < 500 is asked for below, V = |v0| + |v1| +
// |v2|).  A second piece is then off by at most 2^-22 of its factor, or by 2^-25 where it is subnormal, which against
// 64 B >= 64 x 3 x 8^2 is below 2^-28 even after the multiplication by the other factor; without the scaling the subnormal
// pieces of a codebook with |a c| of some hundredths lost whole distances.  So each omitted or rounded term is below 2^-21 of
// 64 B, B = V^2 + 2 V cm + 3 cm^2, and the fp32 accumulation of twelve terms below 2^-19; B also bounds what the reference's own
// fp32 evaluation is off (3 x 2^-24 of a distance <= B).  Two values are so off by less than 2^-17 B against each other; if
// exactly one code lies within that of the smallest approximation it is the reference's choice, and every other (row, patch)
// goes through the exact search (v_search_row) behind the steps, as do all pairs of a patch with cm outside [2^-40, 2^21).
// So the code words stay bit-identical.
//
// CTA = four groups of two warps; a group owns 16 rows (one M tile), its warps search patches 0..31 and 32..63 and share the
// rows in front and behind.  The scales of all patches come first (a patch per warp at a time).
// The B fragments of a patch (8 KB) are built once per CTA and step by all threads, double buffered.  A thread holds 2 rows x 32
// codes of a half patch: minimum by three-input min, then the sign bits of (value - minimum - margin) shifted into a mask.  46 warp
// instructions per (row, patch) against 85 of the exact search, about two per cycle; 0.5 % of the pairs are redone.  129 024
// rows: 800 us with the exact search alone, 646 filtered without the scaling, 664 with it (the latency of the scan;
// 0.5 % more instructions).
constexpr int VM_ROWS = 16;  // rows per group
constexpr int VM_GROUPS = 4;   // per CTA; eight halve the building of fragments but not the time (694 us)
struct CompressScratchVM {
    float p[VM_GROUPS * VM_ROWS][D + 4];   // x as float, then the projection, then (per row) the patch energies
    uint4 b[2][2][256 * 2];                // [buffer][half][code]: k pairs of lanes t = 0..3 (b0, b1 each)
    float2 scale[NP];                      // per patch: its power of two, cm times that (NaN: not for the filter)
    unsigned short code[VM_GROUPS * VM_ROWS][NP];
    alignas(16) unsigned undecided[NP][VM_GROUPS];  // rows of a group that need the exact search, bit 4 g + y: row g + 8 y
};
static_assert(2 * (sizeof(CompressScratchVM) + 1024) <= 228 * 1024, "two CTAs per SM");

__device__ __forceinline__ uint32_t vm_pack(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// The power of two that puts cm into [8, 16), and cm times that; NaN for a patch that the filter does not take.
__device__ __forceinline__ float2 vm_scale(float cm) {
    const unsigned e = __float_as_uint(cm) >> 23, in = min(max(e, 127u - 40u), 127u + 20u);
    const float s = __uint_as_float((2u * 127u + 3u - in) << 23);
    return make_float2(s, e == in ? cm * s : __int_as_float(0x7FFFFFFF));
}

// B fragments of one code (c: its three halfs); alpha: with the patch's power of two.
__device__ __forceinline__ void vm_build(const __half (&c)[3], float alpha, uint4* dst) {
    float q[3], n = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float a = __half2float(c[k]) * alpha;
        n = fmaf(a, a, n);
        q[k] = -2.0f * a;
    }
    const float h0 = __half2float(__float2half(q[0])), h1 = __half2float(__float2half(q[1])), h2 = __half2float(__float2half(q[2]));
    const float n1 = __half2float(__float2half(n)), n2 = __half2float(__float2half(n - n1));
    const uint32_t p01 = vm_pack(h0, h1);
    dst[0] = make_uint4(p01, vm_pack(q[0] - h0, q[1] - h1), vm_pack(h2, n1), vm_pack(q[2] - h2, (n - n1) - n2));
    dst[1] = make_uint4(p01, 0u, vm_pack(h2, n2), 0u);
}

__global__ void __launch_bounds__(VM_GROUPS * 64, 2)
khq_compress_v_mma_kernel(const __half* __restrict__ x, const __half* __restrict__ d_vec,
                          const __half* __restrict__ rotor, const __half* __restrict__ cents,
                          const __half* __restrict__ vq, __half* __restrict__ out_norms,
                          __half* __restrict__ out_r_norms, unsigned char* __restrict__ out_payload,
                          unsigned char* __restrict__ out_shared_meta, int d_val, int n, float alpha,
                          const KhqCompressSeg* __restrict__ segs, int rows_per_seg,
                          long long x_byte_offset) {
    extern __shared__ __align__(16) unsigned char vm_smem[];
    CompressScratchVM& S = *reinterpret_cast<CompressScratchVM*>(vm_smem);
    constexpr int RW = VM_ROWS / 2;  // rows per warp in front and behind
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, grp = warp >> 1, half = warp & 1;
    const int g = lane >> 2, t = lane & 3;
    const float f_s = rsqrtf((float)d_val);
    const int r_first = grp * VM_ROWS + half * RW;  // this warp's rows of the CTA
    const long long l0 = (long long)blockIdx.x * (VM_GROUPS * VM_ROWS) + r_first;
    const int nr = n - l0 >= RW ? RW : (n > l0 ? (int)(n - l0) : 0);

    // the codes a thread prepares for a step: code `tid` of patches step and step + 32
    static_assert(VM_GROUPS * 64 == 256, "a thread per code");
    __half cn[2][3];
    const auto fetch = [&](int step) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const __half* c = vq + ((size_t)(step + 32 * u) * 256 + tid) * 3;
            cn[u][0] = c[0];
            cn[u][1] = c[1];
            cn[u][2] = c[2];
        }
    };
    const auto build = [&](int step) {
#pragma unroll
        for (int u = 0; u < 2; ++u) vm_build(cn[u], alpha * S.scale[step + 32 * u].x, &S.b[step & 1][u][2 * tid]);
    };
    fetch(0);
#pragma unroll 2
    for (int p = warp; p < NP; p += VM_GROUPS * 2) {
        const uint4* cbp = reinterpret_cast<const uint4*>(vq + ((size_t)p * 256 + lane * 8) * 3);
        const uint4 c[3] = {__ldg(cbp), __ldg(cbp + 1), __ldg(cbp + 2)};
        __half2 m = __float2half2_rn(0.0f);
#pragma unroll
        for (int i = 0; i < 12; ++i) m = __hmax2(m, __habs2(reinterpret_cast<const __half2*>(c)[i]));
        // the largest product is the product of the largest: rounding keeps the order
        const float cm = fabsf(__half2float(__hmax(__low2half(m), __high2half(m))) * alpha);
        const unsigned all = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(cm));
        if (lane == 0) S.scale[p] = vm_scale(__uint_as_float(all));
    }
    // ---- front: rows as fp32, in-order sums of squares, projections ----------------------------
#pragma unroll 1
    for (int r = 0; r < RW; ++r) {
        float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
        if (r < nr) {
            long long row;
            const __half* xrow = compress_map_row(x, segs, rows_per_seg, x_byte_offset, l0 + r, row);
            const uint4 raw = *reinterpret_cast<const uint4*>(xrow + lane * 8);
            const __half2* hx = reinterpret_cast<const __half2*>(&raw);
            const float2 x0 = __half22float2(hx[0]), x1 = __half22float2(hx[1]), x2 = __half22float2(hx[2]), x3 = __half22float2(hx[3]);
            lo = make_float4(x0.x, x0.y, x1.x, x1.y);
            hi = make_float4(x2.x, x2.y, x3.x, x3.y);
        }
        *reinterpret_cast<float4*>(&S.p[r_first + r][lane * 8]) = lo;
        *reinterpret_cast<float4*>(&S.p[r_first + r][lane * 8 + 4]) = hi;
    }
    __syncwarp();
    const int cr = lane & (RW - 1);
    float sum_sq = 0.0f;
#pragma unroll 8
    for (int i = 0; i < D; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&S.p[r_first + cr][i]);
        sum_sq = __fmaf_rn(v.x, v.x, sum_sq);
        sum_sq = __fmaf_rn(v.y, v.y, sum_sq);
        sum_sq = __fmaf_rn(v.z, v.z, sum_sq);
        sum_sq = __fmaf_rn(v.w, v.w, sum_sq);
    }
    __syncwarp();
#pragma unroll 1
    for (int r = 0; r < nr; ++r) {
        long long row;
        (void)compress_map_row(x, segs, rows_per_seg, x_byte_offset, l0 + r, row);
        const float norm = sqrtf(__shfl_sync(0xFFFFFFFFu, sum_sq, r) + 1e-8f);
        if (lane == 0) out_norms[row] = __float2half(norm);
        float* pr = S.p[r_first + r];
        float xv[8], proj[8];
        *reinterpret_cast<float4*>(&xv[0]) = *reinterpret_cast<const float4*>(&pr[lane * 8]);
        *reinterpret_cast<float4*>(&xv[4]) = *reinterpret_cast<const float4*>(&pr[lane * 8 + 4]);
        compress_rotate(xv, norm, d_vec, rotor, f_s, lane, proj);
        *reinterpret_cast<float4*>(&pr[lane * 8]) = make_float4(proj[0], proj[1], proj[2], proj[3]);
        *reinterpret_cast<float4*>(&pr[lane * 8 + 4]) = make_float4(proj[4], proj[5], proj[6], proj[7]);
    }
    __syncthreads();
    build(0);
    __syncthreads();
    // ---- code search ---------------------------------------------------------------------------
    const int m_row = grp * VM_ROWS;
#pragma unroll 1
    for (int step = 0; step < NP / 2; ++step) {
        const int buf = step & 1, patch = step + 32 * half;
        if (step + 1 < NP / 2) fetch(step + 1);
        const float vs = S.scale[patch].x, cm = S.scale[patch].y;
        uint32_t a[4];
        float thr[2];
        bool safe[2];
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            const float4 v = *reinterpret_cast<const float4*>(&S.p[m_row + g + 8 * y][patch * 4]);
            const float V = vs * (fabsf(v.x) + fabsf(v.y) + fabsf(v.z));
            thr[y] = fmaf(V, fmaf(2.0f, cm, V), 3.0f * cm * cm) * 0.00048828125f;  // 64 x 2^-17 x B
            safe[y] = V < 500.0f && cm < 16.0f;  // nothing overflows fp16; false for NaN
            const float v64 = 64.0f * vs;
            const float e0 = v64 * ((t & 1) ? v.z : v.x), e1 = (t & 1) ? 64.0f : v64 * v.y;
            const uint32_t hi = vm_pack(e0, e1);
            const float2 hf = __half22float2(*reinterpret_cast<const __half2*>(&hi));
            const uint32_t lo = vm_pack(e0 - hf.x, t == 3 ? 64.0f : e1 - hf.y);
            a[y] = t < 2 ? hi : lo;
            a[2 + y] = t < 2 ? hi : 0u;
        }
        const uint4* bp = S.b[buf][half];
        float best[2];
        uint32_t mask[2], chunk[2];
        bool tie[2];
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
            float acc[16][4];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const uint2 b = reinterpret_cast<const uint2*>(bp)[(ch * 16 + j) * 32 + lane];
                asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                    : "=f"(acc[j][0]), "=f"(acc[j][1]), "=f"(acc[j][2]), "=f"(acc[j][3])
                    : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y), "f"(0.0f));
            }
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                float m4[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {  // eight values each
                    m4[k] = f_min3(acc[4 * k][2 * y], acc[4 * k][2 * y + 1], acc[4 * k + 1][2 * y]);
                    m4[k] = f_min3(m4[k], acc[4 * k + 1][2 * y + 1], acc[4 * k + 2][2 * y]);
                    m4[k] = f_min3(m4[k], acc[4 * k + 2][2 * y + 1], acc[4 * k + 3][2 * y]);
                    m4[k] = fminf(m4[k], acc[4 * k + 3][2 * y + 1]);
                }
                const float m = f_min3(fminf(m4[0], m4[1]), m4[2], m4[3]);
                const float nlim = -(m + thr[y]);
                uint32_t w[2] = {0u, 0u};  // sign bits of the values of tiles 0..7 and 8..15, first value on top
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float d0, d1;
                    f2_unpack(f2_add(f2_pack(acc[j][2 * y], acc[j][2 * y + 1]), f2_pack(nlim, nlim)), d0, d1);
                    w[j >> 3] = __funnelshift_l(__float_as_uint(d0), w[j >> 3], 1);
                    w[j >> 3] = __funnelshift_l(__float_as_uint(d1), w[j >> 3], 1);
                }
                const uint32_t mk = (w[0] << 16) | w[1];
                if (ch == 0) {
                    best[y] = m;
                    mask[y] = mk;
                    chunk[y] = 0;
                    tie[y] = false;
                } else {
                    tie[y] = !(fabsf(m - best[y]) > thr[y]);
                    if (m < best[y]) {
                        best[y] = m;
                        mask[y] = mk;
                        chunk[y] = 128;
                    }
                }
            }
        }
        unsigned redo = 0;  // rows of the tile that need the exact search
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            float m = fminf(best[y], __shfl_xor_sync(0xFFFFFFFFu, best[y], 1));
            m = fminf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 2));
            const int i = __clz((int)mask[y]);  // position of the first candidate among the lane's 32 values
            uint32_t mine = (tie[y] ? 2u : (uint32_t)__popc(mask[y])) << 16;
            mine |= chunk[y] + 8u * (uint32_t)(i >> 1) + 2u * (uint32_t)t + (uint32_t)(i & 1);
            if (!(best[y] <= m + thr[y])) mine = 0u;
            mine += __shfl_xor_sync(0xFFFFFFFFu, mine, 1);
            mine += __shfl_xor_sync(0xFFFFFFFFu, mine, 2);
            const bool one = safe[y] && (mine >> 16) == 1u;
            if (t == 0 && one) S.code[m_row + g + 8 * y][patch] = (unsigned short)(mine & 0xFFFFu);
            redo |= __ballot_sync(0xFFFFFFFFu, t == 0 && !one) << y;  // bit 4 g + y: row g + 8 y
        }
        if (lane == 0) S.undecided[patch][grp] = redo;
        if (step + 1 < NP / 2) build(step + 1);
        __syncthreads();
    }
    // ---- exact search of the undecided pairs, a patch per warp: within the steps it held up the other seven warps -----------
#pragma unroll 1
    for (int p = warp; p < NP; p += VM_GROUPS * 2) {
        const uint4 u = *reinterpret_cast<const uint4*>(S.undecided[p]);
        if ((u.x | u.y | u.z | u.w) == 0u) continue;
        const unsigned long long nalpha2 = f2_pack(-alpha, -alpha);
        unsigned long long cc[3][4];
        v_load_codes(vq, p, lane, cc);
#pragma unroll 1
        for (int gr = 0; gr < VM_GROUPS; ++gr) {
            unsigned redo = S.undecided[p][gr];
            while (redo) {
                const int k = __ffs((int)redo) - 1, r = gr * VM_ROWS + (k >> 2) + 8 * (k & 3);
                redo &= redo - 1;
                v_search_row(S.p[r], S.code[r], p, cc, nalpha2, lane);
            }
        }
    }
    __syncthreads();
    // ---- per row: energies, dim-3 centroid choice, residual, packing ------------------------------
#pragma unroll 1
    for (int r = 0; r < nr; ++r) {
        long long row;
        (void)compress_map_row(x, segs, rows_per_seg, x_byte_offset, l0 + r, row);
        float* pr = S.p[r_first + r];
        float proj[8];
        *reinterpret_cast<float4*>(&proj[0]) = *reinterpret_cast<const float4*>(&pr[lane * 8]);
        *reinterpret_cast<float4*>(&proj[4]) = *reinterpret_cast<const float4*>(&pr[lane * 8 + 4]);
        __syncwarp();  // the energies take the row's place
        v_row_store(proj, *reinterpret_cast<const unsigned*>(&S.code[r_first + r][lane * 2]), row, vq, cents, alpha, out_payload,
                    out_shared_meta, pr, pr + NP, lane);
    }
    __syncwarp();
    // the two energy sums strictly in patch order, the warp's rows at once
    float st = 0.0f, sv = 0.0f;
#pragma unroll 4
    for (int i = 0; i < NP; i += 4) {
        const float4 ta = *reinterpret_cast<const float4*>(&S.p[r_first + cr][i]);
        const float4 tb = *reinterpret_cast<const float4*>(&S.p[r_first + cr][NP + i]);
        st += ta.x; sv += tb.x;
        st += ta.y; sv += tb.y;
        st += ta.z; sv += tb.z;
        st += ta.w; sv += tb.w;
    }
    if (lane < nr) {
        long long row;
        (void)compress_map_row(x, segs, rows_per_seg, x_byte_offset, l0 + lane, row);
        out_r_norms[row] = __float2half(sqrtf(__fdiv_rn(st, sv + 1e-8f)));
    }
}

}  // namespace khq

namespace {
int launch_v_mma(const __half* x, const __half* dv, const __half* ro, const __half* ce, const void* vq, __half* on, __half* orn,
                 unsigned char* op, unsigned char* om, int d, int n, float alpha, const khq::KhqCompressSeg* segs, int rows_per_seg,
                 long long x_byte_offset, cudaStream_t stream) {
    using namespace khq;
    static bool done[64] = {};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return static_cast<int>(err);
    if (dev < 0 || dev >= 64 || !done[dev]) {
        err = cudaFuncSetAttribute(khq_compress_v_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CompressScratchVM));
        if (err != cudaSuccess) return static_cast<int>(err);
        if (dev >= 0 && dev < 64) done[dev] = true;
    }
    khq_compress_v_mma_kernel<<<(unsigned)((n + VM_GROUPS * VM_ROWS - 1) / (VM_GROUPS * VM_ROWS)), VM_GROUPS * 64, sizeof(CompressScratchVM), stream>>>(
        x, dv, ro, ce, static_cast<const __half*>(vq), on, orn, op, om, d, n, alpha, segs, rows_per_seg, x_byte_offset);
    return 0;
}

int compress_launch(const __half* x, const void* d_vec, const void* rotor, const void* centroids,
                    const void* vq_centroids, void* out_mask, void* out_norms, void* out_r_norms,
                    void* out_payload, void* out_shared_meta, int d, int n, float threshold_scale, float alpha,
                    int is_v, const khq::KhqCompressSeg* segs, int rows_per_seg, long long x_byte_offset,
                    cudaStream_t stream) {
    using namespace khq;
    const long long sms = sm_count(), cap = sms * 64;  // grid-stride beyond this
    const auto grid = [&](long long units) {
        long long blocks = (units + CMP_WARPS - 1) / CMP_WARPS;
        return (unsigned)(blocks > cap ? cap : blocks);
    };
    const __half* dv = static_cast<const __half*>(d_vec);
    const __half* ro = static_cast<const __half*>(rotor);
    const __half* ce = static_cast<const __half*>(centroids);
    __half* on = static_cast<__half*>(out_norms);
    __half* orn = static_cast<__half*>(out_r_norms);
    unsigned char* op = static_cast<unsigned char*>(out_payload);
    unsigned char* om = static_cast<unsigned char*>(out_shared_meta);
    if (!is_v && n >= CMP_KROWS_MIN_PER_SM * sms) {
        khq_compress_k_kernel<CMP_KROWS><<<grid(((long long)n + CMP_KROWS - 1) / CMP_KROWS), CMP_WARPS * 32, 0,
                                           stream>>>(x, dv, ro, ce, static_cast<unsigned int*>(out_mask), on, orn, op,
                                                     om, d, n, threshold_scale, segs, rows_per_seg, x_byte_offset);
    } else if (!is_v) {
        khq_compress_k_kernel<1><<<grid(n), CMP_WARPS * 32, 0, stream>>>(
            x, dv, ro, ce, static_cast<unsigned int*>(out_mask), on, orn, op, om, d, n, threshold_scale, segs,
            rows_per_seg, x_byte_offset);
    } else if (compress_v_filtered(n, sms)) {
        const int rc = launch_v_mma(x, dv, ro, ce, vq_centroids, on, orn, op, om, d, n, alpha, segs, rows_per_seg, x_byte_offset, stream);
        if (rc != 0) return rc;
    } else {
        const unsigned blocks = (unsigned)((n + CMP_VROWS - 1) / CMP_VROWS);
        const bool wide = n <= CMP_V16_MAX_PER_SM * sms;
        const auto kernel = wide ? khq_compress_v_kernel<16> : khq_compress_v_kernel<8>;
        kernel<<<blocks, wide ? 512 : 256, 0, stream>>>(x, dv, ro, ce, static_cast<const __half*>(vq_centroids), on, orn, op,
                                                                      om, d, n, alpha, segs, rows_per_seg, x_byte_offset);
    }
    const cudaError_t err = cudaGetLastError();
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}
}  // namespace

extern "C" int launch_khq_compress_fp16(const void* x, const void* d_vec, const void* rotor,
                                        const void* centroids, const void* vq_centroids,
                                        void* out_mask, void* out_norms, void* out_r_norms,
                                        void* out_payload, void* out_shared_meta, int n, int d,
                                        float threshold_scale, float alpha, int is_v,
                                        cudaStream_t stream) {
    using namespace khq;
    if (n <= 0 || d != D) return -100;
    return compress_launch(static_cast<const __half*>(x), d_vec, rotor, centroids, vq_centroids, out_mask,
                           out_norms, out_r_norms, out_payload, out_shared_meta, d, n, threshold_scale,
                           alpha, is_v, nullptr, 1, 0, stream);
}

// Many compression events in one launch: `n_seg` runs of `rows_per_seg` rows (512 = the 128 oldest
// tokens of one sequence's ring), run i read from segs[i].x and written to rows segs[i].row0 .. of
// the output arrays.  `segs` is a device array; x_byte_offset is added to every run's source address
// (a host that keeps K and V rings at a fixed distance uses one table for both launches).  Same
// arithmetic, row by row, as the single launch.
extern "C" int launch_khq_compress_batched_fp16(const void* segs, int n_seg, int rows_per_seg, const void* d_vec,
                                                const void* rotor, const void* centroids, const void* vq_centroids,
                                                void* out_mask, void* out_norms, void* out_r_norms, void* out_payload,
                                                void* out_shared_meta, int d, float threshold_scale, float alpha,
                                                int is_v, long long x_byte_offset, cudaStream_t stream) {
    using namespace khq;
    if (n_seg <= 0 || rows_per_seg <= 0 || d != D || !segs) return -100;
    if ((x_byte_offset & 15) != 0) return -104;
    const long long n = (long long)n_seg * rows_per_seg;
    if (n > 0x7FFFFFFFLL) return -100;
    return compress_launch(nullptr, d_vec, rotor, centroids, vq_centroids, out_mask, out_norms, out_r_norms,
                           out_payload, out_shared_meta, d, (int)n, threshold_scale, alpha, is_v,
                           static_cast<const khq::KhqCompressSeg*>(segs), rows_per_seg, x_byte_offset, stream);
}
