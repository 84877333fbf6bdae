// khq_decode.cu -- two-region KHQ decode attention for sm_100a:
//   khq_attn_compressed_mma_kernel  compressed region, split-K partials (acc, max, sum_exp)
//   khq_attn_reduce_kernel      LSE merge of the split partials
//   khq_window_attn_kernel      raw fp16 ring window
//   khq_merge_gate_kernel       LSE merge of the two regions + sigmoid output gate
// and the launch_khq_* entry points with the reference's signatures.
#include <string.h>

#include "khq_decode.cuh"
#include "khq_launch.cuh"

namespace khq {

// Nonzero once a bounded wait on an asynchronous copy has run out (read by khq_b200_device_status).
__device__ int g_status = 0;

// ------------------------------------------------------------------------------------------
// Tile staging
// ------------------------------------------------------------------------------------------
// Copies `ntok` tokens (4*ntok rows) starting at token `tok0` of every payload array into one
// stage.  Bulk path: thread 0 posts the byte count on the stage's mbarrier and issues eight
// cp.async.bulk copies.  Plain path (odd tail or unaligned arrays): all threads copy with
// 32-bit loads, then thread 0 arrives on the barrier.  The choice is CTA-uniform.
__device__ __forceinline__ void stage_tile(const CompressedKV& P, unsigned char* stage,
                                           uint64_t* bar, int tok0, int ntok, int tid) {
    const size_t r0 = (size_t)tok0 * HKV;
    const int rows = ntok * HKV;
    const unsigned char* src[8] = {
        reinterpret_cast<const unsigned char*>(P.k_mask) + r0 * 64,
        P.k_payload + r0 * K_PAY,
        P.v_payload + r0 * V_PAY,
        reinterpret_cast<const unsigned char*>(P.k_norms) + r0 * 2,
        reinterpret_cast<const unsigned char*>(P.k_r_norms) + r0 * 2,
        reinterpret_cast<const unsigned char*>(P.v_norms) + r0 * 2,
        reinterpret_cast<const unsigned char*>(P.v_r_norms) + r0 * 2,
        P.v_shared_meta + r0 * 4};
    const int dst[8] = {OFF_MASK, OFF_KPAY, OFF_VPAY, OFF_KN, OFF_KRN, OFF_VN, OFF_VRN, OFF_VSM};
    const int bpr[8] = {64, K_PAY, V_PAY, 2, 2, 2, 2, 4};
    const bool bulk = P.bulk_ok && ((tok0 & 1) == 0) && ((ntok & 1) == 0);
    if (bulk) {
        if (tid == 0) {
            mbar_arrive_expect_tx(bar, (uint32_t)(rows * 220));
#pragma unroll
            for (int a = 0; a < 8; ++a)
                bulk_g2s(stage + dst[a], src[a], (uint32_t)(rows * bpr[a]), bar);
        }
    } else {
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const int words = rows * bpr[a] / 4;  // rows is a multiple of 4, so always whole words
            const unsigned int* s = reinterpret_cast<const unsigned int*>(src[a]);
            unsigned int* d = reinterpret_cast<unsigned int*>(stage + dst[a]);
            for (int i = tid; i < words; i += DEC_THREADS) d[i] = s[i];
        }
        fence_proxy_async();
        __syncthreads();
        if (tid == 0) mbar_arrive(bar);
    }
}

// RoPE cos/sin of one tile: entry (t, m) for the position of token tok0 + t and pair m < 32.
// The angle is formed in double so that it stays exact at positions beyond 1e5.
__device__ __forceinline__ void fill_rope(float2* tab, const float* freq, const CompressedKV& P, int tok0, int tid) {
    for (int e = tid; e < TT * 32; e += DEC_THREADS) {
        const int t = e >> 5, m = e & 31;
        double th = (double)token_pos(P, tok0 + t) * (double)freq[m];
        th -= rint(th * 0.15915494309189535) * 6.283185307179586;
        float s, c;
        __sincosf((float)th, &s, &c);
        tab[e] = make_float2(c, s);
    }
}

// ------------------------------------------------------------------------------------------
// Compressed region
// ------------------------------------------------------------------------------------------
// V codebook in shared memory: entry (code, patch) is 4 halfs (3 used) at slot
// code*64 + (patch>>1) + 32*(patch&1).  A lane reads patches 2*lane and 2*lane+1, so the 16
// lanes of an LDS.64 phase always hit 16 different bank pairs whatever their codes are.
__device__ __forceinline__ void load_codebook(unsigned short* vq_s, const __half* vq, int tid) {
    const unsigned int* src = reinterpret_cast<const unsigned int*>(vq);
    for (int w = tid; w < NP * 256 * 3 / 2; w += DEC_THREADS) {
        const unsigned int two = __ldg(src + w);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int hidx = 2 * w + b;
            const int entry = hidx / 3, k = hidx - entry * 3;
            const int patch = entry >> 8, code = entry & 255;
            vq_s[(code * 64 + (patch >> 1) + 32 * (patch & 1)) * 4 + k] = (unsigned short)(two >> (16 * b));
        }
    }
}

// Per-CTA constants of one (sequence, layer): must be followed by __syncthreads().
// Returns nothing; flags[0] ends up 1 when the K rotor is the identity.
__device__ __forceinline__ void setup_tables(unsigned char* smem, const CompressedKV& P, int tid) {
    float* rotor_s = reinterpret_cast<float*>(smem + SM_ROTOR);
    float* freq_s = reinterpret_cast<float*>(smem + SM_FREQ);
    int* flags = reinterpret_cast<int*>(smem + SM_BARS + NSTAGE * 8);
    if (tid < 32) freq_s[tid] = powf(P.rope_base, -2.0f * (float)tid / 64.0f);
    if (tid == 0) flags[0] = 1;  // K rotor is the identity until a thread finds otherwise
    __syncthreads();
    // K rotor -> shared memory as fp32, 36-float stride per owning lane (conflict-free float4)
    for (int e = tid; e < NP * 16; e += DEC_THREADS) {
        const float v = __half2float(P.k_rotor[e]);
        const int patch = e >> 4, idx = e & 15;
        rotor_s[(patch >> 1) * 36 + (patch & 1) * 16 + idx] = v;
        const float want = ((idx >> 2) == (idx & 3)) ? 1.0f : 0.0f;
        if (v != want) flags[0] = 0;
    }
}

// Attention of the six query heads of this warp's kv-head over compressed tokens
// [my_lo, my_hi) of P, accumulated into st (rotated V domain).  All DEC_THREADS threads of the
// CTA call it together; tiles are dealt to the DEC_WPK warps of a kv-head token by token.
// `bar_uses` counts how often each stage barrier has completed so far in this CTA's life (the
// barriers are initialised once per CTA and reused across work items).
template <bool VQS>
__device__ __forceinline__ void compressed_range(unsigned char* smem, const __half* __restrict__ q,
                                                 size_t q_head_stride, const CompressedKV& P, int my_lo,
                                                 int my_hi, float scale, WarpState& st, unsigned& tiles_done) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = warp & 3, sub = warp >> 2;
    float2* rope_tab = reinterpret_cast<float2*>(smem + SM_ROPE);
    const float* rotor_s = reinterpret_cast<const float*>(smem + SM_ROTOR);
    const float* freq_s = reinterpret_cast<const float*>(smem + SM_FREQ);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM_BARS);
    const int* flags = reinterpret_cast<const int*>(smem + SM_BARS + NSTAGE * 8);
    const unsigned short* vq_s = reinterpret_cast<const unsigned short*>(smem + SM_VQ);

    const int base = my_lo & ~1;
    const int ntiles = (my_hi > my_lo) ? (my_hi - base + TT - 1) / TT : 0;
    if (ntiles > 0) fill_rope(rope_tab, freq_s, P, base, tid);

    // per-lane constants
    float cbase[8], dinv[8], qv[NREP][8], c3[2][2];
    {
        const uint4 cr = *reinterpret_cast<const uint4*>(P.cents_k + 2 * D + lane * 8);
        const uint4 dr = *reinterpret_cast<const uint4*>(P.d_k + lane * 8);
        const __half* hc = reinterpret_cast<const __half*>(&cr);
        const __half* hd = reinterpret_cast<const __half*>(&dr);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            cbase[j] = __half2float(hc[j]);
            dinv[j] = (1.0f / 256.0f) / (__half2float(hd[j]) + 1e-8f);
        }
#pragma unroll
        for (int h = 0; h < NREP; ++h) {
            const uint4 qr = *reinterpret_cast<const uint4*>(q + (size_t)(kvh * NREP + h) * q_head_stride + lane * 8);
            const __half* hq = reinterpret_cast<const __half*>(&qr);
#pragma unroll
            for (int j = 0; j < 8; ++j) qv[h][j] = __half2float(hq[j]) * scale;
        }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            c3[p][0] = __half2float(P.cents_v[0 * D + (lane * 2 + p) * 4 + 3]) * P.alpha_v;
            c3[p][1] = __half2float(P.cents_v[1 * D + (lane * 2 + p) * 4 + 3]) * P.alpha_v;
        }
    }

    // ---- prologue: fill NSTAGE-1 stages --------------------------------------------------------
    const unsigned t0 = tiles_done;  // tile i of this range uses stage (t0+i)%NSTAGE
#pragma unroll 1
    for (int i = 0; i < NSTAGE - 1 && i < ntiles; ++i) {
        const int tok0 = base + i * TT;
        const unsigned g = t0 + i;
        stage_tile(P, smem + SM_STAGES + (g % NSTAGE) * STAGE_BYTES, &bars[g % NSTAGE], tok0,
                   min(TT, P.c_len - tok0), tid);
    }
    __syncthreads();
    const bool rotor_identity = flags[0] != 0;

    // ---- main loop ---------------------------------------------------------------------------
#pragma unroll 1
    for (int i = 0; i < ntiles; ++i) {
        const unsigned g = t0 + i;
        const int stg = g % NSTAGE;
        {
            const int nx = i + NSTAGE - 1;
            if (nx < ntiles) {
                const int tok0 = base + nx * TT;
                const unsigned gn = t0 + nx;
                stage_tile(P, smem + SM_STAGES + (gn % NSTAGE) * STAGE_BYTES, &bars[gn % NSTAGE], tok0,
                           min(TT, P.c_len - tok0), tid);
            }
        }
        if (i + 1 < ntiles)
            fill_rope(rope_tab + ((i + 1) & 1) * TT * 32, freq_s, P, base + (i + 1) * TT, tid);
        mbar_wait_bounded(&bars[stg], (uint32_t)((g / NSTAGE) & 1), &g_status);

        const unsigned char* S = smem + SM_STAGES + stg * STAGE_BYTES;
        const float2* rt = rope_tab + (i & 1) * TT * 32;
        const int tile0 = base + i * TT;
#pragma unroll 1
        for (int t = sub; t < TT; t += DEC_WPK) {
            const int s_abs = tile0 + t;
            if (s_abs < my_lo || s_abs >= my_hi) continue;  // warp-uniform
            const int row = t * HKV + kvh;

            // ===== K: code words -> rotated-domain values ===================================
            const unsigned int* kp = reinterpret_cast<const unsigned int*>(S + OFF_KPAY + row * K_PAY);
            const unsigned int mw = reinterpret_cast<const unsigned int*>(S + OFF_MASK + row * 64)[lane >> 1];
            const unsigned int ow = (lane & 1) ? (mw >> 16) : (mw & 0xFFFFu);
            const int cnt = __popc(ow & (ow >> 1) & 0x5555u);
            int incl = cnt;
#pragma unroll
            for (int dlt = 1; dlt < 32; dlt <<= 1) {
                const int tmp = __shfl_up_sync(0xFFFFFFFFu, incl, dlt);
                if (lane >= dlt) incl += tmp;
            }
            int jcur = incl - cnt;  // ordinal of this lane's first outlier
            float mult = (float)kp[0] / 1000.0f;
            if (mult < 0.1f || mult > 10.0f || isnan(mult)) mult = 1.0f;
            const float rscale = hbits2f(reinterpret_cast<const uint16_t*>(S + OFF_KRN)[row]);
            const float knorm = hbits2f(reinterpret_cast<const uint16_t*>(S + OFF_KN)[row]);
            const int j0 = min(jcur, MAX_OUT);
            unsigned int nwin, swin;
            {
                const int nb = 32 + 4 * j0;       // bit offset of residual nibble j0
                nwin = __funnelshift_r(kp[nb >> 5], kp[(nb >> 5) + 1], nb & 31);
                const int sb = 232 + j0;          // bit offset of sign bit j0
                swin = __funnelshift_r(kp[sb >> 5], kp[min((sb >> 5) + 1, 9)], sb & 31);
            }
            const float kscale = P.alpha_k * knorm;
            float y[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const unsigned sym = (ow >> (2 * j)) & 3u;
                const bool is3 = sym == 3u;
                const bool valid = is3 && (jcur < MAX_OUT);
                const float code = valid ? (float)(nwin & 15u) : 0.0f;
                const bool pos_sign = valid && (swin & 1u);
                float mag = (sym != 0u) ? cbase[j] * mult : 0.0f;
                mag = fmaf(code, rscale, mag);
                const bool neg = (sym == 1u) || (is3 && !pos_sign);
                y[j] = (neg ? -mag : mag) * kscale;
                if (valid) { nwin >>= 4; swin >>= 1; }
                jcur += is3 ? 1 : 0;
            }
            // inverse rotor (transpose of the compress-side rotor)
            if (!rotor_identity) {
                float z[8];
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 rr = *reinterpret_cast<const float4*>(&rotor_s[lane * 36 + p * 16 + c * 4]);
                        z[p * 4 + c] = y[p * 4 + 0] * rr.x + y[p * 4 + 1] * rr.y + y[p * 4 + 2] * rr.z +
                                       y[p * 4 + 3] * rr.w;
                    }
#pragma unroll
                for (int j = 0; j < 8; ++j) y[j] = z[j];
            }
            fwht256_lane8(y, lane);
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] *= dinv[j];
            // RoPE on dims 0..63: lanes 0..3 hold m = 8*lane+j, lanes 4..7 hold m+32
            {
                const float2* rl = rt + t * 32 + (lane & 3) * 8;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float other = __shfl_xor_sync(0xFFFFFFFFu, y[j], 4);
                    if (lane < 8) {
                        const float2 cs = rl[j];
                        y[j] = (lane < 4) ? (y[j] * cs.x - other * cs.y) : (other * cs.y + y[j] * cs.x);
                    }
                }
            }
            float sc[NREP];
#pragma unroll
            for (int h = 0; h < NREP; ++h) {
                float a = 0.0f;
#pragma unroll
                for (int j = 0; j < 8; ++j) a = fmaf(qv[h][j], y[j], a);
                sc[h] = a;
            }
            reduce6(sc, lane);
            float pw[NREP];
            softmax_step(st, sc, pw);

            // ===== V: code words -> rotated-domain row ======================================
            const unsigned int* vp = reinterpret_cast<const unsigned int*>(S + OFF_VPAY + row * V_PAY);
            const float vnorm = hbits2f(reinterpret_cast<const uint16_t*>(S + OFF_VN)[row]);
            const float energy = hbits2f(reinterpret_cast<const uint16_t*>(S + OFF_VRN)[row]);
            const float smv = reinterpret_cast<const float*>(S + OFF_VSM)[row];
            const float pre_v = P.alpha_v * vnorm * energy;
            const float pre_res = smv * vnorm * (1.0f / 7.0f);
            const int bo = 24 * (lane & 3);
            const int wi = 3 * (lane >> 2) + (bo >> 5);
            const unsigned int f24 = __funnelshift_r(vp[wi], vp[wi + 1], bo & 31) & 0xFFFFFFu;
            const unsigned int hb = (vp[24 + (lane >> 4)] >> (2 * (lane & 15))) & 3u;
            float v[8];
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const unsigned f = (f24 >> (12 * p)) & 0xFFFu;
                const unsigned code = (f & 0x7Fu) | (((hb >> p) & 1u) << 7);
                if (VQS) {
                    const uint2 e = *reinterpret_cast<const uint2*>(vq_s + (code * 64 + 32 * p + lane) * 4);
                    v[p * 4 + 0] = hbits2f((unsigned short)(e.x & 0xFFFFu)) * pre_v;
                    v[p * 4 + 1] = hbits2f((unsigned short)(e.x >> 16)) * pre_v;
                    v[p * 4 + 2] = hbits2f((unsigned short)(e.y & 0xFFFFu)) * pre_v;
                } else {
                    const unsigned short* e =
                        reinterpret_cast<const unsigned short*>(P.vq) + ((size_t)(lane * 2 + p) * 256 + code) * 3;
                    v[p * 4 + 0] = hbits2f(__ldg(e + 0)) * pre_v;
                    v[p * 4 + 1] = hbits2f(__ldg(e + 1)) * pre_v;
                    v[p * 4 + 2] = hbits2f(__ldg(e + 2)) * pre_v;
                }
                const float c = ((f >> 7) & 1u) ? c3[p][1] : c3[p][0];
                v[p * 4 + 3] = fmaf(c, vnorm, ((float)((f >> 8) & 0xFu) - 8.0f) * pre_res);
            }
            accumulate_v(st, pw, v);
        }
        __syncthreads();  // every warp is done with this stage and this rope buffer
    }

    tiles_done = t0 + (unsigned)ntiles;
}

// Inverse V rotor + FWHT + /16/(d_v+1e-8) of the merged state of the kv-head's heads, each stored as one
// (acc[256], max, sum_exp) record.  Called by one warp per kv-head.
__device__ __forceinline__ void v_epilogue_store(const WarpState& st, const CompressedKV& P, int lane,
                                                 float* const (&ob)[NREP]) {
    float dvi[8];
    {
        const uint4 dr = *reinterpret_cast<const uint4*>(P.d_v + lane * 8);
        const __half* hd = reinterpret_cast<const __half*>(&dr);
#pragma unroll
        for (int j = 0; j < 8; ++j) dvi[j] = (1.0f / 16.0f) / (__half2float(hd[j]) + 1e-8f);
    }
    float rv[2][16];
    {
        const uint4* rp = reinterpret_cast<const uint4*>(P.v_rotor + lane * 32);
        const uint4 r0 = rp[0], r1 = rp[1], r2 = rp[2], r3 = rp[3];
        __half hr[32];
        *reinterpret_cast<uint4*>(&hr[0]) = r0;
        *reinterpret_cast<uint4*>(&hr[8]) = r1;
        *reinterpret_cast<uint4*>(&hr[16]) = r2;
        *reinterpret_cast<uint4*>(&hr[24]) = r3;
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int i = 0; i < 16; ++i) rv[p][i] = __half2float(hr[p * 16 + i]);
    }
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
        float z[8];
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float a = 0.0f;
#pragma unroll
                for (int k = 0; k < 4; ++k) a = fmaf(st.acc[h][p * 4 + k], rv[p][c * 4 + k], a);
                z[p * 4 + c] = a;
            }
        fwht256_lane8(z, lane);
#pragma unroll
        for (int j = 0; j < 8; j += 2)
            *reinterpret_cast<float2*>(ob[h] + lane * 8 + j) = make_float2(z[j] * dvi[j], z[j + 1] * dvi[j + 1]);
        if (lane == 0) {
            ob[h][D] = st.m[h];
            ob[h][D + 1] = st.l[h];
        }
    }
}

// Records of the kernel before are read around L1 (__ldcg): with a dependent launch this kernel may have started before
// they were written.
// LSE merge of `n` partial records `stride` floats apart (acc[D], max, sum) by one block of
// G * D threads: M = max m_i, num = sum acc_i[dd] e^{m_i - M}, den = sum s_i e^{m_i - M}.
// Thread (group g, dim dd) adds records g, g + G, ... in order; the groups' sums are then
// added in group order.  A problem cut over all SMs owns hundreds of records and only H_q blocks merge
// them, so what counts is how many loads a block keeps in flight: the maximum and the weights are
// computed a record per thread, and four groups walk the records side by side.  Valid in threads
// of group 0 on return.
constexpr int MERGE_GROUPS = 4;  // launches with many records per problem; the others use one group
template <int G>
__device__ __forceinline__ float lse_merge_records(const float* __restrict__ base, size_t stride, int n, float& num,
                                                   float& den) {
    constexpr int NT = G * D;
    __shared__ float s_red[NT / 32];
    __shared__ float s_w[NT];
    __shared__ float s_num[G > 1 ? G - 1 : 1][D], s_den[G > 1 ? G - 1 : 1];
    const int tid = threadIdx.x, dd = tid & (D - 1), grp = tid / D;
    float M = NEG_BIG;
    for (int s = tid; s < n; s += NT) M = fmaxf(M, __ldcg(base + s * stride + D));
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) M = fmaxf(M, __shfl_xor_sync(0xFFFFFFFFu, M, m));
    if ((tid & 31) == 0) s_red[tid >> 5] = M;
    __syncthreads();
    M = s_red[0];
#pragma unroll
    for (int w = 1; w < NT / 32; ++w) M = fmaxf(M, s_red[w]);
    num = 0.0f;
    den = 0.0f;
    for (int s0 = 0; s0 < n; s0 += NT) {
        const int cnt = min(NT, n - s0);
        __syncthreads();
        if (tid < cnt) s_w[tid] = __expf(__ldcg(base + (s0 + tid) * stride + D) - M);
        __syncthreads();
#pragma unroll 4
        for (int j = grp; j < cnt; j += G) {
            const float* p = base + (s0 + j) * stride;
            const float w = s_w[j];
            num = fmaf(__ldcg(p + dd), w, num);
            den = fmaf(__ldcg(p + D + 1), w, den);
        }
    }
    if (G > 1) {
        if (grp > 0) {
            s_num[grp - 1][dd] = num;
            if (dd == 0) s_den[grp - 1] = den;
        }
        __syncthreads();
        if (grp == 0) {
#pragma unroll
            for (int g = 0; g < G - 1; ++g) {
                num += s_num[g][dd];
                den += s_den[g];
            }
        }
    }
    return M;
}

// LSE merge over splits: partial (nq, splits, 258) -> out (nq, 258), unnormalised.
template <int G>
__global__ void __launch_bounds__(G * D) khq_attn_reduce_kernel(const float* __restrict__ partial, float* __restrict__ out,
                                                                int num_splits) {
    const int qid = blockIdx.x, d = threadIdx.x;
    pdl_wait();
    pdl_trigger();
    float num, den;
    const float M = lse_merge_records<G>(partial + (size_t)qid * num_splits * PART, (size_t)PART, num_splits, num, den);
    if (d >= D) return;
    float* o = out + (size_t)qid * PART;
    o[d] = num;
    if (d == 0) {
        o[D] = M;
        o[D + 1] = den;
    }
}

// ------------------------------------------------------------------------------------------
// Raw ring window
// ------------------------------------------------------------------------------------------
// Window tokens s = first, first+step, ... < win_hi of this warp: slot (win_start + s) % ring_cap,
// rows token-major (slot*H_kv + kv)*D, K already RoPE'd.  U tokens at a time: their 2 U row loads are in flight together
// and their dot products and warp sums interleave (one token at a time, a token cost a warp a full memory latency plus a
// chain of six warp sums: 0.75 us).
// When new_s >= 0, window token new_s is read from new_k / new_v (one token, H_kv*D halfs each)
// instead of its ring slot: the fused step kernel appends it to the ring while the window runs.
template <int U>
__device__ __forceinline__ void window_range(const __half* __restrict__ q, const __half* __restrict__ ring_k,
                                             const __half* __restrict__ ring_v, int win_start, int first,
                                             int step, int win_hi, int ring_cap, float scale, int kvh,
                                             int lane, WarpState& st, int new_s = -1,
                                             const __half* __restrict__ new_k = nullptr,
                                             const __half* __restrict__ new_v = nullptr) {
    if (first >= win_hi) return;
    uint4 qr[NREP];
#pragma unroll
    for (int h = 0; h < NREP; ++h) qr[h] = *reinterpret_cast<const uint4*>(q + (size_t)(kvh * NREP + h) * 2 * D + lane * 8);
#pragma unroll 1
    for (int s0 = first; s0 < win_hi; s0 += U * step) {
        uint4 kr[U], vr[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int s = s0 + u * step < win_hi ? s0 + u * step : s0;  // past the end: a row that is there, weight 0
            const size_t off = ((size_t)((win_start + s) % ring_cap) * HKV + kvh) * D + lane * 8;
            const bool fresh = (s == new_s);
            kr[u] = *reinterpret_cast<const uint4*>(fresh ? new_k + (size_t)kvh * D + lane * 8 : ring_k + off);
            vr[u] = *reinterpret_cast<const uint4*>(fresh ? new_v + (size_t)kvh * D + lane * 8 : ring_v + off);
        }
        float sc[U][NREP];
        {
            float k8[U][8];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int j = 0; j < 8; ++j) k8[u][j] = __half2float(reinterpret_cast<const __half*>(&kr[u])[j]);
#pragma unroll
            for (int h = 0; h < NREP; ++h) {
                float q8[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) q8[j] = __half2float(reinterpret_cast<const __half*>(&qr[h])[j]) * scale;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    float a = 0.0f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) a = fmaf(q8[j], k8[u][j], a);
                    sc[u][h] = a;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) reduce6(sc[u], lane);
#pragma unroll
        for (int u = 1; u < U; ++u)
            if (s0 + u * step >= win_hi)
#pragma unroll
                for (int h = 0; h < NREP; ++h) sc[u][h] = -1e30f;
#pragma unroll
        for (int h = 0; h < NREP; ++h) {
            float top = sc[0][h];
#pragma unroll
            for (int u = 1; u < U; ++u) top = fmaxf(top, sc[u][h]);
            if (top > st.m[h]) {  // warp-uniform: every lane holds the same scores and maximum
                const float fac = __expf(st.m[h] - top);
                st.l[h] *= fac;
#pragma unroll
                for (int j = 0; j < 8; ++j) st.acc[h][j] *= fac;
                st.m[h] = top;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                sc[u][h] = __expf(sc[u][h] - st.m[h]);
                st.l[h] += sc[u][h];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __half2float(reinterpret_cast<const __half*>(&vr[u])[j]);
            accumulate_v(st, sc[u], v);
        }
    }
}

__device__ __forceinline__ void raw_store(const WarpState& st, int lane, float* const (&ob)[NREP]) {
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
#pragma unroll
        for (int j = 0; j < 8; j += 2)
            *reinterpret_cast<float2*>(ob[h] + lane * 8 + j) = make_float2(st.acc[h][j], st.acc[h][j + 1]);
        if (lane == 0) {
            ob[h][D] = st.m[h];
            ob[h][D + 1] = st.l[h];
        }
    }
}

// One cluster: token s is served by warp (kv, sub) of CTA c when
// s % (cluster_size*DEC_WPK) == c*DEC_WPK + sub.  The heads of the result are dealt to the cluster's warps, which merge the
// per-warp records through distributed shared memory.
constexpr int WIN_SMEM = (DEC_WARPS * MERGE_FLOATS + HQ * PART) * 4;  // one record per warp; the CTA's own heads

// Behind a cluster barrier: head h merged over the records of all warps of the cluster that served its kv-head.
__device__ __forceinline__ HeadAcc window_head(cg::cluster_group& cluster, const float* rec, int csize, int h, int lane) {
    return merge_head<false>(DEC_WPK * csize, lane, [&](int i) {
        return head_of_record(cluster.map_shared_rank(rec, i / DEC_WPK) + (h / NREP + HKV * (i % DEC_WPK)) * MERGE_FLOATS, h % NREP);
    });
}

__global__ void __launch_bounds__(DEC_THREADS, 1)
khq_window_attn_kernel(const __half* __restrict__ q, const __half* __restrict__ ring_k,
                       const __half* __restrict__ ring_v, float* __restrict__ out, int win_start,
                       int win_len, int ring_cap, float scale) {
    extern __shared__ __align__(128) unsigned char smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = warp & 3, sub = warp >> 2;
    const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
    float* rec = reinterpret_cast<float*>(smem);
    pdl_wait();
    pdl_trigger();
    WarpState st;
    st.init();
    window_range<4>(q, ring_k, ring_v, win_start, crank * DEC_WPK + sub, csize * DEC_WPK, win_len, ring_cap, scale,
                    kvh, lane, st);
    store_record(st, rec + warp * MERGE_FLOATS, lane);
    cluster.sync();
#pragma unroll 1
    for (int h = crank + csize * warp; h < HQ; h += csize * DEC_WARPS) store_head(window_head(cluster, rec, csize, h, lane), out + (size_t)h * PART, lane);
    cluster.sync();  // peers must stay resident until their records have been read
}

// ------------------------------------------------------------------------------------------
// Batched decode: many (sequence, layer) problems in one persistent launch
// ------------------------------------------------------------------------------------------
// One CTA per SM pulls work items off an atomic counter.  An item is a token range of one
// problem's compressed region (all four kv-heads) or its raw window; its result is one
// (24, 258) partial in the workspace.  Items arrive ordered by layer so that the layer's
// tables, and the V codebook in shared memory, are reloaded only when the layer changes.
template <bool VQS>
__global__ void __launch_bounds__(DEC_THREADS, 1)
khq_decode_batched_kernel(const KhqSeqDesc* __restrict__ descs, const KhqTablesDesc* __restrict__ tables,
                          const KhqWorkItem* __restrict__ items, int n_items, int* __restrict__ counter,
                          float* __restrict__ partials, float scale, float rope_base, int ring_cap) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_next;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = warp & 3, sub = warp >> 2;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM_BARS);
    if (tid == 0) {
        for (int s = 0; s < NSTAGE; ++s) mbar_init(&bars[s], 1);
        fence_barrier_init();
    }
    int cur_table = -1;
    unsigned tiles_done = 0;
#pragma unroll 1
    while (true) {
        __syncthreads();  // previous item fully retired (merge area, s_next readers)
        if (tid == 0) s_next = atomicAdd(counter, 1);
        __syncthreads();
        const int it = s_next;
        if (it >= n_items) break;
        const KhqWorkItem w = items[it];
        const KhqSeqDesc d = descs[w.desc];
        float* ob[NREP];
#pragma unroll
        for (int h = 0; h < NREP; ++h) ob[h] = partials + ((size_t)w.slot * HQ + kvh * NREP + h) * PART;
        WarpState st;
        st.init();
        if (w.kind == 0) {
            const KhqTablesDesc t = tables[d.table_id];
            CompressedKV P;
            P.k_payload = d.k_payload; P.v_payload = d.v_payload; P.v_shared_meta = d.v_shared_meta;
            P.k_mask = d.k_mask; P.k_norms = d.k_norms; P.k_r_norms = d.k_r_norms;
            P.v_norms = d.v_norms; P.v_r_norms = d.v_r_norms;
            P.cents_k = t.cents_k; P.cents_v = t.cents_v; P.vq = t.vq; P.k_rotor = t.k_rotor;
            P.v_rotor = t.v_rotor; P.d_k = t.d_k; P.d_v = t.d_v;
            P.alpha_k = t.alpha_k; P.alpha_v = t.alpha_v; P.rope_base = rope_base;
            P.start_pos = d.start_pos; P.c_len = d.c_len; P.bulk_ok = 1; P.image = nullptr;
            unpack_pos(d.pos_pack, P);
            if (d.table_id != cur_table) {
                setup_tables(smem, P, tid);
                if (VQS) load_codebook(reinterpret_cast<unsigned short*>(smem + SM_VQ), P.vq, tid);
                cur_table = d.table_id;
            }
            compressed_range<VQS>(smem, d.q_gate, (size_t)2 * D, P, w.lo, w.hi, scale, st, tiles_done);
            merge_cta(st, reinterpret_cast<float*>(smem + SM_MERGE), kvh, sub, lane);
            if (sub == 0) v_epilogue_store(st, P, lane, ob);
        } else {
            window_range<4>(d.q_gate, d.ring_k, d.ring_v, d.win_start, w.lo + sub, DEC_WPK, w.hi, ring_cap, scale, kvh,
                            lane, st);
            merge_cta(st, reinterpret_cast<float*>(smem + SM_MERGE), kvh, sub, lane);
            if (sub == 0) raw_store(st, lane, ob);
        }
    }
}

}  // namespace khq
#include "khq_decode_mma.cuh"
#include "khq_decode_tc5.cuh"
#include "khq_decode_tc5w.cuh"
#include "khq_step.cuh"
namespace khq {

// Per problem and query head: LSE merge of the problem's partial slots, /(den+1e-8), sigmoid
// gate, fp16 store.  grid = n_desc*HQ blocks of G * D threads.
// A problem with few records (the batched serving case: about a dozen).  The block is bound by the latency of
// its loads, so the records are taken eight at a time with all 24 loads of a chunk issued together, and the chunks
// are folded into the running (max, num, den) the way the attention itself folds blocks of tokens.
__global__ void __launch_bounds__(D)
khq_batched_merge_gate_few_kernel(const KhqSeqDesc* __restrict__ descs, const float* __restrict__ partials) {
    constexpr int CH = 8;
    const int di = blockIdx.x / HQ, h = blockIdx.x % HQ, dd = threadIdx.x;
    pdl_wait();
    pdl_trigger();
    const KhqSeqDesc d = descs[di];
    const float* base = partials + ((size_t)d.first_slot * HQ + h) * PART;
    const float gate = __half2float(d.q_gate[(size_t)h * 2 * D + D + dd]);
    float M = NEG_BIG, num = 0.0f, den = 0.0f;
    for (int s0 = 0; s0 < d.n_slots; s0 += CH) {
        float m[CH], l[CH], a[CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const bool in = s0 + i < d.n_slots;
            const float* p = base + (size_t)(in ? s0 + i : s0) * HQ * PART;
            m[i] = in ? __ldcg(p + D) : NEG_BIG;
            l[i] = in ? __ldcg(p + D + 1) : 0.0f;
            a[i] = in ? __ldcg(p + dd) : 0.0f;
        }
        float cm = M;
#pragma unroll
        for (int i = 0; i < CH; ++i) cm = fmaxf(cm, m[i]);
        const float keep = __expf(M - cm);
        num *= keep;
        den *= keep;
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const float w = __expf(m[i] - cm);
            num = fmaf(a[i], w, num);
            den = fmaf(l[i], w, den);
        }
        M = cm;
    }
    const float val = num / (den + 1e-8f);
    d.out[(size_t)h * D + dd] = __float2half(val * (1.0f / (1.0f + __expf(-gate))));
}

template <int G>
__global__ void __launch_bounds__(G * D)
khq_batched_merge_gate_kernel(const KhqSeqDesc* __restrict__ descs, const float* __restrict__ partials) {
    const int di = blockIdx.x / HQ, h = blockIdx.x % HQ, dd = threadIdx.x;
    pdl_wait();
    pdl_trigger();
    const KhqSeqDesc d = descs[di];
    float num, den;
    lse_merge_records<G>(partials + ((size_t)d.first_slot * HQ + h) * PART, (size_t)HQ * PART, d.n_slots, num, den);
    if (dd >= D) return;
    const float val = num / (den + 1e-8f);
    const float g = __half2float(d.q_gate[(size_t)h * 2 * D + D + dd]);
    d.out[(size_t)h * D + dd] = __float2half(val * (1.0f / (1.0f + __expf(-g))));
}

// The same merge without the division and the gate: one unnormalised record (num[256], max, den) per
// (problem, head) into out_partials (n_desc, H_q, 258) -- what a context-parallel rank hands to the exchange.
template <int G>
__global__ void __launch_bounds__(G * D)
khq_batched_merge_partial_kernel(const KhqSeqDesc* __restrict__ descs, const float* __restrict__ partials,
                                 float* __restrict__ out_partials) {
    const int di = blockIdx.x / HQ, h = blockIdx.x % HQ, dd = threadIdx.x;
    pdl_wait();
    pdl_trigger();
    const KhqSeqDesc d = descs[di];
    float num, den;
    const float M = lse_merge_records<G>(partials + ((size_t)d.first_slot * HQ + h) * PART, (size_t)HQ * PART, d.n_slots, num, den);
    if (dd >= D) return;
    float* o = out_partials + ((size_t)di * HQ + h) * PART;
    o[dd] = num;
    if (dd == 0) {
        o[D] = (d.n_slots > 0) ? M : -1e20f;  // a problem without items: the neutral record
        o[D + 1] = den;
    }
}

// Fused tail of a decode step for one sequence: appends the step's token to the three rings (K
// RoPE'd, V, K un-RoPE'd; CTA 0, while every CTA reads that token straight from the inputs), runs
// the raw-window attention over win_len tokens (the new one is the last), then the cluster's warps
// merge the heads they are dealt: the window records, the n_c <= 32 records per head of the compressed region
// (head-major, PART floats each), /(den + 1e-8), sigmoid gate, fp16 store.
// With n_c > 0 the launch before it in the stream has to be the compressed-region kernel of the same step (or its reduction), which
// lets it start only when everything before that is complete, reads no ring and writes nothing but those records: the appends and the
// window part run beside it.
__global__ void __launch_bounds__(DEC_THREADS, 1)
khq_window_step_kernel(const __half* __restrict__ q, __half* __restrict__ ring_k, __half* __restrict__ ring_v,
                       __half* __restrict__ ring_u, const __half* __restrict__ new_k, const __half* __restrict__ new_v,
                       const __half* __restrict__ new_u, const float* __restrict__ part_c, __half* __restrict__ out,
                       int win_start, int win_len, int ring_cap, float scale, int n_c) {
    extern __shared__ __align__(128) unsigned char smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = warp & 3, sub = warp >> 2;
    const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
    const int new_s = new_k != nullptr ? win_len - 1 : -1;  // -1: the token's rows are in the rings already
    float* rec = reinterpret_cast<float*>(smem);
    if (n_c == 0) pdl_wait();
    pdl_trigger();  // what may start now reads nothing but constants before its own wait
    if (crank == 0) {  // ring appends: 3 rows of H_kv*D halfs = 3 x 128 sixteen-byte chunks
        const int slot = (win_start + win_len - 1) % ring_cap;
        const size_t row = (size_t)slot * HKV * D;
        for (int c = tid; c < 3 * (HKV * D / 8); c += DEC_THREADS) {
            const int which = c / (HKV * D / 8), i = c % (HKV * D / 8);
            const __half* src = which == 0 ? new_k : (which == 1 ? new_v : new_u);
            __half* dst = which == 0 ? ring_k : (which == 1 ? ring_v : ring_u);
            if (src != nullptr && dst != nullptr)
                reinterpret_cast<uint4*>(dst + row)[i] = reinterpret_cast<const uint4*>(src)[i];
        }
    }
    WarpState st;
    st.init();
    window_range<4>(q, ring_k, ring_v, win_start, crank * DEC_WPK + sub, csize * DEC_WPK, win_len, ring_cap, scale, kvh,
                    lane, st, new_s, new_k, new_v);
    store_record(st, rec + warp * MERGE_FLOATS, lane);
    cluster.sync();
    // the window part of the heads dealt to this CTA (every csize-th), while the compressed-region kernel may still run
    float* own = rec + DEC_WARPS * MERGE_FLOATS;
#pragma unroll 1
    for (int k = warp; crank + csize * k < HQ; k += DEC_WARPS) store_head(window_head(cluster, rec, csize, crank + csize * k, lane), own + k * PART, lane);
    cluster.sync();  // peers must stay resident until their records have been read
    pdl_wait();
    // a thread finishes two dims of one head: all its loads of the split records are in flight together
    for (int e = tid; e < (HQ - crank + csize - 1) / csize * (D / 2); e += DEC_THREADS) {
        const int k = e / (D / 2), h = crank + csize * k, d = 2 * (e % (D / 2));
        const float2 aw = *reinterpret_cast<const float2*>(own + k * PART + d);
        float M = own[k * PART + D];
        const float mw = M, lw = own[k * PART + D + 1];
        const __half2 hg = *reinterpret_cast<const __half2*>(q + (size_t)h * 2 * D + D + d);
        const float* pc = part_c + (size_t)h * n_c * PART;
        for (int i = 0; i < n_c; ++i) M = fmaxf(M, __ldcg(pc + i * PART + D));
        const float w0 = __expf(mw - M);
        float num0 = aw.x * w0, num1 = aw.y * w0, den = lw * w0;
#pragma unroll 8
        for (int i = 0; i < n_c; ++i) {
            const float w = __expf(__ldcg(pc + i * PART + D) - M);
            const float2 v = __ldcg(reinterpret_cast<const float2*>(pc + i * PART + d));
            num0 = fmaf(v.x, w, num0);
            num1 = fmaf(v.y, w, num1);
            den = fmaf(__ldcg(pc + i * PART + D + 1), w, den);
        }
        const float inv = 1.0f / (den + 1e-8f);
        const float2 gf = __half22float2(hg);
        *reinterpret_cast<__half2*>(out + (size_t)h * D + d) =
            __floats2half2_rn(num0 * inv * (1.0f / (1.0f + __expf(-gf.x))), num1 * inv * (1.0f / (1.0f + __expf(-gf.y))));
    }
}

// LSE merge of the two regions, /(den + 1e-8), sigmoid gate, fp16 store.
__global__ void khq_merge_gate_kernel(const float* __restrict__ attn_c, const float* __restrict__ attn_w,
                                      const __half* __restrict__ q_gate, __half* __restrict__ out, int H_q,
                                      int d_v, int has_w) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= H_q * d_v) return;
    const int h = i / d_v, d = i % d_v;
    const float* cc = attn_c + (size_t)h * (d_v + 2);
    float num = __ldcg(cc + d), den = __ldcg(cc + d_v + 1);
    if (has_w) {
        const float* cw = attn_w + (size_t)h * (d_v + 2);
        const float mc = __ldcg(cc + d_v), mw = __ldcg(cw + d_v);
        const float M = fmaxf(mc, mw);
        const float wc = __expf(mc - M), ww = __expf(mw - M);
        num = num * wc + __ldcg(cw + d) * ww;
        den = den * wc + __ldcg(cw + d_v + 1) * ww;
    }
    const float val = num / (den + 1e-8f);
    const float g = __half2float(q_gate[(size_t)h * 2 * d_v + d_v + d]);
    out[i] = __float2half(val * (1.0f / (1.0f + __expf(-g))));
}

// LSE merge of n_slots slot-major partials (slot, H_q, 258) -> /(den+1e-8) -> sigmoid gate -> fp16.
// Used to finish a context-parallel step from the partials gathered from every GPU.
__global__ void __launch_bounds__(D)
khq_merge_slots_gate_kernel(const float* __restrict__ partials, int n_slots, const __half* __restrict__ q_gate,
                            __half* __restrict__ out) {
    const int h = blockIdx.x, dd = threadIdx.x;
    float M = NEG_BIG;
    for (int s = 0; s < n_slots; ++s) M = fmaxf(M, partials[((size_t)s * HQ + h) * PART + D]);
    float num = 0.0f, den = 0.0f;
    for (int s = 0; s < n_slots; ++s) {
        const float* p = partials + ((size_t)s * HQ + h) * PART;
        const float w = __expf(p[D] - M);
        num = fmaf(p[dd], w, num);
        den = fmaf(p[D + 1], w, den);
    }
    const float val = num / (den + 1e-8f);
    const float g = __half2float(q_gate[(size_t)h * 2 * D + D + dd]);
    out[(size_t)h * D + dd] = __float2half(val * (1.0f / (1.0f + __expf(-g))));
}

// ---- context-parallel exchange over peer memory ----------------------------------------------
// Instead of an all-gather, every GPU stores its partial records straight into every peer's slot
// buffer (plain st.global over NVLink), fences system-wide and raises its flag on that peer to the
// step's epoch; the consumer's merge kernel waits (bounded) for all flags, then merges and gates.
// One CTA per destination GPU.
__global__ void __launch_bounds__(256)
khq_publish_partials_kernel(const float* __restrict__ src, int n_floats, float* const* __restrict__ peer_slots,
                            unsigned int* const* __restrict__ peer_flags, long long dst_offset, int rank,
                            unsigned int epoch) {
    const int p = blockIdx.x;
    float4* dst = reinterpret_cast<float4*>(peer_slots[p] + dst_offset);
    const float4* s4 = reinterpret_cast<const float4*>(src);
    for (int i = threadIdx.x; i < n_floats / 4; i += blockDim.x) dst[i] = s4[i];
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int* flag = peer_flags[p] + rank;
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flag), "r"(epoch) : "memory");
    }
}

// Generic form of the same: `n16` 16-byte units from `src` to byte offset `dst_off` of every peer's
// buffer, then the epoch into word `flag_index` of every peer's flag array.
__global__ void __launch_bounds__(256)
khq_publish_bytes_kernel(const uint4* __restrict__ src, int n16, unsigned char* const* __restrict__ peer_bufs,
                         long long dst_off, unsigned int* const* __restrict__ peer_flags, int flag_index,
                         unsigned int epoch) {
    const int p = blockIdx.x;
    uint4* dst = reinterpret_cast<uint4*>(peer_bufs[p] + dst_off);
    for (int i = threadIdx.x; i < n16; i += blockDim.x) dst[i] = src[i];
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int* flag = peer_flags[p] + flag_index;
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flag), "r"(epoch) : "memory");
    }
}

// One thread waits (bounded) until *flag >= epoch (modulo 2^32): stream-orders the kernels behind it
// after a peer's publish.  Status word 3 when the wait runs out.
__global__ void khq_wait_flag_kernel(const unsigned int* __restrict__ flag, unsigned int epoch, unsigned int max_polls) {
    bool seen = false;
    for (unsigned int it = 0; it < max_polls; ++it) {
        unsigned int v;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if ((int)(v - epoch) >= 0) {
            seen = true;
            break;
        }
        __nanosleep(64);
    }
    if (!seen) atomicExch(&g_status, 3);
}

// The slot merge of khq_merge_slots_gate_kernel, preceded by a bounded wait for the `n_flags`
// producers of this step (flag >= epoch, compared modulo 2^32).  Slots are read around L1 (peers
// wrote them).  A wait that runs out sets the status word to 3 and the CTA still finishes.
__global__ void __launch_bounds__(D)
khq_merge_slots_wait_gate_kernel(const float* __restrict__ partials, const unsigned int* __restrict__ flags, int n_flags,
                                 unsigned int epoch, int n_slots, const __half* __restrict__ q_gate,
                                 __half* __restrict__ out, unsigned int max_polls) {
    const int h = blockIdx.x, dd = threadIdx.x;
    if (dd < n_flags) {
        bool seen = false;
        for (unsigned int it = 0; it < max_polls; ++it) {
            unsigned int v;
            asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flags + dd) : "memory");
            if ((int)(v - epoch) >= 0) {
                seen = true;
                break;
            }
            __nanosleep(64);
        }
        if (!seen) atomicExch(&g_status, 3);
    }
    __syncthreads();
    float M = NEG_BIG;
    for (int s = 0; s < n_slots; ++s) M = fmaxf(M, __ldcv(partials + ((size_t)s * HQ + h) * PART + D));
    float num = 0.0f, den = 0.0f;
    for (int s = 0; s < n_slots; ++s) {
        const float* p = partials + ((size_t)s * HQ + h) * PART;
        const float w = __expf(__ldcv(p + D) - M);
        num = fmaf(__ldcv(p + dd), w, num);
        den = fmaf(__ldcv(p + D + 1), w, den);
    }
    const float val = num / (den + 1e-8f);
    const float g = __half2float(q_gate[(size_t)h * 2 * D + D + dd]);
    out[(size_t)h * D + dd] = __float2half(val * (1.0f / (1.0f + __expf(-g))));
}

__global__ void khq_gather_q_kernel(const __half* __restrict__ q_gate, __half* __restrict__ q_out, int H_q,
                                    int d_v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= H_q * d_v) return;
    q_out[i] = q_gate[(size_t)(i / d_v) * 2 * d_v + (i % d_v)];
}

// ------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------
static inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// Opt in to >48 KB of dynamic shared memory, once per device.
static cudaError_t ensure_smem_attrs() {
    static bool done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if ((e = cudaFuncSetAttribute(khq_decode_batched_kernel<false>, attr, SM_TOTAL)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(khq_decode_batched_kernel<true>, attr, SM_TOTAL_VQ)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(khq_decode_batched_mma_kernel, attr, M2_SM_TOTAL)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(khq_attn_compressed_mma_kernel, attr, M2_SM_TOTAL)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(m3::khq_decode_batched_tc5_kernel, attr, m3::SM_TOTAL)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(m3::khq_decode_batched_tc5w_kernel, attr, m3::SM_TOTAL)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(khq_window_attn_kernel, attr, WIN_SMEM)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(khq_window_step_kernel, attr, WIN_SMEM)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(khq_step_kernel<false>, attr, ST_SM_TOTAL)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(khq_step_kernel<true>, attr, ST_SM_TOTAL)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(khq_step_wide_kernel<false>, attr, SW_TOTAL)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(khq_step_wide_kernel<true>, attr, SW_TOTAL)) != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) done[dev] = true;
    return cudaSuccess;
}

// How many clusters of `c` CTAs of the compressed-attention kernel fit on the device at once.
static int max_clusters(int c) {
    static int cache[64][9] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || c < 1 || c > 8) return 1;
    int& slot = cache[dev][c];
    if (slot == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)c, 1, 1);
        cfg.blockDim = dim3((unsigned)M2_THREADS, 1, 1);
        cfg.dynamicSmemBytes = (size_t)M2_SM_TOTAL;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)c;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, khq_attn_compressed_mma_kernel, &cfg) != cudaSuccess || n <= 0) {
            (void)cudaGetLastError();
            n = sm_count() / c > 0 ? sm_count() / c : 1;
        }
        slot = n;
    }
    return slot;
}

}  // namespace khq

using namespace khq;

static int attn_launch_impl(const void* q, const void* k_payload, const void* v_payload,
                            const void* v_shared_meta, const void* k_mask, const void* k_norms,
                            const void* k_r_norms, const void* v_norms, const void* v_r_norms,
                            const void* centroids_k, const void* centroids_v,
                            const void* vq_centroids, const void* k_rotor, const void* v_rotor,
                            const void* d_vec_k, const void* d_vec_v, void* out_attn,
                            void* out_partial, int num_queries, int num_heads, int L_q, int c_len,
                            int n_rep, float scale, float alpha_k, float alpha_v,
                            float rope_base, int start_pos, int num_splits, int pos_chunk, int pos_stride,
                            bool reduce, const void* image, cudaStream_t stream) {
    if (num_queries <= 0 || c_len <= 0) return -100;
    if (num_splits < 1) num_splits = 1;
    if (num_splits > 1 && out_partial == nullptr) return -101;
    if (n_rep != NREP || num_heads != HQ || L_q < 1 || num_queries != num_heads * L_q) return -103;
    const void* tables[] = {q, centroids_k, centroids_v, vq_centroids, k_rotor, v_rotor, d_vec_k, d_vec_v};
    for (const void* t : tables)
        if (!aligned(t, 16)) return -104;
    const void* arrays[] = {k_payload, v_payload, v_shared_meta, k_mask, k_norms, k_r_norms, v_norms, v_r_norms};
    bool bulk_ok = true;
    for (const void* a : arrays) {
        if (!aligned(a, 4)) return -104;
        bulk_ok = bulk_ok && aligned(a, 16);
    }
    if (!aligned(out_attn, 8) || (out_partial && !aligned(out_partial, 8))) return -104;
    cudaError_t err = ensure_smem_attrs();
    if (err != cudaSuccess) return static_cast<int>(err);

    CompressedKV P;
    P.k_payload = static_cast<const unsigned char*>(k_payload);
    P.v_payload = static_cast<const unsigned char*>(v_payload);
    P.v_shared_meta = static_cast<const unsigned char*>(v_shared_meta);
    P.k_mask = static_cast<const unsigned int*>(k_mask);
    P.k_norms = static_cast<const __half*>(k_norms);
    P.k_r_norms = static_cast<const __half*>(k_r_norms);
    P.v_norms = static_cast<const __half*>(v_norms);
    P.v_r_norms = static_cast<const __half*>(v_r_norms);
    P.cents_k = static_cast<const __half*>(centroids_k);
    P.cents_v = static_cast<const __half*>(centroids_v);
    P.vq = static_cast<const __half*>(vq_centroids);
    P.k_rotor = static_cast<const __half*>(k_rotor);
    P.v_rotor = static_cast<const __half*>(v_rotor);
    P.d_k = static_cast<const __half*>(d_vec_k);
    P.d_v = static_cast<const __half*>(d_vec_v);
    P.alpha_k = alpha_k;
    P.alpha_v = alpha_v;
    P.rope_base = rope_base;
    P.start_pos = start_pos;
    P.c_len = c_len;
    P.bulk_ok = bulk_ok ? 1 : 0;
    P.pos_chunk = pos_chunk;
    P.pos_stride = pos_stride;
    P.image = static_cast<const unsigned char*>(image);

    for (int l = 0; l < L_q; ++l) {
        const int s_limit = (L_q > 1) ? (c_len < l + 1 ? c_len : l + 1) : c_len;
        const int per = (s_limit + num_splits - 1) / num_splits;
        // CTAs per split (a portable cluster of at most 8), by estimated time in units of 0.16 us: waves x (per-CTA
        // set-up + tokens per CTA in whole 48-token rounds), waves = splits / clusters of that size that fit on the GPU at
        // once (clusters are placed inside a GPC, so fewer than SMs / size fit).
        int cluster = 1;
        long long best = -1;
        for (int c = 1; c <= 8; ++c) {
            const int tpc = (per + c - 1) / c;
            const long long waves = (num_splits + max_clusters(c) - 1) / max_clusters(c);
            const long long cost = waves * (70 + (tpc + M2_TT - 1) / M2_TT * M2_TT);
            if (best < 0 || cost < best) {
                best = cost;
                cluster = c;
            }
            if (tpc <= M2_TT) break;  // more CTAs would only add set-ups
        }
        err = launch_pdl(khq_attn_compressed_mma_kernel, (unsigned)(num_splits * cluster), (unsigned)cluster,
                         (size_t)M2_SM_TOTAL, stream, (unsigned)M2_THREADS, static_cast<const __half*>(q), P,
                         static_cast<float*>(out_attn), static_cast<float*>(out_partial), num_splits, L_q,
                         l, s_limit, scale);
        if (err != cudaSuccess) return static_cast<int>(err);
    }
    if (num_splits > 1 && reduce) {
        if (num_splits > 32)
            err = launch_pdl(khq_attn_reduce_kernel<MERGE_GROUPS>, (unsigned)num_queries, 0, 0, stream, MERGE_GROUPS * D,
                             static_cast<const float*>(out_partial), static_cast<float*>(out_attn), num_splits);
        else
            err = launch_pdl(khq_attn_reduce_kernel<1>, (unsigned)num_queries, 0, 0, stream, D,
                             static_cast<const float*>(out_partial), static_cast<float*>(out_attn), num_splits);
        if (err != cudaSuccess) return static_cast<int>(err);
    }
    return 0;
}

extern "C" int launch_khq_attn_fp16(const void* q, const void* k_payload, const void* v_payload,
                                    const void* v_shared_meta, const void* k_mask, const void* k_norms,
                                    const void* k_r_norms, const void* v_norms, const void* v_r_norms,
                                    const void* centroids_k, const void* centroids_v,
                                    const void* vq_centroids, const void* k_rotor, const void* v_rotor,
                                    const void* d_vec_k, const void* d_vec_v, void* out_attn,
                                    void* out_partial, int num_queries, int num_heads, int L_q, int c_len,
                                    int stride_s, int n_rep, float scale, float alpha_k, float alpha_v,
                                    float rope_base, int start_pos, int num_splits, cudaStream_t stream) {
    (void)stride_s;
    return attn_launch_impl(q, k_payload, v_payload, v_shared_meta, k_mask, k_norms, k_r_norms, v_norms, v_r_norms,
                            centroids_k, centroids_v, vq_centroids, k_rotor, v_rotor, d_vec_k, d_vec_v, out_attn, out_partial,
                            num_queries, num_heads, L_q, c_len, n_rep, scale, alpha_k, alpha_v, rope_base, start_pos,
                            num_splits, 0, 0, true, nullptr, stream);
}

// launch_khq_attn_fp16 over a slice that holds every G-th `pos_chunk`-token chunk of a longer context
// (chunk-cyclic context partition over G GPUs): token s of the arrays sits at absolute position
// start_pos + (s / pos_chunk) * pos_stride + s % pos_chunk.  pos_chunk must be even and positive,
// pos_stride >= pos_chunk; -103 otherwise.  No counterpart in the reference (it serves one GPU).
extern "C" int launch_khq_attn_strided_fp16(const void* q, const void* k_payload, const void* v_payload,
                                            const void* v_shared_meta, const void* k_mask, const void* k_norms,
                                            const void* k_r_norms, const void* v_norms, const void* v_r_norms,
                                            const void* centroids_k, const void* centroids_v,
                                            const void* vq_centroids, const void* k_rotor, const void* v_rotor,
                                            const void* d_vec_k, const void* d_vec_v, void* out_attn,
                                            void* out_partial, int num_queries, int num_heads, int L_q, int c_len,
                                            int n_rep, float scale, float alpha_k, float alpha_v, float rope_base,
                                            int start_pos, int num_splits, int pos_chunk, int pos_stride,
                                            cudaStream_t stream) {
    if (pos_chunk <= 0 || (pos_chunk & 1) || pos_stride < pos_chunk) return -103;
    return attn_launch_impl(q, k_payload, v_payload, v_shared_meta, k_mask, k_norms, k_r_norms, v_norms, v_r_norms,
                            centroids_k, centroids_v, vq_centroids, k_rotor, v_rotor, d_vec_k, d_vec_v, out_attn, out_partial,
                            num_queries, num_heads, L_q, c_len, n_rep, scale, alpha_k, alpha_v, rope_base, start_pos,
                            num_splits, pos_chunk, pos_stride, true, nullptr, stream);
}

// CTAs of the one cluster that runs a raw window: a warp takes four tokens at a time.
static unsigned window_cluster(int win_len) {
    const int c = (win_len + DEC_WPK * 4 - 1) / (DEC_WPK * 4);
    return (unsigned)(c < 1 ? 1 : c > 8 ? 8 : c);
}

extern "C" int launch_khq_window_attn_fp16(const void* q, const void* ring_k, const void* ring_v,
                                           void* out_attn, int win_start, int win_len, int ring_cap,
                                           int H_q, int H_kv, int d, float scale, cudaStream_t stream) {
    if (H_q <= 0 || win_len <= 0) return -100;
    if (H_q != HQ || H_kv != HKV || d != D || ring_cap <= 0) return -103;
    if (!aligned(q, 16) || !aligned(ring_k, 16) || !aligned(ring_v, 16) || !aligned(out_attn, 8)) return -104;
    cudaError_t err = ensure_smem_attrs();
    if (err != cudaSuccess) return static_cast<int>(err);
    err = launch_pdl(khq_window_attn_kernel, window_cluster(win_len), window_cluster(win_len), (size_t)WIN_SMEM, stream,
                     (unsigned)DEC_THREADS, static_cast<const __half*>(q), static_cast<const __half*>(ring_k),
                     static_cast<const __half*>(ring_v), static_cast<float*>(out_attn), win_start, win_len, ring_cap, scale);
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

extern "C" int launch_khq_merge_gate_fp16(const void* attn_c, const void* attn_w, const void* q_gate,
                                          void* out, int H_q, int d, int has_w, cudaStream_t stream) {
    if (H_q <= 0 || d <= 0) return -100;
    const int total = H_q * d, threads = 256;
    const cudaError_t err = launch_pdl(khq_merge_gate_kernel, (unsigned)((total + threads - 1) / threads), 0, 0, stream,
                                       (unsigned)threads, static_cast<const float*>(attn_c), static_cast<const float*>(attn_w),
                                       static_cast<const __half*>(q_gate), static_cast<__half*>(out), H_q, d, has_w);
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

// One decode step of one sequence in two or three launches: compressed-region attention over
// c_len tokens (launch_khq_attn_fp16 with its arguments; skipped when c_len == 0), then the fused
// ring append + window attention + merge + gate kernel.  win_len counts the step's own token,
// which is appended at slot (win_start + win_len - 1) % ring_cap.
// k_roped == v_new == NULL: the token's rows are in the rings already (a pre-step appended them).
static int decode_step_impl(
    const void* q_gate, const void* k_roped, const void* v_new, const void* k_unroped, void* ring_k, void* ring_v,
    void* ring_u, const void* k_payload, const void* v_payload, const void* v_shared_meta, const void* k_mask,
    const void* k_norms, const void* k_r_norms, const void* v_norms, const void* v_r_norms, const void* centroids_k,
    const void* centroids_v, const void* vq_centroids, const void* k_rotor, const void* v_rotor, const void* d_vec_k,
    const void* d_vec_v, void* attn_c, void* attn_partial, void* out, int c_len, int win_start, int win_len, int ring_cap,
    int num_splits, float scale, float alpha_k, float alpha_v, float rope_base, const void* image, cudaStream_t stream) {
    const void* al[] = {q_gate, k_roped, v_new, k_unroped, ring_k, ring_v, ring_u, out};
    for (const void* p : al)
        if (p && !aligned(p, 16)) return -104;
    if (!aligned(attn_c, 8)) return -104;
    // the tail merges up to 32 split records per head itself
    const bool tail_merges = num_splits > 1 && num_splits <= 32;
    if (c_len > 0) {
        const int rc = attn_launch_impl(q_gate, k_payload, v_payload, v_shared_meta, k_mask, k_norms, k_r_norms, v_norms, v_r_norms,
                                        centroids_k, centroids_v, vq_centroids, k_rotor, v_rotor, d_vec_k, d_vec_v, attn_c, attn_partial,
                                        HQ, HQ, 1, c_len, NREP, scale, alpha_k, alpha_v, rope_base, 0, num_splits, 0, 0, !tail_merges, image, stream);
        if (rc != 0) return rc;
    }
    cudaError_t err = ensure_smem_attrs();
    if (err != cudaSuccess) return static_cast<int>(err);
    const float* part_c = static_cast<const float*>(tail_merges ? attn_partial : attn_c);
    // Nothing may be launched between the attention above and this: see the kernel.
    err = launch_pdl(khq_window_step_kernel, window_cluster(win_len), window_cluster(win_len), (size_t)WIN_SMEM,
                     stream, (unsigned)DEC_THREADS, static_cast<const __half*>(q_gate), static_cast<__half*>(ring_k),
                     static_cast<__half*>(ring_v), static_cast<__half*>(ring_u), static_cast<const __half*>(k_roped),
                     static_cast<const __half*>(v_new), static_cast<const __half*>(k_unroped), part_c, static_cast<__half*>(out),
                     win_start, win_len, ring_cap, scale, c_len > 0 ? (tail_merges ? num_splits : 1) : 0);
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

extern "C" int launch_khq_decode_step_fp16(
    const void* q_gate, const void* k_roped, const void* v_new, const void* k_unroped, void* ring_k, void* ring_v,
    void* ring_u, const void* k_payload, const void* v_payload, const void* v_shared_meta, const void* k_mask,
    const void* k_norms, const void* k_r_norms, const void* v_norms, const void* v_r_norms, const void* centroids_k,
    const void* centroids_v, const void* vq_centroids, const void* k_rotor, const void* v_rotor, const void* d_vec_k,
    const void* d_vec_v, void* attn_c, void* attn_partial, void* out, int c_len, int win_start, int win_len, int ring_cap,
    int num_splits, float scale, float alpha_k, float alpha_v, float rope_base, cudaStream_t stream) {
    if (!q_gate || !k_roped || !v_new || !ring_k || !ring_v || !attn_c || !out || win_len <= 0 || c_len < 0) return -100;
    if (ring_cap <= 0 || win_len > ring_cap) return -103;
    return decode_step_impl(q_gate, k_roped, v_new, k_unroped, ring_k, ring_v, ring_u, k_payload, v_payload, v_shared_meta, k_mask,
                            k_norms, k_r_norms, v_norms, v_r_norms, centroids_k, centroids_v, vq_centroids, k_rotor, v_rotor,
                            d_vec_k, d_vec_v, attn_c, attn_partial, out, c_len, win_start, win_len, ring_cap, num_splits, scale,
                            alpha_k, alpha_v, rope_base, nullptr, stream);
}

// One decode step of one layer from a context that keeps the layer's addresses: compression event if due, compressed-region
// attention, and the fused tail (mirrored in include/khq_b200.h).
struct khq_layer_ctx {
    const void *d_k, *cents_k, *rotor_k, *d_v, *cents_v, *rotor_v, *vq;
    void *ring_k, *ring_v, *ring_u;
    void *k_mask, *k_payload, *k_norms, *k_r_norms, *v_payload, *v_norms, *v_r_norms, *v_shared_meta;
    void *attn_c, *attn_partial;
    const void* prepared;
    float ts_k, alpha_k, ts_v, alpha_v, rope_base;
    int ring_cap;
};
static_assert(sizeof(khq_layer_ctx) == 21 * 8 + 24, "ABI");
extern "C" int launch_khq_compress_fp16(const void*, const void*, const void*, const void*, const void*, void*, void*, void*, void*,
                                        void*, int, int, float, float, int, cudaStream_t);

// Shape of a step: csize 0, khq_step_kernel, else khq_step_wide_kernel with clusters of csize CTAs; n_comp clusters (per kv-head) on the
// compressed region and blocks of 16 tokens per CTA.  Measured on 148 SMs, a layer of a chain of steps, us:
//     compressed tokens          384   1024   1536   2176   3072   4096   8192  16384  32768  131072
//     one block per CTA          12.0   15.8   18.1   21.4   27.9   29.5   44.0   67.2    114     370
//     wide, 14 clusters of 8     18.9   20.9   21.0   21.6   23.0   23.4   29.3   40.3   59.4     177
//     wide, 31 clusters of 4     19.6   22.1   23.3   22.9   25.1   25.3   31.5   39.5   57.9     165
//     two kernels (before)       20.4   23.4          25.8          29.9   37.5   48.4            209
// The first as long as every CTA has one block and not all of the device is taken: at 2176 tokens (136 blocks, 576 CTAs, four on an SM) it
// is as fast in this chain, but leaves a pre-step between two layers no room to start (30.3 us a layer, 24.3 with the wide
// one; 1792 tokens: 21.3 and 23.9).  Clusters live inside a GPC, so fewer fit on the
// device than SMs / size (measured 15 of 8 and 33 of 4, the occupancy query does not know); one is the window's.
static void step_shape(int c_len, int& csize, int& n_comp, int& per_cta) {
    const int blocks = (c_len + M2_BT - 1) / M2_BT, sms = sm_count();
    const auto at_least = [](int n) { return n < 1 ? 1 : n > ST_MAX_RECORDS - 1 ? ST_MAX_RECORDS - 1 : n; };
    int most = at_least(4 * sms / (HKV * ST_CLUSTER) - 4);
    csize = 0;
    if (blocks > most * ST_CLUSTER) {
        csize = 8;
        most = at_least(sms / 8 - 4);
        if (blocks > 1024) {
            csize = 4;
            most = at_least(sms / 4 - 5);
        }
    }
    const int ctas = csize ? csize : ST_CLUSTER;
    per_cta = (blocks + most * ctas - 1) / (most * ctas);
    n_comp = blocks > 0 ? (blocks + per_cta * ctas - 1) / (per_cta * ctas) : 0;
}

// The compression event of a step, if due: moves the regions on by 128 tokens.
static int layer_event(const khq_layer_ctx* L, int& c_len, int& win_len, int compress, cudaStream_t stream) {
    constexpr int CHUNK = 128;
    if (!compress) return 0;
    // the 128 oldest raw tokens, contiguous in the ring; the step's own token is not among them
    const int s0 = c_len % L->ring_cap, row = c_len * HKV;
    if (win_len <= CHUNK || s0 + CHUNK > L->ring_cap) return -103;
    const auto at = [](void* p, size_t bytes) { return static_cast<void*>(static_cast<char*>(p) + bytes); };
    const size_t src = (size_t)s0 * HKV * D * sizeof(__half);
    // K first: it zeroes the shared meta rows that the V launch then fills
    int rc = launch_khq_compress_fp16(at(L->ring_u, src), L->d_k, L->rotor_k, L->cents_k, L->cents_k, at(L->k_mask, (size_t)row * 64),
                                      at(L->k_norms, (size_t)row * 2), at(L->k_r_norms, (size_t)row * 2),
                                      at(L->k_payload, (size_t)row * K_PAY), at(L->v_shared_meta, (size_t)row * 4), CHUNK * HKV, D,
                                      L->ts_k, L->alpha_k, 0, stream);
    if (rc != 0) return rc;
    rc = launch_khq_compress_fp16(at(L->ring_v, src), L->d_v, L->rotor_v, L->cents_v, L->vq, at(L->k_mask, (size_t)row * 64),
                                  at(L->v_norms, (size_t)row * 2), at(L->v_r_norms, (size_t)row * 2),
                                  at(L->v_payload, (size_t)row * V_PAY), at(L->v_shared_meta, (size_t)row * 4), CHUNK * HKV, D,
                                  L->ts_v, L->alpha_v, 1, stream);
    if (rc != 0) return rc;
    c_len += CHUNK;
    win_len -= CHUNK;
    return 0;
}

extern "C" int launch_khq_layer_step(const khq_layer_ctx* L, const void* q_gate, const void* k_roped, const void* v_new,
                                     const void* k_unroped, void* out, int c_len, int win_len, int compress, int num_splits,
                                     float scale, cudaStream_t stream) {
    if (!L || !q_gate || !out || win_len <= 0 || c_len < 0 || !L->attn_c || !aligned(L->prepared, 128) || (k_roped == nullptr) != (v_new == nullptr)) return -100;
    if (L->ring_cap <= 0 || win_len > L->ring_cap) return -103;
    const int rc = layer_event(L, c_len, win_len, compress, stream);
    if (rc != 0) return rc;
    return decode_step_impl(q_gate, k_roped, v_new, k_unroped, L->ring_k, L->ring_v, L->ring_u, L->k_payload, L->v_payload,
                            L->v_shared_meta, L->k_mask, L->k_norms, L->k_r_norms, L->v_norms, L->v_r_norms, L->cents_k, L->cents_v,
                            L->vq, L->rotor_k, L->rotor_v, L->d_k, L->d_v, L->attn_c, L->attn_partial, out, c_len,
                            c_len % L->ring_cap, win_len, L->ring_cap, num_splits, scale, L->alpha_k, L->alpha_v, L->rope_base, L->prepared, stream);
}

extern "C" int launch_khq_layer_token(const khq_layer_ctx* L, void* counters, const void* q_gate, const void* k_roped, const void* v_new,
                                      const void* k_unroped, void* out, int c_len, int win_len, int compress, float scale,
                                      cudaStream_t stream) {
    if (!L || !counters || !q_gate || !out || win_len <= 0 || c_len < 0 || !L->prepared || !L->attn_partial ||
        (k_roped == nullptr) != (v_new == nullptr))
        return -100;
    if (L->ring_cap <= 0 || win_len > L->ring_cap) return -103;
    const void* al[] = {q_gate, k_roped, v_new, k_unroped, out, L->ring_k, L->ring_v, L->ring_u, L->attn_partial, L->cents_k, L->rotor_k, L->rotor_v, L->d_k, L->d_v};
    for (const void* p : al)
        if (!aligned(p, 16)) return -104;
    if (!aligned(L->prepared, 128) || !aligned(counters, 4)) return -104;
    const void* arrays[] = {L->k_payload, L->v_payload, L->v_shared_meta, L->k_mask, L->k_norms, L->k_r_norms, L->v_norms, L->v_r_norms};
    for (const void* a : arrays)
        if (!aligned(a, 4)) return -104;
    const int rc = layer_event(L, c_len, win_len, compress, stream);
    if (rc != 0) return rc;
    cudaError_t err = ensure_smem_attrs();
    if (err != cudaSuccess) return static_cast<int>(err);
    StepArgs A = {};
    CompressedKV& P = A.kv;
    P.k_payload = static_cast<const unsigned char*>(L->k_payload);
    P.v_payload = static_cast<const unsigned char*>(L->v_payload);
    P.v_shared_meta = static_cast<const unsigned char*>(L->v_shared_meta);
    P.k_mask = static_cast<const unsigned int*>(L->k_mask);
    P.k_norms = static_cast<const __half*>(L->k_norms);
    P.k_r_norms = static_cast<const __half*>(L->k_r_norms);
    P.v_norms = static_cast<const __half*>(L->v_norms);
    P.v_r_norms = static_cast<const __half*>(L->v_r_norms);
    P.cents_k = static_cast<const __half*>(L->cents_k);
    P.k_rotor = static_cast<const __half*>(L->rotor_k);
    P.v_rotor = static_cast<const __half*>(L->rotor_v);
    P.d_k = static_cast<const __half*>(L->d_k);
    P.d_v = static_cast<const __half*>(L->d_v);
    P.alpha_k = L->alpha_k;
    P.alpha_v = L->alpha_v;
    P.rope_base = L->rope_base;
    P.c_len = c_len;
    P.image = static_cast<const unsigned char*>(L->prepared);
    A.q = static_cast<const __half*>(q_gate);
    A.ring_k = static_cast<__half*>(L->ring_k);
    A.ring_v = static_cast<__half*>(L->ring_v);
    A.ring_u = static_cast<__half*>(L->ring_u);
    A.new_k = static_cast<const __half*>(k_roped);
    A.new_v = static_cast<const __half*>(v_new);
    A.new_u = static_cast<const __half*>(k_unroped);
    A.out = static_cast<__half*>(out);
    A.sums = static_cast<float*>(L->attn_partial);
    A.ml = reinterpret_cast<float2*>(A.sums + ST_MAX_RECORDS * HQ * D);
    A.counters = static_cast<int*>(counters);
    A.win_start = c_len % L->ring_cap;
    A.win_len = win_len;
    A.ring_cap = L->ring_cap;
    A.scale = scale;
    P.cents_v = static_cast<const __half*>(L->cents_v);
    P.vq = static_cast<const __half*>(L->vq);
    bool bulk_ok = true;
    for (const void* a : arrays) bulk_ok = bulk_ok && aligned(a, 16);
    P.bulk_ok = bulk_ok ? 1 : 0;
    A.wide = aligned(L->k_mask, 16) && aligned(L->k_payload, 8) && aligned(L->v_payload, 8);
    int csize, n_comp;
    step_shape(c_len, csize, n_comp, A.blocks_per_cta);
    A.n_records = n_comp + 1;
    if (csize == 0)
        err = launch_pdl(khq_step_kernel<false>, (unsigned)(A.n_records * HKV * ST_CLUSTER), (unsigned)ST_CLUSTER, (size_t)ST_SM_TOTAL, stream,
                         (unsigned)ST_THREADS, A, StepBatch{});
    else
        err = launch_pdl(khq_step_wide_kernel<false>, (unsigned)(A.n_records * csize), (unsigned)csize, (size_t)SW_TOTAL, stream, (unsigned)M2_THREADS, A,
                         StepBatch{});
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

// The newest rows of a prompt into the three rings, row by row at slot = token % ring_cap.  Grid (16-byte vectors, 3 rings).  One
// launch instead of up to six copies: short prompts are bound by launches (a 2 KB row per token and ring, 1.5 us).
// It copies beside the kernel before and waits for that at its end only.  launch_khq_layer_prefill puts it directly behind the attention,
// which lets it start when everything before that is complete and shares nothing with it but inputs that both read, or behind the
// compression, which ends before it starts.
__global__ void __launch_bounds__(256)
khq_ring_fill_kernel(const uint4* __restrict__ k_roped, const uint4* __restrict__ v, const uint4* __restrict__ k_unroped,
                     uint4* __restrict__ ring_k, uint4* __restrict__ ring_v, uint4* __restrict__ ring_u, int first, int tokens,
                     int ring_cap) {
    constexpr int ROW = HKV * D / 8;
    pdl_trigger();  // the kernel behind reads nothing but constants before its own wait
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= tokens * ROW) {
        pdl_wait();
        return;
    }
    const int token = first + i / ROW;
    const uint4* src = blockIdx.y == 0 ? k_roped : blockIdx.y == 1 ? v : k_unroped;
    uint4* dst = blockIdx.y == 0 ? ring_k : blockIdx.y == 1 ? ring_v : ring_u;
    dst[(size_t)(token % ring_cap) * ROW + i % ROW] = src[(size_t)token * ROW + i % ROW];
    pdl_wait();
}

extern "C" int launch_khq_gqa_prefill_fp16(const void*, const void*, const void*, void*, int, int, int, int, int, float, long long,
                                           long long, long long, cudaStream_t);

extern "C" int launch_khq_layer_prefill(const khq_layer_ctx* L, const void* q_gate, const void* k_unroped, const void* k_roped,
                                        const void* v, void* out, int T, int n_chunks, float scale, cudaStream_t stream) {
    constexpr int CHUNK = 128;
    if (!L || !q_gate || !k_unroped || !k_roped || !v || !out || T <= 0 || n_chunks < 0 || n_chunks > T / CHUNK) return -100;
    if (L->ring_cap <= 0) return -103;
    if (!aligned(k_unroped, 16) || !aligned(L->ring_k, 16) || !aligned(L->ring_v, 16) || !aligned(L->ring_u, 16)) return -104;
    int rc = launch_khq_gqa_prefill_fp16(q_gate, k_roped, v, out, 1, T, HQ, HKV, D, scale, (long long)T * HQ * 2 * D,
                                         (long long)T * HKV * D, (long long)T * HQ * D, stream);
    if (rc != 0) return rc;
    if (n_chunks > 0) {  // K first: it zeroes the shared meta rows that the V launch then fills
        const int rows = n_chunks * CHUNK * HKV;
        rc = launch_khq_compress_fp16(k_unroped, L->d_k, L->rotor_k, L->cents_k, L->cents_k, L->k_mask, L->k_norms, L->k_r_norms,
                                      L->k_payload, L->v_shared_meta, rows, D, L->ts_k, L->alpha_k, 0, stream);
        if (rc != 0) return rc;
        rc = launch_khq_compress_fp16(v, L->d_v, L->rotor_v, L->cents_v, L->vq, L->k_mask, L->v_norms, L->v_r_norms, L->v_payload,
                                      L->v_shared_meta, rows, D, L->ts_v, L->alpha_v, 1, stream);
        if (rc != 0) return rc;
    }
    const int tokens = T < L->ring_cap ? T : L->ring_cap;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((tokens * (HKV * D / 8) + 255) / 256), 3, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, khq_ring_fill_kernel, static_cast<const uint4*>(k_roped), static_cast<const uint4*>(v),
                                               static_cast<const uint4*>(k_unroped), static_cast<uint4*>(L->ring_k),
                                               static_cast<uint4*>(L->ring_v), static_cast<uint4*>(L->ring_u), T - tokens, tokens,
                                               L->ring_cap);
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

extern "C" int launch_khq_gather_q_fp16(const void* q_gate, void* q_out, int H_q, int d,
                                        cudaStream_t stream) {
    if (H_q <= 0 || d <= 0) return -100;
    const int total = H_q * d, threads = 256;
    khq_gather_q_kernel<<<(total + threads - 1) / threads, threads, 0, stream>>>(
        static_cast<const __half*>(q_gate), static_cast<__half*>(q_out), H_q, d);
    const cudaError_t err = cudaGetLastError();
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

// ------------------------------------------------------------------------------------------
// Batched decode entry points (no counterpart in the reference)
// ------------------------------------------------------------------------------------------
extern "C" size_t khq_b200_decode_workspace_bytes(int n_slots_total) {
    if (n_slots_total < 0) n_slots_total = 0;
    return 256 + (size_t)n_slots_total * HQ * PART * sizeof(float);
}


// SM count for the planner's default item size.  The planner itself makes no CUDA call that can
// fail the plan: when no device is current or the query fails it plans for 148 SMs.
static int plan_sm_count() {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) {
        (void)cudaGetLastError();
        return 148;
    }
    return v;
}

// ---- host planner -----------------------------------------------------------------------------
// The CTAs of the persistent kernels pull items off one counter in array order, so a plan is judged
// by the makespan of list scheduling on `sms` workers, in units of 61 ns (half a compressed token).  Measured on
// launches of 148 equal items: 6.1 us per round of 48 tokens (each of the three groups one block of 16), 3.7 us for a last round
// of one block and 4.9 of two, 9.2 us per item (query set-up, records, their merge); a raw window takes 0.18 us a
// token and 12 us an item when its rows come from HBM.
#include <algorithm>
#include <functional>
#include <queue>
#include <vector>

namespace {
constexpr int PLAN_ROUND = 48;        // compressed tokens
constexpr int PLAN_WINDOW_TOKENS = 3;  // a window is cut so that its pieces stay below a third of a compressed piece, in tokens
long long plan_cost(int kind, int n) {
    if (kind) return 200 + 3LL * n;
    const int r = n % PLAN_ROUND;
    return 150 + 2LL * (n - r) + (r ? 60 + r * 36 / PLAN_ROUND : 0);
}

struct PlanPiece {
    int problem, lo, hi;
};

struct PlanRule {
    int kind;   // 0: guided self-scheduling (cap, floor), windows whole; 1: piece counts per problem (pieces, win_pieces); 2: a list
    int cap, floor_;
    const std::vector<int>* pieces;
    const std::vector<int>* win_pieces;
    const std::vector<PlanPiece>* list = nullptr;
};

// Walks the items of a plan in launch order: fn(problem, kind, lo, hi).
template <class F>
void plan_walk(const PlanRule& rule, const int* c_len, const int* win_len, int n_desc, int sms, F fn) {
    long long remaining = 0;
    for (int i = 0; i < n_desc; ++i) remaining += c_len[i] > 0 ? c_len[i] : 0;
    // every raw window first (they need no tables): the last items of a launch are then small pieces
    for (int i = 0; i < n_desc; ++i) {
        const int wl = win_len[i];
        if (wl <= 0) continue;
        const int wp = rule.win_pieces ? (*rule.win_pieces)[i] : 1;
        const int per = (wl + wp - 1) / wp;
        for (int lo = 0; lo < wl; lo += per) fn(i, 1, lo, lo + per < wl ? lo + per : wl);
    }
    if (rule.kind == 2) {
        for (const PlanPiece& p : *rule.list) fn(p.problem, 0, p.lo, p.hi);
        return;
    }
    for (int i = 0; i < n_desc; ++i) {
        const int cl = c_len[i] > 0 ? c_len[i] : 0;
        if (rule.kind == 0) {
            // tokens_per_item while more than 2 x SMs such items remain in the launch, then
            // remaining / (2 x SMs), down to the floor: the last items handed out are small
            for (int lo = 0; lo < cl;) {
                long long size = remaining / (2LL * sms);
                if (size > rule.cap) size = rule.cap;
                size = (size / rule.floor_) * rule.floor_;
                if (size < rule.floor_) size = rule.floor_;
                const int left = cl - lo;
                if (left < size + rule.floor_ / 2) size = left;  // a short remainder joins the last piece
                fn(i, 0, lo, lo + (int)size);
                lo += (int)size;
                remaining -= size;
            }
        } else if (cl > 0) {
            const int pieces = (*rule.pieces)[i];
            const int per = (((cl + pieces - 1) / pieces) + 1) & ~1;  // equal pieces, each starting on an even token
            for (int lo = 0; lo < cl; lo += per) fn(i, 0, lo, lo + per < cl ? lo + per : cl);
        }
    }
}

long long plan_makespan(const PlanRule& rule, const int* c_len, const int* win_len, int n_desc, int sms) {
    std::priority_queue<long long, std::vector<long long>, std::greater<long long>> free_at;
    for (int w = 0; w < sms; ++w) free_at.push(0);
    long long end = 0;
    plan_walk(rule, c_len, win_len, n_desc, sms, [&](int, int kind, int lo, int hi) {
        const long long t = free_at.top() + plan_cost(kind, hi - lo);
        free_at.pop();
        free_at.push(t);
        if (t > end) end = t;
    });
    return end;
}

// `total` pieces over the problems such that the largest piece is as small as possible (every problem
// with tokens gets one; the next piece always goes to the problem whose pieces are the largest now).
bool plan_even_pieces(const int* c_len, int n_desc, int total, int max_piece, std::vector<int>& pieces) {
    pieces.assign(n_desc, 0);
    std::priority_queue<std::pair<double, int>> largest;
    int used = 0;
    for (int i = 0; i < n_desc; ++i)
        if (c_len[i] > 0) {
            pieces[i] = 1;
            ++used;
            largest.push({(double)c_len[i], i});
        }
    if (used == 0 || used > total) return false;
    for (; used < total; ++used) {
        const int i = largest.top().second;
        if (c_len[i] / (pieces[i] + 1) < 24) break;  // nothing left worth cutting
        largest.pop();
        ++pieces[i];
        largest.push({(double)c_len[i] / pieces[i], i});
    }
    return largest.top().first <= (double)max_piece;
}

// Pieces that fill every worker up to `limit`: the worker that is free first takes as many whole rounds of the problem at hand as fit
// (it is the one the kernel's counter serves next), the rest of the problem goes to the next worker, and a worker that a
// problem's end left with time takes the first piece of a later one.  False: the tokens do not fit.
bool plan_fill(const int* c_len, const int* win_len, const std::vector<int>& win_pieces, int n_desc, int sms, int max_piece, long long limit,
               std::vector<PlanPiece>& list) {
    list.clear();
    std::priority_queue<long long, std::vector<long long>, std::greater<long long>> free_at;
    for (int w = 0; w < sms; ++w) free_at.push(0);
    const PlanRule windows = {2, 0, 0, nullptr, &win_pieces, &list};  // (the list is empty)
    plan_walk(windows, c_len, win_len, n_desc, sms, [&](int, int kind, int lo, int hi) {
        const long long t = free_at.top() + plan_cost(kind, hi - lo);
        free_at.pop();
        free_at.push(t);
    });
    for (int i = 0; i < n_desc; ++i)
        for (int lo = 0, left = c_len[i]; left > 0;) {
            const long long t = free_at.top();
            long long size = (limit - t - plan_cost(0, 0)) / 2 / PLAN_ROUND * PLAN_ROUND;
            if (size > max_piece) size = max_piece / PLAN_ROUND * PLAN_ROUND;
            if (left <= size + PLAN_ROUND / 2) size = left;  // a short rest joins the piece
            else if (size < 2 * PLAN_ROUND) return false;    // not worth an item
            list.push_back({i, lo, lo + (int)size});
            free_at.pop();
            free_at.push(t + plan_cost(0, (int)size));
            lo += (int)size;
            left -= (int)size;
        }
    return true;
}
}  // namespace

// Cuts every problem into one item for its raw window and items of its compressed region.  Candidates: guided self-scheduling with a 96- or a 48-token floor, one, two or three
// waves of equal pieces (a launch small enough that every CTA gets one to three pieces is balanced
// best by exactly that), and pieces that fill every worker; the one with the shortest simulated makespan is written out.
extern "C" int khq_b200_plan_decode(const int* c_len, const int* win_len, int n_desc, int tokens_per_item,
                                    void* items_out, int max_items, int* first_slot, int* n_slots) {
    if (n_desc < 0 || !c_len || !win_len) return -100;
    const int sms = plan_sm_count();
    long long total = 0;
    for (int i = 0; i < n_desc; ++i) total += c_len[i] > 0 ? c_len[i] : 0;
    const bool auto_size = tokens_per_item <= 0;
    if (auto_size) {
        long long t = total / (2LL * sms);  // the guided rule's own first size
        if (t < 48) t = 48;
        if (t > 8192) t = 8192;  // ~1.2 ms of work: an item costs ~12 us whatever its size
        tokens_per_item = (int)t;
    }
    tokens_per_item = ((tokens_per_item + 95) / 96) * 96;  // a multiple of every generation's staging tile (24, 32 tokens)

    std::vector<int> pieces[3], win_pieces[3];
    std::vector<PlanPiece> filled;
    PlanRule best = {0, tokens_per_item, 96, nullptr, nullptr};
    // A launch of many waves is planned by the guided rule as it stands (its tail is a fraction of a percent);
    // smaller ones compare the candidates.
    if (total <= 8LL * sms * tokens_per_item) {
        long long best_t = plan_makespan(best, c_len, win_len, n_desc, sms);
        auto consider = [&](const PlanRule& r) {
            const long long t = plan_makespan(r, c_len, win_len, n_desc, sms);
            if (t < best_t) {
                best_t = t;
                best = r;
            }
        };
        consider(PlanRule{0, tokens_per_item, 48, nullptr, nullptr});
        // an explicit tokens_per_item stays an upper bound on every piece
        const int max_piece = auto_size ? 8256 : tokens_per_item;
        long long work = total;
        for (int i = 0; i < n_desc; ++i) work += (long long)PLAN_WINDOW_TOKENS * (win_len[i] > 0 ? win_len[i] : 0);
        for (int k = 1; k <= 3; ++k) {
            // k items per SM of about work / (k x SMs) each: a raw window that costs more than that is cut too
            const long long target = std::max<long long>(work / ((long long)k * sms), 48);
            std::vector<int>& wp = win_pieces[k - 1];
            wp.assign(n_desc, 0);
            int n_win = 0;
            for (int i = 0; i < n_desc; ++i)
                if (win_len[i] > 0) {
                    long long c = ((long long)PLAN_WINDOW_TOKENS * win_len[i] + target / 2) / target;
                    c = std::min<long long>(std::max<long long>(c, 1), std::max(win_len[i] / 16, 1));
                    wp[i] = (int)c;
                    n_win += (int)c;
                }
            if (plan_even_pieces(c_len, n_desc, k * sms - n_win, max_piece, pieces[k - 1]))
                consider(PlanRule{1, 0, 0, &pieces[k - 1], &wp});
        }
        // Filled workers: some 1.2 items per SM instead of the guided rule's six, or of equal pieces of which the workers that took the
        // windows have one less.  Not for launches whose guided items are at the cap (2 x 8192 tokens per SM, 2 ms): their
        // small last items also even out what the SMs differ by, and cost little there.
        if (total < 2LL * sms * 8192) {
            long long cost = 0;
            plan_walk(PlanRule{2, 0, 0, nullptr, &win_pieces[0], &filled}, c_len, win_len, n_desc, sms,
                      [&](int, int kind, int lo, int hi) { cost += plan_cost(kind, hi - lo); });
            for (int i = 0; i < n_desc; ++i) cost += c_len[i] > 0 ? plan_cost(0, c_len[i]) : 0;
            const long long least = cost / sms + plan_cost(0, 0);
            for (int step = 0; step < 8; ++step)  // 1.5 % more each time
                if (plan_fill(c_len, win_len, win_pieces[0], n_desc, sms, max_piece, least + least * step * 3 / 200, filled)) {
                    consider(PlanRule{2, 0, 0, nullptr, &win_pieces[0], &filled});
                    break;
                }
        }
    }

    // slots are numbered problem by problem (a problem's partial records are contiguous, its window first);
    // the array order is the launch order: all windows, then the pieces in problem order
    std::vector<int> count(n_desc, 0), next(n_desc, 0);
    int n = 0;
    plan_walk(best, c_len, win_len, n_desc, sms, [&](int i, int, int, int) {
        ++count[i];
        ++n;
    });
    for (int i = 0, at = 0; i < n_desc; ++i) {
        next[i] = at;
        if (first_slot) first_slot[i] = at;
        if (n_slots) n_slots[i] = count[i];
        at += count[i];
    }
    KhqWorkItem* items = static_cast<KhqWorkItem*>(items_out);
    int pos = 0;
    plan_walk(best, c_len, win_len, n_desc, sms, [&](int i, int kind, int lo, int hi) {
        if (items && pos < max_items) {
            KhqWorkItem w = {i, kind, lo, hi, next[i], 0, 0, 0};
            items[pos] = w;
        }
        ++next[i];
        ++pos;
    });
    return n;  // > max_items means the items buffer was too small
}

// The counters of a batch's step kernels at the end of its workspace: one per problem and head.
static size_t step_counter_bytes(int n_desc) { return ((size_t)n_desc * HQ * sizeof(int) + 255) / 256 * 256; }

// A small batch as clusters of the step kernels (khq_step.cuh), mirrored in include/khq_b200.h: where every CTA has one block
// (khq_step_kernel), else where the clusters that fit on the device take the compressed regions in one or two rounds of 48 tokens per
// CTA, three for a single sequence; beyond, the persistent kernel's finer items and 148 CTAs win.  Measured per layer of a serving
// chain with its pre-step, us, persistent kernel and merge / this: sequences of compressed tokens 1 x 0: 18.5 / 10.7, 1 x 768: 28.3 /
// 18.4, 2 x 128: 26.6 / 16.7, 12 x ~20: 46.4 / 24.2 (one block); 1 x 2304: 33.4 / 28.7, 3 of 128 to 1536: 33.8 / 29.5, 6 x ~256: 38.4 /
// 32.0 (a round); 6 x ~790: 44.1 / 40.4, 1 x 7680: 42.3 / 38.2 (two); 1 x 15872: 50.5 / 44.5, but 2 x 4736: 41.4 / 43.9 and 4 x ~2500:
// 42.3 / 44.2 (three).  Returns the kernel (5: khq_step_kernel, 6:
// khq_step_wide_kernel) and the number of items, or 0 for a batch that is better off with the items of khq_b200_plan_decode.
extern "C" int khq_b200_plan_steps(const int* c_len, const int* win_len, int n_desc, void* items, int max_items, int* n_items, int* first_slot,
                                   int* n_slots) {
    if (!c_len || !win_len || n_desc <= 0 || !items || !n_items || !first_slot || !n_slots) return -100;
    const int most = plan_sm_count() / 8 - 3;  // clusters of eight CTAs that run side by side; as many sets of four clusters of khq_step_kernel
    for (int i = 0; i < n_desc; ++i)
        if (c_len[i] < 0 || win_len[i] <= 0) return 0;
    int mode = 0, per = 0;
    const auto clusters = [&](int p) {
        int n = 0;
        for (int i = 0; i < n_desc; ++i) {
            const int k = ((c_len[i] + M2_BT - 1) / M2_BT + p * ST_CLUSTER - 1) / (p * ST_CLUSTER);
            if (k + 1 > ST_MAX_RECORDS) return max_items + most + 1;
            n += k + 1;
        }
        return n;
    };
    if (clusters(1) <= most) mode = 5, per = 1;
    for (int p = 3; mode == 0 && p <= (n_desc == 1 ? 9 : 6); p += 3)
        if (clusters(p) <= most) mode = 6, per = p;
    if (mode == 0 || clusters(per) > max_items) return 0;
    KhqWorkItem* w = static_cast<KhqWorkItem*>(items);
    int n = 0;
    for (int i = 0; i < n_desc; ++i) {
        const int blocks = (c_len[i] + M2_BT - 1) / M2_BT, k = (blocks + per * ST_CLUSTER - 1) / (per * ST_CLUSTER);
        first_slot[i] = n;
        n_slots[i] = k + 1;
        for (int j = 0; j <= k; ++j, ++n) w[n] = KhqWorkItem{i, j < k ? 0 : 1, j * per * ST_CLUSTER, per, n, first_slot[i], k + 1, 0};
    }
    *n_items = n;
    return mode;
}

// The item counter of a persistent launch.  A kernel, because a memset between two kernels keeps the launch of the second one from
// overlapping the end of the first.
__global__ void khq_zero_counter_kernel(int* counter) {
    pdl_trigger();
    pdl_wait();
    if (threadIdx.x == 0) *counter = 0;
}

static int decode_batched_impl(const void* descs, const void* tables, const void* items, int n_desc, int n_items,
                               void* workspace, size_t workspace_bytes, int n_slots_total, float scale, float rope_base,
                               int ring_cap, int codebook_in_smem, float* out_partials, const void* images, cudaStream_t stream) {
    if (n_desc <= 0 || n_items <= 0 || !descs || !tables || !items || !workspace) return -100;
    if (workspace_bytes < khq_b200_decode_workspace_bytes(n_slots_total) || ring_cap <= 0) return -105;
    if (!aligned(workspace, 256)) return -104;
    cudaError_t err = ensure_smem_attrs();
    if (err != cudaSuccess) return static_cast<int>(err);
    int* counter = static_cast<int*>(workspace);
    float* partials = reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + 256);
    if (codebook_in_smem == 5 || codebook_in_smem == 6) {  // items of khq_b200_plan_steps
        if (!images || out_partials) return -103;
        const size_t counters = step_counter_bytes(n_desc);
        if (workspace_bytes % 256 != 0 || workspace_bytes < khq_b200_decode_workspace_bytes(n_slots_total) + counters) return -105;
        StepBatch B;
        B.descs = static_cast<const KhqSeqDesc*>(descs);
        B.tables = static_cast<const KhqTablesDesc*>(tables);
        B.images = static_cast<const unsigned char* const*>(images);
        B.items = static_cast<const KhqWorkItem*>(items);
        B.sums = partials;
        B.ml = reinterpret_cast<float2*>(partials + (size_t)n_slots_total * HQ * D);
        B.counters = reinterpret_cast<int*>(static_cast<unsigned char*>(workspace) + workspace_bytes - counters);
        B.scale = scale;
        B.rope_base = rope_base;
        B.ring_cap = ring_cap;
        if (codebook_in_smem == 5)
            err = launch_pdl(khq_step_kernel<true>, (unsigned)(n_items * HKV * ST_CLUSTER), (unsigned)ST_CLUSTER, (size_t)ST_SM_TOTAL, stream,
                             (unsigned)ST_THREADS, StepArgs{}, B);
        else
            err = launch_pdl(khq_step_wide_kernel<true>, (unsigned)(n_items * ST_CLUSTER), (unsigned)ST_CLUSTER, (size_t)SW_TOTAL, stream,
                             (unsigned)M2_THREADS, StepArgs{}, B);
        return (err == cudaSuccess) ? 0 : static_cast<int>(err);
    }
    const int grid = n_items < sm_count() ? n_items : sm_count();
    const bool vqs = codebook_in_smem != 0, mma = codebook_in_smem == 2 || codebook_in_smem < 0;
    if (!mma || n_items > grid) {  // the default kernel takes its first item without the counter
        err = launch_pdl(khq_zero_counter_kernel, 1, 0, 0, stream, 32u, counter);
        if (err != cudaSuccess) return static_cast<int>(err);
    }
    if (codebook_in_smem == 4)
        m3::khq_decode_batched_tc5w_kernel<<<grid, m3::W_THREADS, m3::SM_TOTAL, stream>>>(
            static_cast<const KhqSeqDesc*>(descs), static_cast<const KhqTablesDesc*>(tables),
            static_cast<const KhqWorkItem*>(items), n_items, counter, partials, scale, rope_base, ring_cap);
    else if (codebook_in_smem == 3)
        m3::khq_decode_batched_tc5_kernel<<<grid, m3::THREADS, m3::SM_TOTAL, stream>>>(
            static_cast<const KhqSeqDesc*>(descs), static_cast<const KhqTablesDesc*>(tables),
            static_cast<const KhqWorkItem*>(items), n_items, counter, partials, scale, rope_base, ring_cap);
    else if (mma)
        err = launch_pdl(khq_decode_batched_mma_kernel, (unsigned)grid, 0, (size_t)M2_SM_TOTAL, stream, (unsigned)M2_THREADS,
                         static_cast<const KhqSeqDesc*>(descs), static_cast<const KhqTablesDesc*>(tables),
                         static_cast<const KhqWorkItem*>(items), n_items, counter, partials, scale, rope_base, ring_cap,
                         static_cast<const unsigned char* const*>(images));
    else if (vqs)
        khq_decode_batched_kernel<true><<<grid, DEC_THREADS, SM_TOTAL_VQ, stream>>>(
            static_cast<const KhqSeqDesc*>(descs), static_cast<const KhqTablesDesc*>(tables),
            static_cast<const KhqWorkItem*>(items), n_items, counter, partials, scale, rope_base, ring_cap);
    else
        khq_decode_batched_kernel<false><<<grid, DEC_THREADS, SM_TOTAL, stream>>>(
            static_cast<const KhqSeqDesc*>(descs), static_cast<const KhqTablesDesc*>(tables),
            static_cast<const KhqWorkItem*>(items), n_items, counter, partials, scale, rope_base, ring_cap);
    if (err == cudaSuccess) err = cudaGetLastError();
    if (err != cudaSuccess) return static_cast<int>(err);
    const KhqSeqDesc* dd = static_cast<const KhqSeqDesc*>(descs);
    const bool many = n_items > 32 * n_desc;  // many records per problem
    const unsigned blocks = (unsigned)(n_desc * HQ);
    if (out_partials) {
        if (many) err = launch_pdl(khq_batched_merge_partial_kernel<MERGE_GROUPS>, blocks, 0, 0, stream, MERGE_GROUPS * D, dd, partials, out_partials);
        else err = launch_pdl(khq_batched_merge_partial_kernel<1>, blocks, 0, 0, stream, D, dd, partials, out_partials);
    } else {
        if (many) err = launch_pdl(khq_batched_merge_gate_kernel<MERGE_GROUPS>, blocks, 0, 0, stream, MERGE_GROUPS * D, dd, partials);
        else err = launch_pdl(khq_batched_merge_gate_few_kernel, blocks, 0, 0, stream, D, dd, partials);
    }
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

extern "C" int launch_khq_decode_batched_fp16(const void* descs, const void* tables, const void* items,
                                              int n_desc, int n_items, void* workspace,
                                              size_t workspace_bytes, int n_slots_total, float scale,
                                              float rope_base, int ring_cap, int codebook_in_smem,
                                              cudaStream_t stream) {
    return decode_batched_impl(descs, tables, items, n_desc, n_items, workspace, workspace_bytes, n_slots_total, scale,
                               rope_base, ring_cap, codebook_in_smem, nullptr, nullptr, stream);
}

// The same launch with the tables' images (device array of pointers by table_id, see launch_khq_prepare_tables).
extern "C" int launch_khq_decode_batched_prepared_fp16(const void* descs, const void* tables, const void* images, const void* items,
                                                       int n_desc, int n_items, void* workspace, size_t workspace_bytes,
                                                       int n_slots_total, float scale, float rope_base, int ring_cap,
                                                       int codebook_in_smem, cudaStream_t stream) {
    return decode_batched_impl(descs, tables, items, n_desc, n_items, workspace, workspace_bytes, n_slots_total, scale,
                               rope_base, ring_cap, codebook_in_smem, nullptr, images, stream);
}

extern "C" size_t khq_b200_prepared_bytes(void) { return (M2_IMG_BYTES + 127) / 128 * 128; }

// Orders an image before everything behind it in the stream.  A step's kernels are launched with the programmatic attribute: one
// of them may start before what is in front of its predecessor has completed, and khq_attn_compressed_mma_kernel reads the image
// before its wait.  This kernel starts when the image is complete and visible (an ordinary launch), and as it has no trigger, a
// kernel behind it starts when it has ended, and what is behind that one later still.
__global__ void khq_after_prepare_kernel() {}

// A layer's tables in the form the decode kernels use them, once per layer: see include/khq_b200.h.
extern "C" int launch_khq_prepare_tables(const void* tables_desc, float rope_base, void* image, cudaStream_t stream) {
    if (!tables_desc || !image) return -100;
    const KhqTablesDesc& t = *static_cast<const KhqTablesDesc*>(tables_desc);  // host memory
    const void* ptrs[] = {t.cents_k, t.cents_v, t.vq, t.k_rotor, t.v_rotor, t.d_k, t.d_v};
    for (const void* p : ptrs)
        if (!p || !aligned(p, 16)) return p ? -104 : -100;
    if (!aligned(image, 128)) return -104;
    CompressedKV P = {};
    P.cents_k = t.cents_k;
    P.cents_v = t.cents_v;
    P.vq = t.vq;
    P.k_rotor = t.k_rotor;
    P.d_k = t.d_k;
    P.alpha_k = t.alpha_k;
    P.alpha_v = t.alpha_v;
    P.rope_base = rope_base;
    khq_prepare_tables_kernel<<<1, M2_THREADS, 0, stream>>>(P, static_cast<unsigned char*>(image));
    khq_after_prepare_kernel<<<1, 1, 0, stream>>>();
    return static_cast<int>(cudaGetLastError());
}

// The same launch, ending in one unnormalised record (acc[256], max, sum) per (problem, head) in
// out_partials (n_desc, H_q, 258) fp32 instead of the gated fp16 outputs: the share of a context-parallel
// rank.  Descriptors may carry chunk-cyclic positions (pos_pack; generations 1 and 2).
extern "C" int launch_khq_decode_batched_partial_fp16(const void* descs, const void* tables, const void* items,
                                                      int n_desc, int n_items, void* workspace, size_t workspace_bytes,
                                                      int n_slots_total, float scale, float rope_base, int ring_cap,
                                                      int codebook_in_smem, void* out_partials, cudaStream_t stream) {
    if (!out_partials || !aligned(out_partials, 8)) return out_partials ? -104 : -100;
    return decode_batched_impl(descs, tables, items, n_desc, n_items, workspace, workspace_bytes, n_slots_total, scale,
                               rope_base, ring_cap, codebook_in_smem, static_cast<float*>(out_partials), nullptr, stream);
}

// Per-sequence state of a batch engine that changes every step and is the same for all layers
// (mirrored in include/khq_b200.h).
struct KhqSeqDyn {
    int c_len, start_pos, win_start, win_len, first_slot, n_slots, r0, r1;
};
static_assert(sizeof(KhqSeqDyn) == 32, "ABI");

// descs: layer-major (layer * n_seq + sequence); the pointers stay, the eight ints follow dyn[sequence].
__global__ void khq_update_descs_kernel(khq::KhqSeqDesc* __restrict__ descs, const KhqSeqDyn* __restrict__ dyn, int n_seq,
                                        int n_layers) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n_seq * n_layers) return;
    const KhqSeqDyn d = dyn[idx % n_seq];
    khq::KhqSeqDesc* o = descs + idx;
    o->c_len = d.c_len;
    o->start_pos = d.start_pos;
    o->win_start = d.win_start;
    o->win_len = d.win_len;
    o->first_slot = d.first_slot;
    o->n_slots = d.n_slots;
}

// After a decode step has moved the sequences on (tokens appended, compression events fired), one
// launch rewrites the step-dependent fields of every layer's descriptors from one small table.
extern "C" int launch_khq_update_descs(void* descs, const void* dyn, int n_seq, int n_layers, cudaStream_t stream) {
    if (!descs || !dyn || n_seq <= 0 || n_layers <= 0) return -100;
    const int total = n_seq * n_layers;
    khq_update_descs_kernel<<<(total + 255) / 256, 256, 0, stream>>>(static_cast<khq::KhqSeqDesc*>(descs),
                                                                    static_cast<const KhqSeqDyn*>(dyn), n_seq, n_layers);
    const cudaError_t err = cudaGetLastError();
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

// ------------------------------------------------------------------------------------------
// Compressed-region attention without a caller-supplied partial buffer
// ------------------------------------------------------------------------------------------
// Split partials of launch_khq_attn_static_fp16 live here instead of in a buffer the caller
// allocates: 24 query heads x at most 32 splits x 258 floats = 792 576 bytes, held by every GPU
// that loads the library until the process exits.
constexpr int STATIC_MAX_SPLITS = 32;
static __device__ __align__(256) float g_static_partials[khq::HQ * STATIC_MAX_SPLITS * khq::PART];

// Device address of g_static_partials on the current device.  In host code the array's name is
// only a handle for the runtime, not an address a kernel can use, so the address is looked up
// once per device (with that device current) and cached.
static cudaError_t static_partials_address(float** out) {
    static float* cached[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (cached[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_partials);
        if (e != cudaSuccess) return e;
        cached[dev] = static_cast<float*>(p);
    }
    *out = cached[dev];
    return cudaSuccess;
}

extern "C" int launch_khq_attn_static_fp16(const void* q, const void* k_payload, const void* v_payload,
                                           const void* v_shared_meta, const void* k_mask,
                                           const void* k_norms, const void* k_r_norms, const void* v_norms,
                                           const void* v_r_norms, const void* centroids_k,
                                           const void* centroids_v, const void* vq_centroids,
                                           const void* k_rotor, const void* v_rotor, const void* d_vec_k,
                                           const void* d_vec_v, void* out_attn, int num_queries,
                                           int num_heads, int L_q, int c_len, int n_rep, float scale,
                                           float alpha_k, float alpha_v, float rope_base, int start_pos,
                                           int num_splits, cudaStream_t stream) {
    if (num_queries <= 0 || c_len <= 0) return -100;
    // The static array is sized for one decode query row per head and at most 32 splits.
    if (L_q != 1 || num_queries != khq::HQ || num_splits > STATIC_MAX_SPLITS) return -106;
    float* partials = nullptr;
    const cudaError_t e = static_partials_address(&partials);
    if (e != cudaSuccess) return static_cast<int>(e);
    return launch_khq_attn_fp16(q, k_payload, v_payload, v_shared_meta, k_mask, k_norms, k_r_norms, v_norms,
                                v_r_norms, centroids_k, centroids_v, vq_centroids, k_rotor, v_rotor, d_vec_k,
                                d_vec_v, out_attn, partials, num_queries, num_heads, L_q, c_len, c_len, n_rep,
                                scale, alpha_k, alpha_v, rope_base, start_pos, num_splits, stream);
}

extern "C" int launch_khq_merge_slots_gate_fp16(const void* partials, int n_slots, const void* q_gate,
                                                void* out, int H_q, int d, cudaStream_t stream) {
    if (n_slots <= 0 || !partials || !q_gate || !out) return -100;
    if (H_q != HQ || d != D) return -103;
    khq_merge_slots_gate_kernel<<<HQ, D, 0, stream>>>(static_cast<const float*>(partials), n_slots,
                                                      static_cast<const __half*>(q_gate),
                                                      static_cast<__half*>(out));
    const cudaError_t err = cudaGetLastError();
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

// Kernels of the current device may only dereference another GPU's memory (an IPC mapping is made
// in the exporting device's context) once peer access from the current device to it is enabled.
extern "C" int khq_b200_enable_peer_access(int peer_device) {
    int cur = 0;
    cudaError_t e = cudaGetDevice(&cur);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (peer_device == cur) return 0;
    int can = 0;
    e = cudaDeviceCanAccessPeer(&can, cur, peer_device);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (!can) return -109;
    e = cudaDeviceEnablePeerAccess(peer_device, 0);
    if (e == cudaErrorPeerAccessAlreadyEnabled) {
        (void)cudaGetLastError();
        return 0;
    }
    return (e == cudaSuccess) ? 0 : static_cast<int>(e);
}

// ---- peer-visible buffers (CUDA IPC), for the exchange above -----------------------------------
// khq_b200_peer_alloc: cudaMalloc + zero fill on the current device and the 64-byte IPC handle
// of the allocation.  khq_b200_peer_open: maps another process's allocation for the CURRENT
// device (peer access between the two GPUs is enabled by the open itself).  Both return 0 or a
// positive cudaError_t; -100 for null arguments.
extern "C" int khq_b200_peer_alloc(size_t bytes, void** ptr_out, unsigned char* handle_out) {
    if (!ptr_out || !handle_out || bytes == 0) return -100;
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    e = cudaMemset(p, 0, bytes);
    cudaIpcMemHandle_t h;
    if (e == cudaSuccess) e = cudaIpcGetMemHandle(&h, p);
    if (e != cudaSuccess) {
        cudaFree(p);
        return static_cast<int>(e);
    }
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "IPC handle size");
    memcpy(handle_out, &h, 64);
    *ptr_out = p;
    return 0;
}
extern "C" int khq_b200_peer_open(const unsigned char* handle, void** ptr_out) {
    if (!handle || !ptr_out) return -100;
    cudaIpcMemHandle_t h;
    memcpy(&h, handle, 64);
    void* p = nullptr;
    const cudaError_t e = cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess);
    if (e != cudaSuccess) return static_cast<int>(e);
    *ptr_out = p;
    return 0;
}
extern "C" int khq_b200_peer_close(void* ptr) {
    if (!ptr) return -100;
    const cudaError_t e = cudaIpcCloseMemHandle(ptr);
    return (e == cudaSuccess) ? 0 : static_cast<int>(e);
}
extern "C" int khq_b200_peer_free(void* ptr) {
    if (!ptr) return -100;
    const cudaError_t e = cudaFree(ptr);
    return (e == cudaSuccess) ? 0 : static_cast<int>(e);
}
// Blocking 4-byte writes / reads through the runtime (no kernel): lets a host check a mapping before
// any kernel dereferences it.
extern "C" int khq_b200_peer_poke(void* dst, unsigned int value) {
    const cudaError_t e = cudaMemcpy(dst, &value, 4, cudaMemcpyHostToDevice);
    return (e == cudaSuccess) ? 0 : static_cast<int>(e);
}
extern "C" int khq_b200_peer_peek(const void* src, unsigned int* value_out) {
    if (!value_out) return -100;
    const cudaError_t e = cudaMemcpy(value_out, src, 4, cudaMemcpyDeviceToHost);
    return (e == cudaSuccess) ? 0 : static_cast<int>(e);
}

extern "C" int launch_khq_publish_partials_fp32(const void* src, int n_records, const void* peer_slots,
                                                const void* peer_flags, int world, int rank, int first_slot,
                                                long long parity_offset_records, unsigned int epoch, cudaStream_t stream) {
    if (!src || !peer_slots || !peer_flags || n_records <= 0 || world <= 0 || rank < 0 || rank >= world || first_slot < 0)
        return -100;
    if (!aligned(src, 16)) return -104;
    const long long off = (parity_offset_records + first_slot) * (long long)(HQ * PART);
    khq_publish_partials_kernel<<<(unsigned)world, 256, 0, stream>>>(
        static_cast<const float*>(src), n_records * HQ * PART, static_cast<float* const*>(peer_slots),
        static_cast<unsigned int* const*>(peer_flags), off, rank, epoch);
    const cudaError_t err = cudaGetLastError();
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

extern "C" int launch_khq_publish_bytes(const void* src, size_t bytes, const void* peer_bufs, long long dst_byte_offset,
                                        const void* peer_flags, int flag_index, int world, unsigned int epoch,
                                        cudaStream_t stream) {
    if (!src || !peer_bufs || !peer_flags || bytes == 0 || world <= 0 || flag_index < 0 || dst_byte_offset < 0) return -100;
    if (!aligned(src, 16) || (bytes & 15) != 0 || (dst_byte_offset & 15) != 0) return -104;
    khq_publish_bytes_kernel<<<(unsigned)world, 256, 0, stream>>>(
        static_cast<const uint4*>(src), (int)(bytes / 16), static_cast<unsigned char* const*>(peer_bufs), dst_byte_offset,
        static_cast<unsigned int* const*>(peer_flags), flag_index, epoch);
    const cudaError_t err = cudaGetLastError();
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

extern "C" int launch_khq_wait_flag(const void* flag, unsigned int epoch, unsigned int max_polls, cudaStream_t stream) {
    if (!flag) return -100;
    khq_wait_flag_kernel<<<1, 1, 0, stream>>>(static_cast<const unsigned int*>(flag), epoch, max_polls ? max_polls : (1u << 22));
    const cudaError_t err = cudaGetLastError();
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

extern "C" int launch_khq_merge_slots_wait_gate_fp16(const void* partials, const void* flags, int n_flags,
                                                     unsigned int epoch, int n_slots, const void* q_gate, void* out,
                                                     int H_q, int d, unsigned int max_polls, cudaStream_t stream) {
    if (n_slots <= 0 || n_flags < 0 || n_flags > D || !partials || !flags || !q_gate || !out) return -100;
    if (H_q != HQ || d != D) return -103;
    khq_merge_slots_wait_gate_kernel<<<HQ, D, 0, stream>>>(
        static_cast<const float*>(partials), static_cast<const unsigned int*>(flags), n_flags, epoch, n_slots,
        static_cast<const __half*>(q_gate), static_cast<__half*>(out), max_polls ? max_polls : (1u << 22));
    const cudaError_t err = cudaGetLastError();
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}

// The library keeps process-wide cells (the state slots below, cached symbol addresses, per-device
// attribute caches).  Like the reference library (src/csrc/qmv_sm75_kernel.cu:17-22) it pins itself
// at load time so that a host that dlcloses it between calls finds them again.
#include <dlfcn.h>
__attribute__((constructor)) static void khq_b200_pin_self() {
    Dl_info info;
    if (dladdr(reinterpret_cast<const void*>(&khq_b200_pin_self), &info) && info.dli_fname)
        (void)dlopen(info.dli_fname, RTLD_NOW | RTLD_GLOBAL | RTLD_NODELETE);
}

static void* g_khq_slots[3] = {nullptr, nullptr, nullptr};
extern "C" void* khq_state_slot(int which) {
    if (which < 0 || which > 2) which = 0;
    return static_cast<void*>(&g_khq_slots[which]);
}
extern "C" int bonsai_cuda_sm75_init(void) { return 0; }
extern "C" const char* khq_b200_version(void) { return "khq-b200 0.1 sm_100a"; }
extern "C" int khq_b200_device_status_clear(void) {
    int v = 0;
    cudaError_t err = cudaMemcpyFromSymbol(&v, khq::g_status, sizeof(int));
    if (err != cudaSuccess) return -static_cast<int>(err);
    const int zero = 0;
    err = cudaMemcpyToSymbol(khq::g_status, &zero, sizeof(int));
    return (err == cudaSuccess) ? v : -static_cast<int>(err);
}
extern "C" int khq_b200_device_status(void) {
    int v = 0;
    const cudaError_t err = cudaMemcpyFromSymbol(&v, khq::g_status, sizeof(int));
    return (err == cudaSuccess) ? v : -static_cast<int>(err);
}
