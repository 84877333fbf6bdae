// khq_step.cuh -- one decode step of one (sequence, layer) as one kernel: ring appends, compressed region, raw window, merge and
// gate.  Included by khq_decode.cu.
//
// A step of a short context is a chain of latencies, not work: through the throughput kernel (a warp decodes 16 tokens of a
// kv-head from code words to V sums, ~2100 instructions) and a window kernel behind it, a layer with 384 + 128 tokens took 20.4 us:
// 1.3 to start, 2.7 query build, 7.5 for the one block that a warp gets, 4.6 records and their merge, 4.6 for the kernel
// boundary and the merge of both regions.  12.0 us so:
//   * khq_step_kernel: a CTA is four warps that share blocks of 16 tokens of one kv-head.  K side: warp w decodes mask words 4t + w (its
//     four k-steps), the rotor tiles 2w and 2w + 1 meet in shared memory, warp w finishes the rotary pairs of tiles w and w + 4, and
//     the partial scores are added up; every warp then has all weights and takes patches 8g + 2w, 8g + 2w + 1 of V.  Query
//     fragments (four k-steps) and V sums of a warp fit its registers: no tensor memory.
//   * A cluster's CTAs push each head's sums into the shared memory of the CTA that owns the head (bulk copies that count on
//     the owner's barrier: 0.7 us; pulled by loads, 24 records took 9 us), which merges them and, for the compressed region,
//     applies the inverse V transform.
//   * The raw window is one more cluster per kv-head of the same grid: Q K^T on mma.sync, weights and P V in fp32 (st_window has the reason).
//   * No second kernel: the clusters' records go to global memory, and for each head the warp that arrives last (a counter per
//     head) merges them, divides and gates.  No block ever waits for another cluster.
// khq_step_wide_kernel is the same around the throughput kernel's CTA, for contexts where a 16-token block per CTA would take
// several rounds (step_shape has the line and both sides).  Where its 18 us of a short context go (384 + 128 tokens): 1.6 start, 3.5
// query build, 6.7 the block, 2.2 records and their merge in the CTA, 1 push, 0.8 merge, 1.4 counter, 1.6 the last merge.
#pragma once

namespace khq {

constexpr int ST_PARTS = 4;                     // warps of a CTA: they share a block of 16 tokens of one kv-head
constexpr int ST_THREADS = 32 * ST_PARTS;
constexpr int ST_CLUSTER = 8;                   // CTAs that split the tokens of a kv-head; the first NREP of them own a head each
constexpr int ST_MAX_RECORDS = 32;              // records per head
constexpr int ST_REC = D + 28;                  // a head's sums, four floats of padding after every 32 (bank conflicts)
constexpr int ST_RECV = ST_REC + 8;             // ... its maximum and sum of weights, and padding

// Shared memory of khq_step_kernel.  A staged block: mask words, K payload and V payload of 16 rows.
constexpr int ST_KPAY = M2_BT * 64, ST_VPAY = ST_KPAY + M2_BT * K_PAY;
constexpr int ST_STAGE = ST_VPAY + M2_BT * V_PAY + 128;       // a decode reads up to 34 words from a K payload row on
constexpr int ST_SM_X = 2 * ST_STAGE;                         // exchange: rotor tiles [8][32] float4, partial scores [4][32] float4
constexpr int ST_X_BYTES = (8 + ST_PARTS) * 32 * 16;
constexpr int ST_SM_SMALL = ST_SM_X + ST_X_BYTES;             // the image's small tables
constexpr int ST_SM_ROT = ST_SM_SMALL + M2_SMALL_BYTES;       // rotor fragments: [hi | lo][k-step][lane] of 16 bytes
constexpr int ST_SM_RSC = ST_SM_ROT + 16 * 32 * 32;           // per parity of the block: 16 rows x 2 float4
constexpr int ST_SM_RSTEP = ST_SM_RSC + 2 * 16 * 32;          // cos / sin of 16 positions of each rotary pair
constexpr int ST_SM_RECV = ST_SM_RSTEP + 256;                 // the owned head's records of the cluster's CTAs
constexpr int ST_SM_BAR = ST_SM_RECV + ST_CLUSTER * ST_RECV * 4;
constexpr int ST_SM_ARGS = ST_SM_BAR + 16;  // of a batch
constexpr int ST_SM_TOTAL = ST_SM_ARGS + 320;
constexpr int ST_SM_SEND = 0;                                 // the CTA's records, behind the last block
static_assert(ST_X_BYTES == NREP * D * 4, "the query build's scratch aliases the exchange buffers");
static_assert(NREP * ST_RECV * 4 <= ST_SM_SMALL, "the records alias the stages and exchange buffers");
static_assert(ST_STAGE % 16 == 0 && ST_KPAY % 16 == 0 && ST_VPAY % 16 == 0 && ST_SM_X % 16 == 0 && ST_SM_RECV % 16 == 0 && ST_SM_BAR % 8 == 0 &&
                  (ST_RECV * 4) % 16 == 0, "alignment");

struct StepArgs {
    CompressedKV kv;  // with an image
    const __half* q;  // (24, 512): query and gate
    __half *ring_k, *ring_v, *ring_u;
    const __half *new_k, *new_v, *new_u;  // the step's token; new_k == nullptr: it is in the rings already
    __half* out;
    float* sums;      // (records, 24, 256)
    float2* ml;       // (records, 24): maximum, sum of weights
    int* counters;    // 24, zero before and after a launch
    int win_start, win_len, ring_cap;
    int n_records;    // clusters (of khq_step_kernel: per kv-head)
    int rec;          // a batch: this cluster's record; otherwise record 0 .. n_records - 2 are the compressed region's clusters
    int comp;         // a batch: whether that is the compressed region's
    int block0;       // a batch: the cluster's first block of 16 tokens
    int blocks_per_cta;
    int wide;         // masks on 16 bytes, payloads on 8
    float scale;
};
constexpr int ST_ARGS_BYTES = 320;
static_assert(sizeof(StepArgs) <= ST_ARGS_BYTES && sizeof(StepArgs) % 8 == 0, "shared memory of a batch");
// A batch (khq_b200_plan_steps): item i is cluster i (of khq_step_kernel: clusters 4i .. 4i + 3, one per kv-head).
struct StepBatch {
    const KhqSeqDesc* descs;  // all with the same tables
    const KhqTablesDesc* tables;
    const unsigned char* const* images;
    const KhqWorkItem* items;  // kind 0 / 1, lo: first block, hi: blocks per CTA, slot: record, r0: the problem's first one, r1: its number
    float* sums;
    float2* ml;
    int* counters;  // (problems, 24)
    float scale, rope_base;
    int ring_cap;
};
// The layer's constants, which may be read ahead of the kernel's wait, and the item.
__device__ __forceinline__ void st_fill_constants(StepArgs& A, const StepBatch& B) {
    const int id = B.descs[0].table_id;
    const KhqTablesDesc& t = B.tables[id];
    A.kv.cents_k = t.cents_k; A.kv.cents_v = t.cents_v; A.kv.vq = t.vq; A.kv.k_rotor = t.k_rotor;
    A.kv.v_rotor = t.v_rotor; A.kv.d_k = t.d_k; A.kv.d_v = t.d_v;
    A.kv.alpha_k = t.alpha_k; A.kv.alpha_v = t.alpha_v; A.kv.rope_base = B.rope_base;
    A.kv.image = B.images[id];
}
__device__ __forceinline__ void st_fill_item(StepArgs& A, const StepBatch& B, int item) {
    const KhqWorkItem w = B.items[item];
    const KhqSeqDesc& d = B.descs[w.desc];
    A.kv.k_payload = d.k_payload; A.kv.v_payload = d.v_payload; A.kv.v_shared_meta = d.v_shared_meta;
    A.kv.k_mask = d.k_mask; A.kv.k_norms = d.k_norms; A.kv.k_r_norms = d.k_r_norms;
    A.kv.v_norms = d.v_norms; A.kv.v_r_norms = d.v_r_norms;
    A.kv.start_pos = d.start_pos; A.kv.c_len = d.c_len;
    const auto off = [](const void* p) { return (uint32_t)reinterpret_cast<uintptr_t>(p); };
    A.kv.bulk_ok = ((off(d.k_payload) | off(d.v_payload) | off(d.v_shared_meta) | off(d.k_mask) | off(d.k_norms) | off(d.k_r_norms) |
                     off(d.v_norms) | off(d.v_r_norms)) & 15u) == 0u;
    A.wide = (off(d.k_mask) & 15u) == 0u && ((off(d.k_payload) | off(d.v_payload)) & 7u) == 0u;
    unpack_pos(d.pos_pack, A.kv);
    A.q = d.q_gate;
    A.ring_k = const_cast<__half*>(d.ring_k);
    A.ring_v = const_cast<__half*>(d.ring_v);
    A.ring_u = nullptr;
    A.new_k = A.new_v = A.new_u = nullptr;
    A.out = d.out;
    A.sums = B.sums + (size_t)w.r0 * HQ * D;
    A.ml = B.ml + (size_t)w.r0 * HQ;
    A.counters = B.counters + w.desc * HQ;
    A.win_start = d.win_start;
    A.win_len = d.win_len;
    A.ring_cap = B.ring_cap;
    A.n_records = w.r1;
    A.rec = w.slot - w.r0;
    A.comp = w.kind == 0;
    A.block0 = w.lo;
    A.blocks_per_cta = w.hi;
    A.scale = B.scale;
}

__device__ __forceinline__ void st_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// The address of `p` (own shared memory) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t st_map(const void* p, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
// Own shared memory to a CTA of the cluster; its barrier counts the bytes.
__device__ __forceinline__ void st_push(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(smem_u32(src)),
                 "r"(bytes), "r"(bar)
                 : "memory");
}
template <int BYTES>
__device__ __forceinline__ void st_copy(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}
// ---- staging: the rows of `n` tokens from tok0 of kv-head kvh (asynchronous copies) ------------------------------------------
struct StepScalars {  // of row lane & 15
    uint16_t kn, krn, vn, vrn;
    float vsm;
};
template <int BYTES, int ROW>
__device__ __forceinline__ void st_copy_rows(unsigned char* dst, const unsigned char* src, size_t r0, int n, int tid) {
    constexpr int PER = ROW / BYTES;
    for (int c = tid; c < n * PER; c += ST_THREADS) st_copy<BYTES>(dst + c * BYTES, src + (r0 + (size_t)(c / PER) * HKV) * ROW + (c % PER) * BYTES);
}
__device__ __forceinline__ void st_stage(const CompressedKV& P, unsigned char* stage, int tok0, int n, int kvh, bool wide, int tid, StepScalars& sc) {
    const size_t r0 = (size_t)tok0 * HKV + kvh;
    const unsigned char* mask = reinterpret_cast<const unsigned char*>(P.k_mask);
    if (wide) {
        st_copy_rows<16, 64>(stage, mask, r0, n, tid);
        st_copy_rows<8, K_PAY>(stage + ST_KPAY, P.k_payload, r0, n, tid);
        st_copy_rows<8, V_PAY>(stage + ST_VPAY, P.v_payload, r0, n, tid);
    } else {
        st_copy_rows<4, 64>(stage, mask, r0, n, tid);
        st_copy_rows<4, K_PAY>(stage + ST_KPAY, P.k_payload, r0, n, tid);
        st_copy_rows<4, V_PAY>(stage + ST_VPAY, P.v_payload, r0, n, tid);
    }
    const size_t r = r0 + (size_t)min(tid & 15, n - 1) * HKV;
    sc.kn = reinterpret_cast<const uint16_t*>(P.k_norms)[r];
    sc.krn = reinterpret_cast<const uint16_t*>(P.k_r_norms)[r];
    sc.vn = reinterpret_cast<const uint16_t*>(P.v_norms)[r];
    sc.vrn = reinterpret_cast<const uint16_t*>(P.v_r_norms)[r];
    sc.vsm = reinterpret_cast<const float*>(P.v_shared_meta)[r];
}

// ---- query side: fragments of the warp's four k-steps (q1.x, q1.y, q2.x, q2.y, then their low-order halves) ------------
struct StepQueryTables {  // constants of the model
    uint4 rotor[4], d;
    uint2 cents[4];
    __device__ __forceinline__ void load(const CompressedKV& P, int part, int lane) {
        const int g = lane >> 2, t = lane & 3;
        const uint4* rp = reinterpret_cast<const uint4*>(P.k_rotor + lane * 32);
#pragma unroll
        for (int i = 0; i < 4; ++i) rotor[i] = rp[i];
        d = *reinterpret_cast<const uint4*>(P.d_k + lane * 8);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            cents[i] = g < NREP ? *reinterpret_cast<const uint2*>(P.cents_k + 2 * D + 64 * t + 4 * (4 * part + i)) : make_uint2(0u, 0u);
    }
};

__device__ __forceinline__ void st_load_query(uint4 (&qraw)[2], uint32_t (&qr)[2], const __half* __restrict__ q, int kvh, int part, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int i = 0; i < 2; ++i)  // heads part and part + 4
        if (i == 0 || part < NREP - 4) qraw[i] = *reinterpret_cast<const uint4*>(q + (size_t)(kvh * NREP + part + 4 * i) * 2 * D + lane * 8);
    {  // raw rotary query: dims 8 part + 2t, + 1 and 32 dims on
        const __half* qh = q + (size_t)(kvh * NREP + (g < NREP ? g : 0)) * 2 * D + 8 * part + 2 * t;
        qr[0] = g < NREP ? *reinterpret_cast<const uint32_t*>(qh) : 0u;
        qr[1] = g < NREP ? *reinterpret_cast<const uint32_t*>(qh + 32) : 0u;
    }
}
__device__ __forceinline__ void st_build_query(uint32_t (&qf)[4][8], const uint4 (&qraw)[2], const StepQueryTables& qt, int part, int lane,
                                               float* scratch) {
    const int g = lane >> 2, t = lane & 3;
    float dv[8];
    const __half* hd = reinterpret_cast<const __half*>(&qt.d);
    const __half* hr = reinterpret_cast<const __half*>(qt.rotor);
#pragma unroll
    for (int j = 0; j < 8; ++j) dv[j] = (lane >= 8) ? __fdividef(1.0f / 256.0f, __half2float(hd[j]) + 1e-8f) : 0.0f;
    // q~ = R^T H256 (q * dinv * [dim >= 64])
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (i == 1 && part >= NREP - 4) break;
        const int h = part + 4 * i;
        const __half* hq = reinterpret_cast<const __half*>(&qraw[i]);
        float x[8], y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = __half2float(hq[j]) * dv[j];
        fwht256_lane8(x, lane);
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float a = 0.0f;
#pragma unroll
                for (int c = 0; c < 4; ++c) a = fmaf(__half2float(hr[p * 16 + c * 4 + r]), x[p * 4 + c], a);
                y[p * 4 + r] = a;
            }
        *reinterpret_cast<float4*>(scratch + h * D + m2_q_chunk(h, 2 * lane)) = make_float4(y[0], y[1], y[2], y[3]);
        *reinterpret_cast<float4*>(scratch + h * D + m2_q_chunk(h, 2 * lane + 1)) = make_float4(y[4], y[5], y[6], y[7]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f}, c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (g < NREP) {
            const float4 qq = *reinterpret_cast<const float4*>(scratch + g * D + m2_q_chunk(g, 16 * t + 4 * part + i));
            const __half* hc = reinterpret_cast<const __half*>(&qt.cents[i]);
            v[0] = qq.x; v[1] = qq.z; v[2] = qq.y; v[3] = qq.w;  // dims 64t + 4s + {0, 2, 1, 3}
            c[0] = __half2float(hc[0]); c[1] = __half2float(hc[2]); c[2] = __half2float(hc[1]); c[3] = __half2float(hc[3]);
        }
        m2_pack_hilo(v[0] * c[0], v[1] * c[1], qf[i][0], qf[i][4]);
        m2_pack_hilo(v[2] * c[2], v[3] * c[3], qf[i][1], qf[i][5]);
        m2_pack_hilo(v[0], v[1], qf[i][2], qf[i][6]);
        m2_pack_hilo(v[2], v[3], qf[i][3], qf[i][7]);
    }
    __syncthreads();  // the exchange buffers alias the scratch
}

// ---- K side of a block: the warp's mask word of rows g and g + 8, all quarters --------------------------------------------
struct StepWord {
    uint32_t word, first, cnt;  // ordinal of its first outlier in the row, number of outliers
    const uint32_t* kp;
};
struct StepKSums {
    float cs[4], cs2[4], cu[2][4];
};
__device__ __forceinline__ bool st_open(StepWord (&sw)[2], const unsigned char* __restrict__ S, int part, int lane, int valid_hi) {
    const int g = lane >> 2, t = lane & 3;
    bool odd = false;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int row = g + 8 * x;
        sw[x].kp = reinterpret_cast<const uint32_t*>(S + ST_KPAY + row * K_PAY);
        uint4 m = *reinterpret_cast<const uint4*>(S + row * 64 + 16 * t);
        if (g + 8 * x >= valid_hi) m = make_uint4(0u, 0u, 0u, 0u);
        const uint32_t b0 = m.x & (m.x >> 1) & 0x55555555u, b1 = m.y & (m.y >> 1) & 0x55555555u, b2 = m.z & (m.z >> 1) & 0x55555555u,
                       b3 = m.w & (m.w >> 1) & 0x55555555u;
        const uint32_t n01 = __popc(b0 | (b1 << 1)), total = n01 + __popc(b2 | (b3 << 1));
        uint32_t incl = total;
        uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, 1);
        if (t >= 1) incl += up;
        up = __shfl_up_sync(0xFFFFFFFFu, incl, 2);
        if (t >= 2) incl += up;
        const uint32_t even = __popc(part < 2 ? b0 : b2), own = part == 0 ? b0 : part == 1 ? b1 : part == 2 ? b2 : b3;
        sw[x].word = part == 0 ? m.x : part == 1 ? m.y : part == 2 ? m.z : m.w;
        sw[x].first = incl - total + (part >= 2 ? n01 : 0u) + ((part & 1) ? even : 0u);
        sw[x].cnt = __popc(own);
        odd = odd || sw[x].cnt > 8u || sw[x].first + sw[x].cnt > (uint32_t)MAX_OUT;
    }
    return odd;
}
template <bool ANY>
__device__ __forceinline__ void st_word(const StepWord& sw, uint32_t (&t2)[8], uint32_t (&c2)[8]) {
    if (ANY && (sw.cnt > 8u || sw.first + sw.cnt > (uint32_t)MAX_OUT)) {
        khq3::kq_word_slow(sw.word, sw.first, sw.kp, t2, c2);
        return;
    }
    khq3::KQuarter q;
    const uint32_t* c = sw.kp + 1 + (sw.first >> 3);
    q.c0 = khq3::k3_funnel_r(c[0], c[1], (4u * sw.first) & 31u);
    const uint32_t sb = 232u + sw.first;
    q.neg = ~khq3::k3_funnel_r(sw.kp[sb >> 5], sw.kp[(sb >> 5) + 1u], sb & 31u);
    q.c1 = q.c2 = 0u;
    khq3::kq_word(q, sw.word, sw.cnt, t2, c2);
}
template <bool ANY>
__device__ __forceinline__ void st_k_part(const StepWord (&sw)[2], const uint32_t (&qf)[4][8], const uint4* __restrict__ rot,
                                          const float (&ratio)[2], StepKSums& ks) {
    uint32_t ta[8], xa[8], tb[8], xb[8];
    st_word<ANY>(sw[0], ta, xa);
    st_word<ANY>(sw[1], tb, xb);
    if (ANY) __syncwarp();
    float cur[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint32_t a1[4] = {ta[q], tb[q], ta[4 + q], tb[4 + q]};
        const uint32_t ax[4] = {xa[q], xb[q], xa[4 + q], xb[4 + q]};
        const uint4 rh = rot[32 * q], rl = rot[16 * 32 + 32 * q];
        if (q == 0) {
            m2_mma0(ks.cs, a1, qf[q][0], qf[q][1]);
            m2_mma0(ks.cs2, ax, qf[q][2], qf[q][3]);
        } else {
            m2_mma(ks.cs, a1, qf[q][0], qf[q][1]);
            m2_mma(ks.cs2, ax, qf[q][2], qf[q][3]);
        }
        float (&cu)[4] = ks.cu[q >> 1];
        if ((q & 1) == 0) {
            m2_mma0(cu, a1, rh.x, rh.y);
            m2_mma0(cur, ax, rh.z, rh.w);
        } else {
            m2_mma(cu, a1, rh.x, rh.y);
            m2_mma(cur, ax, rh.z, rh.w);
        }
        m2_mma_lo(ks.cs, a1, qf[q][4], qf[q][5]);
        m2_mma_lo(ks.cs2, ax, qf[q][6], qf[q][7]);
        m2_mma_lo(cu, a1, rl.x, rl.y);
        m2_mma_lo(cur, ax, rl.z, rl.w);
        if (q & 1) {
            m2_fma2(cu[0], cu[1], ratio[0], ratio[0], cur[0], cur[1], cu[0], cu[1]);
            m2_fma2(cu[2], cu[3], ratio[1], ratio[1], cur[2], cur[3], cu[2], cu[3]);
        }
    }
}
struct StepFragments {
    uint32_t qf[4][8];
};
// Words with more than eight outliers, rows past the format's 50: out of line (see m2_k_gemm_odd).
__device__ __noinline__ void st_k_part_odd(const StepWord& w0, const StepWord& w1, const StepFragments& f, const uint4* rot, float ratio0,
                                           float ratio1, StepKSums& out) {
    const StepWord sw[2] = {w0, w1};
    const StepFragments fr = f;
    const float ratio[2] = {ratio0, ratio1};
    StepKSums ks;
    st_k_part<true>(sw, fr.qf, rot, ratio, ks);
    out = ks;
}

// Running state of a warp: thread (g, t) holds heads 2t, 2t + 1.  The four warps of a kv-head hold the same weights state and
// their own dims of the V sums (o: see M2State).
struct StepState {
    float o[5][4];
    float m[2], l[2], p2[2], top[2];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) o[i][j] = 0.0f;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            m[e] = top[e] = NEG_BIG;
            l[e] = p2[e] = 0.0f;
        }
    }
};
// Weights of a block from its scores (rows g and g + 8, heads 2t and 2t + 1); the sums follow the reference (see M2_SLACK).
template <int N>
__device__ __forceinline__ void st_weights(StepState& st, const float (&sc)[2][2], const bool (&valid)[2], float slack, float (&pw)[2][2]) {
    bool raise = false;
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            st.top[e] = fmaxf(st.top[e], sc[x][e]);
            raise = raise || sc[x][e] > st.m[e] + slack;
        }
    if (__any_sync(0xFFFFFFFFu, raise)) {
        float corr[2];
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
#pragma unroll
        for (int i = 0; i < N; ++i) {
            st.o[i][0] *= corr[0];
            st.o[i][1] *= corr[1];
            st.o[i][2] *= corr[0];
            st.o[i][3] *= corr[1];
        }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        pw[0][e] = valid[0] ? __expf(sc[0][e] - st.m[e]) : 0.0f;
        pw[1][e] = valid[1] ? __expf(sc[1][e] - st.m[e]) : 0.0f;
        st.l[e] += pw[0][e] + pw[1][e];
    }
}

// Cosines and sines of a thread's rotary pairs 8 part + 2t, + 1 at the positions of rows g and g + 8: cos, cos, sin, sin.
__device__ __forceinline__ void st_rope_seed(float4 (&rope)[2], const CompressedKV& P, const float* freq, int part, int lane, int tok0) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        float c[2], s[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            double th = (double)token_pos(P, tok0 + g + 8 * x) * (double)freq[8 * part + 2 * t + e];
            th -= rint(th * 0.15915494309189535) * 6.283185307179586;
            __sincosf((float)th, &s[e], &c[e]);
        }
        rope[x] = make_float4(c[0], c[1], s[0], s[1]);
    }
}

// One staged block of 16 tokens.
__device__ __forceinline__ void st_block(const unsigned char* __restrict__ S, unsigned char* __restrict__ smem, const float4 (&rope)[2], int part,
                                         int lane, int valid_hi, int parity, const StepFragments& f, const uint32_t (&qr)[2], const CompressedKV& P,
                                         float scale, const StepScalars& row_sc, StepState& st) {
    const int g = lane >> 2, t = lane & 3;
    float4* rsc = reinterpret_cast<float4*>(smem + ST_SM_RSC) + parity * 32;
    float4* xt = reinterpret_cast<float4*>(smem + ST_SM_X);
    float4* xs = xt + 8 * 32;
    const uint4* rot = reinterpret_cast<const uint4*>(smem + ST_SM_ROT) + 4 * part * 32 + lane;
    // this warp's V codes, two patches of four tokens; their codebook entries come from L2 while the K side runs (the codebook in shared
    // memory would leave room for one CTA per SM, and none for the next layer's)
    uint32_t f24[4];
    uint2 ent[2][4];  // (d0, d1), (d2, -)
    {
        const unsigned char* vq = P.image + M2_IMG_VQ8 + (8 * g + 2 * part) * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const unsigned char* row = S + ST_VPAY + (2 * t + (i & 1) + 8 * (i >> 1)) * V_PAY;
            const uint32_t* w = reinterpret_cast<const uint32_t*>(row) + 3 * g + (3 * part >> 2);
            f24[i] = __funnelshift_r(w[0], w[1], 8 * (3 * part & 3));
            const uint32_t hb = ((uint32_t)row[96 + g] >> (2 * part)) << 7;  // bits 7 and 8: the pair's high code bits
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t code = ((u ? f24[i] >> 12 : f24[i]) & 0x7Fu) | ((u ? hb >> 1 : hb) & 0x80u);
                ent[u][i] = __ldg(reinterpret_cast<const uint2*>(vq + code * (NP * 8) + 8 * u));
            }
        }
    }
    StepWord sw[2];
    const bool odd = st_open(sw, S, part, lane, valid_hi);
    float ratio[2];
    {  // a row's scalars: every warp needs the ratio; warp 0 leaves the score scales, warp 1 the V scales
        const int r16 = lane & 15;
        float mult = (float)*reinterpret_cast<const uint32_t*>(S + ST_KPAY + r16 * K_PAY) / 1000.0f;
        if (mult < 0.1f || mult > 10.0f || isnan(mult)) mult = 1.0f;
        const float rs = 16777216.0f * hbits2f(row_sc.krn);
        const float rr = rs / mult;
        ratio[0] = __shfl_sync(0xFFFFFFFFu, rr, g);
        ratio[1] = __shfl_sync(0xFFFFFFFFu, rr, g + 8);
        if (lane < 16) {
            const bool in = r16 < valid_hi;
            if (part == 0) {
                const float kn = P.alpha_k * scale * hbits2f(row_sc.kn);
                rsc[2 * r16] = make_float4(kn * mult, kn * rs, 0.0f, 0.0f);
            } else if (part == 1) {
                const float vn = hbits2f(row_sc.vn), en = hbits2f(row_sc.vrn);
                const float s1 = P.alpha_v * vn * en, s3 = row_sc.vsm * vn * (1.0f / 7.0f);
                const bool large = in && !(fmaxf(fmaxf(fabsf(s1), fabsf(s3)), vn) < M2_SLACK_SCALES);
                rsc[2 * r16 + 1] = in ? make_float4(s1, vn, s3, large ? 1.0f : 0.0f) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
    }
    StepKSums ks;
    if (!__any_sync(0xFFFFFFFFu, odd)) {
        st_k_part<false>(sw, f.qf, rot, ratio, ks);
    } else {
        const StepWord s0 = sw[0], s1 = sw[1];
        const StepFragments fm = f;
        StepKSums ksm;
        st_k_part_odd(s0, s1, fm, rot, ratio[0], ratio[1], ksm);
        ks = ksm;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) xt[(2 * part + i) * 32 + lane] = make_float4(ks.cu[i][0], ks.cu[i][1], ks.cu[i][2], ks.cu[i][3]);
    __syncthreads();
    // ---- rotary part: rest of H64 for tiles part and part + 4, /d, rotation, dot with the raw query ----
    float sc4[4];
    {
        const float* dinv = reinterpret_cast<const float*>(smem + ST_SM_SMALL) + (M2_SM_DINV - M2_SM_FREQ) / 4 + 8 * part + 2 * t;
        const float2 dlo = *reinterpret_cast<const float2*>(dinv), dhi = *reinterpret_cast<const float2*>(dinv + 32);
        const float s1 = (part & 1) ? -1.0f : 1.0f, s2 = (part & 2) ? -1.0f : 1.0f, s3 = s1 * s2;
        float a[4], b[4];
        const auto fold = [&](int j0, float (&r)[4]) {
            const float4 v0 = xt[j0 * 32 + lane], v1 = xt[(j0 + 1) * 32 + lane], v2 = xt[(j0 + 2) * 32 + lane], v3 = xt[(j0 + 3) * 32 + lane];
            m2_fma2(r[0], r[1], v1.x, v1.y, s1, s1, v0.x, v0.y);
            m2_fma2(r[2], r[3], v1.z, v1.w, s1, s1, v0.z, v0.w);
            m2_fma2(r[0], r[1], v2.x, v2.y, s2, s2, r[0], r[1]);
            m2_fma2(r[2], r[3], v2.z, v2.w, s2, s2, r[2], r[3]);
            m2_fma2(r[0], r[1], v3.x, v3.y, s3, s3, r[0], r[1]);
            m2_fma2(r[2], r[3], v3.z, v3.w, s3, s3, r[2], r[3]);
        };
        fold(0, a);
        fold(4, b);
        float lo[4], hi[4];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const float4 rc = rope[x];
            float z0, z1, w0, w1, u0, u1;
            m2_add2(z0, z1, a[2 * x], a[2 * x + 1], b[2 * x], b[2 * x + 1]);
            m2_sub2(w0, w1, a[2 * x], a[2 * x + 1], b[2 * x], b[2 * x + 1]);
            m2_mul2(z0, z1, z0, z1, dlo.x, dlo.y);
            m2_mul2(w0, w1, w0, w1, dhi.x, dhi.y);
            m2_mul2(u0, u1, w0, w1, -rc.z, -rc.w);
            m2_fma2(lo[2 * x], lo[2 * x + 1], z0, z1, rc.x, rc.y, u0, u1);
            m2_mul2(u0, u1, w0, w1, rc.x, rc.y);
            m2_fma2(hi[2 * x], hi[2 * x + 1], z0, z1, rc.z, rc.w, u0, u1);
        }
        uint32_t ah[4], al[4];
        m2_pack_hilo(lo[0], lo[1], ah[0], al[0]);
        m2_pack_hilo(lo[2], lo[3], ah[1], al[1]);
        m2_pack_hilo(hi[0], hi[1], ah[2], al[2]);
        m2_pack_hilo(hi[2], hi[3], ah[3], al[3]);
        float cr[4];
        m2_mma0(cr, ah, qr[0], qr[1]);
        m2_mma_lo(cr, al, qr[0], qr[1]);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const float2 sp = *reinterpret_cast<const float2*>(rsc + 2 * (g + 8 * x));
#pragma unroll
            for (int e = 0; e < 2; ++e) sc4[2 * x + e] = fmaf(sp.x, ks.cs[2 * x + e] + cr[2 * x + e], sp.y * ks.cs2[2 * x + e]);
        }
    }
    xs[part * 32 + lane] = make_float4(sc4[0], sc4[1], sc4[2], sc4[3]);
    __syncthreads();
    // ================================ softmax over the block ====================================
    float sc[2][2], pw[2][2];
    bool valid[2];
    float4 vs[2];
    {
        const float4 p0 = xs[lane], p1 = xs[32 + lane], p2 = xs[64 + lane], p3 = xs[96 + lane];
        const float tot[4] = {(p0.x + p1.x) + (p2.x + p3.x), (p0.y + p1.y) + (p2.y + p3.y), (p0.z + p1.z) + (p2.z + p3.z),
                              (p0.w + p1.w) + (p2.w + p3.w)};
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            valid[x] = g + 8 * x < valid_hi;
            vs[x] = rsc[2 * (g + 8 * x) + 1];
#pragma unroll
            for (int e = 0; e < 2; ++e) sc[x][e] = valid[x] ? tot[2 * x + e] : -1e30f;
        }
    }
    const float slack = __any_sync(0xFFFFFFFFu, vs[0].w + vs[1].w != 0.0f) ? 0.0f : M2_SLACK;
    st_weights<5>(st, sc, valid, slack, pw);
    uint32_t pb[3][2], pl_[3][2];  // three scaled variants of P (dims 0..2, centroid sign, residual field), hi and lo, tokens = k
#pragma unroll
    for (int e = 0; e < 2; ++e) st.p2[e] = fmaf(pw[1][e], vs[1].y, fmaf(pw[0][e], vs[0].y, st.p2[e]));
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        uint32_t hi, lo;
        m2_pack_hilo(pw[x][0] * vs[x].x, pw[x][1] * vs[x].x, hi, lo);
        pb[0][x] = m2_movmatrix_t(hi);
        pl_[0][x] = m2_movmatrix_t(lo);
        m2_pack_hilo(pw[x][0] * vs[x].y, pw[x][1] * vs[x].y, hi, lo);
        pb[1][x] = m2_movmatrix_t(hi);
        pl_[1][x] = m2_movmatrix_t(lo);
        m2_pack_hilo(pw[x][0] * vs[x].z, pw[x][1] * vs[x].z, hi, lo);
        pb[2][x] = m2_movmatrix_t(hi);
        pl_[2][x] = m2_movmatrix_t(lo);
    }
    // ================================ V side: O^T += V^T P^T (see m2_block) =====================
    uint32_t lo[6], hi[6];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        lo[3 * u + 0] = __byte_perm(ent[u][0].x, ent[u][1].x, 0x5410);
        lo[3 * u + 1] = __byte_perm(ent[u][0].x, ent[u][1].x, 0x7632);
        lo[3 * u + 2] = __byte_perm(ent[u][0].y, ent[u][1].y, 0x5410);
        hi[3 * u + 0] = __byte_perm(ent[u][2].x, ent[u][3].x, 0x5410);
        hi[3 * u + 1] = __byte_perm(ent[u][2].x, ent[u][3].x, 0x7632);
        hi[3 * u + 2] = __byte_perm(ent[u][2].y, ent[u][3].y, 0x5410);
    }
    const uint32_t b01l = __byte_perm(f24[0], f24[1], 0x5410), b01h = __byte_perm(f24[2], f24[3], 0x5410);
    const uint32_t b2l = __byte_perm(f24[0], f24[1], 0x7632), b2h = __byte_perm(f24[2], f24[3], 0x7632);
    const uint32_t da[4] = {m2_field_lo(b01l >> 8), m2_field_hi(b2l), m2_field_lo(b01h >> 8), m2_field_hi(b2h)};
    const uint32_t ca[4] = {m2_sign(b01l << 8), m2_sign(b2l << 12), m2_sign(b01h << 8), m2_sign(b2h << 12)};
#pragma unroll
    for (int jj = 0; jj < 3; ++jj) {
        const uint32_t a[4] = {lo[2 * jj], lo[2 * jj + 1], hi[2 * jj], hi[2 * jj + 1]};
        m2_mma(st.o[jj], a, pb[0][0], pb[0][1]);
        m2_mma_lo(st.o[jj], a, pl_[0][0], pl_[0][1]);
    }
    m2_mma(st.o[3], da, pb[2][0], pb[2][1]);
    m2_mma_lo(st.o[3], da, pl_[2][0], pl_[2][1]);
    m2_mma(st.o[4], ca, pb[1][0], pb[1][1]);
    m2_mma_lo(st.o[4], ca, pl_[1][0], pl_[1][1]);
}

// The CTA's share of the compressed region: blocks of 16 tokens from block0 on.  Leaves the warp's dims 32g + 8 part .. + 7 of heads
// 2t, 2t + 1 in val, relative to the largest score m, and the sum of weights l.
__device__ __forceinline__ void st_compressed(unsigned char* smem, const StepArgs& A, int block0, int nblk, const StepQueryTables& qt,
                                              float4 (&rope)[2], int tid, int kvh, int part, int lane, float (&val)[2][8], float (&m)[2],
                                              float (&l)[2]) {
    const CompressedKV& P = A.kv;
    StepScalars now, next;
    const auto stage = [&](int i, StepScalars& sc) {
        const int tok0 = (block0 + i) * M2_BT;
        st_stage(P, smem + (i & 1) * ST_STAGE, tok0, min(M2_BT, P.c_len - tok0), kvh, A.wide != 0, tid, sc);
    };
    StepFragments f;
    uint32_t qr[2];
    uint4 qraw[2];
    st_load_query(qraw, qr, A.q, kvh, part, lane);  // the longer chain first
    if (nblk > 0) stage(0, now);
    st_build_query(f.qf, qraw, qt, part, lane, reinterpret_cast<float*>(smem + ST_SM_X));
    StepState st;
    st.init();
#pragma unroll 1
    for (int i = 0; i < nblk; ++i) {
        const int tok0 = (block0 + i) * M2_BT;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();  // and every warp is behind block i - 1
        next = now;
        if (i + 1 < nblk) stage(i + 1, next);
        st_block(smem + (i & 1) * ST_STAGE, smem, rope, part, lane, min(P.c_len - tok0, M2_BT), i & 1, f, qr, P, A.scale, now, st);
        now = next;
        if (i + 1 < nblk) {
            if (P.pos_chunk == 0 && (i + 1) % M2_ROPE_RESEED != 0) {
                const float4 d = reinterpret_cast<const float4*>(smem + ST_SM_RSTEP)[4 * part + (lane & 3)];
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float4 a = rope[x];
                    rope[x] = make_float4(a.x * d.x - a.z * d.z, a.y * d.y - a.w * d.w, a.z * d.x + a.x * d.z, a.w * d.y + a.y * d.w);
                }
            } else {
                st_rope_seed(rope, P, reinterpret_cast<const float*>(smem + ST_SM_SMALL), part, lane, tok0 + M2_BT);
            }
        }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
        for (int x = 4; x <= 16; x <<= 1) {
            st.l[e] += __shfl_xor_sync(0xFFFFFFFFu, st.l[e], x);
            st.p2[e] += __shfl_xor_sync(0xFFFFFFFFu, st.p2[e], x);
            st.top[e] = fmaxf(st.top[e], __shfl_xor_sync(0xFFFFFFFFu, st.top[e], x));
        }
        const float fin = __expf(st.m[e] - st.top[e]);
        m[e] = st.top[e];
        l[e] = st.l[e] * fin;
        const float2* c3 = reinterpret_cast<const float2*>(smem + ST_SM_SMALL + (M2_SM_C3 - M2_SM_FREQ)) + 8 * (lane >> 2) + 2 * part;
#pragma unroll
        for (int idx = 0; idx < 6; ++idx) val[e][4 * (idx / 3) + idx % 3] = fin * st.o[idx >> 1][2 * (idx & 1) + e];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const float2 c = c3[u];
            val[e][4 * u + 3] = fin * fmaf(c.x, st.p2[e], fmaf(c.y, st.o[4][2 * u + e], st.o[3][2 * u + e]));
        }
    }
}

// The CTA's share of the raw window: blocks of 16 tokens rank, rank + ctas, ...  Q K^T on mma.sync (fp16 rows as they are, exact products, fp32
// sums; the order of the 64 dims in a contraction is free, so a thread takes 16 contiguous dims of K and Q with 16-byte loads).  The
// weights and P V stay in fp32 on the CUDA cores, lane = 4 dims of 8 of the block's tokens: as a pair of fp16 operands a weight was held to 3e-8
// of the largest one, and where one token with a small V row takes the attention the output is the sum of just those others (200
// tokens, relative error of the output where the others' weights are 2e-4 together: 4.2e-3, 1.7e-6: 0.27; so 2.1e-4 for both, the
// output's own rounding; 16 layers of 384 + 128 tokens 185.5 us with the operands in fp16, 183.3 so).  out: dims 64 part + 4 (lane & 15) .. + 3
// of heads 3 (lane >> 4) .. + 2.
constexpr int ST_WIN_P = (M2_BT + 1) * 8;  // floats per warp: the block's weights, token by token, and the factors of the sums so far
static_assert(ST_PARTS * ST_WIN_P * 4 <= ST_SM_X, "the window's weights take the stages' place");
__device__ __forceinline__ void st_window(unsigned char* smem, const StepArgs& A, int rank, int ctas, int kvh, int part, int lane,
                                          float (&out)[3][4], float (&m)[2], float (&l)[2]) {
    const int g = lane >> 2, t = lane & 3, half = lane >> 4;
    float4* xs = reinterpret_cast<float4*>(smem + ST_SM_X);
    float* wp = reinterpret_cast<float*>(smem) + part * ST_WIN_P;
    const int blocks = (A.win_len + M2_BT - 1) / M2_BT, new_s = A.new_k != nullptr ? A.win_len - 1 : -1;
    uint4 qv[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
    if (g < NREP) {
        const uint4* qp = reinterpret_cast<const uint4*>(A.q + (size_t)(kvh * NREP + g) * 2 * D + 64 * part + 16 * t);
        qv[0] = qp[0];
        qv[1] = qp[1];
    }
    StepState st;
    st.init();
    float o[NREP][4];
#pragma unroll
    for (int h = 0; h < NREP; ++h)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[h][j] = 0.0f;
    int turn = 0;
#pragma unroll 1
    for (int b = rank; b < blocks; b += ctas, turn ^= 1) {
        const int slot0 = (A.win_start + M2_BT * b) % A.ring_cap, last = A.win_len - 1 - M2_BT * b;
        const auto row = [&](const __half* ring, const __half* fresh, int i) {
            i = min(i, last);  // past the end: a row that is there, weight 0
            int slot = slot0 + i;
            if (slot >= A.ring_cap) slot = A.ring_cap >= M2_BT ? slot - A.ring_cap : slot % A.ring_cap;
            return (M2_BT * b + i == new_s ? fresh : ring + (size_t)slot * HKV * D) + kvh * D + 64 * part;
        };
        uint4 kv[2][2];
        uint2 vv[8];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const uint4* kp = reinterpret_cast<const uint4*>(row(A.ring_k, A.new_k, g + 8 * x) + 16 * t);
            kv[x][0] = kp[0];
            kv[x][1] = kp[1];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) vv[i] = *reinterpret_cast<const uint2*>(row(A.ring_v, A.new_v, 8 * half + i) + 4 * (lane & 15));
        float s4[4];
        const uint32_t *k0 = reinterpret_cast<const uint32_t*>(kv[0]), *k1 = reinterpret_cast<const uint32_t*>(kv[1]);
        const uint32_t* qw = reinterpret_cast<const uint32_t*>(qv);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t a[4] = {k0[2 * i], k1[2 * i], k0[2 * i + 1], k1[2 * i + 1]};
            if (i == 0) m2_mma0(s4, a, qw[0], qw[1]);
            else m2_mma(s4, a, qw[2 * i], qw[2 * i + 1]);
        }
        float4* x = xs + turn * ST_PARTS * 32;  // two buffers: one barrier a block
        x[part * 32 + lane] = make_float4(s4[0], s4[1], s4[2], s4[3]);
        __syncthreads();
        const float4 p0 = x[lane], p1 = x[32 + lane], p2 = x[64 + lane], p3 = x[96 + lane];
        const float tot[4] = {(p0.x + p1.x) + (p2.x + p3.x), (p0.y + p1.y) + (p2.y + p3.y), (p0.z + p1.z) + (p2.z + p3.z),
                              (p0.w + p1.w) + (p2.w + p3.w)};
        float sc[2][2], pw[2][2];
        bool valid[2];
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            valid[y] = g + 8 * y <= last;
#pragma unroll
            for (int e = 0; e < 2; ++e) sc[y][e] = valid[y] ? A.scale * tot[2 * y + e] : -1e30f;
        }
        const float before[2] = {st.m[0], st.m[1]};
        st_weights<0>(st, sc, valid, 0.0f, pw);
        if (t < 3) {
#pragma unroll
            for (int y = 0; y < 2; ++y) *reinterpret_cast<float2*>(wp + (g + 8 * y) * 8 + 2 * t) = make_float2(pw[y][0], pw[y][1]);
            if (g == 0) *reinterpret_cast<float2*>(wp + M2_BT * 8 + 2 * t) = make_float2(__expf(before[0] - st.m[0]), __expf(before[1] - st.m[1]));
        }
        __syncwarp();
        const auto weights = [&](int i, float (&w)[NREP]) {
            const float4 a = *reinterpret_cast<const float4*>(wp + i * 8);
            const float2 c = *reinterpret_cast<const float2*>(wp + i * 8 + 4);
            w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = c.x; w[5] = c.y;
        };
        float w[NREP];
        if (b != rank) {
            weights(M2_BT, w);
#pragma unroll
            for (int h = 0; h < NREP; ++h) {
                m2_mul2(o[h][0], o[h][1], o[h][0], o[h][1], w[h], w[h]);
                m2_mul2(o[h][2], o[h][3], o[h][2], o[h][3], w[h], w[h]);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            weights(8 * half + i, w);
            const float2 va = __half22float2(*reinterpret_cast<const __half2*>(&vv[i].x)), vb = __half22float2(*reinterpret_cast<const __half2*>(&vv[i].y));
#pragma unroll
            for (int h = 0; h < NREP; ++h) {
                m2_fma2(o[h][0], o[h][1], va.x, va.y, w[h], w[h], o[h][0], o[h][1]);
                m2_fma2(o[h][2], o[h][3], vb.x, vb.y, w[h], w[h], o[h][2], o[h][3]);
            }
        }
    }
    // both halves of the tokens: three heads each
#pragma unroll
    for (int h = 0; h < 3; ++h)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float other = __shfl_xor_sync(0xFFFFFFFFu, half ? o[h][j] : o[h + 3][j], 16);
            out[h][j] = (half ? o[h + 3][j] : o[h][j]) + other;
        }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
        for (int y = 4; y <= 16; y <<= 1) st.l[e] += __shfl_xor_sync(0xFFFFFFFFu, st.l[e], y);
        m[e] = st.m[e];
        l[e] = st.l[e];
    }
}

// The warp's share of head h, record `rec` of n: with several records the warp that arrives last merges them all; then the division
// and the gate.
__device__ __forceinline__ void st_finish_head(const StepArgs& A, int h, int rec, int lane, HeadAcc& a, const uint4& gate) {
    const int n = A.n_records;
    if (n > 1) {
        float* r = A.sums + ((size_t)rec * HQ + h) * D + lane * 8;
        __stcg(reinterpret_cast<float4*>(r), make_float4(a.a[0], a.a[1], a.a[2], a.a[3]));
        __stcg(reinterpret_cast<float4*>(r + 4), make_float4(a.a[4], a.a[5], a.a[6], a.a[7]));
        float2* ml_of = A.ml + h;
        if (lane == 0) __stcg(ml_of + rec * HQ, make_float2(a.m, a.l));
        __syncwarp();
        int order = 0;
        if (lane == 0) {
            __threadfence();
            order = atomicAdd(A.counters + h, 1);
            __threadfence();
        }
        __syncwarp();  // the other lanes read the records behind lane 0's fence (a shuffle orders no memory)
        if (__shfl_sync(0xFFFFFFFFu, order, 0) != n - 1) return;
        if (lane == 0) A.counters[h] = 0;
        constexpr int AHEAD = 6;  // records whose sums are on their way beside the maxima
        const float* base = A.sums + (size_t)h * D + lane * 8;
        float2 ml = make_float2(NEG_BIG, 0.0f);
        if (lane < n) ml = __ldcg(ml_of + lane * HQ);
        float4 v[AHEAD][2];
        const auto fetch = [&](int i, int at) {
            const float4* p = reinterpret_cast<const float4*>(base + (size_t)min(at, n - 1) * HQ * D);
            v[i][0] = __ldcg(p);
            v[i][1] = __ldcg(p + 1);
        };
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) fetch(i, i);
        float M = ml.x;
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) M = fmaxf(M, __shfl_xor_sync(0xFFFFFFFFu, M, k));
        const float w = __expf(ml.x - M);  // 0 for lanes without a record
        float den = ml.y * w;
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) den += __shfl_xor_sync(0xFFFFFFFFu, den, k);
        a.l = den;
#pragma unroll
        for (int j = 0; j < 8; ++j) a.a[j] = 0.0f;
        for (int i0 = 0; i0 < n; i0 += AHEAD) {
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                const float wi = __shfl_sync(0xFFFFFFFFu, w, min(i0 + i, 31));
                const float x[8] = {v[i][0].x, v[i][0].y, v[i][0].z, v[i][0].w, v[i][1].x, v[i][1].y, v[i][1].z, v[i][1].w};
                if (i0 + i < n)
#pragma unroll
                    for (int j = 0; j < 8; ++j) a.a[j] = fmaf(x[j], wi, a.a[j]);
                if (i0 + AHEAD < n) fetch(i, i0 + AHEAD + i);
            }
        }
    }
    const float inv_den = 1.0f / (a.l + 1e-8f);
    const __half2* hg = reinterpret_cast<const __half2*>(&gate);
    uint4 o;
    __half2* ho = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 gf = __half22float2(hg[j]);
        ho[j] = __floats2half2_rn(a.a[2 * j] * inv_den * (1.0f / (1.0f + __expf(-gf.x))), a.a[2 * j + 1] * inv_den * (1.0f / (1.0f + __expf(-gf.y))));
    }
    *reinterpret_cast<uint4*>(A.out + (size_t)h * D + lane * 8) = o;
}

// grid = 4 kv-heads x n_records clusters, the last four serve the window; or four clusters per item of a batch.
template <bool BATCH>
__global__ void __launch_bounds__(ST_THREADS, 4) khq_step_kernel(const __grid_constant__ StepArgs one, const __grid_constant__ StepBatch batch) {
    extern __shared__ __align__(128) unsigned char smem[];
    StepArgs& filled = *reinterpret_cast<StepArgs*>(smem + ST_SM_ARGS);
    const StepArgs& A = BATCH ? filled : one;
    const int tid = threadIdx.x, part = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    const int rank = (int)blockIdx.x % ST_CLUSTER, cl = (int)blockIdx.x / ST_CLUSTER, kvh = cl % HKV;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + ST_SM_BAR);
    float* recv = reinterpret_cast<float*>(smem + ST_SM_RECV);
    if (tid == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
        mbar_arrive_expect_tx(bar, ST_CLUSTER * ST_RECV * 4);
        if (BATCH) st_fill_constants(filled, batch);
    }
    __syncthreads();
    st_cluster_arrive();  // waited for before the first push: the peers' barriers are there
    StepQueryTables qt;
    float4 rope[2];
    if (BATCH || cl / HKV < A.n_records - 1) {  // constants of the model: fetched while the kernel in front still runs
        qt.load(A.kv, part, lane);
        const uint4* src = reinterpret_cast<const uint4*>(A.kv.image + M2_IMG_ROT);
        uint4* dst = reinterpret_cast<uint4*>(smem + ST_SM_ROT);
#pragma unroll
        for (int e = tid; e < 16 * 32; e += ST_THREADS) {
            dst[e] = __ldg(src + 2 * e);
            dst[16 * 32 + e] = __ldg(src + 2 * e + 1);
        }
        const uint4* small = reinterpret_cast<const uint4*>(A.kv.image + M2_IMG_SMALL);
        for (int e = tid; e < M2_SMALL_BYTES / 16; e += ST_THREADS) reinterpret_cast<uint4*>(smem + ST_SM_SMALL)[e] = __ldg(small + e);
        const float* freq = reinterpret_cast<const float*>(A.kv.image + M2_IMG_SMALL);
        if (!BATCH) st_rope_seed(rope, A.kv, freq, part, lane, (cl / HKV * ST_CLUSTER + rank) * A.blocks_per_cta * M2_BT);
        if (tid < 32) {
            double th = (double)M2_BT * (double)freq[tid] * 0.3183098861837907;  // half turns
            th -= 2.0 * rint(0.5 * th);
            float* o = reinterpret_cast<float*>(smem + ST_SM_RSTEP) + 4 * (tid >> 1) + (tid & 1);
            sincospif((float)th, &o[2], &o[0]);
        }
    }
    st_cluster_wait();
    pdl_wait();
    pdl_trigger();
    if (BATCH) {
        if (tid == 0) st_fill_item(filled, batch, cl / HKV);
        __syncthreads();
    }
    const int rec = BATCH ? A.rec : cl / HKV;
    const bool comp = BATCH ? A.comp != 0 : rec < A.n_records - 1;
    const int block0 = BATCH ? A.block0 + rank * A.blocks_per_cta : (rec * ST_CLUSTER + rank) * A.blocks_per_cta;
    const int nblk = comp ? min(max((A.kv.c_len + M2_BT - 1) / M2_BT - block0, 0), A.blocks_per_cta) : 0;
    if (BATCH && nblk > 0) st_rope_seed(rope, A.kv, reinterpret_cast<const float*>(smem + ST_SM_SMALL), part, lane, block0 * M2_BT);
    float val[2][8], win[3][4], m[2], l[2];
    if (comp) {
        st_compressed(smem, A, block0, nblk, qt, rope, tid, kvh, part, lane, val, m, l);
    } else {
        if (rank < 3) {  // ring appends: the kv-head's part of one ring's row
            const size_t at = (size_t)((A.win_start + A.win_len - 1) % A.ring_cap) * HKV * D + kvh * D;
            const __half* src = rank == 0 ? A.new_k : rank == 1 ? A.new_v : A.new_u;
            __half* dst = rank == 0 ? A.ring_k : rank == 1 ? A.ring_v : A.ring_u;
            if (tid < D / 8 && src != nullptr && dst != nullptr) reinterpret_cast<uint4*>(dst + at)[tid] = reinterpret_cast<const uint4*>(src + kvh * D)[tid];
        }
        st_window(smem, A, rank, ST_CLUSTER, kvh, part, lane, win, m, l);
    }
    // ---- each head's sums to the CTA that owns it ------------------------------------------------
    const int g = lane >> 2, t = lane & 3;
    float* send = reinterpret_cast<float*>(smem + ST_SM_SEND);
    __syncthreads();  // the records alias what the last block was read from
    if (comp) {
        const int d0 = 32 * g + 8 * part;
        if (t < 3)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float4* to = reinterpret_cast<float4*>(send + (2 * t + e) * ST_RECV + d0 + 4 * (d0 >> 5));
                to[0] = make_float4(val[e][0], val[e][1], val[e][2], val[e][3]);
                to[1] = make_float4(val[e][4], val[e][5], val[e][6], val[e][7]);
            }
    } else {
        const int d0 = 64 * part + 4 * (lane & 15);
#pragma unroll
        for (int h = 0; h < 3; ++h)
            *reinterpret_cast<float4*>(send + (3 * (lane >> 4) + h) * ST_RECV + d0 + 4 * (d0 >> 5)) = make_float4(win[h][0], win[h][1], win[h][2], win[h][3]);
    }
    if (t < 3 && g == 0 && part == 0)
#pragma unroll
        for (int e = 0; e < 2; ++e) *reinterpret_cast<float2*>(send + (2 * t + e) * ST_RECV + ST_REC) = make_float2(m[e], l[e]);
    fence_proxy_async();
    __syncthreads();
    if (tid < NREP) st_push(st_map(recv + rank * ST_RECV, tid), send + tid * ST_RECV, ST_RECV * 4, st_map(bar, tid));
    if (part == 0 && rank < NREP) {  // the owned head
        const int h = kvh * NREP + rank;
        VInverse inv;
        if (comp) inv.load(A.kv, lane);
        const uint4 gate = *reinterpret_cast<const uint4*>(A.q + (size_t)h * 2 * D + D + lane * 8);
        mbar_wait_bounded(bar, 0u, &g_status);
        HeadAcc a = merge_head<true, ST_CLUSTER>(ST_CLUSTER, lane, [&](int i) {
            const float* r = recv + i * ST_RECV;
            return HeadRec{r, r + ST_REC, r + ST_REC + 1};
        });
        if (comp) inv.apply(a.a, lane);
        st_finish_head(A, h, rec, lane, a, gate);
    }
    st_cluster_arrive();  // no CTA ends before its records have been read
    st_cluster_wait();
}

// The same step for longer contexts: a CTA has all kv-heads and twelve warps, each on its own 16-token blocks (m2_compressed_range), and
// one cluster of the same grid has the window (window_range).  The three warps of a kv-head are merged inside the CTA, the rest
// is as above.  One more cluster barrier than there: the received records take the codebook's place.
constexpr int SW_SEND = M2_SM_VQ, SW_RECV = SW_SEND + 32 * 1024;
constexpr int SW_ARGS = (M2_SM_TOTAL + 15) / 16 * 16, SW_TOTAL = SW_ARGS + ST_ARGS_BYTES;  // of a batch
static_assert(SW_TOTAL <= 226 * 1024 && HQ * ST_RECV * 4 <= 32 * 1024 && SW_RECV + HQ * ST_RECV * 4 <= M2_SM_ROPE && SW_SEND % 16 == 0, "records take the codebook's place");
template <bool BATCH>
__global__ void __launch_bounds__(M2_THREADS, 1) khq_step_wide_kernel(const __grid_constant__ StepArgs one, const __grid_constant__ StepBatch batch) {
    extern __shared__ __align__(128) unsigned char smem[];
    StepArgs& filled = *reinterpret_cast<StepArgs*>(smem + SW_ARGS);
    const StepArgs& A = BATCH ? filled : one;
    __shared__ __align__(8) uint64_t s_bar;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31, kvh = warp & 3, sub = warp >> 2;
    const int csize = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), cl = (int)blockIdx.x / csize, owned = HQ / csize;
    const bool tables = BATCH || cl < A.n_records - 1;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + M2_SM_BARS);
    uint32_t* tm_slot = reinterpret_cast<uint32_t*>(smem + M2_SM_TMSLOT);
    if (tid == 0) {
        for (int s = 0; s < M2_BAR_SMALL; ++s) mbar_init(&bars[s], HKV);
        for (int s = M2_BAR_SMALL; s < M2_NBARS; ++s) mbar_init(&bars[s], 1);
        mbar_init(&s_bar, 1);
        fence_barrier_init();
        mbar_arrive_expect_tx(&s_bar, HQ * ST_RECV * 4);
        if (BATCH) st_fill_constants(filled, batch);
    }
    if (tables) m2_tm_alloc(tm_slot, warp);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tables ? __shfl_sync(0xFFFFFFFFu, *tm_slot, 0) : 0u;
    VInverse inv;
    M2QueryTables qt;
    if (tables) {
        m2_load_tables(smem, A.kv, tmem, tid, warp, lane);  // constants of the model: while the kernel in front still runs
        qt.load(A.kv, sub, lane);
    }
    pdl_wait();
    pdl_trigger();
    if (BATCH) {
        if (tid == 0) st_fill_item(filled, batch, cl);
        __syncthreads();
    }
    const int rec = BATCH ? A.rec : cl;
    const bool comp = BATCH ? A.comp != 0 : tables;
    if (comp) {
        unsigned blocks_done = 0;
        const int block0 = BATCH ? A.block0 + rank * A.blocks_per_cta : (int)blockIdx.x * A.blocks_per_cta;
        const int lo = min(M2_BT * block0, A.kv.c_len), hi = min(lo + M2_BT * A.blocks_per_cta, A.kv.c_len);
        m2_compressed_range(smem, A.q, (size_t)2 * D, A.kv, lo, hi, A.scale, blocks_done, tmem, qt, 1u, inv);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    } else {
        if (BATCH) {  // the tables that it has no use for: no copy outlives the kernel, none lands in what follows
            mbar_wait_bounded(&bars[M2_BAR_SMALL], 0u, &g_status);
            mbar_wait_bounded(&bars[M2_BAR_VQ], 0u, &g_status);
        }
        if (rank < 3) {  // ring appends: one ring per CTA
            const size_t at = (size_t)((A.win_start + A.win_len - 1) % A.ring_cap) * HKV * D;
            const __half* src = rank == 0 ? A.new_k : rank == 1 ? A.new_v : A.new_u;
            __half* dst = rank == 0 ? A.ring_k : rank == 1 ? A.ring_v : A.ring_u;
            if (tid < HKV * D / 8 && src != nullptr && dst != nullptr) reinterpret_cast<uint4*>(dst + at)[tid] = reinterpret_cast<const uint4*>(src)[tid];
        }
        WarpState ws;
        ws.init();
        window_range<4>(A.q, A.ring_k, A.ring_v, A.win_start, rank * M2_WPK + sub, csize * M2_WPK, A.win_len, A.ring_cap, A.scale, kvh, lane, ws,
                        A.new_k != nullptr ? A.win_len - 1 : -1, A.new_k, A.new_v);
        m2_store_record(ws, reinterpret_cast<float*>(smem + M2_SM_STAGES) + warp * M2_REC_FLOATS, lane);
        __syncthreads();
    }
    st_cluster_arrive();  // this CTA's codebook is not needed any more
    {
        const float* recs = reinterpret_cast<const float*>(smem + M2_SM_STAGES);
        HeadAcc a[2];  // two heads per warp, side by side
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int h = warp + k * (HQ / 2);
            a[k] = merge_head<true, M2_WPK>(M2_WPK, lane, [&](int i) { return m2_head_of_record(recs + (h / NREP + HKV * i) * M2_REC_FLOATS, h % NREP); });
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            float* r = reinterpret_cast<float*>(smem + SW_SEND) + (warp + k * (HQ / 2)) * ST_RECV;
            float4* to = reinterpret_cast<float4*>(r + lane * 8 + 4 * (lane >> 2));
            to[0] = make_float4(a[k].a[0], a[k].a[1], a[k].a[2], a[k].a[3]);
            to[1] = make_float4(a[k].a[4], a[k].a[5], a[k].a[6], a[k].a[7]);
            if (lane == 0) *reinterpret_cast<float2*>(r + ST_REC) = make_float2(a[k].m, a[k].l);
        }
    }
    fence_proxy_async();
    __syncthreads();
    if (tables) m2_tm_free(tmem, warp);
    st_cluster_wait();
    float* recv = reinterpret_cast<float*>(smem + SW_RECV);
    if (tid < HQ)
        st_push(st_map(recv + (tid / csize * csize + rank) * ST_RECV, tid % csize), smem + SW_SEND + tid * ST_RECV * 4, ST_RECV * 4,
                st_map(&s_bar, tid % csize));
    if (warp < owned) {
        const int h = rank + csize * warp;
        const uint4 gate = *reinterpret_cast<const uint4*>(A.q + (size_t)h * 2 * D + D + lane * 8);
        mbar_wait_bounded(&s_bar, 0u, &g_status);
        HeadAcc a = merge_head<true>(csize, lane, [&](int i) {
            const float* r = recv + (warp * csize + i) * ST_RECV;
            return HeadRec{r, r + ST_REC, r + ST_REC + 1};
        });
        if (comp) inv.apply(a.a, lane);
        st_finish_head(A, h, rec, lane, a, gate);
    }
    st_cluster_arrive();  // no CTA ends before its records have been read
    st_cluster_wait();
}

}  // namespace khq
