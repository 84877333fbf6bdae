// khq_prefill_pair.cuh -- the causal GQA prefill of khq_prefill_tc5.cu on CTA pairs (tcgen05 cta_group::2), for prompts of many row
// blocks.  Included by it.
//
// A pair of CTAs on two SMs takes 128 query rows of two neighbouring heads of one kv head, which attend the same keys: one
// instruction is M 256 over both (rows 0-127: the first CTA's head), and each CTA keeps half of the K tile (64 of 128 keys) and
// half of the V tile (128 of 256 head dims).  That halves what a CTA loads from L2 and makes room for two K and two V tiles:
// with one of each, a tile's K came some 600 cycles late.
//
// What bounds it: the tensor pipe and, in long runs, the power limit.  64 cycles per Q K^T step and 128 per P V step, 2050 a tile of
// 128 keys, was measured for these instructions back to back (also with one CTA); the kernel takes 2230 where the limit does not
// slow it.  On the way there from 2820:
//   * Two groups of four softmax warps take the tiles in turn, a thread per row.  A tile's weights take 1800 cycles from its scores (a
//     thread per row: no exchange of maxima; 16 ex2 a cycle are 1024 of them), which one group could not hide.
//   * P reaches the MMA warp in two halves of 64 keys.
//   * The MMA warp tests the barriers of its next step in front of the last instructions of the current one: a wait costs 300 to 600
//     cycles, more than the pipe has queued.
//   * Its operands stay in uniform registers (umma2_ss).
// Around a row block (some 30 tiles at T = 8192, 6 at 1500): barriers and tensor memory are set up while Q and K load; half of the gates
// have buffers of their own, the others land in the Q buffer once the last Q K^T has read it; the sigmoids of the first half are
// evaluated while the last P V runs.
// 4 x 8192: 2.67 -> 2.35 ms alone, 3.0-3.2 -> 2.45-2.7 in a row (box and power limit); 9 x 1531: 385 -> 355 us; 8 x 2048: 553 -> 492.
#pragma once

namespace khq_prefill5 {
namespace pair {

constexpr int TILE_BYTES = 64 * D * 2;  // a CTA's share of a K or V tile
constexpr int OFF_Q = 0;                // later two pieces of the gates, then of the outputs
constexpr int OFF_K = OFF_Q + Q_BYTES;
constexpr int OFF_V = OFF_K + 2 * TILE_BYTES;
constexpr int OFF_STG = OFF_V + 2 * TILE_BYTES;   // the first two pieces of the gates, then of the outputs
constexpr int OFF_MREF = OFF_STG + 2 * STG_BYTES;  // float [2 groups][128 rows]: the reference behind the group's last tile
constexpr int OFF_LSUM = OFF_MREF + 2 * 128 * 4;  // float [2 groups][128 rows]
constexpr int OFF_BARS = OFF_LSUM + 2 * 128 * 4;
enum Bar {  // K, V, S and P V by tile parity
    B_KFULL = 0, B_VFULL = 2, B_SFULL = 4, B_PVDONE = 6, B_PREADY = 8 /* [parity][half of the keys] */, B_QFULL = 12, B_QFREE = 13, B_PEER = 14,
    B_MREF = 15 /* [group][lane quarter] */, B_LSUM = 23 /* [lane quarter] */, B_GFULL = 27 /* [piece] */, B_OUT = 31 /* [piece] */, B_COUNT = 35
};
constexpr int OFF_SLOT = OFF_BARS + B_COUNT * 8;
constexpr int SMEM = OFF_SLOT + 16;
static_assert(2 * STG_BYTES <= Q_BYTES && SMEM <= 227 * 1024, "shared memory");
__host__ __device__ constexpr int off_piece(int c) { return c < 2 ? OFF_STG + c * STG_BYTES : OFF_Q + (c - 2) * STG_BYTES; }

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// (d0, d1) = (a0, a1) m + c and (s0, s1) += (a0, a1), one packed instruction each
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float m, float c) {
    asm("{.reg .b64 a, m, c, d; mov.b64 a, {%2, %3}; mov.b64 m, {%4, %4}; mov.b64 c, {%5, %5}; fma.rn.f32x2 d, a, m, c; mov.b64 {%0, %1}, d;}"
        : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(m), "f"(c));
}
__device__ __forceinline__ void add2(float& s0, float& s1, float a0, float a1) {
    asm("{.reg .b64 a, s; mov.b64 a, {%2, %3}; mov.b64 s, {%0, %1}; add.rn.f32x2 s, s, a; mov.b64 {%0, %1}, s;}" : "+f"(s0), "+f"(s1) : "f"(a0), "f"(a1));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
                 "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
                 : "memory");
}
// The MMA warp stays together and one lane issues (`one`): its descriptors are then values of the whole warp, kept and stepped in uniform
// registers.  With one lane alone inside a branch each instruction's operands had to be moved there one by one, which took about as
// long as the pipe takes for the instruction, or longer by the luck of the code's placement (4 x 8192: 2.42 ms, 2.49 to 2.95).
template <int ACC>
__device__ __forceinline__ void umma2_ss(uint32_t one, uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .b64 da, db;\n\t.reg .pred p, q;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "setp.ne.u32 p, %6, 0;\n\tsetp.ne.u32 q, %7, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "n"(ACC), "r"(one)
        : "memory");
}
__device__ __forceinline__ void umma2_ts(uint32_t one, uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .b64 db;\n\t.reg .pred p, q;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.u32 p, %5, 0;\n\tsetp.ne.u32 q, %6, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(one)
        : "memory");
}
// Arrives at this barrier of both CTAs once the instructions issued so far have completed.
__device__ __forceinline__ void umma2_commit(uint32_t one, uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
        "h"((uint16_t)3), "r"(one)
        : "memory");
}
// The address of `bar` in the pair's first CTA.
__device__ __forceinline__ uint32_t in_leader(uint64_t* bar) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(bar)));
    return r;
}
__device__ __forceinline__ void arrive_leader(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(in_leader(bar)) : "memory");
}
// A load into this CTA's shared memory whose bytes count at a barrier of the pair's first CTA.
__device__ __forceinline__ void load_for_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c1, int c2, int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5, "
        "%6, %7}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}
// Of the MMA warp's barriers too: the other CTA's arrivals announce tensor-memory contents and asynchronous copies, which the tcgen05
// fences and the copies' byte counts order, not ordinary memory.  Acquiring at cluster scope cost 4 to 8 %.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// Item of a pair: (batch, kv head) groups one after the other, the heaviest row blocks first inside a group: what is in flight then
// streams the K and V rows of one or two groups, which stay in L2, and the hardware's scheduler evens out the triangle.
// q_gate (B, T, H_q, 2D), out (B, T, H_q, D) through their tensor maps; grid = 2 x row blocks x H_q / 2 x B.
template <bool BF16>
__global__ void __launch_bounds__(NTHREADS, 1)
khq_gqa_prefill_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                            const __grid_constant__ CUtensorMap tm_g, const __grid_constant__ CUtensorMap tm_o, int T, int H_q, int H_kv,
                            float scale_log2e) {
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BARS);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_SLOT);
    float* mref = reinterpret_cast<float*>(smem + OFF_MREF);
    float* lsum = reinterpret_cast<float*>(smem + OFF_LSUM);
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    const int rank = (int)(blockIdx.x & 1);  // the pair's first CTA has the MMA thread
    int* status = &g_prefill_status;
    if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled layouts need a 1024-byte aligned base; the same in both CTAs
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int nqb = (T + BR - 1) / BR, sets = H_q / H_kv / 2;  // head pairs of a kv head
    const int group = (int)(blockIdx.x >> 1) / (sets * nqb), idx = (int)(blockIdx.x >> 1) % (sets * nqb);
    const int qb = nqb - 1 - idx / sets, b = group / H_kv, kvh = group % H_kv, h = kvh * 2 * sets + idx % sets * 2 + rank;
    const int q0 = qb * BR, n_tiles = qb + 1, last = n_tiles - 1;  // causal: key tiles 0..qb
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            khq::mbar_init(&bars[B_KFULL + s], 1);
            khq::mbar_init(&bars[B_VFULL + s], 1);
            khq::mbar_init(&bars[B_SFULL + s], 1);
            khq::mbar_init(&bars[B_PVDONE + s], 1);
        }
        khq::mbar_init(&bars[B_QFULL], 1);
        khq::mbar_init(&bars[B_QFREE], 1);
        khq::mbar_init(&bars[B_PEER], 1);
        // one elected arrival per softmax warp of both CTAs: separate arrivals on one barrier serialise
        for (int q = 0; q < 4; ++q) {
            khq::mbar_init(&bars[B_PREADY + q], 2 * NSOFT / 64);
            khq::mbar_init(&bars[B_LSUM + q], 2);  // the two warps of a lane quarter
            khq::mbar_init(&bars[B_GFULL + q], 1);
            khq::mbar_init(&bars[B_OUT + q], NSOFT / 32);
        }
        for (int q = 0; q < 8; ++q) khq::mbar_init(&bars[B_MREF + q], 1);
        khq::fence_barrier_init();
    } else if (warp == 8 && lane < 3) {
        prefetch_map(lane == 0 ? &tm_q : lane == 1 ? &tm_k : &tm_v);
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();  // the barriers of both CTAs are there
    // Everything above overlaps the kernel before; tensor memory is only taken once that kernel has finished (it may still have
    // to allocate its own on this SM).
    khq::pdl_wait();
    khq::pdl_trigger();
    const uint32_t sbase = smem_u32(smem);
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(TM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    // tensor memory is there; the loads do not wait for that
    if (warp == 8 || warp == 10 || warp == 11) asm volatile("bar.arrive 1, %0;" ::"n"(NTHREADS) : "memory");
    else asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory");
    tc_fence_after();

    if (warp == 8) {
        // ================================ producer of Q and K: the CTA's 64 keys of a tile as [4 groups][64 keys][128 B] ==========
        if (lane == 0) {
            if (rank == 0) khq::mbar_arrive_expect_tx(&bars[B_QFULL], 2 * Q_BYTES);
            load_for_pair(sbase + OFF_Q, &tm_q, in_leader(&bars[B_QFULL]), q0, 0, h, b);
            int g = 0;
            for (; g < n_tiles; ++g) {
                const int s = g & 1;
                if (g >= 2 && !khq::mbar_wait_bounded(&bars[B_SFULL + s], (uint32_t)(((g >> 1) - 1) & 1), status)) break;
                if (rank == 0) khq::mbar_arrive_expect_tx(&bars[B_KFULL + s], 2 * TILE_BYTES);
                load_for_pair(sbase + OFF_K + s * TILE_BYTES, &tm_k, in_leader(&bars[B_KFULL + s]), g * BC + rank * 64, 0, kvh, b);
            }
            // nothing may still be in flight when the pair leaves: the first CTA waits for the loads of both
            if (rank == 0) {
                khq::mbar_wait_bounded(&bars[B_QFULL], 0u, status);
                for (int i = max(0, g - 2); i < g; ++i) khq::mbar_wait_bounded(&bars[B_KFULL + (i & 1)], (uint32_t)((i >> 1) & 1), status);
            }
        }
    } else if (warp == 10) {
        // ================================ producer of V: the CTA's 128 head dims as [2 groups][128 keys][128 B] ===================
        if (lane == 0) {
            int g = 0;
            for (; g < n_tiles; ++g) {
                const int s = g & 1;
                if (g >= 2 && !khq::mbar_wait_bounded(&bars[B_PVDONE + s], (uint32_t)(((g >> 1) - 1) & 1), status)) break;
                if (rank == 0) khq::mbar_arrive_expect_tx(&bars[B_VFULL + s], 2 * TILE_BYTES);
                load_for_pair(sbase + OFF_V + s * TILE_BYTES, &tm_v, in_leader(&bars[B_VFULL + s]), g * BC, 2 * rank, kvh, b);
            }
            if (rank == 0)
                for (int i = max(0, g - 2); i < g; ++i) khq::mbar_wait_bounded(&bars[B_VFULL + (i & 1)], (uint32_t)((i >> 1) & 1), status);
        }
    } else if (warp == 9) {
        // ================================ MMA issuer ==============================================
        const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);
        if (rank == 1 && lane == 0) arrive_leader(&bars[B_PEER]);
        if (rank == 0) {
            const uint32_t one = elect_one();
            constexpr uint32_t IDESC_S = instr_desc(2 * BR, BC, false, BF16), IDESC_O = instr_desc(2 * BR, D, true, BF16);
            constexpr uint32_t HI = desc_hi(1024);  // Q, K (K-major) and V (MN-major): 1024 bytes between 8-row groups
            const uint32_t q_lo = desc_lo(sbase + OFF_Q, 16), k_lo = desc_lo(sbase + OFF_K, 16);
            const uint32_t v_lo = desc_lo(sbase + OFF_V, 128 * 128);  // leading offset: the next 64-column group
            bool ok = true;
            // A wait costs this thread some 300 cycles even when its barrier completed long ago, and the pipe holds only a few
            // instructions ahead.  So a barrier is tested in front of the last instructions before its use, and waited for only if
            // that came out negative.
            uint32_t k_there = 0, p_there = 0, v_there = 0;
            const auto need = [&](uint32_t there, uint64_t* bar, uint32_t parity) {
                if (ok && !__any_sync(0xFFFFFFFFu, there)) ok = warp_wait(bar, parity, status);
            };
            // S[g & 1] = Q K^T of tile g; behind it come the weights of tile g - 1
            const auto issue_qk = [&](int g) {
                const uint32_t s_tmem = tmem + TM_S + (uint32_t)(g & 1) * BC;
                need(k_there, &bars[B_KFULL + (g & 1)], (uint32_t)((g >> 1) & 1));
                if (!ok) return;
                tc_fence_after();
                const uint32_t k_at = k_lo + (uint32_t)(g & 1) * (TILE_BYTES >> 4);
#pragma unroll
                for (int ks = 0; ks < 16; ++ks) {
                    // byte offsets / 16: next 64-dim group = rows * 128 bytes, next K step = 32 bytes
                    const uint32_t oa = (uint32_t)((ks >> 2) * (BR * 128) + (ks & 3) * 32) >> 4;
                    const uint32_t ob = (uint32_t)((ks >> 2) * (64 * 128) + (ks & 3) * 32) >> 4;
                    if (ks == 0) umma2_ss<0>(one, s_tmem, q_lo + oa, HI, k_at + ob, HI, IDESC_S);
                    else umma2_ss<1>(one, s_tmem, q_lo + oa, HI, k_at + ob, HI, IDESC_S);
                    if (ks == 11 && g > 0) {
                        p_there = mbar_test(&bars[B_PREADY + 2 * ((g - 1) & 1)], (uint32_t)(((g - 1) >> 1) & 1));
                        v_there = mbar_test(&bars[B_VFULL + ((g - 1) & 1)], (uint32_t)(((g - 1) >> 1) & 1));
                    }
                }
                umma2_commit(one, &bars[B_SFULL + (g & 1)]);
                if (g == last) umma2_commit(one, &bars[B_QFREE]);
            };
            ok = warp_wait(&bars[B_PEER], 0u, status) && warp_wait(&bars[B_QFULL], 0u, status);
            if (ok) issue_qk(0);
            for (int g = 0; ok && g < n_tiles; ++g) {
                const int s = g & 1;
                const uint32_t par = (uint32_t)((g >> 1) & 1);
                k_there &= (uint32_t)(g > 0);
                p_there = v_there = 0;
                if (g < last) issue_qk(g + 1);
                need(p_there, &bars[B_PREADY + 2 * s], par);
                need(v_there, &bars[B_VFULL + s], par);
                if (!ok) break;
                tc_fence_after();
                const uint32_t v_at = v_lo + (uint32_t)s * (TILE_BYTES >> 4), p_tmem = tmem + TM_S + (uint32_t)s * BC;
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) {
                    if (kk == 4) {  // the other half of the keys: its weights come while the first half is multiplied
                        need(p_there, &bars[B_PREADY + 2 * s + 1], par);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    umma2_ts(one, tmem + TM_O, p_tmem + kk * 8, v_at + ((uint32_t)(kk * 2048) >> 4), HI, IDESC_O, kk > 0 ? 1u : (uint32_t)(g > 0));  // 16 keys = 2048 bytes
                    if (kk == 1) p_there = mbar_test(&bars[B_PREADY + 2 * s + 1], par);
                    if (kk == 5) k_there = mbar_test(&bars[B_KFULL + s], (uint32_t)(((g + 2) >> 1) & 1));  // of tile g + 2
                }
                if (!ok) break;
                umma2_commit(one, &bars[B_PVDONE + s]);
            }
        }
    } else if (warp == 11) {
        // ================================ gates in, outputs out: four pieces of 64 columns ==========
        if (lane == 0) {
            int loads = 0;
            const auto load = [&](int c) {
                khq::mbar_arrive_expect_tx(&bars[B_GFULL + c], STG_BYTES);
                tma_load_5d(sbase + off_piece(c), &tm_g, &bars[B_GFULL + c], q0, c, h, b);
                ++loads;
            };
            load(0);
            load(1);
            tma_prefetch_5d(&tm_g, q0, 2, h, b);
            tma_prefetch_5d(&tm_g, q0, 3, h, b);
            if (khq::mbar_wait_bounded(&bars[B_QFREE], 0u, status)) {  // the last Q K^T has read Q
                load(2);
                load(3);
            }
            for (int c = 0; c < loads; ++c) {
                if (!khq::mbar_wait_bounded(&bars[B_OUT + c], 0u, status)) break;
                tma_store_5d(&tm_o, sbase + off_piece(c), q0, c, h, b);
            }
            for (int c = 0; c < loads; ++c) khq::mbar_wait_bounded(&bars[B_GFULL + c], 0u, status);
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
    } else {
        // ================================ softmax + epilogue ======================================
        // Group 0 (warps 0-3) has the even tiles, group 1 (warps 4-7) the odd ones; a thread owns a row (all 128 keys of its tiles, and
        // half the columns of O in the epilogue).  The groups' reference maxima follow one another through shared memory, warp by
        // warp: the two warps of a lane quarter have the same rows.
        const uint32_t tmem = *tmem_slot;
        const int grp = warp >> 2, quarter = warp & 3, r = tid & 127, row = q0 + r;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
        bool ok = true;
        float m_l = -1e30f, l_run = 0.0f;  // the sum of this group's tiles and the reference that it is against
        for (int g = grp; g < n_tiles; g += 2) {
            // the reference behind the tile before, mostly there by now: ahead of the scores
            float before = 0.0f;
            if (g > 0) {
                ok = __all_sync(0xFFFFFFFFu, khq::mbar_wait_bounded(&bars[B_MREF + 4 * (grp ^ 1) + quarter], (uint32_t)(((g - 1) >> 1) & 1), status));
                if (!ok) break;
                before = mref[(grp ^ 1) * 128 + r];
            }
            ok = __all_sync(0xFFFFFFFFu, khq::mbar_wait_bounded(&bars[B_SFULL + grp], (uint32_t)((g >> 1) & 1), status));
            if (!ok) break;
            tc_fence_after();
            const uint32_t s_addr = lane_base + TM_S + (uint32_t)grp * BC;
            uint32_t sr[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + 32 * c, sr[c]);
            tmem_ld_wait();
            const int k0 = g * BC;
            // raw scores; masked entries (key after the row, or past the prompt) become -inf-like
            if ((k0 + BC - 1 > q0) || (k0 + BC > T)) {
#pragma unroll
                for (int c = 0; c < BC; ++c)
                    if (k0 + c > row || k0 + c >= T) sr[c >> 5][c & 31] = __float_as_uint(-1e30f);
            }
            float mx4[4] = {-1e30f, -1e30f, -1e30f, -1e30f};
#pragma unroll
            for (int c = 0; c < BC; c += 2)
                mx4[(c >> 1) & 3] = max3(mx4[(c >> 1) & 3], __uint_as_float(sr[c >> 5][c & 31]), __uint_as_float(sr[(c + 1) >> 5][(c + 1) & 31]));
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2e;  // scale > 0
            // the reference follows the maximum only when that has grown by more than 2^8
            const bool grow = g > 0 && mx > before + RESCALE_LOG2;
            const float m_used = g > 0 && !grow ? before : mx, factor = grow ? exp2f(before - mx) : 1.0f;
            mref[grp * 128 + r] = m_used;
            __syncwarp();
            if (lane == 0) khq::mbar_arrive(&bars[B_MREF + 4 * grp + quarter]);
            if (__any_sync(0xFFFFFFFFu, grow)) {
                // O may only be touched between P V of the previous tile and P V of this one.  The
                // completion barriers alternate between two mbarriers so that a thread may skip
                // phases: barrier (g-1)&1 last completed for tile g-3 (certainly, since Q K^T of
                // this tile was issued behind P V of tile g-2) and cannot complete for tile g+1
                // before this thread's own arrival for tile g.
                ok = __all_sync(0xFFFFFFFFu, khq::mbar_wait_bounded(&bars[B_PVDONE + ((g - 1) & 1)],
                                                                  (uint32_t)(((g - 1) >> 1) & 1), status));
                if (!ok) break;
                tc_fence_after();
#pragma unroll 1
                for (int c0 = 0; c0 < D; c0 += 16) {
                    uint32_t orr[16];
                    tmem_ld16(lane_base + TM_O + c0, orr);
                    tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 16; ++q) orr[q] = __float_as_uint(__uint_as_float(orr[q]) * factor);
                    tmem_st16(lane_base + TM_O + c0, orr);
                }
            }
            // p = 2^(s*scale - m): one fused multiply-add and one ex2 per score; P (16-bit pairs) over the S buffer it came from, in
            // two halves of 64 keys that the MMA thread takes as they come
            float rs[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const float neg_m = -m_used;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t pk[32];
#pragma unroll
                for (int c = 0; c < 64; c += 2) {
                    const uint32_t* sc = &sr[2 * h + (c >> 5)][c & 31];
                    float x0, x1;
                    fma2(x0, x1, __uint_as_float(sc[0]), __uint_as_float(sc[1]), scale_log2e, neg_m);
                    const float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
                    add2(rs[c & 2], rs[(c & 2) + 1], p0, p1);
                    pk[c >> 1] = pack2<BF16>(p0, p1);
                }
                tmem_st32(s_addr + h * 32, pk);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_leader(&bars[B_PREADY + 2 * grp + h]);
            }
            l_run = (m_l == m_used ? l_run : l_run * exp2f(m_l - m_used)) + ((rs[0] + rs[1]) + (rs[2] + rs[3]));
            m_l = m_used;
        }
        // ---- epilogue -----------------------------------------------------------------------------
        // Pieces of 64 columns, 32 per thread.  Gates and outputs pass through shared memory (128-byte swizzle, free of bank conflicts) and
        // TMA: a thread owns a row, so its own global accesses would take a line each.
        const auto chunk = [&](int c, int q) { return reinterpret_cast<uint4*>(smem + off_piece(c) + r * 128 + (((grp * 4 + q) ^ (r & 7)) << 4)); };
        const auto sigmoids = [&](int c, float (&s)[32]) {
            if (ok) ok = __all_sync(0xFFFFFFFFu, khq::mbar_wait_bounded(&bars[B_GFULL + c], 0u, status));
            if (!ok) return;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 v = *chunk(c, q);
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = unpack2<BF16>(w[e]);
                    s[8 * q + 2 * e] = sigmoid(f.x);
                    s[8 * q + 2 * e + 1] = sigmoid(f.y);
                }
            }
        };
        float sg[2][32];  // the first two pieces while the last P V runs
#pragma unroll
        for (int c = 0; c < 2; ++c) sigmoids(c, sg[c]);
        // the last tile's reference, then both groups' sums against it
        if (ok && grp != (last & 1))
            ok = khq::mbar_wait_bounded(&bars[B_MREF + 4 * (last & 1) + quarter], (uint32_t)((last >> 1) & 1), status);
        const float m_end = mref[(last & 1) * 128 + r];
        l_run = m_l == m_end ? l_run : l_run * exp2f(m_l - m_end);
        lsum[grp * 128 + r] = l_run;
        __syncwarp();
        if (lane == 0) khq::mbar_arrive(&bars[B_LSUM + quarter]);
        if (ok) ok = khq::mbar_wait_bounded(&bars[B_LSUM + quarter], 0u, status);
        if (ok) l_run += lsum[(grp ^ 1) * 128 + r];
        if (ok) ok = khq::mbar_wait_bounded(&bars[B_PVDONE + (last & 1)], (uint32_t)((last >> 1) & 1), status);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (ok) {
            tc_fence_after();
            const float inv = 1.0f / (l_run + 1e-9f);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t o[32];
                tmem_ld32(lane_base + TM_O + c * 64 + grp * 32, o);
                float late[32];
                if (c >= 2) sigmoids(c, late);
                tmem_ld_wait();
                const float (&s)[32] = c < 2 ? sg[c < 2 ? c : 0] : late;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        w[e] = pack2<BF16>(__uint_as_float(o[8 * q + 2 * e]) * inv * s[8 * q + 2 * e],
                                           __uint_as_float(o[8 * q + 2 * e + 1]) * inv * s[8 * q + 2 * e + 1]);
                    *chunk(c, q) = make_uint4(w[0], w[1], w[2], w[3]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) khq::mbar_arrive(&bars[B_OUT + c]);
            }
        }
    }
    // ---- teardown: every thread arrives here, with or without a failed wait ----------------------
    tc_fence_before();
    __syncwarp();
    cluster_arrive();
    cluster_wait();  // no CTA leaves while the other's loads, products or arrivals concern it
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(*tmem_slot), "n"(TM_COLS) : "memory");
}

}  // namespace pair
}  // namespace khq_prefill5
