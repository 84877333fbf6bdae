// khq_prefill_tc5.cu -- causal GQA prefill attention with sigmoid output gate on the fifth
// generation tensor cores (tcgen05.mma, accumulators in tensor memory, operands staged by TMA).
//
// Same math and the same tensors as the warp-level kernel in khq_prefill.cu (the reference's
// fp16-KV attention, src/kernels/elementwise_sm75.mojo:1140-1231, applied to all prompt rows at
// once): out[t,h,:] = softmax_{u<=t}(q[t,h].K[u,h/6]*scale) V[u,h/6] * sigmoid(gate[t,h,:]).
//
// A work item = 128 query rows of one query head; key tiles of 128.  A CTA works through one item
// (long prompts: one CTA per item, left to the hardware scheduler) or through several (short
// prompts: one persistent CTA per SM; the producers and the MMA thread then run ahead into the
// next item while the softmax warps finish the epilogue of the current one).  Twelve warps:
//   warps 0-7  softmax, two threads per query row (warp w and warp w+4 share the tensor-memory
//              lane quarter w%4 and a scheduler): a row's S and O live in tensor-memory lane i,
//              so there are no shuffles; the two threads of a row take 64 keys of a tile each
//              and swap their half maxima (and, at the end, half sums) through shared memory.
//              Per tile a thread reads 64 S columns with tcgen05.ld and writes P (fp16 pairs, 32
//              columns) back over the S buffer with tcgen05.st; O is rescaled lazily (only when
//              the running max grew by more than 2^8); the epilogue normalises and gates.
//   warp 11    brings the gates into shared memory in pieces and stores the outputs that take their
//              place (a softmax thread owns a row: its own global accesses would cost a line each,
//              16 000 of the 45 000 cycles of an item of 11 tiles; 9 x 1531 rows 386 -> 373 us,
//              32 x 512: 290 -> 270).
//   warps 8,10 producers: one thread each issues the TMA loads of Q and the K tiles (warp 8, a
//              K tile in two halves of 128 head dims, each released as soon as the Q K^T steps
//              that read it have completed) and of the V tiles (warp 10, two halves of 64 keys,
//              each released when the P V steps that read it have completed).
//   warp 9     MMA: one lane issues S = Q K^T (M128 N128 K256, A = Q from shared memory) for
//              tile j+1, then O += P V (M128 N256 K128, A = P from tensor memory) for tile j;
//              tcgen05.commit signals the mbarriers.
// Tensor memory columns: O [0,256), S/P ping [256,384), S/P pong [384,512).  An A operand in
// tensor memory is row = lane, 16 consecutive K elements = 8 columns of fp16 pairs.
// Why these shapes: back to back the pipe takes 64 cycles for a Q K^T step (N 128) and 128 for a P V step (N 256); 64-key tiles
// would issue twice the instructions for the same work.  Tensor memory (512 columns) holds O plus two 128-key S buffers, which
// leaves no room for Q, so Q stays in shared memory.
// Prompts of many row blocks go to CTA pairs instead (khq_prefill_pair.cuh); this kernel has the short ones, where a row's two
// threads shorten the chain of the few tiles of an item, and odd numbers of query heads per kv head.
//
// Shared-memory operand layout: the 128-byte-swizzle canonical layouts.  A 5-D tensor map
// {64 halfs, row, 64-column group, head, batch} with 128-byte swizzle makes TMA write a
// (rows x 256) tile as sub-tiles [group][row][128 bytes], 16-byte chunk c of row r at
// r*128 + ((c ^ (r & 7)) << 4).  Descriptors over it:
//   K-major  (Q, K): stride-dim byte offset (between 8-row groups) = 1024; a K step of 16 halfs
//                 advances the start address by 32 bytes inside a group, then to the next group;
//   MN-major (V as the B operand of P V, keys are the contraction dim): leading-dim byte offset
//                 (between 64-column groups) = rows*128, stride-dim byte offset (between 8-key
//                 groups) = 1024; a K step of 16 keys advances the start address by 2048 bytes.
// Every wait is bounded; a wait that runs out sets a status word the host can read and the CTA
// falls through to the teardown (tensor memory is always released).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include "khq_common.cuh"
#include "khq_launch.cuh"

namespace khq_prefill5 {

using khq::smem_u32;

constexpr int D = 256;
constexpr int BR = 128;     // query rows per CTA
constexpr int BC = 128;     // keys per tile
constexpr int NSOFT = 256;  // softmax threads: two per query row, 64 of a tile's 128 keys each
constexpr int NTHREADS = NSOFT + 128;
constexpr int Q_BYTES = BR * D * 2;        // 64 KB
constexpr int KHALF_BYTES = BC * 128 * 2;  // 32 KB: 128 keys x 128 head dims (two 64-dim groups)
constexpr int VHALF_BYTES = 64 * D * 2;    // 32 KB: 64 keys x 256 head dims (four 64-dim groups)
constexpr int OFF_Q = 0;
constexpr int OFF_K = OFF_Q + Q_BYTES;
constexpr int OFF_V = OFF_K + 2 * KHALF_BYTES;
constexpr int STG_BYTES = BR * 64 * 2;     // gate / output piece: 128 rows x 64 columns
constexpr int OFF_STG = OFF_V + 2 * VHALF_BYTES;
constexpr int OFF_XCHG = OFF_STG + 2 * STG_BYTES;  // float [2 parities][2 halves][128 rows]
constexpr int OFF_BARS = OFF_XCHG + 2 * 2 * 128 * 4;
constexpr int SMEM_BYTES = OFF_BARS + 256;
constexpr uint32_t TM_COLS = 512, TM_O = 0, TM_S = 256;
// Up to half a row tile the epilogue reads gates and writes outputs straight from and to global memory: its lines (one per thread)
// are few then, and the pieces through shared memory one after the other take longer (one prompt of 57 rows: 10.3 us against
// 11.2; of 128 rows 12.8 against 11.4).
constexpr int DIRECT_MAX_T = BR / 2;
constexpr float RESCALE_LOG2 = 8.0f;

enum Bar {
    B_KFULL = 0, B_VFULL = 2, B_KEMPTY = 4, B_VEMPTY = 6, B_SFULL = 8, B_QFULL = 10, B_PREADY = 11, B_PVDONE = 12,
    B_XCHG = 14, B_QEMPTY = 18, B_OFREE = 19, B_PREADY2 = 20, B_GFULL = 21, B_OUT = 23,
    B_COUNT = 25
};
static_assert(B_COUNT * 8 <= 240, "barriers overlap the tensor-memory slot");

__device__ int g_prefill_status = 0;

// ---- descriptors ---------------------------------------------------------------------------------
// Shared-memory matrix descriptor (64 bits): start address, leading and stride byte offsets (all in
// 16-byte units; bits 0-13, 16-29, 32-45), descriptor version 1 in bits 46-47, layout type 2
// (128-byte swizzle) in bits 61-63.  It is assembled from a low and a high word, see desc_lo/desc_hi.
// Instruction descriptor for kind::f16: fp32 accumulate, fp16 A and B, A K-major, M = 128 (256: a CTA pair).
// (A/B format field: 0 = fp16, 1 = bf16, bits 7-9 and 10-12.)
__host__ __device__ constexpr uint32_t instr_desc(int m, int n, bool b_mn_major, bool bf16) {
    return (1u << 4) | (bf16 ? ((1u << 7) | (1u << 10)) : 0u) | (b_mn_major ? (1u << 16) : 0u) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}
// Two floats -> one 32-bit word of the 16-bit storage type (round to nearest even), and back.
template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    if (BF16) {
        const __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&t);
    }
    const __half2 t = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&t);
}
template <bool BF16>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
    if (BF16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
}

// ---- tcgen05 / TMA wrappers ----------------------------------------------------------------------
// The issuing warp is on the critical path: the 64-bit descriptors are assembled from a
// precomputed low word (start address and leading offset; the caller adds the K-step offset, which
// never carries out of the 14-bit address field) and a constant high word.  umma_ss: A and B from
// shared memory; umma_ts: A from tensor memory (row = lane, fp16 pairs, 8 columns per K step of 16).
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr, uint32_t lbo) {
    return ((addr & 0x3FFFFu) >> 4) | (((lbo >> 4) & 0x3FFFu) << 16);
}
__host__ __device__ constexpr uint32_t desc_hi(uint32_t sbo) {
    return ((sbo >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);  // version 1 (bit 46), 128-byte swizzle (bits 61-63)
}
// All lanes of the MMA warp call these and one of them issues (`one`): the operands are then values of the whole warp, which the
// compiler keeps and steps in uniform registers (see khq_prefill_pair.cuh).
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(r));
    return r;
}
template <int ACC>
__device__ __forceinline__ void umma_ss(uint32_t one, uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                        uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .b64 da, db;\n\t.reg .pred p, q;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "setp.ne.u32 p, %6, 0;\n\tsetp.ne.u32 q, %7, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "n"(ACC), "r"(one)
        : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t one, uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .b64 db;\n\t.reg .pred p, q;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.u32 p, %5, 0;\n\tsetp.ne.u32 q, %6, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(one)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t one, uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)), "r"(one)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
        "%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 1 / (1 + e^-x): four instructions, two of them approximations of 2^-22 relative error; subnormal terms are below the sum's rounding
// (and below 2^-126 of the result).
__device__ __forceinline__ float sigmoid(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(1.0f + ex2_approx(x * -1.4426950408889634f)));
    return y;
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
        "%29,%30,%31};" ::"r"(r[0]),
        "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
        "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
        "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// A piece of the gates to L2; a piece of the outputs from shared memory.
__device__ __forceinline__ void tma_prefetch_5d(const CUtensorMap* map, int c1, int c2, int c3, int c4) {
    asm volatile("cp.async.bulk.prefetch.tensor.5d.L2.global.tile [%0, {%1, %2, %3, %4, %5}];" ::"l"(reinterpret_cast<uint64_t>(map)),
                 "r"(0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
                 : "memory");
}
__device__ __forceinline__ void tma_store_5d(const CUtensorMap* map, uint32_t src, int c1, int c2, int c3, int c4) {
    asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(src), "r"(0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// One 5-D tiled TMA load of a single CTA; coordinate 0 is always 0, so the 16-byte rule holds.
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int c1, int c2,
                                            int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, "
        "%6, %7}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}

// Bounded wait on up to three barriers at once.  A satisfied mbarrier wait still costs a ~250-cycle
// round trip, so the MMA warp polls the barriers of a step together (the polls overlap) instead
// of one after the other; a barrier found complete stays "done" (its next phase cannot complete
// before this thread moves on).
__device__ __forceinline__ uint32_t mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok;
}
// Waits of a whole warp: all lanes go on together.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, int* status) {
    for (uint32_t it = 0; it < (1u << 22); ++it)
        if (__any_sync(0xFFFFFFFFu, khq::mbar_try_wait(bar, parity))) return true;
    atomicExch(status, 1);
    return false;
}
template <int N>
__device__ __forceinline__ bool mbar_wait_all_bounded(uint64_t* const (&bar)[N], const uint32_t (&parity)[N], int* status) {
    uint32_t done = 0;
    for (uint32_t it = 0; it < (1u << 22); ++it) {
        uint32_t got[N];
#pragma unroll
        for (int i = 0; i < N; ++i) got[i] = mbar_test(bar[i], parity[i]);
#pragma unroll
        for (int i = 0; i < N; ++i) done |= (uint32_t)__any_sync(0xFFFFFFFFu, got[i]) << i;
        if (done == (1u << N) - 1u) return true;
        bool parked = false;  // park (a blocking try_wait) on the first barrier that is still open
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (!parked && !((done >> i) & 1u)) {
                if (__any_sync(0xFFFFFFFFu, khq::mbar_try_wait(bar[i], parity[i]))) done |= 1u << i;
                parked = true;
            }
        if (done == (1u << N) - 1u) return true;
    }
    atomicExch(status, 1);
    return false;
}

// Eight columns: O normalised, times the sigmoids of the gates g, as 16-bit values.
template <bool BF16>
__device__ __forceinline__ uint4 gated(const uint32_t* o, float inv, const uint4& g) {
    const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
    uint32_t ow[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 gf = unpack2<BF16>(gw[e]);
        ow[e] = pack2<BF16>(__uint_as_float(o[2 * e]) * inv * sigmoid(gf.x), __uint_as_float(o[2 * e + 1]) * inv * sigmoid(gf.y));
    }
    return make_uint4(ow[0], ow[1], ow[2], ow[3]);
}

// ---- the kernel ----------------------------------------------------------------------------------
// A work item = 128 query rows of one (batch, head); the last row block attends the most keys.  CTA c
// takes one item per round of `grid` items, the c-th of even rounds and the c-th from the end of odd
// rounds; with one CTA per item there is a single round and the item is the CTA index.
struct Item {
    int q0, h, b, kvh, n_tiles;
};
template <bool PERSIST>
__device__ __forceinline__ bool get_item(int ordinal, int T, int H_q, int H_kv, int batch, int group_major, Item& it) {
    if (!PERSIST && ordinal > 0) return false;  // one item per CTA: the item is the CTA index
    const int nqb = (T + BR - 1) / BR;
    const int per = H_q * batch;
    // boustrophedon over the item list: in odd rounds the CTAs take the items in reverse, so that
    // every CTA's share of the triangular workload stays within one round's spread
    const long long lane_in_round = (ordinal & 1) ? (long long)(gridDim.x - 1 - blockIdx.x) : (long long)blockIdx.x;
    const long long w = lane_in_round + (long long)ordinal * gridDim.x;
    if (w >= (long long)nqb * per) return false;
    int qb;
    if (group_major) {
        // one (batch, kv head) group after the other, heaviest row blocks first inside a group:
        // the CTAs in flight then stream the K/V rows of one or two groups, which stay in L2
        const int n_rep = H_q / H_kv, per_group = n_rep * nqb;
        const int grp = (int)(w / per_group), idx = (int)(w % per_group);
        qb = nqb - 1 - idx / n_rep;
        it.b = grp / H_kv;
        it.kvh = grp % H_kv;
        it.h = it.kvh * n_rep + idx % n_rep;
    } else {
        // heaviest first over everything: consecutive items have (almost) the same size
        qb = nqb - 1 - (int)(w / per);
        const int rem = (int)(w % per);
        it.h = rem % H_q;
        it.b = rem / H_q;
        it.kvh = it.h / (H_q / H_kv);
    }
    it.q0 = qb * BR;
    it.n_tiles = min((T + BC - 1) / BC, qb + 1);  // causal: key tiles 0..qb (BR == BC)
    return true;
}

// grid = min(items, SMs) persistent CTAs for short prompts, one CTA per item for long ones (the
// launcher decides; a CTA simply works through the items its index selects).  q_gate (B, T, H_q, 2D), out (B, T, H_q, D); Q, K and V
// operands come through their tensor maps.  Per-tile barriers are indexed by g, the running count of
// tiles this CTA has processed over all its items, so that the producers and the MMA thread run
// ahead into the next item while the softmax warps are still in the epilogue of the current one.
template <bool PERSIST, bool BF16>
__global__ void __launch_bounds__(NTHREADS, 1)
khq_gqa_prefill_tc5_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                           const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_g,
                           const __grid_constant__ CUtensorMap tm_o, const __half* __restrict__ q_gate,
                           __half* __restrict__ out, long long q_bs, long long o_bs, int T, int H_q, int H_kv, int batch, int group_major,
                           float scale_log2e) {
    const bool direct = !PERSIST && T <= DIRECT_MAX_T;  // gates and outputs without shared memory
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BARS);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_BARS + 240);
    float* xchg = reinterpret_cast<float*>(smem + OFF_XCHG);
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    int* status = &g_prefill_status;
    if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled layouts need a 1024-byte aligned base
        if (tid == 0) atomicExch(status, 2);
        return;
    }

    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            khq::mbar_init(&bars[B_KFULL + s], 1);
            khq::mbar_init(&bars[B_VFULL + s], 1);
            khq::mbar_init(&bars[B_KEMPTY + s], 1);
            khq::mbar_init(&bars[B_VEMPTY + s], 1);
            khq::mbar_init(&bars[B_SFULL + s], 1);
            khq::mbar_init(&bars[B_PVDONE + s], 1);
        }
        khq::mbar_init(&bars[B_QFULL], 1);
        khq::mbar_init(&bars[B_QEMPTY], 1);
        // one elected arrival per softmax warp: 256 separate arrivals on one barrier serialise
        // Two "P ready" barriers, used alternately: a softmax warp may finish tile g+1 (its S is
        // computed ahead) before a slower warp has arrived for tile g, and its arrival must not be
        // counted for tile g.  It cannot get two tiles ahead: S of tile g+2 is issued after tile g's
        // barrier has completed.
        khq::mbar_init(&bars[B_PREADY], NSOFT / 32);
        khq::mbar_init(&bars[B_PREADY2], NSOFT / 32);
        khq::mbar_init(&bars[B_OFREE], NSOFT / 32);
        for (int q = 0; q < 2; ++q) {
            khq::mbar_init(&bars[B_GFULL + q], 1);
            khq::mbar_init(&bars[B_OUT + q], NSOFT / 32);
        }
        for (int q = 0; q < 4; ++q) khq::mbar_init(&bars[B_XCHG + q], 2);  // the two warps of a lane quarter
        khq::fence_barrier_init();
    }
    // Everything above overlaps the kernel before; tensor memory is only taken once that kernel has finished (it may still have
    // to allocate its own on this SM).
    khq::pdl_wait();
    khq::pdl_trigger();
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "n"(TM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);
    const uint32_t sbase = smem_u32(smem);

    if (warp == 8) {
        // ================================ producer of Q and K ======================================
        // K tile = two halves by head dim (groups 0-1 and 2-3), each [2 groups][128 keys][128 B].
        // The Q buffer is reloaded for the next item once the MMA thread has committed the last
        // Q K^T of the current one.
        if (lane == 0) {
            int g = 0, items = 0, halves = 0;
            bool ok = true;
            Item it;
            for (int i = 0; ok && get_item<PERSIST>(i, T, H_q, H_kv, batch, group_major, it); ++i) {
                if (i > 0 && !khq::mbar_wait_bounded(&bars[B_QEMPTY], (uint32_t)((i - 1) & 1), status)) break;
                khq::mbar_arrive_expect_tx(&bars[B_QFULL], Q_BYTES);
                tma_load_5d(sbase + OFF_Q, &tm_q, &bars[B_QFULL], it.q0, 0, it.h, it.b);
                items = i + 1;
                for (int j = 0; ok && j < it.n_tiles; ++j, ++g) {
                    for (int hf = 0; hf < 2; ++hf) {
                        if (g >= 1 && !khq::mbar_wait_bounded(&bars[B_KEMPTY + hf], (uint32_t)((g - 1) & 1), status)) {
                            ok = false;
                            break;
                        }
                        khq::mbar_arrive_expect_tx(&bars[B_KFULL + hf], KHALF_BYTES);
                        tma_load_5d(sbase + OFF_K + hf * KHALF_BYTES, &tm_k, &bars[B_KFULL + hf], j * BC, 2 * hf, it.kvh, it.b);
                        halves = 2 * g + hf + 1;
                    }
                }
            }
            // nothing this thread started may still be in flight when the CTA leaves
            if (items > 0) khq::mbar_wait_bounded(&bars[B_QFULL], (uint32_t)((items - 1) & 1), status);
            for (int i = max(0, halves - 2); i < halves; ++i)
                khq::mbar_wait_bounded(&bars[B_KFULL + (i & 1)], (uint32_t)((i >> 1) & 1), status);
        }
    } else if (warp == 10) {
        // ================================ producer of V ============================================
        // V tile = two halves by key (64 keys each), each [4 groups][64 keys][128 B].
        if (lane == 0) {
            int g = 0, halves = 0;
            bool ok = true;
            Item it;
            for (int i = 0; ok && get_item<PERSIST>(i, T, H_q, H_kv, batch, group_major, it); ++i) {
                for (int j = 0; ok && j < it.n_tiles; ++j, ++g) {
                    for (int hf = 0; hf < 2; ++hf) {
                        if (g >= 1 && !khq::mbar_wait_bounded(&bars[B_VEMPTY + hf], (uint32_t)((g - 1) & 1), status)) {
                            ok = false;
                            break;
                        }
                        khq::mbar_arrive_expect_tx(&bars[B_VFULL + hf], VHALF_BYTES);
                        tma_load_5d(sbase + OFF_V + hf * VHALF_BYTES, &tm_v, &bars[B_VFULL + hf], j * BC + hf * 64, 0, it.kvh,
                                    it.b);
                        halves = 2 * g + hf + 1;
                    }
                }
            }
            for (int i = max(0, halves - 2); i < halves; ++i)
                khq::mbar_wait_bounded(&bars[B_VFULL + (i & 1)], (uint32_t)((i >> 1) & 1), status);
        }
    } else if (warp == 9) {
        // ================================ MMA issuer ==============================================
        {
            const uint32_t one = elect_one();
            constexpr uint32_t IDESC_S = instr_desc(BR, BC, false, BF16);
            constexpr uint32_t IDESC_O = instr_desc(BR, D, true, BF16);
            constexpr uint32_t HI_K = desc_hi(1024);  // Q, K (K-major) and V (MN-major): 1024 bytes between 8-row groups
            const uint32_t q_lo = desc_lo(sbase + OFF_Q, 16), k_lo = desc_lo(sbase + OFF_K, 16);
            const uint32_t v_lo = desc_lo(sbase + OFF_V, 64 * 128);  // leading offset: the next 64-column group
            bool ok = true;
            auto issue_qk = [&](int g) {  // S[g & 1] = Q K^T of the tile with running index g
                const uint32_t s_tmem = tmem + TM_S + (uint32_t)(g & 1) * BC;
                uint64_t* const kb[2] = {&bars[B_KFULL], &bars[B_KFULL + 1]};
                const uint32_t kp[2] = {(uint32_t)(g & 1), (uint32_t)(g & 1)};
                ok = ok && mbar_wait_all_bounded(kb, kp, status);
                if (!ok) return;
                tc_fence_after();
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk) {
                        const int ks = hf * 8 + kk;
                        // byte offsets / 16: next 64-dim group = rows*128 bytes, next K step = 32 bytes
                        const uint32_t oa = (uint32_t)((ks >> 2) * (BR * 128) + (ks & 3) * 32) >> 4;
                        const uint32_t ob = (uint32_t)(hf * KHALF_BYTES + (kk >> 2) * (BC * 128) + (kk & 3) * 32) >> 4;
                        if (ks == 0) umma_ss<0>(one, s_tmem, q_lo + oa, HI_K, k_lo + ob, HI_K, IDESC_S);
                        else umma_ss<1>(one, s_tmem, q_lo + oa, HI_K, k_lo + ob, HI_K, IDESC_S);
                    }
                    umma_commit(one, &bars[B_KEMPTY + hf]);
                }
                umma_commit(one, &bars[B_SFULL + (g & 1)]);
            };
            Item it, nx;
            bool have = get_item<PERSIST>(0, T, H_q, H_kv, batch, group_major, it);
            int g = 0;
            if (have) {
                ok = warp_wait(&bars[B_QFULL], 0u, status);
                if (ok) issue_qk(0);
                if (PERSIST && ok && it.n_tiles == 1) umma_commit(one, &bars[B_QEMPTY]);
            }
            for (int i = 0; have && ok; ++i) {
                const bool have_nx = get_item<PERSIST>(i + 1, T, H_q, H_kv, batch, group_major, nx);
                for (int j = 0; ok && j < it.n_tiles; ++j, ++g) {
                    // run ahead: Q K^T of the next tile, which may be the first tile of the next item
                    const bool same_item = j + 1 < it.n_tiles;
                    if (same_item || have_nx) {
                        if (!same_item) ok = warp_wait(&bars[B_QFULL], (uint32_t)((i + 1) & 1), status);
                        if (ok) issue_qk(g + 1);
                        // once the last Q K^T of an item is out, its Q buffer may be reloaded
                        const bool last_qk = same_item ? (j + 2 == it.n_tiles) : (nx.n_tiles == 1);
                        if (PERSIST && ok && last_qk) umma_commit(one, &bars[B_QEMPTY]);
                    }
                    if (!ok) break;
                    uint64_t* const pb[3] = {&bars[(g & 1) ? B_PREADY2 : B_PREADY], &bars[B_VFULL], &bars[B_VFULL + 1]};
                    const uint32_t pp[3] = {(uint32_t)((g >> 1) & 1), (uint32_t)(g & 1), (uint32_t)(g & 1)};
                    ok = mbar_wait_all_bounded(pb, pp, status);
                    // the first P V of an item overwrites O: the previous item's epilogue must have read it
                    if (PERSIST && ok && j == 0 && i > 0)
                        ok = warp_wait(&bars[B_OFREE], (uint32_t)((i - 1) & 1), status);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t p_tmem = tmem + TM_S + (uint32_t)(g & 1) * BC;
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            const uint32_t ob = (uint32_t)(hf * VHALF_BYTES + kk * 2048) >> 4;  // 16 keys = 2048 bytes
                            umma_ts(one, tmem + TM_O, p_tmem + (hf * 4 + kk) * 8, v_lo + ob, HI_K, IDESC_O,
                                    (hf > 0 || kk > 0) ? 1u : (uint32_t)(j > 0));
                        }
                        if (hf == 1) umma_commit(one, &bars[B_PVDONE + (g & 1)]);
                        umma_commit(one, &bars[B_VEMPTY + hf]);
                    }
                }
                it = nx;
                have = have_nx;
            }
        }
    } else if (warp == 11) {
        // ================================ gates in, outputs out =====================================
        // Four pieces of 64 columns per item through two buffers: the gates of a piece come in, the softmax warps overwrite them
        // with the outputs, the piece is stored and the buffer takes the piece after the next (of the next item, too).
        if (lane == 0 && !direct) {
            Item in, st;
            int i_in = 0, c_in = 0, loads = 0, n = 0;
            bool more = get_item<PERSIST>(0, T, H_q, H_kv, batch, group_major, in), ok = true;
            const auto load_next = [&]() {
                if (!more) return;
                const int b = loads & 1;
                khq::mbar_arrive_expect_tx(&bars[B_GFULL + b], STG_BYTES);
                tma_load_5d(sbase + OFF_STG + b * STG_BYTES, &tm_g, &bars[B_GFULL + b], in.q0, c_in, in.h, in.b);
                if (c_in < 2) tma_prefetch_5d(&tm_g, in.q0, c_in + 2, in.h, in.b);
                ++loads;
                if (++c_in == 4) {
                    c_in = 0;
                    more = get_item<PERSIST>(++i_in, T, H_q, H_kv, batch, group_major, in);
                }
            };
            load_next();
            load_next();
            for (int i = 0; ok && get_item<PERSIST>(i, T, H_q, H_kv, batch, group_major, st); ++i) {
                for (int c = 0; c < 4; ++c, ++n) {
                    ok = khq::mbar_wait_bounded(&bars[B_OUT + (n & 1)], (uint32_t)((n >> 1) & 1), status);
                    if (!ok) break;
                    tma_store_5d(&tm_o, sbase + OFF_STG + (n & 1) * STG_BYTES, st.q0, c, st.h, st.b);
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    load_next();
                }
            }
            // nothing this thread started may still be in flight when the CTA leaves
            for (int k = max(0, loads - 2); k < loads; ++k)
                khq::mbar_wait_bounded(&bars[B_GFULL + (k & 1)], (uint32_t)((k >> 1) & 1), status);
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
    } else {
        // ================================ softmax + epilogue ======================================
        // Two threads per query row: half 0 (warps 0-3) takes keys 0-63 of a tile and columns 0-127
        // of O, half 1 (warps 4-7) keys 64-127 and columns 128-255.  Both warps of a row sit on the
        // same tensor-memory lane quarter (warp % 4) and on the same scheduler.
        const int half = warp >> 2, r = tid & 127;
        const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        uint64_t* xbar = &bars[B_XCHG + (warp & 3)];
        int g = 0, x = 0, n = 0;  // running tile index; running phase of the exchange barrier; running epilogue piece
        bool ok = true;
        Item it;
        for (int i = 0; ok && get_item<PERSIST>(i, T, H_q, H_kv, batch, group_major, it); ++i) {
            const int q0 = it.q0, row = q0 + r;
            float m_used = -1e30f, l_run = 0.0f;
            for (int j = 0; j < it.n_tiles; ++j, ++g, ++x) {
                ok = __all_sync(0xFFFFFFFFu, khq::mbar_wait_bounded(&bars[B_SFULL + (g & 1)], (uint32_t)((g >> 1) & 1), status));
                if (!ok) break;
                tc_fence_after();
                const uint32_t s_addr = lane_base + TM_S + (uint32_t)(g & 1) * BC;
                uint32_t sr[2][32];
                tmem_ld32(s_addr + half * 64, sr[0]);
                tmem_ld32(s_addr + half * 64 + 32, sr[1]);
                tmem_ld_wait();
                const int k0 = j * BC + half * 64;
                // raw scores; masked entries (key after the row, or past the prompt) become -inf-like
                if ((k0 + 63 > q0) || (k0 + 64 > T)) {
#pragma unroll
                    for (int c = 0; c < 64; ++c)
                        if (k0 + c > row || k0 + c >= T) sr[c >> 5][c & 31] = __float_as_uint(-1e30f);
                }
                float mx4[4] = {-1e30f, -1e30f, -1e30f, -1e30f};
#pragma unroll
                for (int c = 0; c < 64; ++c) mx4[c & 3] = fmaxf(mx4[c & 3], __uint_as_float(sr[c >> 5][c & 31]));
                float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                // the row maximum over all 128 keys: swap half maxima with the partner thread
                xchg[((x & 1) * 2 + half) * 128 + r] = mx;
                __syncwarp();
                if (lane == 0) khq::mbar_arrive(xbar);
                ok = __all_sync(0xFFFFFFFFu, khq::mbar_wait_bounded(xbar, (uint32_t)(x & 1), status));
                if (!ok) break;
                mx = fmaxf(mx, xchg[((x & 1) * 2 + (half ^ 1)) * 128 + r]) * scale_log2e;  // scale > 0
                float factor = 1.0f;
                bool grow = false;
                if (j == 0) {
                    m_used = mx;
                } else if (mx > m_used + RESCALE_LOG2) {
                    factor = exp2f(m_used - mx);
                    m_used = mx;
                    grow = true;
                }
                // p = 2^(s*scale - m): one fused multiply-add and one ex2 per score
                float rs4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                uint32_t pk[32];
                const float neg_m = -m_used;
#pragma unroll
                for (int c = 0; c < 64; c += 2) {
                    const float p0 = ex2_approx(fmaf(__uint_as_float(sr[c >> 5][c & 31]), scale_log2e, neg_m));
                    const float p1 = ex2_approx(fmaf(__uint_as_float(sr[(c + 1) >> 5][(c + 1) & 31]), scale_log2e, neg_m));
                    rs4[(c >> 1) & 3] += p0 + p1;
                    pk[c >> 1] = pack2<BF16>(p0, p1);
                }
                const float rs = (rs4[0] + rs4[1]) + (rs4[2] + rs4[3]);
                l_run = l_run * factor + rs;
                if (j > 0 && __any_sync(0xFFFFFFFFu, grow)) {
                    // O may only be touched between P V of the previous tile and P V of this one.  The
                    // completion barriers alternate between two mbarriers so that a thread may skip
                    // phases: barrier (g-1)&1 last completed for tile g-3 (certainly, since Q K^T of
                    // this tile was issued behind P V of tile g-2) and cannot complete for tile g+1
                    // before this thread's own arrival for that tile.
                    ok = __all_sync(0xFFFFFFFFu, khq::mbar_wait_bounded(&bars[B_PVDONE + ((g - 1) & 1)],
                                                                      (uint32_t)(((g - 1) >> 1) & 1), status));
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll 1
                    for (int c0 = half * 128; c0 < half * 128 + 128; c0 += 32) {
                        uint32_t orr[32];
                        tmem_ld32(lane_base + TM_O + c0, orr);
                        tmem_ld_wait();
#pragma unroll
                        for (int q = 0; q < 32; ++q) orr[q] = __float_as_uint(__uint_as_float(orr[q]) * factor);
                        tmem_st32(lane_base + TM_O + c0, orr);
                    }
                }
                // P (fp16 pairs) over the S buffer it came from: keys 64*half.. -> columns 32*half..
                // (the partner has read its S columns: it passed the exchange barrier after its load)
                tmem_st32(s_addr + half * 32, pk);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) khq::mbar_arrive(&bars[(g & 1) ? B_PREADY2 : B_PREADY]);
            }
            if (!ok) break;
            // ---- epilogue of the item -------------------------------------------------------------
            const bool live = row < T;
            uint4 g4[PERSIST ? 1 : 16];  // direct: this thread's 128 gate values, all loads ahead of the final waits
            if (!PERSIST && direct && live) {
                const __half* gate = q_gate + it.b * q_bs + (long long)row * H_q * 2 * D + (long long)it.h * 2 * D + D + half * 128;
#pragma unroll
                for (int q = 0; q < (PERSIST ? 1 : 16); ++q) g4[q] = __ldg(reinterpret_cast<const uint4*>(gate) + q);
            }
            // row sum over both halves (one more phase of the exchange barrier)
            xchg[((x & 1) * 2 + half) * 128 + r] = l_run;
            __syncwarp();
            if (lane == 0) khq::mbar_arrive(xbar);
            ok = khq::mbar_wait_bounded(xbar, (uint32_t)(x & 1), status);
            if (ok) l_run += xchg[((x & 1) * 2 + (half ^ 1)) * 128 + r];
            ++x;
            if (ok) ok = khq::mbar_wait_bounded(&bars[B_PVDONE + ((g - 1) & 1)], (uint32_t)(((g - 1) >> 1) & 1), status);
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok) break;
            tc_fence_after();
            const float inv = 1.0f / (l_run + 1e-9f);
            if constexpr (!PERSIST) {
                if (direct) {
                    __half* op = out + it.b * o_bs + (long long)(live ? row : 0) * H_q * D + (long long)it.h * D + half * 128;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint32_t orr[32];
                        tmem_ld32(lane_base + TM_O + half * 128 + c * 32, orr);
                        tmem_ld_wait();
                        if (live) {
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                *reinterpret_cast<uint4*>(op + c * 32 + q * 8) = gated<BF16>(orr + 8 * q, inv, g4[c * 4 + q]);
                        }
                    }
                    break;
                }
            }
            // Pieces of 64 columns, 32 per thread.  Gates and outputs pass through shared memory (128-byte swizzle, free of bank
            // conflicts) and TMA: a thread owns a row, so its own global accesses would take a line each (16 400 cycles per
            // item for 64 KB in and 64 KB out).
#pragma unroll 1
            for (int c = 0; c < 4; ++c, ++n) {
                uint32_t orr[32];
                tmem_ld32(lane_base + TM_O + c * 64 + half * 32, orr);
                ok = __all_sync(0xFFFFFFFFu, khq::mbar_wait_bounded(&bars[B_GFULL + (n & 1)], (uint32_t)((n >> 1) & 1), status));
                tmem_ld_wait();
                if (!ok) break;
                if (PERSIST && c == 3) {  // O has been read: the next item's first P V may overwrite it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) khq::mbar_arrive(&bars[B_OFREE]);
                }
                unsigned char* const prow = smem + OFF_STG + (n & 1) * STG_BYTES + r * 128;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint4* const at = reinterpret_cast<uint4*>(prow + (((half * 4 + q) ^ (r & 7)) << 4));
                    *at = gated<BF16>(orr + 8 * q, inv, *at);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) khq::mbar_arrive(&bars[B_OUT + (n & 1)]);
            }
        }
    }
    // ---- teardown: every thread arrives here, with or without a failed wait ----------------------
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TM_COLS) : "memory");
    }
}

}  // namespace khq_prefill5
#include "khq_prefill_pair.cuh"

// ---- host side -----------------------------------------------------------------------------------
namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// Tensor map over a (batch, T, heads, row_halfs) fp16 tensor that exposes, per (head, batch), a
// T x 256 matrix as {64 halfs, T rows, 4 column groups}; a box is `box_rows` rows x `box_groups`
// column groups of one head.
int make_map(CUtensorMap* map, const void* base, int T, int heads, int batch, long long row_halfs,
             long long head_halfs, long long batch_halfs, int box_rows, int box_groups, bool bf16) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return -107;
    if (batch == 1) batch_halfs = (long long)T * row_halfs;
    const cuuint64_t dims[5] = {64, (cuuint64_t)T, 4, (cuuint64_t)heads, (cuuint64_t)batch};
    const cuuint64_t strides[4] = {(cuuint64_t)row_halfs * 2, 128, (cuuint64_t)head_halfs * 2, (cuuint64_t)batch_halfs * 2};
    const cuuint32_t box[5] = {64, (cuuint32_t)box_rows, (cuuint32_t)box_groups, 1, 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    for (cuuint64_t st : strides)
        if (st % 16 != 0) return -104;
    const CUresult r = fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -108;
}

}  // namespace

static int g_tc5_items_per_cta = 0, g_tc5_pairs = 0;

// 0 = CTA pairs by the size of the prompts, 1 = wherever the heads allow it, 2 = never.
extern "C" int khq_b200_prefill_pairs(int mode) {
    if (mode < 0 || mode > 2) return -100;
    g_tc5_pairs = mode;
    return 0;
}

// 0 = choose by prompt length, 1 = one item per CTA, n > 1 = n items per CTA (a large n gives
// the fully persistent grid).  Returns -100 for a negative value.
extern "C" int khq_b200_prefill_tc5_items_per_cta(int n) {
    if (n < 0) return -100;
    g_tc5_items_per_cta = n;
    return 0;
}

namespace {
// Whether CTA pairs take the items of two neighbouring heads of a kv head together.  From nine row blocks on, below that the chain of an
// item's few tiles counts (T = 1000: 16 prompts 353 us either way, 4 prompts 92.8 against 91.7), and from 2.25 items per SM on, so that
// the epilogue of one item runs beside the tiles of others (T = 1531: one prompt 41.5 us against 39.1, two 85.0 against 85.8, nine
// 355 against 373; one of 2000: 58 against 62; 8 x 2048: 492 against 533; 4 x 8192 in a row, both at the power limit: 2.45 to 2.84 ms
// against 2.65 to 2.97).
// A work distribution of the single-CTA kernel that was asked for (`forced`) asks for that kernel; only khq_b200_prefill_pairs(1) is stronger.
bool use_pair(int row_blocks, long long items, int n_rep, int sms, int forced) {
    if (n_rep % 2 != 0 || g_tc5_pairs == 2) return false;
    return g_tc5_pairs == 1 || (forced == 0 && row_blocks > 8 && 4 * items > 9LL * sms);
}

int launch_tc5(const void* q_gate, const void* k, const void* v, void* out, int batch, int T, int H_q, int H_kv, int d,
               float scale, long long q_batch_stride, long long kv_batch_stride, long long out_batch_stride,
               cudaStream_t stream, bool bf16) {
    using namespace khq_prefill5;
    if (batch <= 0 || T <= 0 || H_q <= 0 || H_kv <= 0) return -100;
    if (d != D || H_q % H_kv != 0) return -103;
    const void* ptrs[] = {q_gate, k, v, out};
    for (const void* p : ptrs)
        if ((reinterpret_cast<uintptr_t>(p) & 15) != 0) return -104;
    if (batch > 1 && ((q_batch_stride | kv_batch_stride | out_batch_stride) & 7) != 0) return -104;
    static bool attr_done[64] = {};
    static int sm_count[64] = {};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return static_cast<int>(err);
    if (dev < 0 || dev >= 64) return -100;
    if (!attr_done[dev]) {
        const void* kernels[4] = {(const void*)khq_gqa_prefill_tc5_kernel<true, false>, (const void*)khq_gqa_prefill_tc5_kernel<false, false>,
                                  (const void*)khq_gqa_prefill_tc5_kernel<true, true>, (const void*)khq_gqa_prefill_tc5_kernel<false, true>};
        for (const void* kf : kernels) {
            err = cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
            if (err != cudaSuccess) return static_cast<int>(err);
        }
        for (const void* kf : {(const void*)pair::khq_gqa_prefill_pair_kernel<false>, (const void*)pair::khq_gqa_prefill_pair_kernel<true>}) {
            err = cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, pair::SMEM);
            if (err != cudaSuccess) return static_cast<int>(err);
        }
        err = cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
        if (err != cudaSuccess) return static_cast<int>(err);
        attr_done[dev] = true;
    }
    const int nqb = (T + BR - 1) / BR;
    const long long items = (long long)nqb * H_q * batch;
    // khq_b200_prefill_tc5_items_per_cta(n) or KHQ_PREFILL_ITEMS_PER_CTA (read once) ask for the kernel without pairs and its mode:
    // 1 = one item per CTA, larger = that many items per CTA (the setter wins; 0 = automatic).
    static int env_forced = -1;
    if (env_forced < 0) {
        const char* e = getenv("KHQ_PREFILL_ITEMS_PER_CTA");
        env_forced = e ? atoi(e) : 0;
        if (env_forced < 0) env_forced = 0;
    }
    const int forced = g_tc5_items_per_cta > 0 ? g_tc5_items_per_cta : env_forced;
    const bool pairs = use_pair(nqb, items, H_q / H_kv, sm_count[dev], forced);
    // The kernel without pairs, for what those leave (short prompts, few items, odd numbers of query heads per kv head).  Short prompts: a
    // persistent grid of one CTA per SM, each working through its items and overlapping one item's epilogue with the next one's first
    // tiles.  Longer ones: one CTA per item, one (batch, kv head) group after the other, heaviest first, which leaves the balancing of
    // the triangular workload to the hardware's dynamic CTA scheduler and runs the leaner instantiation of the kernel.  It wins above
    // 24 row blocks, and above 16 where a CTA has few items to even out its share.  Persistent / one per item, us, 20 query heads on
    // 4 kv heads: 32 x 300: 130 / 168; 4 x 1000: 74 / 82; 8 x 2048: 406 / 408; 2 x 2300: 132 / 136; 1 x 2500: 83 / 77; 1 x 3000:
    // 105 / 97; 4 x 3000: 435 / 411; 1 x 4000: 185 / 170; 4 x 4096: 757 / 716; 2 x 8192: 1413 / 1187.
    long long ctas;  // without pairs
    int group_major = 0;
    if (forced == 1 || (forced == 0 && (nqb > 24 || (nqb > 16 && items <= 16LL * sm_count[dev])))) {
        ctas = items;
        group_major = 1;
    } else if (forced > 1) {
        ctas = (items + forced - 1) / forced;
        if (ctas < sm_count[dev]) ctas = items < sm_count[dev] ? items : sm_count[dev];
    } else {
        ctas = items < sm_count[dev] ? items : sm_count[dev];
    }
    CUtensorMap mq, mk, mv, mg, mo;
    int rc = make_map(&mq, q_gate, T, H_q, batch, (long long)H_q * 2 * D, 2 * D, q_batch_stride, BR, 4, bf16);
    if (rc == 0) rc = make_map(&mk, k, T, H_kv, batch, (long long)H_kv * D, D, kv_batch_stride, pairs ? 64 : BC, pairs ? 4 : 2, bf16);
    if (rc == 0) rc = make_map(&mv, v, T, H_kv, batch, (long long)H_kv * D, D, kv_batch_stride, pairs ? BC : 64, pairs ? 2 : 4, bf16);
    if (!pairs && ctas == items && T <= DIRECT_MAX_T) {  // gates and outputs go without maps, which take the host some time
        mg = mo = mq;
    } else {
        if (rc == 0) rc = make_map(&mg, static_cast<const __half*>(q_gate) + D, T, H_q, batch, (long long)H_q * 2 * D, 2 * D, q_batch_stride, BR, 1, bf16);
        if (rc == 0) rc = make_map(&mo, out, T, H_q, batch, (long long)H_q * D, D, out_batch_stride, BR, 1, bf16);
    }
    if (rc != 0) return rc;
    const float sl2 = scale * 1.4426950408889634f;
    if (pairs) {
        err = khq::launch_pdl(bf16 ? pair::khq_gqa_prefill_pair_kernel<true> : pair::khq_gqa_prefill_pair_kernel<false>, (unsigned)items, 2u, (size_t)pair::SMEM,
                              stream, (unsigned)NTHREADS, mq, mk, mv, mg, mo, T, H_q, H_kv, sl2);
        return (err == cudaSuccess) ? 0 : static_cast<int>(err);
    }
    const unsigned grid = (unsigned)ctas;
    const __half* qp = static_cast<const __half*>(q_gate);  // 16-bit storage; the kernel converts per its type flag
    __half* op = static_cast<__half*>(out);
#define KHQ_TC5_LAUNCH(PERSIST, BF16)                                                                                  \
    err = khq::launch_pdl(khq_gqa_prefill_tc5_kernel<PERSIST, BF16>, grid, 0, SMEM_BYTES, stream, (unsigned)NTHREADS, mq, mk, mv, mg, mo, qp, op, \
                          q_batch_stride, out_batch_stride, T, H_q, H_kv, batch, group_major, sl2)
    if (ctas == items) {
        if (bf16) KHQ_TC5_LAUNCH(false, true);
        else KHQ_TC5_LAUNCH(false, false);
    } else {
        if (bf16) KHQ_TC5_LAUNCH(true, true);
        else KHQ_TC5_LAUNCH(true, false);
    }
#undef KHQ_TC5_LAUNCH
    return (err == cudaSuccess) ? 0 : static_cast<int>(err);
}
}  // namespace

// Same arguments as launch_khq_gqa_prefill_fp16.  Returns -107 when the driver offers no tensor-map
// encoder and -108 when it refuses these shapes.
extern "C" int launch_khq_gqa_prefill_tc5_fp16(const void* q_gate, const void* k, const void* v, void* out, int batch,
                                               int T, int H_q, int H_kv, int d, float scale,
                                               long long q_batch_stride, long long kv_batch_stride,
                                               long long out_batch_stride, cudaStream_t stream) {
    return launch_tc5(q_gate, k, v, out, batch, T, H_q, H_kv, d, scale, q_batch_stride, kv_batch_stride, out_batch_stride,
                      stream, false);
}

// The same attention over bf16 tensors (bf16 operands and P, fp32 accumulation, bf16 output).
extern "C" int launch_khq_gqa_prefill_bf16(const void* q_gate, const void* k, const void* v, void* out, int batch, int T,
                                           int H_q, int H_kv, int d, float scale, long long q_batch_stride,
                                           long long kv_batch_stride, long long out_batch_stride, cudaStream_t stream) {
    return launch_tc5(q_gate, k, v, out, batch, T, H_q, H_kv, d, scale, q_batch_stride, kv_batch_stride, out_batch_stride,
                      stream, true);
}

// Reads and clears the status word of the tcgen05 prefill kernel on the current device
// (synchronises the device): 0 = clean, 1 = a bounded wait ran out, 2 = misaligned shared memory.
extern "C" int khq_b200_prefill_status(void) {
    int st = 0;
    if (cudaMemcpyFromSymbol(&st, khq_prefill5::g_prefill_status, sizeof(int)) != cudaSuccess) return -1;
    if (st != 0) {
        const int zero = 0;
        cudaMemcpyToSymbol(khq_prefill5::g_prefill_status, &zero, sizeof(int));
    }
    return st;
}
