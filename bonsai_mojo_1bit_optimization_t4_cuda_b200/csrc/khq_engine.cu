// khq_engine.cu -- host side of a batch engine's token step: copies, pre-step, compression events and attention of all layers
// issued from one native call.  (From Python the same calls cost about 100 us per layer, more than the GPU needs for them
// below some dozens of sequences.)
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <new>

#include "khq_b200.h"

namespace {
constexpr int HKV = 4, HQ = 24, D = 256, KV = HKV * D, QG = HQ * 2 * D, CHUNK_ROWS = 128 * HKV;
}  // namespace

// Streams and events of one engine: nothing of it is shared with another engine.
struct khq_engine {
    int device;
    cudaStream_t in, out;                       // host -> device and device -> host copies, beside the kernels
    struct Chunk {
        cudaEvent_t ready, done;                // a chunk of layers: inputs landed, outputs computed
    };
    Chunk* chunks;
    int n_chunks;
    cudaEvent_t begin, end, control[2];
    bool control_used[2];
};

extern "C" int khq_b200_engine_destroy(khq_engine* e) {
    if (!e) return -100;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != e->device) cudaSetDevice(e->device);
    // The caller frees the step's buffers behind this call, and no allocator knows of the copies: wait for them.  The output copies
    // follow the step's kernels.  (Relaxed: waiting for these streams does not concern a capture on another one.)
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    for (int i = 0; i < 2; ++i)
        if (e->control_used[i]) cudaEventSynchronize(e->control[i]);
    if (e->in) cudaStreamSynchronize(e->in);
    if (e->out) cudaStreamSynchronize(e->out);
    cudaThreadExchangeStreamCaptureMode(&mode);
    for (int i = 0; i < e->n_chunks; ++i) {
        cudaEventDestroy(e->chunks[i].ready);
        cudaEventDestroy(e->chunks[i].done);
    }
    delete[] e->chunks;
    cudaEvent_t more[] = {e->begin, e->end, e->control[0], e->control[1]};
    for (cudaEvent_t v : more)
        if (v) cudaEventDestroy(v);
    if (e->in) cudaStreamDestroy(e->in);
    if (e->out) cudaStreamDestroy(e->out);
    if (dev != e->device) cudaSetDevice(dev);
    delete e;
    return 0;
}

extern "C" int khq_b200_engine_create(khq_engine** out) {
    if (!out) return -100;
    khq_engine* e = new (std::nothrow) khq_engine();
    if (!e) return -100;
    cudaError_t err = cudaGetDevice(&e->device);
    const auto event = [&](cudaEvent_t* v) {
        if (err == cudaSuccess) err = cudaEventCreateWithFlags(v, cudaEventDisableTiming);
    };
    if (err == cudaSuccess) err = cudaStreamCreateWithFlags(&e->in, cudaStreamNonBlocking);
    if (err == cudaSuccess) err = cudaStreamCreateWithFlags(&e->out, cudaStreamNonBlocking);
    event(&e->begin);
    event(&e->end);
    event(&e->control[0]);
    event(&e->control[1]);
    if (err != cudaSuccess) {
        khq_b200_engine_destroy(e);
        return static_cast<int>(err);
    }
    *out = e;
    return 0;
}

// Events for at least n chunks: created by the first step, as many as its chunks of layers.
static cudaError_t have_chunks(khq_engine* e, int n) {
    if (n <= e->n_chunks) return cudaSuccess;
    khq_engine::Chunk* more = new (std::nothrow) khq_engine::Chunk[n];
    if (!more) return cudaErrorMemoryAllocation;
    for (int i = 0; i < e->n_chunks; ++i) more[i] = e->chunks[i];
    delete[] e->chunks;
    e->chunks = more;
    while (e->n_chunks < n) {
        khq_engine::Chunk c = {};
        cudaError_t err = cudaEventCreateWithFlags(&c.ready, cudaEventDisableTiming);
        if (err != cudaSuccess) return err;
        err = cudaEventCreateWithFlags(&c.done, cudaEventDisableTiming);
        if (err != cudaSuccess) {
            cudaEventDestroy(c.ready);
            return err;
        }
        more[e->n_chunks++] = c;
    }
    return cudaSuccess;
}

extern "C" int khq_b200_engine_wait_control(khq_engine* e, int parity) {
    if (!e || parity < 0 || parity > 1) return -100;
    return e->control_used[parity] ? static_cast<int>(cudaEventSynchronize(e->control[parity])) : 0;
}

extern "C" int launch_khq_engine_step(khq_engine* e, const khq_engine_layer* layers, const khq_engine_step* s, khq_stream_t stream) {
    if (!e || !layers || !s || s->n_layers <= 0 || s->n_seq <= 0) return -100;
    const int L = s->n_layers, B = s->n_seq;
    const int per = s->layers_per_chunk <= 0 ? 1 : s->layers_per_chunk < L ? s->layers_per_chunk : L, chunks = (L + per - 1) / per;
    cudaError_t err = have_chunks(e, chunks);
    if (err != cudaSuccess) return static_cast<int>(err);
    const auto ok = [&](cudaError_t r) {
        if (err == cudaSuccess) err = r;
        return err == cudaSuccess;
    };
    // the step's control block in one copy
    ok(cudaMemcpyAsync(s->d_control, s->h_control, s->control_bytes, cudaMemcpyHostToDevice, stream));
    ok(cudaEventRecord(e->control[s->parity], stream));
    e->control_used[s->parity] = true;
    // the copies start behind everything queued so far: the previous step's readers of the inputs and writers of the outputs
    ok(cudaEventRecord(e->begin, stream));
    ok(cudaStreamWaitEvent(e->in, e->begin, 0));
    if (err != cudaSuccess) return static_cast<int>(err);
    const size_t q_row = (size_t)B * QG * 2, kv_row = (size_t)B * KV * 2, o_row = (size_t)B * HQ * D * 2;
    const auto stage = [&](int c) {  // inputs of chunk c: three copies, whatever the number of its layers
        const size_t l0 = (size_t)c * per, n = l0 + per <= (size_t)L ? per : L - l0;
        ok(cudaMemcpyAsync(static_cast<char*>(s->d_q) + l0 * q_row, static_cast<const char*>(s->h_q) + l0 * q_row, n * q_row, cudaMemcpyHostToDevice, e->in));
        ok(cudaMemcpyAsync(static_cast<char*>(s->d_k) + l0 * kv_row, static_cast<const char*>(s->h_k) + l0 * kv_row, n * kv_row, cudaMemcpyHostToDevice, e->in));
        ok(cudaMemcpyAsync(static_cast<char*>(s->d_v) + l0 * kv_row, static_cast<const char*>(s->h_v) + l0 * kv_row, n * kv_row, cudaMemcpyHostToDevice, e->in));
        ok(cudaEventRecord(e->chunks[c].ready, e->in));
    };
    stage(0);
    int rc = launch_khq_update_descs(s->descs, s->d_dyn, B, L, stream);
    if (rc != 0) return rc;
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) stage(c + 1);
        if (!ok(cudaStreamWaitEvent(stream, e->chunks[c].ready, 0))) return static_cast<int>(err);
        const int hi = (c + 1) * per < L ? (c + 1) * per : L;
        for (int l = c * per; l < hi; ++l) {
            const khq_engine_layer& y = layers[l];
            rc = launch_khq_prestep_batched_fp16(static_cast<char*>(s->d_q) + l * q_row, static_cast<char*>(s->d_k) + l * kv_row,
                                                 static_cast<char*>(s->d_v) + l * kv_row, y.q_norm, y.k_norm, y.ring_k, y.ring_v, y.ring_u,
                                                 (long long)s->ring_cap * KV, s->d_slots, s->d_pos, B, HQ, HKV, D, s->rotary_dim, s->rope_theta,
                                                 s->rms_eps, y.q_norm ? 1 : 0, stream);
            if (rc != 0) return rc;
            if (s->n_events > 0) {
                const void* segs = static_cast<const char*>(s->d_segs) + (size_t)l * B * sizeof(khq_compress_seg);
                rc = launch_khq_compress_batched_fp16(segs, s->n_events, CHUNK_ROWS, y.d_k, y.rotor_k, y.cents_k, y.cents_k, y.k_mask, y.k_norms,
                                                      y.k_r_norms, y.k_payload, y.v_shared_meta, D, y.ts_k, y.alpha_k, 0, 0, stream);
                if (rc != 0) return rc;
                rc = launch_khq_compress_batched_fp16(segs, s->n_events, CHUNK_ROWS, y.d_v, y.rotor_v, y.cents_v, y.vq, y.k_mask, y.v_norms,
                                                      y.v_r_norms, y.v_payload, y.v_shared_meta, D, y.ts_v, y.alpha_v, 1,
                                                      static_cast<const char*>(y.ring_v) - static_cast<const char*>(y.ring_u), stream);
                if (rc != 0) return rc;
            }
            rc = launch_khq_decode_batched_prepared_fp16(static_cast<const char*>(s->descs) + (size_t)l * B * sizeof(khq_seq_desc), s->tables, s->images, s->d_items, B,
                                                s->n_items, s->workspace, s->workspace_bytes, s->n_items, s->scale, s->rope_theta, s->ring_cap,
                                                s->codebook_in_smem, stream);
            if (rc != 0) return rc;
        }
        ok(cudaEventRecord(e->chunks[c].done, stream));
        ok(cudaStreamWaitEvent(e->out, e->chunks[c].done, 0));
        const size_t l0 = (size_t)c * per;
        ok(cudaMemcpyAsync(static_cast<char*>(s->h_out) + l0 * o_row, static_cast<const char*>(s->d_out) + l0 * o_row, (hi - l0) * o_row,
                           cudaMemcpyDeviceToHost, e->out));
    }
    // the caller synchronises its stream before it reads the outputs
    ok(cudaEventRecord(e->end, e->out));
    ok(cudaStreamWaitEvent(stream, e->end, 0));
    return static_cast<int>(err);
}
