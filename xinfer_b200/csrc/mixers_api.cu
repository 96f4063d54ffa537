// C-ABI entry points for the per-layer mixer ops, with the reference's own op signatures (fp16 overloads,
// cudaStream_t for sycl::queue&), so that each kernel of mixers.cu can be checked on its own against the
// cases the reference's tests hold:
//   rmsnorm, rmsnorm_residual       src/ops/rmsnorm.h:9-42
//   rope                            src/ops/rope.h:14-34
//   attention_write_kv_cache        src/ops/attention.h:38-58
//   sdpa_causal_cached              src/ops/attention.h:89-113
//   causal_conv1d_silu              src/targets/qwen3_8/linear_attn.h:15-21
//   recurrent_gated_delta_net       src/targets/qwen3_8/linear_attn.h:41-58
// They run the product kernels (the ones the speculative step and the chunked prefill launch), not separate test
// kernels; the stateful ops update their state in the call, as the reference's do.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <mutex>

#include "../../include/xinfer_b200.h"
#include "mixers.h"
#include "w4a16.h"

namespace {

constexpr int kMaxDevices = 64;

// Scratch of the stand-alone entry points, a block per device and op (the speculative decoder has its own).  A block is taken at
// the most that any call with the same heads needs (39 MB for the attention and 32 MB for the delta rule at the 27B shapes), so it
// stays where it is whatever the row counts.  Other heads may need a larger one.  Then the old one is kept, since a captured graph
// may hold it; sizes are powers of two, so that all of an op's blocks together are less than twice the largest.
struct MixerScratch {
    float* buf = nullptr;
    size_t bytes = 0, refused = SIZE_MAX;  // `refused`: the smallest request that there was no memory for
};
enum ScratchOf { kAttention, kDelta, kConvState, kScratches };
MixerScratch g_scratch[kMaxDevices][kScratches];
std::mutex g_mu;

// `bytes`: what this call needs; `most`: what any call with these heads needs.
int scratch(ScratchOf which, size_t bytes, size_t most, float** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return XINFER_ERR_NO_DEVICE;
    std::lock_guard<std::mutex> lock(g_mu);
    MixerScratch& m = g_scratch[dev][which];
    for (size_t want : {most, bytes}) {  // (on a full device the call still gets what it needs)
        if (m.bytes >= want) break;
        if (want == most && most != bytes && want >= m.refused) continue;
        size_t size = size_t{1} << 20;
        while (size < want) size *= 2;
        float* buf = nullptr;
        if (cudaMalloc(reinterpret_cast<void**>(&buf), size) == cudaSuccess) {
            m.buf = buf;
            m.bytes = size;
            break;
        }
        cudaGetLastError();
        if (want < m.refused) m.refused = want;
    }
    if (m.bytes < bytes) return XINFER_ERR_OUT_OF_MEMORY;
    *out = m.buf;
    return XINFER_OK;
}

int ok_or_cuda(int rc) {
    if (rc == 0) return XINFER_OK;
    xb::set_last_error(cudaGetErrorString(cudaGetLastError()));
    return rc == -2 ? XINFER_ERR_INVALID_ARGUMENT : XINFER_ERR_CUDA;
}

}  // namespace

extern "C" {

int xinfer_rmsnorm_f16(xinfer_stream_t s, void* out, const void* in, const float* weight, int64_t num_tokens,
                       int64_t hidden_size, float eps) {
    if (num_tokens <= 0 || hidden_size <= 0) return XINFER_NOOP_INVALID_SHAPE;
    if (!out || !in || !weight) return XINFER_ERR_INVALID_ARGUMENT;
    return ok_or_cuda(xb::rmsnorm_rows(static_cast<cudaStream_t>(s), static_cast<__half*>(out), hidden_size,
                                       static_cast<const __half*>(in), weight, static_cast<int>(num_tokens),
                                       static_cast<int>(hidden_size), eps));
}

int xinfer_rmsnorm_residual_f16(xinfer_stream_t s, void* out, void* residual, const void* in, const float* weight,
                                int64_t num_tokens, int64_t hidden_size, float eps) {
    if (num_tokens <= 0 || hidden_size <= 0) return XINFER_NOOP_INVALID_SHAPE;
    if (!out || !residual || !in || !weight) return XINFER_ERR_INVALID_ARGUMENT;
    return ok_or_cuda(xb::add_rmsnorm_rows(static_cast<cudaStream_t>(s), static_cast<__half*>(out), static_cast<__half*>(residual),
                                           static_cast<const __half*>(in), weight, static_cast<int>(num_tokens),
                                           static_cast<int>(hidden_size), eps));
}

int xinfer_rope_f16(xinfer_stream_t s, void* q_ptr, void* k_ptr, int64_t num_tokens, int64_t num_q_heads,
                    int64_t num_kv_heads, int64_t head_dim, const int64_t* positions_dev, float theta, int64_t rotary_dim) {
    if (num_tokens <= 0 || num_q_heads < 0 || num_kv_heads < 0 || num_q_heads + num_kv_heads == 0) return XINFER_NOOP_INVALID_SHAPE;
    if (head_dim != 256 || rotary_dim < 0 || rotary_dim > 256 || rotary_dim % 2 || !positions_dev || !(theta > 0.f) ||
        (num_q_heads > 0 && !q_ptr) || (num_kv_heads > 0 && !k_ptr))
        return XINFER_ERR_INVALID_ARGUMENT;
    // in place: each (row, head) block reads its 256 values before it writes them
    return ok_or_cuda(xb::attn_prep_ex(static_cast<cudaStream_t>(s), static_cast<__half*>(q_ptr), nullptr, nullptr,
                                       static_cast<const __half*>(q_ptr), static_cast<const __half*>(k_ptr), nullptr, nullptr,
                                       nullptr, nullptr, 1, static_cast<int>(num_tokens), static_cast<int>(num_q_heads),
                                       static_cast<int>(num_kv_heads), 1ll << 40, 0.f, theta, static_cast<int>(rotary_dim), 256,
                                       reinterpret_cast<const long long*>(positions_dev), 0, static_cast<__half*>(k_ptr)));
}

int xinfer_attention_write_kv_cache_f16(xinfer_stream_t s, void* k_cache, void* v_cache, const void* K_in, const void* V_in,
                                        int64_t start_pos, int64_t num_tokens, int64_t num_kv_heads, int64_t head_dim,
                                        int64_t max_seq_len) {
    if (num_tokens <= 0 || num_kv_heads <= 0) return XINFER_NOOP_INVALID_SHAPE;
    if (!k_cache || !v_cache || !K_in || !V_in || head_dim != 256 || start_pos < 0 || start_pos > INT32_MAX)
        return XINFER_ERR_INVALID_ARGUMENT;
    // the reference throws std::out_of_range when the rows do not fit a bounded cache (src/ops/attention.cpp:95-99)
    if (max_seq_len > 0 && start_pos + num_tokens > max_seq_len) return XINFER_ERR_INVALID_ARGUMENT;
    const long long cap = max_seq_len > 0 ? max_seq_len : (1ll << 40);
    return ok_or_cuda(xb::attn_prep_ex(static_cast<cudaStream_t>(s), nullptr, static_cast<__half*>(k_cache),
                                       static_cast<__half*>(v_cache), nullptr, static_cast<const __half*>(K_in),
                                       static_cast<const __half*>(V_in), nullptr, nullptr, nullptr, 1,
                                       static_cast<int>(num_tokens), 0, static_cast<int>(num_kv_heads), cap, 0.f, 1.0e7f, 0, 256,
                                       nullptr, static_cast<int>(start_pos), nullptr));
}

int xinfer_sdpa_causal_cached_f16(xinfer_stream_t s, void* out, const void* Q, const void* k_cache, const void* v_cache,
                                  int64_t start_pos, int64_t num_q_tokens, int64_t num_q_heads, int64_t num_kv_heads,
                                  int64_t head_dim, float scale, int64_t max_seq_len) {
    if (num_q_tokens <= 0 || num_q_heads <= 0 || num_kv_heads <= 0) return XINFER_NOOP_INVALID_SHAPE;
    if (!out || !Q || !k_cache || !v_cache || head_dim != 256 || num_q_heads % num_kv_heads || start_pos < 0 ||
        start_pos + num_q_tokens > INT32_MAX)
        return XINFER_ERR_INVALID_ARGUMENT;
    if (max_seq_len > 0 && start_pos + num_q_tokens > max_seq_len) return XINFER_ERR_INVALID_ARGUMENT;
    const int hq = static_cast<int>(num_q_heads), hkv = static_cast<int>(num_kv_heads);
    const int group = hq / hkv;
    if (group > 32) return XINFER_ERR_INVALID_ARGUMENT;
    int *status = nullptr, num_sms = 0;
    int rc = xb::device_facts(&status, &num_sms);
    if (rc != XINFER_OK) return rc;
    xb::AttnTiles a;
    a.k_cache = static_cast<const __half*>(k_cache);
    a.v_cache = static_cast<const __half*>(v_cache);
    a.hq = hq;
    a.hkv = hkv;
    a.scale = scale > 0.f ? scale : 1.0f / sqrtf(256.0f);  // src/ops/attention.cpp:165-167
    // pieces of rows that keep the count of (128-row tile, 64-key block) units of a launch well inside 32 bits
    const int64_t tile_pos = 128 / group, blocks = (start_pos + num_q_tokens) / 64 + 1;
    int64_t piece = (int64_t{1} << 29) / (blocks * hkv) * tile_pos;
    constexpr int64_t kMostRows = 65536;
    piece = piece < tile_pos ? tile_pos : (piece < kMostRows ? piece : kMostRows);
    const int most = static_cast<int>(num_q_tokens < piece ? num_q_tokens : piece);
    rc = scratch(kAttention, xb::attn_tile_scratch_bytes(1, most, hq, hkv, num_sms), xb::attn_tile_scratch_bytes(1, kMostRows, hq, hkv, num_sms),
                 &a.scratch);
    if (rc != XINFER_OK) return rc;
    for (int64_t t0 = 0; t0 < num_q_tokens; t0 += piece) {
        a.rows_per_seq = static_cast<int>(num_q_tokens - t0 < piece ? num_q_tokens - t0 : piece);
        a.ctx_base = static_cast<int>(start_pos + t0);
        a.cache_rows = a.cache_stride = start_pos + t0 + a.rows_per_seq;
        a.out = static_cast<__half*>(out) + t0 * hq * 256;
        a.q = static_cast<const __half*>(Q) + t0 * hq * 256;
        rc = xb::attn_tiles(static_cast<cudaStream_t>(s), a, num_sms, status);
        if (rc != 0) return ok_or_cuda(rc);
    }
    return XINFER_OK;
}

int xinfer_causal_conv1d_silu_f16(xinfer_stream_t s, void* out_qkv, const void* in_qkv, const float* conv_w, int64_t seq_len,
                                  float* conv_state, int64_t num_channels) {
    // the reference throws std::invalid_argument on num_channels <= 0 before it looks at anything else
    // (src/targets/qwen3_8/linear_attn.cpp, causal_conv1d_silu; tests/test_decode_graph.cpp:27-35)
    if (num_channels <= 0 || num_channels > INT32_MAX) return XINFER_ERR_INVALID_ARGUMENT;
    if (seq_len <= 0) return XINFER_NOOP_INVALID_SHAPE;
    if (!out_qkv || !in_qkv || !conv_w) return XINFER_ERR_INVALID_ARGUMENT;
    // pieces that 32-bit positions reach; the state carries from one to the next
    constexpr int64_t kPiece = int64_t{1} << 30;
    float* state = conv_state;
    if (!state && seq_len > kPiece) {
        const size_t bytes = 3 * sizeof(float) * static_cast<size_t>(num_channels);
        const int rc = scratch(kConvState, bytes, bytes, &state);
        if (rc != XINFER_OK) return rc;
        if (cudaMemsetAsync(state, 0, bytes, static_cast<cudaStream_t>(s)) != cudaSuccess) return ok_or_cuda(-1);
    }
    for (int64_t t0 = 0; t0 < seq_len; t0 += kPiece) {
        const int rows = static_cast<int>(seq_len - t0 < kPiece ? seq_len - t0 : kPiece);
        const int r = xb::conv1d_chunk(static_cast<cudaStream_t>(s), static_cast<__half*>(out_qkv) + t0 * num_channels,
                                       static_cast<const __half*>(in_qkv) + t0 * num_channels, conv_w, state, 1, rows,
                                       static_cast<int>(num_channels));
        if (r != 0) return ok_or_cuda(r);
    }
    return XINFER_OK;
}

int xinfer_recurrent_gated_delta_net_f16(xinfer_stream_t s, void* out, const void* qkv, const void* z, const void* b,
                                         const void* a, const float* A_log, const float* dt_bias, const float* norm_weight,
                                         float* state_buffer, int64_t seq_len, int zero_state, int64_t num_v_heads,
                                         int64_t num_k_heads) {
    if (seq_len <= 0) return XINFER_NOOP_INVALID_SHAPE;
    // The reference refuses every shape but its compiled one (48 v heads, 16 k heads, 128 x 128 state;
    // src/targets/qwen3_8/linear_attn.cpp:163-181, tests/test_decode_graph.cpp:37-49); the kernel here takes any
    // head counts with v_heads a multiple of k_heads and refuses the rest the same way.
    if (num_v_heads <= 0 || num_k_heads <= 0 || num_v_heads % num_k_heads) return XINFER_ERR_INVALID_ARGUMENT;
    if (!out || !qkv || !z || !b || !a || !A_log || !dt_bias || !norm_weight || !state_buffer) return XINFER_ERR_INVALID_ARGUMENT;
    const int hv = static_cast<int>(num_v_heads), hk = static_cast<int>(num_k_heads);
    int *status = nullptr, num_sms = 0;
    int rc = xb::device_facts(&status, &num_sms);
    if (rc != XINFER_OK) return rc;
    if (xb::gdn_chunk_aligned(out, qkv, z, state_buffer)) {
        // pieces of 1024 rows bound the scratch (32 MB at 48 heads)
        const int64_t piece = 1024, ch = 2 * static_cast<int64_t>(hk) * 128 + static_cast<int64_t>(hv) * 128, vd = static_cast<int64_t>(hv) * 128;
        float* blocks = nullptr;
        const int most = static_cast<int>(seq_len < piece ? seq_len : piece);
        rc = scratch(kDelta, xb::gdn_chunk_scratch_bytes(1, most, hv), xb::gdn_chunk_scratch_bytes(1, static_cast<int>(piece), hv), &blocks);
        if (rc != XINFER_OK) return rc;
        for (int64_t t0 = 0; t0 < seq_len; t0 += piece) {
            const int rows = static_cast<int>(seq_len - t0 < piece ? seq_len - t0 : piece);
            const int r = xb::gdn_chunk(static_cast<cudaStream_t>(s), static_cast<__half*>(out) + t0 * vd, static_cast<const __half*>(qkv) + t0 * ch,
                                        static_cast<const __half*>(z) + t0 * vd, static_cast<const __half*>(b) + t0 * hv,
                                        static_cast<const __half*>(a) + t0 * hv, A_log, dt_bias, norm_weight, state_buffer, 1, rows, hv, hk,
                                        blocks, num_sms, zero_state && t0 == 0);
            if (r != 0) return ok_or_cuda(r);
        }
        return XINFER_OK;
    }
    // pointers that the vector accesses of the chunk kernel do not fit: eight tokens a launch through the step's kernel
    const size_t pk = static_cast<size_t>(hv) * 8 * 128;
    float* scr = nullptr;
    const size_t pending = (2 * pk + static_cast<size_t>(hv) * 8) * sizeof(float);
    rc = scratch(kDelta, pending, xb::gdn_chunk_scratch_bytes(1, 1024, hv), &scr);
    if (rc != XINFER_OK) return rc;
    float *pend_k = scr, *pend_d = scr + pk, *pend_g = scr + 2 * pk;
    cudaStream_t st = static_cast<cudaStream_t>(s);
    if (zero_state &&
        cudaMemsetAsync(state_buffer, 0, static_cast<size_t>(hv) * 128 * 128 * sizeof(float), st) != cudaSuccess)
        return ok_or_cuda(-1);
    const int64_t ch = 2 * static_cast<int64_t>(hk) * 128 + static_cast<int64_t>(hv) * 128, vd = static_cast<int64_t>(hv) * 128;
    const __half *q = static_cast<const __half*>(qkv), *zz = static_cast<const __half*>(z), *bb = static_cast<const __half*>(b),
                 *aa = static_cast<const __half*>(a);
    __half* o = static_cast<__half*>(out);
    int prev = 0;
    for (int64_t t0 = 0; t0 < seq_len; t0 += 8) {
        const int rows = static_cast<int>(seq_len - t0 < 8 ? seq_len - t0 : 8);
        rc = xb::gdn_spec(st, o + t0 * vd, q + t0 * ch, zz + t0 * vd, bb + t0 * hv, aa + t0 * hv, A_log, dt_bias, norm_weight,
                          state_buffer, pend_k, pend_d, pend_g, nullptr, 1, rows, prev, hv, hk, prev, 0, 0, num_sms);
        if (rc != 0) return ok_or_cuda(rc);
        prev = rows;
    }
    return ok_or_cuda(xb::gdn_spec(st, o, q, zz, bb, aa, A_log, dt_bias, norm_weight, state_buffer, pend_k, pend_d, pend_g, nullptr,
                                   1, 0, prev, hv, hk, prev, 0, 0, num_sms));
}

/* ---- plain device memory and streams, for hosts that do not link the CUDA runtime themselves --------------- */
int xinfer_device_alloc(size_t bytes, void** out) {
    if (!out) return XINFER_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (bytes == 0) return XINFER_OK;
    if (cudaMalloc(out, bytes) != cudaSuccess) {
        cudaGetLastError();
        return XINFER_ERR_OUT_OF_MEMORY;
    }
    return XINFER_OK;
}
void xinfer_device_free(void* p) {
    if (p) cudaFree(p);
}
int xinfer_stream_create(xinfer_stream_t* out) {
    if (!out) return XINFER_ERR_INVALID_ARGUMENT;
    cudaStream_t st = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return ok_or_cuda(-1);
    *out = st;
    return XINFER_OK;
}
void xinfer_stream_destroy(xinfer_stream_t s) {
    if (s) cudaStreamDestroy(static_cast<cudaStream_t>(s));
}
int xinfer_stream_synchronize(xinfer_stream_t s) {
    return cudaStreamSynchronize(static_cast<cudaStream_t>(s)) == cudaSuccess ? XINFER_OK : ok_or_cuda(-1);
}

}  // extern "C"
