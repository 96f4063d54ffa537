// Internal interface of the per-layer glue kernels (mixers.cu).  Rows are (sequence b, position i),
// i < rows_per_seq; every function is asynchronous on the stream and returns 0 or a negative code.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stddef.h>

namespace xb {

// perm_out (here and below): write the output with every block of eight features in the order the int4 unpack of
// the W4A16 kernel yields them, (0,4,1,5,2,6,3,7): such a buffer is only good as the X of a projection launched
// with kTcXPermuted (w4a16.h).
int rmsnorm_rows(cudaStream_t s, __half* out, long long ld_out, const __half* in, const float* w, int rows, int hidden,
                 float eps, int perm_out = 0);
// x = embedding rows (bf16 table) of the tokens, out = rmsnorm(x) * w
int embed_norm_rows(cudaStream_t s, __half* out, __half* x, const void* table_bf16, const long long* tokens, const float* w, int rows,
                    int hidden, long long vocab, float eps, int perm_out = 0);
// cat[row] = [rmsnorm(embedding of tokens[row]) * embed_norm ; rmsnorm(hidden_rows[row]) * hidden_norm], and on the way
// token_copy[row * token_ld] = tokens[row] and pos_out[row] = pos_in[row] + pos_add (each if its target is given)
struct HeadInput {
    __half* cat = nullptr;  // [rows][2 hidden]
    const void* table_bf16 = nullptr;
    const long long* tokens = nullptr;
    long long vocab = 0;
    const float *embed_norm = nullptr, *hidden_norm = nullptr;
    const __half* hidden_rows = nullptr;
    long long* token_copy = nullptr;
    int token_ld = 1;
    const int* pos_in = nullptr;
    int* pos_out = nullptr;
    int pos_add = 0;
};
int head_input_rows(cudaStream_t s, const HeadInput& h, int rows, int hidden, float eps, int perm_out = 0);
// x = half(x + delta) in place, out = rmsnorm(x) * w
int add_rmsnorm_rows(cudaStream_t s, __half* out, __half* x, const __half* delta, const float* w, int rows, int hidden,
                     float eps, int perm_out = 0);

// q/k head RMSNorm + partial RoPE + KV-cache write.  Caches are [batch][max_seq][hkv][256] fp16.
int attn_prep(cudaStream_t s, __half* q_out, __half* k_cache, __half* v_cache, const __half* q_gate, const __half* k_in,
              const __half* v_in, const float* q_norm_w, const float* k_norm_w, const int* ctx, int batch,
              int rows_per_seq, int hq, int hkv, long long max_seq, float eps, float rope_theta, int rope_dim);
// The same kernel with its optional pieces spelled out (the stand-alone op entry points): query heads
// `q_head_stride` halves apart in q_in, null norm weights skip the head norm, `positions` (per row) or `ctx_base`
// (when ctx is null) give the positions, null caches skip the write and the rotated keys go to `k_out`.
int attn_prep_ex(cudaStream_t s, __half* q_out, __half* k_cache, __half* v_cache, const __half* q_in, const __half* k_in,
                 const __half* v_in, const float* q_norm_w, const float* k_norm_w, const int* ctx, int batch,
                 int rows_per_seq, int hq, int hkv, long long max_seq, float eps, float rope_theta, int rope_dim,
                 int q_head_stride, const long long* positions, int ctx_base, __half* k_out);
// Causal GQA attention over the cache (row i of sequence b sees keys below ctx[b] + i + 1), then * sigmoid(gate).
struct AttnTiles {
    __half* out = nullptr;             // [batch][rows_per_seq][hq][256]
    const __half *q = nullptr, *k_cache = nullptr, *v_cache = nullptr;  // 16-byte aligned
    const __half* q_gate = nullptr;    // [batch][rows_per_seq][hq][512], the gate in the upper 256, 16-byte aligned; null: no gate
    const int* ctx = nullptr;          // per sequence; null: ctx_base
    int ctx_base = 0;
    int batch = 1, rows_per_seq = 1, hq = 1, hkv = 1;  // hq / hkv <= 128
    // rows of a sequence's cache that hold keys (what is behind a row's own limit must still be finite), and its row stride
    long long cache_rows = 0, cache_stride = 0;
    float scale = 1.f;
    int perm_out = 0;                  // see perm_out of rmsnorm_rows
    int early = 0;                     // see below
    float* scratch = nullptr;          // attn_tile_scratch_bytes
};
size_t attn_tile_scratch_bytes(int batch, int rows_per_seq, int hq, int hkv, int num_sms);
int attn_tiles(cudaStream_t s, const AttnTiles& a, int num_sms, int* status);

// state [batch][3][channels], pending [batch][8][channels] fp32.  The first min(n_commit[b], prev_rows) pending
// inputs of the previous call are committed to the state before the new rows are processed (n_commit null:
// nc_base of them).  rows_per_seq = 0 only commits.  early_state = 1 (both kernels): state, pending updates and
// weights were NOT written by the launch directly in front of this one in the stream, so the kernel may fetch
// them while that launch is still running (programmatic dependent launch).
//
// early / early_state: the kernel reads its context lengths and the keys below them, or its state, pending updates and n_commit
// (conv1d_spec also writes its state), before it waits for the launch in front of it.  Kernels of the step signal their
// dependents first and wait afterwards, so several launches may be under way at once, and "some launches ago" says nothing.
// What is read early must have been written before a launch of this stream that signals only after its own wait
// (build_verify_tokens; any launch or copy outside programmatic dependent launch), with that launch in front of this one.
int conv1d_spec(cudaStream_t s, __half* out, const __half* in, const float* conv_w, float* state, float* pending,
                const int* n_commit, int batch, int rows_per_seq, int prev_rows, int channels, int nc_base = 0,
                int early_state = 0);
// state [batch][hv][128][128], pend_k / pend_d [batch][hv][8][128], pend_g [batch][hv][8] fp32; rows_per_seq <= 8
int gdn_spec(cudaStream_t s, __half* out, const __half* qkv, const __half* z, const __half* b, const __half* a,
             const float* A_log, const float* dt_bias, const float* norm_w, float* state, float* pend_k, float* pend_d,
             float* pend_g, const int* n_commit, int batch, int rows_per_seq, int prev_rows, int hv, int hk, int nc_base,
             int early_state, int perm_out, int num_sms);

// The convolution and the gated delta rule over all rc positions of a prefill chunk in one launch each (rows
// [sequence][position], every row kept, the state read once and written back once; nothing pending afterwards).  A null
// convolution state means zeros; zero_state starts the recurrence from zeros.
int conv1d_chunk(cudaStream_t s, __half* out, const __half* in, const float* conv_w, float* state, int batch, int rc,
                 int channels);
int gdn_chunk(cudaStream_t s, __half* out, const __half* qkv, const __half* z, const __half* b, const __half* a,
              const float* A_log, const float* dt_bias, const float* norm_w, float* state, int batch, int rc, int hv, int hk,
              void* scratch, int num_sms, int zero_state = 0);
size_t gdn_chunk_scratch_bytes(int batch, int rc, int hv);  // of `scratch`, 16-byte aligned
// Whether the vector accesses of gdn_chunk fit these pointers.
bool gdn_chunk_aligned(const void* out, const void* qkv, const void* z, const void* state);

int spec_commit(cudaStream_t s, const void* accept_records, const long long* draft_tokens, int batch, int k,
                int rows_per_seq, int* ctx, int* n_commit, long long* cur_tok, long long* emitted, int* emitted_n,
                __half* h_last, const __half* hidden_rows, int hidden);
int build_verify_tokens(cudaStream_t s, long long* out, const long long* cur_tok, const long long* draft, int batch,
                        int k);
int fill_int(cudaStream_t s, int* p, int n, int v);

}  // namespace xb
