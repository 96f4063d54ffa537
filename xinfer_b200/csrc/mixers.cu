// Per-layer glue of the speculative decode / verify step: embedding lookup, RMSNorm (+ residual add),
// the full-attention mixer (q/k head norm, partial RoPE, KV-cache write, split-KV GQA attention over an
// fp16 cache, sigmoid output gate) and the Gated-DeltaNet mixer (causal conv1d + SiLU, gated delta-rule
// recurrence with fused gated RMSNorm).
//
// Semantics follow the reference's kernels; every fp16 rounding point of the reference is kept so
// that a CPU restatement of the reference agrees to the last fp16 bit in most elements:
//   embed_tokens_lookup            src/targets/qwen3_8/forward.cpp:17-64
//   rmsnorm                        src/ops/rmsnorm.cpp:15-82
//   add_inplace (fp16)             src/ops/elementwise.cpp:213-236
//   q/gate split, sigmoid gating   src/targets/qwen3_8/forward.cpp:145-151, 217-226
//   rope                           src/ops/rope.cpp:12-62
//   attention_write_kv_cache       src/ops/attention.cpp:84-116
//   sdpa_causal_cached             src/ops/attention.cpp:151-243
//   causal_conv1d_silu             src/targets/qwen3_8/linear_attn.cpp:37-122
//   recurrent_gated_delta_net      src/targets/qwen3_8/linear_attn.cpp:144-343
//
// What is different is the batching and the speculative state handling, which the reference does not
// have: rows are (sequence b, position i) with i < R, R = 1 while drafting and k+1 while verifying;
// sequence b sees keys below ctx[b] + i + 1; and the recurrent states (DeltaNet S, conv window) are
// committed lazily: a step stores its per-token updates, and the NEXT step first replays the
// n_commit[b] accepted ones onto the stored state, bit-identically, before it processes new tokens.
// Nothing is copied or restored when draft tokens are rejected.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

#include "launch.cuh"
#include "mixers.h"
#include "ptx_sm100.cuh"
#include "silu.cuh"

namespace xb {

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Outputs that feed a W4A16 projection can be written with every block of eight features in the order the int4
// unpack yields them, (0,4,1,5,2,6,3,7), which saves the projection kernel its in-flight rewrite of the staged
// activations.  perm8: where feature n goes;  perm8_vec: eight consecutive features (one 16-byte vector) reordered.
__device__ __forceinline__ int perm8(int n) {
    const int k = n & 7;
    return (n & ~7) | ((k < 4) ? 2 * k : 2 * (k - 4) + 1);
}
__device__ __forceinline__ uint4 perm8_vec(const uint4& v) {
    // halves (h0 h1 | h2 h3 | h4 h5 | h6 h7) -> (h0 h4 | h1 h5 | h2 h6 | h3 h7)
    uint4 o;
    o.x = __byte_perm(v.x, v.z, 0x5410);
    o.y = __byte_perm(v.x, v.z, 0x7632);
    o.z = __byte_perm(v.y, v.w, 0x5410);
    o.w = __byte_perm(v.y, v.w, 0x7632);
    return o;
}

// block-wide sum for up to 1024 threads; every thread gets the result
__device__ __forceinline__ float block_sum(float v, float* smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) smem[warp] = v;
    __syncthreads();
    float t = (lane < nw) ? smem[lane] : 0.f;
    t = warp_sum(t);
    return t;
}

// ------------------------------------------------------------------------------- RMSNorm family
// out = rmsnorm(x) * w, where x is read
//   from `x`                                                  (plain)
//   as half(x + delta), also written back to x                (residual add, then norm)
//   from row `tokens[row]` of the bf16 table, also written to x when x is given   (embedding, then norm)
// `out` may have a wider row (ld_out) and a column offset so that two norms can fill one concatenated row.
// One or two such jobs per launch (blockIdx.y).  Bound by latency at a step's 1 to 32 rows (2.3 us a launch): what counts
// is the number of launches and of dependent trips to memory.  An embedding of its own, 2 bytes per load, took 10 us.
struct NormJob {
    __half* out;
    __half* x;
    const __half* delta;
    const float* w;
    const uint16_t* table;    // embedding rows (bf16), or null
    const long long* tokens;  // one per row
    long long vocab;          // tokens outside [0, vocab) read as zeros
    long long* token_copy;    // tokens[row] also goes to token_copy[row * token_ld], if given
    int token_ld;
    const int* pos_in;        // pos_out[row] = pos_in[row] + pos_add, if given
    int* pos_out;
    int pos_add;
};

// The table row of a job's token (null: none, or no table); the first thread keeps the job's books.
__device__ __forceinline__ const uint16_t* norm_tokens(const NormJob& job, long long row, int hidden) {
    const long long tok = job.tokens[row];
    if (threadIdx.x == 0) {
        if (job.token_copy) job.token_copy[row * job.token_ld] = tok;
        if (job.pos_out) job.pos_out[row] = job.pos_in[row] + job.pos_add;
    }
    return (tok >= 0 && (job.vocab <= 0 || tok < job.vocab)) ? job.table + tok * hidden : nullptr;
}
__device__ __forceinline__ __half bf16_to_half(uint32_t bits) { return __float2half_rn(__uint_as_float(bits << 16)); }

constexpr int kNormNarrow = 2048, kNormPairs = 6144;
// TABLE: some job of the launch reads the embedding table.  VECS: most 8-element vectors of a thread: four of 256 threads (and the path for
// rows that are not vectors), two of up to 512, or one of up to 1024.  FEW: no row shares its SM.  Bound by latency, then by the rows in flight.
// One vector a thread is the shorter way through a row, which is what counts as long as every row has an SM to itself, and where 256
// threads would not all have one (a launch of two jobs has two blocks a row, and that is what is counted): 5120 features with the residual added, 1 row 2.30 -> 1.84 us, 32 rows 2.57 -> 2.13, 148 rows 2.58 -> 2.24;
// 1024 features, 2796 rows 8.9 -> 4.9.  (0.07 to 0.12 us of it since the compiler may use 64 registers, where otherwise it fits two rows of 1024
// threads on an SM; with many narrow rows those are worth as much: 1024 features, 2796 rows 4.47 against 4.71.)  With more rows the 640
// threads of a wide row leave an SM three rows at a time: 1024 x 5120 5.93 us with four vectors, 6.83 with one.
// Two vectors, the weights read behind the sum (another trip to L2, but 40 registers in place of 77), put four rows of 5120 or 6144 features on an
// SM in place of three and leave no thread idle: where rows are many, and where four an SM are a single wave.  5120 features with the residual
// added: 296..444 rows 3.8 us with four vectors and 4.5 with two, 445..592 5.2 and 4.4, 740 5.9 and 6.4, 1480 9.8 and 9.1, 2796 17.7 and 15.9;
// 2560 features, 740 rows 4.3 and 4.7, 2796 11.8 and 8.0.  At 7168 and more, two rows an SM, 740 rows 5.3 and 6.1, 2796 15.8 and 16.2; at 2048
// one vector is better up to 1024 rows (3.1 and 3.9).
template <bool TABLE, int VECS, bool FEW>
__global__ void __launch_bounds__(VECS == 1 ? 1024 : VECS == 2 ? 512 : 256, VECS == 2 ? 3 : FEW ? 1 : 0) rmsnorm_kernel(const __grid_constant__ NormJob job0, const __grid_constant__ NormJob job1,
                                                      long long ld_out, int hidden, float eps, int perm_out) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ __align__(16) float red[32];  // of every warp
    const NormJob& job = TABLE && blockIdx.y ? job1 : job0;
    const bool table = TABLE && job.table;
    const float* w = job.w;
    const long long row = blockIdx.x;
    __half* xr = job.x ? job.x + row * hidden : nullptr;
    const __half* dr = job.delta ? job.delta + row * hidden : nullptr;
    __half* orow = job.out + row * ld_out;
    const int nvec = hidden >> 3;
    constexpr bool kLateW = VECS == 2;
    const bool vec_ok = (hidden & 7) == 0 && nvec <= VECS * static_cast<int>(blockDim.x) &&
                        ((reinterpret_cast<uintptr_t>(xr) | reinterpret_cast<uintptr_t>(orow) | reinterpret_cast<uintptr_t>(dr) |
                          reinterpret_cast<uintptr_t>(job.table) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
    if (vec_ok) {
        // The norm weights do not depend on the previous kernel in the stream: they are fetched before waiting
        // for it, so that only the activations' latency is left on the critical path.
        float4 wv[VECS][2];
#pragma unroll
        for (int it = 0; it < VECS; ++it) {
            const int i = threadIdx.x + it * (VECS == 2 ? blockDim.x : 256);
            if (i < nvec && !kLateW) {
                wv[it][0] = __ldg(reinterpret_cast<const float4*>(w + i * 8));
                wv[it][1] = __ldg(reinterpret_cast<const float4*>(w + i * 8 + 4));
            }
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const uint16_t* tr = table ? norm_tokens(job, row, hidden) : nullptr;
        // one pass: each thread keeps its 8-element vectors (VECS at most) in registers.  Every load goes out before the first
        // value is used and before any store (which the compiler must take for a possible alias of the later loads): with
        // the residual stored in between, each further vector was another trip to memory (2.9 us a launch against 2.5).
        uint4 v[VECS], dv[VECS];
#pragma unroll
        for (int it = 0; it < VECS; ++it) {
            const int i = threadIdx.x + it * (VECS == 2 ? blockDim.x : 256);
            if (i < nvec) {
                if (!table) v[it] = *reinterpret_cast<const uint4*>(xr + i * 8);
                else v[it] = tr ? __ldg(reinterpret_cast<const uint4*>(tr + i * 8)) : make_uint4(0u, 0u, 0u, 0u);
                if (dr) dv[it] = *reinterpret_cast<const uint4*>(dr + i * 8);
            }
        }
        float ss = 0.f;
#pragma unroll
        for (int it = 0; it < VECS; ++it) {
            const int i = threadIdx.x + it * (VECS == 2 ? blockDim.x : 256);
            if (i < nvec) {
                __half2* h = reinterpret_cast<__half2*>(&v[it]);
                if (table) {
                    const uint32_t e[4] = {v[it].x, v[it].y, v[it].z, v[it].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) h[j] = __halves2half2(bf16_to_half(e[j] & 0xFFFFu), bf16_to_half(e[j] >> 16));
                }
                if (dr) {
                    const __half2* dh = reinterpret_cast<const __half2*>(&dv[it]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 a = __half22float2(h[j]), b = __half22float2(dh[j]);
                        h[j] = __halves2half2(__float2half_rn(a.x + b.x), __float2half_rn(a.y + b.y));
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 a = __half22float2(h[j]);
                    ss = fmaf(a.y, a.y, fmaf(a.x, a.x, ss));
                }
            }
        }
        ss = warp_sum(ss);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
        if (VECS <= 2 && threadIdx.x < 32 && threadIdx.x >= (blockDim.x >> 5)) red[threadIdx.x] = 0.f;
        __syncthreads();
        float total = 0.f;
#pragma unroll
        for (int w = 0; w < (VECS == 1 ? 32 : VECS == 2 ? 16 : 8); w += 8) {
            const float4 r0 = *reinterpret_cast<const float4*>(red + w), r1 = *reinterpret_cast<const float4*>(red + w + 4);
            total += ((r0.x + r1.x) + (r0.z + r1.z)) + ((r0.y + r1.y) + (r0.w + r1.w));
        }
        const float r = 1.0f / sqrtf(total / static_cast<float>(hidden) + eps);
#pragma unroll
        for (int it = 0; it < VECS; ++it) {
            const int i = threadIdx.x + it * (VECS == 2 ? blockDim.x : 256);
            if (i < nvec) {
                if (xr && (dr || table)) *reinterpret_cast<uint4*>(xr + i * 8) = v[it];
                const __half2* h = reinterpret_cast<const __half2*>(&v[it]);
                const float4 w0 = kLateW ? __ldg(reinterpret_cast<const float4*>(w + i * 8)) : wv[it][0];
                const float4 w1 = kLateW ? __ldg(reinterpret_cast<const float4*>(w + i * 8 + 4)) : wv[it][1];
                const float ww[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
                uint4 o;
                __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 a = __half22float2(h[j]);
                    oh[j] = __halves2half2(__float2half_rn(a.x * r * ww[2 * j]), __float2half_rn(a.y * r * ww[2 * j + 1]));
                }
                *reinterpret_cast<uint4*>(orow + i * 8) = perm_out ? perm8_vec(o) : o;
            }
        }
        return;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint16_t* tr = table ? norm_tokens(job, row, hidden) : nullptr;
    auto element = [&](int i) { return table ? (tr ? bf16_to_half(tr[i]) : __float2half_rn(0.f)) : xr[i]; };
    float ss = 0.f;
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
        __half e = element(i);
        if (dr) e = __float2half_rn(__half2float(e) + __half2float(dr[i]));
        if (xr && (dr || table)) xr[i] = e;
        const float v = __half2float(e);
        ss += v * v;
    }
    const float total = block_sum(ss, red);
    const float r = 1.0f / sqrtf(total / static_cast<float>(hidden) + eps);
    for (int i = threadIdx.x; i < hidden; i += blockDim.x)
        orow[(perm_out && (hidden & 7) == 0) ? perm8(i) : i] = __float2half_rn(__half2float(xr ? xr[i] : element(i)) * r * w[i]);
}

// ------------------------------------------------------------------------------- attention prologue
// A rotation is two products and a sum; one product is rounded before the sum, and left to the compiler it was another one in each of
// the two forms below.  Here it is the sine's, in both.  Calls of more than 4096 heads, which have only ever had the second form, keep
// what that gave them: the cosine's for a pair's second value (SINE_FUSED).
template <bool SINE_FUSED>
__device__ __forceinline__ float rotated(bool second, float v0, float v1, float c, float s) {
    if (!second) return fmaf(v0, c, -__fmul_rn(v1, s));
    return SINE_FUSED ? fmaf(v0, s, __fmul_rn(v1, c)) : fmaf(v1, c, __fmul_rn(v0, s));
}

// One block per (row, head slot); head slots 0..Hq-1 are query heads, Hq..Hq+Hkv-1 key heads,
// Hq+Hkv..Hq+2Hkv-1 value heads.  256 threads = head_dim.
// Generalisations used by the stand-alone op entry points: `q_head_stride` is the distance between query
// heads in q_in (512 for the interleaved [q | gate] block, 256 for plain queries); a null norm weight skips
// that head norm; `positions` (one per row) overrides ctx[b] + i; a null ctx means context length ctx_base; a
// null cache pointer skips the write (the rotated key then goes to k_out, if given).
__global__ void __launch_bounds__(256) attn_prep_kernel(__half* q_out, __half* k_cache, __half* v_cache,
                                                        const __half* q_gate, const __half* k_in, const __half* v_in,
                                                        const float* q_norm_w, const float* k_norm_w, const int* ctx,
                                                        int rows_per_seq, int hq, int hkv, long long max_seq,
                                                        float eps, float log_theta, int rope_dim, int q_head_stride,
                                                        const long long* positions, int ctx_base, __half* k_out) {
    griddep_prologue();
    __shared__ float red[32];
    __shared__ float vals[256];
    const int row = blockIdx.x;
    const int slot = blockIdx.y;
    const int d = threadIdx.x;
    const int b = row / rows_per_seq, i = row % rows_per_seq;
    const long long pos = positions ? positions[row] : static_cast<long long>(ctx ? ctx[b] : ctx_base) + i;
    const bool in_cache = pos >= 0 && pos < max_seq;
    if (slot >= hq + hkv) {  // value head: plain copy into the cache
        const int h = slot - hq - hkv;
        if (in_cache && v_cache && v_in)
            v_cache[((static_cast<long long>(b) * max_seq + pos) * hkv + h) * 256 + d] =
                v_in[(static_cast<long long>(row) * hkv + h) * 256 + d];
        return;
    }
    const bool is_q = slot < hq;
    const int h = is_q ? slot : slot - hq;
    // the reference first copies q out of the interleaved [q | gate] head block (fp16, exact)
    const float x = is_q ? __half2float(q_gate[(static_cast<long long>(row) * hq + h) * q_head_stride + d])
                         : __half2float(k_in[(static_cast<long long>(row) * hkv + h) * 256 + d]);
    const float* w = is_q ? q_norm_w : k_norm_w;
    float normed = x;
    if (w) {
        const float total = block_sum(x * x, red);
        const float r = 1.0f / sqrtf(total / 256.0f + eps);
        // rounding point: the head RMSNorm writes fp16
        normed = __half2float(__float2half_rn(x * r * w[d]));
    }
    vals[d] = normed;
    __syncthreads();
    float outv = normed;
    const int half_rot = rope_dim / 2;
    if (d < rope_dim) {
        const int pair = d < half_rot ? d : d - half_rot;
        const float freq = expf(-static_cast<float>(2 * pair) * (1.0f / static_cast<float>(rope_dim)) * log_theta);
        const float angle = static_cast<float>(pos) * freq;
        const float c = cosf(angle), s = sinf(angle);
        const float v0 = vals[pair], v1 = vals[pair + half_rot];
        outv = rotated<false>(d >= half_rot, v0, v1, c, s);
    }
    const __half o = __float2half_rn(outv);
    if (is_q) {
        q_out[(static_cast<long long>(row) * hq + h) * 256 + d] = o;
    } else if (k_cache) {
        if (in_cache) k_cache[((static_cast<long long>(b) * max_seq + pos) * hkv + h) * 256 + d] = o;
    } else if (k_out) {
        k_out[(static_cast<long long>(row) * hkv + h) * 256 + d] = o;
    }
}

// The same for many heads: a warp per (row, head slot), eight slots of a row per block; lane l holds dims l, l + 32, ...  Same
// sums in the same order.  No block barriers, and a prompt's heads are two waves of blocks instead of fourteen: 512 rows and 24
// query heads 13.9 -> 5 us.  A warp's own chain is longer: 32 heads of 32 rows take 5.6 us against 3.6.
template <bool SINE_FUSED>
__global__ void __launch_bounds__(256) attn_prep_rows_kernel(__half* q_out, __half* k_cache, __half* v_cache,
                                                        const __half* q_gate, const __half* k_in, const __half* v_in,
                                                        const float* q_norm_w, const float* k_norm_w, const int* ctx,
                                                        int rows_per_seq, int hq, int hkv, long long max_seq,
                                                        float eps, float log_theta, int rope_dim, int q_head_stride,
                                                        const long long* positions, int ctx_base, __half* k_out) {
    griddep_prologue();
    __shared__ float sh[8][256];
    __shared__ float2 sh_cs[8][128];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row = blockIdx.x;
    const int slot = blockIdx.y * 8 + warp;
    if (slot >= hq + 2 * hkv) return;
    const int b = row / rows_per_seq, i = row % rows_per_seq;
    const long long pos = positions ? positions[row] : static_cast<long long>(ctx ? ctx[b] : ctx_base) + i;
    const bool in_cache = pos >= 0 && pos < max_seq;
    if (slot >= hq + hkv) {  // value head: plain copy into the cache
        const int h = slot - hq - hkv;
        if (in_cache && v_cache && v_in) {
            __half* to = v_cache + ((static_cast<long long>(b) * max_seq + pos) * hkv + h) * 256 + lane;
            const __half* from = v_in + (static_cast<long long>(row) * hkv + h) * 256 + lane;
            __half v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = from[32 * j];
#pragma unroll
            for (int j = 0; j < 8; ++j) to[32 * j] = v[j];
        }
        return;
    }
    const bool is_q = slot < hq;
    const int h = is_q ? slot : slot - hq;
    // the reference first copies q out of the interleaved [q | gate] head block (fp16, exact)
    const __half* from = is_q ? q_gate + (static_cast<long long>(row) * hq + h) * q_head_stride : k_in + (static_cast<long long>(row) * hkv + h) * 256;
    const float* w = is_q ? q_norm_w : k_norm_w;
    float x[8], weight[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        x[j] = __half2float(from[lane + 32 * j]);
        weight[j] = w ? w[lane + 32 * j] : 0.f;
    }
    // the pairs' rotations, while the values are on their way (rolled: eight copies of sinf and cosf cost more in instruction
    // fetches than they do)
    const int half_rot = rope_dim / 2;
    float2* cs = sh_cs[warp];
#pragma unroll 1
    for (int pair = lane; pair < rope_dim - half_rot; pair += 32) {
        const float freq = expf(-static_cast<float>(2 * pair) * (1.0f / static_cast<float>(rope_dim)) * log_theta);
        const float angle = static_cast<float>(pos) * freq;
        cs[pair] = make_float2(cosf(angle), sinf(angle));
    }
    if (w) {
        float sq[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) sq[j] = warp_sum(x[j] * x[j]);
        const float total = ((sq[0] + sq[4]) + (sq[2] + sq[6])) + ((sq[1] + sq[5]) + (sq[3] + sq[7]));
        const float r = 1.0f / sqrtf(total / 256.0f + eps);
        // rounding point: the head RMSNorm writes fp16
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = __half2float(__float2half_rn(x[j] * r * weight[j]));
    }
    float* vals = sh[warp];
#pragma unroll
    for (int j = 0; j < 8; ++j) vals[lane + 32 * j] = x[j];
    __syncwarp();
    __half* to = is_q ? q_out + (static_cast<long long>(row) * hq + h) * 256
                 : k_cache ? k_cache + ((static_cast<long long>(b) * max_seq + pos) * hkv + h) * 256
                           : k_out ? k_out + (static_cast<long long>(row) * hkv + h) * 256 : nullptr;
    const bool store = is_q || (k_cache ? in_cache : k_out != nullptr);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int d = lane + 32 * j;
        float outv = x[j];
        if (d < rope_dim) {
            const int pair = d < half_rot ? d : d - half_rot;
            const float c = cs[pair].x, s = cs[pair].y;
            const float v0 = vals[pair], v1 = vals[pair + half_rot];
            outv = rotated<SINE_FUSED>(d >= half_rot, v0, v1, c, s);
        }
        if (store) to[d] = __float2half_rn(outv);
    }
}

// ------------------------------------------------------------------------------- causal conv1d + SiLU
// One thread per (sequence, channel).  state [B][3][C] holds the last three committed inputs; pending
// [B][Rmax][C] the raw inputs of the previous step, of which the first n_commit[b] were accepted.
__global__ void conv1d_spec_kernel(__half* out, const __half* in, const float* conv_w, float* state, float* pending,
                                   const int* n_commit, int rows_per_seq, int prev_rows, int channels, int nc_base,
                                   int early_state) {
    // early_state: state, pending inputs and weights are read, and the committed state written, before waiting for the kernel
    // in front of this one, from which only `in` comes (mixers.h says when that is sound).  0: everything waits.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!early_state) asm volatile("griddepcontrol.wait;" ::: "memory");
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (c >= channels) return;
    float* st = state + static_cast<long long>(b) * 3 * channels;
    float* pd = pending + static_cast<long long>(b) * 8 * channels;
    int nc = n_commit ? n_commit[b] : nc_base;
    if (nc > prev_rows) nc = prev_rows;
    // the last three inputs, with the accepted ones of the previous step behind the committed ones
    float s0 = nc < 3 ? st[nc * channels + c] : pd[(nc - 3) * channels + c];
    float s1 = nc < 2 ? st[(nc + 1) * channels + c] : pd[(nc - 2) * channels + c];
    float s2 = nc < 1 ? st[2 * channels + c] : pd[(nc - 1) * channels + c];
    st[c] = s0;
    st[channels + c] = s1;
    st[2 * channels + c] = s2;
    const float w0 = conv_w[c * 4], w1 = conv_w[c * 4 + 1], w2 = conv_w[c * 4 + 2], w3 = conv_w[c * 4 + 3];
    if (early_state) asm volatile("griddepcontrol.wait;" ::: "memory");
    // all rows (eight at most) are requested before the first is used: one trip to memory instead of one per row
    __half xs[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (i < rows_per_seq) xs[i] = in[(static_cast<long long>(b) * rows_per_seq + i) * channels + c];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (i >= rows_per_seq) break;
        const long long row = static_cast<long long>(b) * rows_per_seq + i;
        const float x = __half2float(xs[i]);
        const float sum = w0 * s0 + w1 * s1 + w2 * s2 + w3 * x;
        out[row * channels + c] = __float2half_rn(silu(sum));
        pd[i * channels + c] = x;
        s0 = s1;
        s1 = s2;
        s2 = x;
    }
}

// ------------------------------------------------------------------------------- two fp32 operations per instruction
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float sum_f32x2(uint64_t a) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a));
    return lo + hi;
}

// ------------------------------------------------------------------------------- Gated DeltaNet recurrence
// One CTA per (v head, sequence).  pend_k [B][Hv][8][128] normalised keys, pend_d [B][Hv][8][128] deltas, pend_g [B][Hv][8]
// decay factors of the previous step: replaying the accepted ones of them touches each state element with the same two
// operations in the same order every time, and gives the committed state.
//
// The state streams through: element by element it is replayed, written back and multiplied with the keys and queries of
// all tokens, and the recurrence itself is solved on those products.  With G_t the product of the decay factors up to t,
//     delta_t = beta_t (v_t - G_t k_t.S - sum_{s<t} (G_t / G_s) (k_t.k_s) delta_s)
//     out_t   =             G_t q_t.S + sum_{s<=t} (G_t / G_s) (q_t.k_s) delta_s
// (the factors G_t / G_s are products of the decays in between, never quotients).  Thread (part, j) takes 128 / PARTS rows
// of column j, BATCH at a time with the next BATCH in flight; TOKENS >= rows_per_seq.
//
// A pass is latency with few heads and memory with many (128 KB of state moved per head).  PARTS = 4, BATCH = 32: every
// load of a head is in flight at once.  PARTS = 2, BATCH = 16: three CTAs per SM, so that 384 heads (48 heads, eight
// sequences, 50 MB) are one wave.  A kernel that kept the state in registers through the tokens needed 64 registers and
// 512 threads a head, ran those 384 heads in two waves and paid a barrier per token: 23.3 us against 13.0, and with one
// sequence of four tokens 11.8 against 6.7.
constexpr int kGdnTokens = 8;  // rows_per_seq at most, and entries of the pending buffers

// sum of squares of 128 values, lane l holding l, l + 32, l + 64 and l + 96
__device__ __forceinline__ float warp_sum_sq(const float (&v)[4]) {
    float s[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] = warp_sum(v[i] * v[i]);
    return ((s[0] + s[1]) + s[2]) + s[3];
}

template <int PARTS, int BATCH, int TOKENS>
__global__ void __launch_bounds__(128 * PARTS, PARTS == 2 ? (TOKENS <= 4 ? 3 : 2) : 1) gdn_spec_kernel(
    __half* out, const __half* qkv, const __half* z, const __half* bb, const __half* aa, const float* A_log,
    const float* dt_bias, const float* norm_w, float* state, float* pend_k, float* pend_d, float* pend_g,
    const int* n_commit, int rows_per_seq, int prev_rows, int hv, int hk, int nc_base, int early_state, int perm_out) {
    // early_state: the recurrent state, the previous step's pending updates and the per-head constants (written by this layer's
    // kernel of the previous pass, and by the commit at the end of the previous step) are requested BEFORE waiting for the
    // kernel in front of this one, from which only q/k/v/z/b/a come (mixers.h says when that is sound).  0: everything waits.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!early_state) asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int kRows = 128 / PARTS, kThreads = 128 * PARTS, kWarps = 4 * PARTS;
    static_assert(TOKENS <= kWarps, "a warp per token");
    __shared__ __align__(16) float sh_q[TOKENS][128], sh_k[TOKENS][128], sh_pk[kGdnTokens][128];
    __shared__ float sh_v[TOKENS][128], sh_z[TOKENS][128], sh_pd[kGdnTokens][128], sh_pg[kGdnTokens];
    __shared__ float sums[PARTS][TOKENS][128];
    __shared__ float sh_nw[128], sh_beta[TOKENS], sh_eg[TOKENS];
    __shared__ float gram[2][TOKENS][TOKENS];  // k_t.k_s and q_t.k_s
    const int h = blockIdx.x, b = blockIdx.y;
    const int j = threadIdx.x & 127, part = threadIdx.x >> 7;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i0 = part * kRows;
    const int h_k = h / (hv / hk);
    const int channels = 2 * hk * 128 + hv * 128;
    const int value_dim = hv * 128;
    float* S = state + (static_cast<long long>(b) * hv + h) * (128 * 128) + i0 * 128 + j;
    const long long pbase = (static_cast<long long>(b) * hv + h) * kGdnTokens;

    float next[BATCH];
#pragma unroll
    for (int i = 0; i < BATCH; ++i) next[i] = S[i * 128];
    int nc = n_commit ? n_commit[b] : nc_base;
    if (nc > prev_rows) nc = prev_rows;
    for (int e = threadIdx.x; e < nc * 128; e += kThreads) {
        sh_pk[0][e] = pend_k[pbase * 128 + e];
        sh_pd[0][e] = pend_d[pbase * 128 + e];
    }
    if (threadIdx.x < nc) sh_pg[threadIdx.x] = pend_g[pbase + threadIdx.x];
    if (part == 0) sh_nw[j] = norm_w[j];
    if (early_state) asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---- per-token quantities that do not depend on the state: one warp per token
    if (warp < TOKENS) {
        const int t = warp;
        float q[4] = {}, k[4] = {}, v[4] = {}, zz[4] = {};  // (zeros beyond rows_per_seq)
        if (t < rows_per_seq) {
            const long long row = static_cast<long long>(b) * rows_per_seq + t;
            const __half* cur = qkv + row * channels;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int d = lane + 32 * i;
                q[i] = __half2float(cur[h_k * 128 + d]);
                k[i] = __half2float(cur[hk * 128 + h_k * 128 + d]);
                v[i] = __half2float(cur[2 * hk * 128 + h * 128 + d]);
                zz[i] = __half2float(z[row * value_dim + h * 128 + d]);
            }
            if (lane == 0) {
                const float b_val = __half2float(bb[row * hv + h]);
                const float a_val = __half2float(aa[row * hv + h]) + dt_bias[h];
                const float softplus = (a_val > 20.0f) ? a_val : logf(1.0f + expf(a_val));
                sh_beta[t] = 1.0f / (1.0f + expf(-b_val));
                sh_eg[t] = expf(-expf(A_log[h]) * softplus);
            }
        }
        const float q_sq = warp_sum_sq(q), k_sq = warp_sum_sq(k);
        const float rq = 1.0f / sqrtf(q_sq + 1e-6f), rk = 1.0f / sqrtf(k_sq + 1e-6f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int d = lane + 32 * i;
            sh_q[t][d] = (q[i] * rq) * 0.08838834764f;
            sh_k[t][d] = k[i] * rk;
            sh_v[t][d] = v[i];
            sh_z[t][d] = silu(zz[i]);
        }
    }
    __syncthreads();

    // ---- the state streams through
    uint64_t ks[TOKENS], qs[TOKENS];  // sums over the even and the odd rows
#pragma unroll
    for (int t = 0; t < TOKENS; ++t) ks[t] = qs[t] = 0;
#pragma unroll 1
    for (int r0 = 0; r0 < kRows; r0 += BATCH) {
        uint64_t cur[BATCH / 2];
#pragma unroll
        for (int i = 0; i < BATCH / 2; ++i) cur[i] = pack_f32x2(next[2 * i], next[2 * i + 1]);
        if (r0 + BATCH < kRows) {
#pragma unroll
            for (int i = 0; i < BATCH; ++i) next[i] = S[(r0 + BATCH + i) * 128];
        }
        if (nc > 0) {
#pragma unroll 1
            for (int t = 0; t < nc; ++t) {  // the previous step's accepted updates
                const uint64_t eg = pack_f32x2(sh_pg[t], sh_pg[t]), dj = pack_f32x2(sh_pd[t][j], sh_pd[t][j]);
                const ulonglong2* k4 = reinterpret_cast<const ulonglong2*>(&sh_pk[t][i0 + r0]);
#pragma unroll
                for (int m = 0; m < BATCH / 4; ++m) {
                    const ulonglong2 kk = k4[m];
                    cur[2 * m] = fma_f32x2(kk.x, dj, mul_f32x2(cur[2 * m], eg));
                    cur[2 * m + 1] = fma_f32x2(kk.y, dj, mul_f32x2(cur[2 * m + 1], eg));
                }
            }
#pragma unroll
            for (int i = 0; i < BATCH / 2; ++i) {
                S[(r0 + 2 * i) * 128] = __uint_as_float(static_cast<uint32_t>(cur[i]));
                S[(r0 + 2 * i + 1) * 128] = __uint_as_float(static_cast<uint32_t>(cur[i] >> 32));
            }
        }
#pragma unroll
        for (int m = 0; m < BATCH / 4; ++m) {
#pragma unroll
            for (int t = 0; t < TOKENS; ++t) {
                const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(&sh_k[t][i0 + r0 + 4 * m]);
                const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(&sh_q[t][i0 + r0 + 4 * m]);
                ks[t] = fma_f32x2(cur[2 * m + 1], kk.y, fma_f32x2(cur[2 * m], kk.x, ks[t]));
                qs[t] = fma_f32x2(cur[2 * m + 1], qq.y, fma_f32x2(cur[2 * m], qq.x, qs[t]));
            }
        }
    }
#pragma unroll
    for (int t = 0; t < TOKENS; ++t) sums[part][t][j] = sum_f32x2(ks[t]);
    // products among the tokens: k or q of a token with the keys up to it
    for (int e = warp; e < 2 * TOKENS; e += kWarps) {
        const int t = e >> 1;
        const float* a = (e & 1) ? sh_q[t] : sh_k[t];
        const float a0 = a[lane], a1 = a[lane + 32], a2 = a[lane + 64], a3 = a[lane + 96];
        for (int u = 0; u <= t && t < rows_per_seq; ++u) {
            const float g = warp_sum((a0 * sh_k[u][lane] + a1 * sh_k[u][lane + 32]) + (a2 * sh_k[u][lane + 64] + a3 * sh_k[u][lane + 96]));
            if (lane == 0) gram[e & 1][t][u] = g;
        }
    }
    __syncthreads();
    float kS[TOKENS];
    auto column_sum = [&](int t) {
        float v = sums[0][t][j] + sums[1][t][j];
        if constexpr (PARTS == 4) v += sums[2][t][j] + sums[3][t][j];
        return v;
    };
    if (part == 0) {
#pragma unroll
        for (int t = 0; t < TOKENS; ++t) kS[t] = column_sum(t);
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < TOKENS; ++t) sums[part][t][j] = sum_f32x2(qs[t]);
    __syncthreads();

    // ---- the recurrence on the products; part 0 keeps the deltas
    if (part == 0) {
        float delta[TOKENS], decay[TOKENS];  // decay[u]: from token u to the present one
        float G = 1.f;
#pragma unroll
        for (int t = 0; t < TOKENS; ++t) {
            if (t >= rows_per_seq) break;
            const float eg = sh_eg[t];
            G *= eg;
            float mem = G * kS[t], att = G * column_sum(t);
#pragma unroll
            for (int u = 0; u < t; ++u) {
                decay[u] *= eg;
                const float d = decay[u] * delta[u];
                mem += gram[0][t][u] * d;
                att += gram[1][t][u] * d;
            }
            decay[t] = 1.f;
            delta[t] = (sh_v[t][j] - mem) * sh_beta[t];
            sums[0][t][j] = att + gram[1][t][t] * delta[t];
            pend_d[(pbase + t) * 128 + j] = delta[t];
            if (j == 0) pend_g[pbase + t] = eg;
        }
    } else if (part == 1) {
        for (int t = 0; t < rows_per_seq; ++t) pend_k[(pbase + t) * 128 + j] = sh_k[t][j];
    }
    __syncthreads();

    // ---- gated RMSNorm of every token's output: one warp per token
    if (warp < rows_per_seq) {
        const int t = warp;
        const float* at = sums[0][t];
        const float a[4] = {at[lane], at[lane + 32], at[lane + 64], at[lane + 96]};
        const float sq = warp_sum_sq(a);
        const float inv_std = 1.0f / sqrtf(sq / 128.0f + 1e-6f);
        __half* orow = out + (static_cast<long long>(b) * rows_per_seq + t) * value_dim + h * 128;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int d = lane + 32 * i;
            orow[perm_out ? perm8(d) : d] = __float2half_rn(a[i] * inv_std * sh_nw[d] * sh_z[t][d]);
        }
    }
}

// ------------------------------------------------------------------------------- the same two mixers over a prompt chunk
// Prefill keeps every row, so there is nothing to replay or to hold back.  Rows are [sequence][position].
//
// The convolution has no recurrence on its outputs (y_p needs the inputs p-3 .. p only): a thread takes V channels and
// SPAN consecutive positions with the window in registers.  The threads of the first positions are the only readers of
// the state and also the ones that replace it by the chunk's last three inputs, so one launch does both.  512 x 10240 in 9.7 us
// (its 21 MB take 3.2 at the copy's rate; 11.9 with the weights loaded one by one).
// SPAN 0: all positions, when the output overwrites the input (a position's inputs are its neighbours').  A store may not pass the
// loads behind it, so the inputs are read kAhead positions at a time there too: 512 x 10240 in 65 us, four channels a thread in 86,
// position by position in 172.
constexpr int kAhead = 8, kConvNarrowBlocks = 3;
template <int V, int SPAN>
__global__ void __launch_bounds__(128) conv1d_chunk_kernel(__half* out, const __half* in, const float* conv_w, float* state, int rc,
                                                           int channels) {
    griddep_prologue();
    const int c = (blockIdx.z * 128 + threadIdx.x) * V;
    const int b = blockIdx.y, p0 = blockIdx.x * SPAN;
    const long long seq0 = static_cast<long long>(b) * rc;
    if (c >= channels) return;
    // (a channel's four weights in one load: one by one, sixteen bytes apart, the lanes' requests were more than the activations')
    float w[V][4];
    if ((reinterpret_cast<uintptr_t>(conv_w) & 15) == 0) {
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const float4 q = __ldg(reinterpret_cast<const float4*>(conv_w) + c + e);
            w[e][0] = q.x;
            w[e][1] = q.y;
            w[e][2] = q.z;
            w[e][3] = q.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < V; ++e) {
#pragma unroll
            for (int t = 0; t < 4; ++t) w[e][t] = conv_w[(c + e) * 4 + t];
        }
    }
    float* st = state ? state + static_cast<long long>(b) * 3 * channels : nullptr;
    struct alignas(2 * V) Vec { __half h[V]; };
    auto load = [&](int p, float (&x)[V]) {  // the input at position p; negative: the state's slot 3 + p
        if (p >= 0) {
            const Vec v = *reinterpret_cast<const Vec*>(in + (seq0 + p) * channels + c);
#pragma unroll
            for (int e = 0; e < V; ++e) x[e] = __half2float(v.h[e]);
        } else {
#pragma unroll
            for (int e = 0; e < V; ++e) x[e] = st ? st[(3 + p) * static_cast<long long>(channels) + c + e] : 0.f;
        }
    };
    float x0[V], x1[V], x2[V], tail[3][V];
    load(p0 - 3, x0);
    load(p0 - 2, x1);
    load(p0 - 1, x2);
    if (p0 == 0 && st) {
#pragma unroll
        for (int t = 0; t < 3; ++t) load(rc - 3 + t, tail[t]);
    }
    auto emit = [&](int p, const float (&x)[V]) {
        Vec o;
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const float sum = w[e][0] * x0[e] + w[e][1] * x1[e] + w[e][2] * x2[e] + w[e][3] * x[e];
            o.h[e] = __float2half_rn(silu(sum));
            x0[e] = x1[e];
            x1[e] = x2[e];
            x2[e] = x[e];
        }
        *reinterpret_cast<Vec*>(out + (seq0 + p) * channels + c) = o;
    };
    // eight positions requested before the first is used
    const int p1 = SPAN > 0 ? p0 + SPAN : rc;
#pragma unroll 1
    for (int p = p0; p < p1; p += kAhead) {
        Vec raw[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i)
            if (p + i < rc) raw[i] = *reinterpret_cast<const Vec*>(in + (seq0 + p + i) * channels + c);
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            if (p + i < rc) {
                float x[V];
#pragma unroll
                for (int e = 0; e < V; ++e) x[e] = __half2float(raw[i].h[e]);
                emit(p + i, x);
            }
        }
    }
    if (p0 == 0 && st) {
#pragma unroll
        for (int t = 0; t < 3; ++t) {
#pragma unroll
            for (int e = 0; e < V; ++e) st[t * static_cast<long long>(channels) + c + e] = tail[t][e];
        }
    }
}

// The delta rule over a chunk: rc sequential tokens, so what counts is the latency of a token and how few instructions it
// takes.  The columns of a head's 128 x 128 state do not interact, so a head is eight CTAs of 16 columns (one cluster; with
// one sequence 48 heads alone would be 48 SMs), and inside a CTA a warp owns four columns by itself - eight lanes per
// column, 16 rows each, in registers - and runs its tokens without any barrier:
//   both dot products of a token are taken on the old state S, together:    ks = k.S, qs = q.S   (three shuffles each)
//   delta = (v - g ks) beta;    out = g qs + (q.k) delta = q.(g S + k delta);    S = g S + k delta
// At most kGdnWalkRows tokens, whose q, k, v, norms and gates are all in shared memory before the first is walked.  The gated
// RMSNorm of the outputs spans the head's 128 columns: every CTA sends its sums of squares to the other seven through
// distributed shared memory, and writes its state back while the cluster barrier completes.
// For short chunks; a token costs 0.6 us.
// Up to here the token-by-token kernel is the faster one (16 rows: 13 us against 15 for the launches of the blocked form).
constexpr int kGdnWalkRows = 16;
constexpr int kGdnCols = 16, kGdnSlices = 128 / kGdnCols, kGdnThreads = kGdnCols * 8;

__global__ void __cluster_dims__(kGdnSlices, 1, 1) __launch_bounds__(kGdnThreads) gdn_walk_kernel(
    __half* out, const __half* qkv, const __half* z, const __half* bb, const __half* aa, const float* A_log, const float* dt_bias,
    const float* norm_w, float* state, int rc, int hv, int hk, int zero_state) {
    cluster_arrive();  // (a CTA may write into another one's shared memory once that one has started)
    griddep_prologue();
    __shared__ __align__(16) float sh_q[kGdnWalkRows][128], sh_k[kGdnWalkRows][128];
    __shared__ float sh_v[kGdnWalkRows][kGdnCols], sh_out[kGdnWalkRows][kGdnCols + 1];
    __shared__ float4 sh_gate[kGdnWalkRows];           // decay, beta, q.k
    __shared__ float sh_sq[kGdnSlices][kGdnWalkRows];  // sums of squares of the outputs, by column slice
    __shared__ float sh_s[128][kGdnCols + 1];
    const int slice = blockIdx.x % kGdnSlices, h = blockIdx.x / kGdnSlices, b = blockIdx.y;
    const long long seq0 = static_cast<long long>(b) * rc;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cl = lane >> 3, rg = lane & 7, col = warp * 4 + cl;  // rows of a lane: 4 (rg + 8 m) + e, m, e = 0..3
    const int h_k = h / (hv / hk), channels = 2 * hk * 128 + hv * 128, value_dim = hv * 128;
    const int col0 = slice * kGdnCols;
    // the output columns of this thread: token tid / 8, columns 2 (tid % 8) and the next
    const int ot = tid >> 3, oc = (tid & 7) * 2;

    // ---- the state slice, through shared memory so that global accesses are whole 64-byte rows
    float* S = state + (static_cast<long long>(b) * hv + h) * (128 * 128) + col0;
    uint64_t s2[8];
    if (zero_state) {
#pragma unroll
        for (int i = 0; i < 8; ++i) s2[i] = 0;
    } else {
#pragma unroll
        for (int i = 0; i < 128 * kGdnCols / (4 * kGdnThreads); ++i) {
            const int idx = i * kGdnThreads + tid, row = idx >> 2, c4 = (idx & 3) * 4;
            const float4 v = *reinterpret_cast<const float4*>(S + row * 128 + c4);
            sh_s[row][c4] = v.x; sh_s[row][c4 + 1] = v.y; sh_s[row][c4 + 2] = v.z; sh_s[row][c4 + 3] = v.w;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = 4 * (rg + 8 * (i >> 1)) + 2 * (i & 1);
            s2[i] = pack_f32x2(sh_s[row][col], sh_s[row + 1][col]);
        }
    }
    const float exp_a_log = expf(A_log[h]), dtb = dt_bias[h];
    const float nw0 = norm_w[col0 + oc], nw1 = norm_w[col0 + oc + 1];

    // ---- the inputs: each warp takes q and k of four tokens, the CTA its 16 values per token, 16 threads the gates
    uint2 rq[kGdnWalkRows / 4], rk[kGdnWalkRows / 4];
#pragma unroll
    for (int u = 0; u < kGdnWalkRows / 4; ++u) {
        const int t = warp + 4 * u;
        if (t < rc) {
            const __half* cur = qkv + (seq0 + t) * channels + h_k * 128 + lane * 4;
            rq[u] = *reinterpret_cast<const uint2*>(cur);
            rk[u] = *reinterpret_cast<const uint2*>(cur + hk * 128);
        }
    }
    if (ot < rc) {
        const long long row = seq0 + ot;
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(qkv + row * channels + 2 * hk * 128 + h * 128 + col0 + oc));
        sh_v[ot][oc] = v.x;
        sh_v[ot][oc + 1] = v.y;
        if ((tid & 7) == 0) {
            const float a_val = __half2float(aa[row * hv + h]) + dtb;
            const float softplus = (a_val > 20.0f) ? a_val : logf(1.0f + expf(a_val));
            sh_gate[ot].x = expf(-exp_a_log * softplus);
            sh_gate[ot].y = 1.0f / (1.0f + expf(-__half2float(bb[row * hv + h])));
        }
    }
#pragma unroll
    for (int u = 0; u < kGdnWalkRows / 4; ++u) {
        const int t = warp + 4 * u;
        if (t < rc) {
            const float2 qa = __half22float2(*reinterpret_cast<const __half2*>(&rq[u].x)), qb = __half22float2(*reinterpret_cast<const __half2*>(&rq[u].y));
            const float2 ka = __half22float2(*reinterpret_cast<const __half2*>(&rk[u].x)), kb = __half22float2(*reinterpret_cast<const __half2*>(&rk[u].y));
            const float q_sq = warp_sum(qa.x * qa.x + qa.y * qa.y + qb.x * qb.x + qb.y * qb.y);
            const float k_sq = warp_sum(ka.x * ka.x + ka.y * ka.y + kb.x * kb.x + kb.y * kb.y);
            const float iq = 1.0f / sqrtf(q_sq + 1e-6f), ik = 1.0f / sqrtf(k_sq + 1e-6f);
            const float4 qn = make_float4((qa.x * iq) * 0.08838834764f, (qa.y * iq) * 0.08838834764f, (qb.x * iq) * 0.08838834764f,
                                          (qb.y * iq) * 0.08838834764f);
            const float4 kn = make_float4(ka.x * ik, ka.y * ik, kb.x * ik, kb.y * ik);
            const float qk = warp_sum(qn.x * kn.x + qn.y * kn.y + qn.z * kn.z + qn.w * kn.w);
            *reinterpret_cast<float4*>(&sh_q[t][lane * 4]) = qn;
            *reinterpret_cast<float4*>(&sh_k[t][lane * 4]) = kn;
            if (lane == 0) sh_gate[t].z = qk;
        }
    }
    __syncthreads();

    // ---- the tokens
#pragma unroll 1
    for (int t = 0; t < rc; ++t) {
        const float4 gate = sh_gate[t];
        const float v = sh_v[t][col];
        uint64_t k2[8], ks0 = 0, ks1 = 0, qs0 = 0, qs1 = 0;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(&sh_k[t][4 * (rg + 8 * m)]);
            const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(&sh_q[t][4 * (rg + 8 * m)]);
            k2[2 * m] = kk.x;
            k2[2 * m + 1] = kk.y;
            ks0 = fma_f32x2(s2[2 * m], kk.x, ks0);
            ks1 = fma_f32x2(s2[2 * m + 1], kk.y, ks1);
            qs0 = fma_f32x2(s2[2 * m], qq.x, qs0);
            qs1 = fma_f32x2(s2[2 * m + 1], qq.y, qs1);
        }
        float ks = sum_f32x2(ks0) + sum_f32x2(ks1), qs = sum_f32x2(qs0) + sum_f32x2(qs1);
#pragma unroll
        for (int off = 1; off < 8; off <<= 1) {
            ks += __shfl_xor_sync(0xffffffffu, ks, off);
            qs += __shfl_xor_sync(0xffffffffu, qs, off);
        }
        const float delta = (v - gate.x * ks) * gate.y;
        const uint64_t d2 = pack_f32x2(delta, delta), g2 = pack_f32x2(gate.x, gate.x);
#pragma unroll
        for (int i = 0; i < 8; ++i) s2[i] = fma_f32x2(k2[i], d2, mul_f32x2(s2[i], g2));
        if (rg == 0) sh_out[t][col] = gate.x * qs + gate.z * delta;
    }
    __syncthreads();

    // ---- sums of squares: eight threads per token, the r-th of them sends to CTA r of the cluster
    const float o0 = ot < rc ? sh_out[ot][oc] : 0.f, o1 = ot < rc ? sh_out[ot][oc + 1] : 0.f;
    float sq = o0 * o0 + o1 * o1;
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
    cluster_wait();
    st_shared_cluster_f32(mapa_shared_cluster(smem_u32(&sh_sq[slice][ot]), tid & 7), sq);
    cluster_arrive();

#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = 4 * (rg + 8 * (i >> 1)) + 2 * (i & 1);
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(s2[i]));
        sh_s[row][col] = lo;
        sh_s[row + 1][col] = hi;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 128 * kGdnCols / (4 * kGdnThreads); ++i) {
        const int idx = i * kGdnThreads + tid, row = idx >> 2, c4 = (idx & 3) * 4;
        *reinterpret_cast<float4*>(S + row * 128 + c4) = make_float4(sh_s[row][c4], sh_s[row][c4 + 1], sh_s[row][c4 + 2], sh_s[row][c4 + 3]);
    }
    cluster_wait();
    if (ot < rc) {
        float total = 0.f;
#pragma unroll
        for (int r = 0; r < kGdnSlices; ++r) total += sh_sq[r][ot];
        const float inv_std = 1.0f / sqrtf(total / 128.0f + 1e-6f);
        const long long at = (seq0 + ot) * value_dim + h * 128 + col0 + oc;
        const float2 zv = __half22float2(*reinterpret_cast<const __half2*>(z + at));
        const float y0 = o0 * inv_std * nw0 * silu(zv.x), y1 = o1 * inv_std * nw1 * silu(zv.y);
        *reinterpret_cast<__half2*>(out + at) = __floats2half2_rn(y0, y1);
    }
}

// ------------------------------------------------------------------------------- the delta rule over longer chunks
// Blocks of 16 tokens on the tensor cores.  With G_i the product of the decay factors of a block's tokens 0 .. i (kept as
// sums of logarithms, so only ratios <= 1 are ever formed) and S0 the state in front of the block, the recurrence unrolls to
//   delta = (I + L)^-1 diag(beta) (V - diag(G) K S0),     L_ij = beta_i G_i / G_j (k_i.k_j)   for j < i
//   O = diag(G) Q S0 + P delta,                           P_ij = G_i / G_j (q_i.k_j)          for j <= i
//   S = G_15 S0 + K^T diag(G_15 / G_j) delta
// which is the same arithmetic, token for token, in another order (the blocked form of the delta rule published as
// "Parallelizing Linear Transformers with the Delta Rule over Sequence Length", Yang et al. 2024).  What does not involve the
// state - (I + L)^-1 - I, P, the norms and the decays - is computed for all blocks of all heads at once by
// gdn_block_kernel, a warp per block; gdn_scan_kernel then walks the blocks.
//
// Everything keeps fp32's precision: k and q enter as their raw fp16 values (their norms are row factors), every other
// operand x as two fp16 values, hi = rn(x) and mid = rn(2^11 (x - hi)); the products with mid are summed apart and scaled back.
// Together they hold x to 2^-24 of itself from 2^-12 upwards and to 2^-36 below, so what is proportional to the state is carried
// times a power of two f, which a warp chooses for its sixteen value columns: when the largest of f |S| and f beta |v| of the
// coming block has left [2^-4, 2], f brings it back to [1/2, 1).  The rule enlarges nothing (beta <= 1, |k| <= 1), so f |delta|
// stays below 32 inside a block and its product with 1 / |k| <= 1000 inside fp16.  (A fixed factor of 2^-4 before: states of
// 1e-4 were carried to 1e-4 of themselves, a key near zero beside large values or a state above 2^20 gave NaN.  The choice costs 4
// of the scan's 46 us at 512 tokens.)  What falls by more than 2^12 within sixteen tokens is, in those, held to 2^-36 of where it
// came from.  delta is (r + ((I + L)^-1 - I) r): the tensor core's sums, which truncate, only get the smaller part.
// (With tf32 operands the same kernel ran at a quarter of the rate: mma.sync of that type does 90 multiply-adds per clock and SM.)
// Transposed products (state S^T, with the value columns as the MMA's rows) let a warp keep its 16 x 128 slice of the state
// in accumulators that are A operands as they stand.
// Bound by the latency of a block, one warp per scheduler, so nothing that the next block does not wait for stays in the walk:
// it leaves the raw outputs in fp32, and gdn_norm_kernel does their gated RMSNorm, which spans all columns of a head, for all
// tokens at once (with a cluster adding up the squares inside the walk the scan took 145 us).
// 512 tokens, one sequence, 48 heads: 61 us, 1.5 ms through the step's kernel eight tokens a launch, 300 us with
// gdn_walk_kernel.
constexpr int kScanBlock = 16, kScanWarps = 2, kScanCols = 16 * kScanWarps, kScanSlices = 128 / kScanCols, kScanPitch = 136;
constexpr float kMidUp = 2048.0f, kMidDown = 1.0f / 2048.0f;
struct GdnBlock {                         // one block of one head, written by gdn_block_kernel
    __half t[2][kScanBlock][kScanBlock];  // (I + L)^-1 - I: rn(x), rn(2^11 (x - hi))
    __half p[2][kScanBlock][kScanBlock];
    float4 coef[kScanBlock];              // per token: beta_i G_i / |k_i|, G_i / (|q_i| sqrt(128)), G_15 / G_i / |k_i|, beta_i
    float decay, most, pad[2];            // G_15; the largest beta_i |v_i|
};

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Two values as fp16 pairs hi and mid.
__device__ __forceinline__ void split_f16x2(float x, float y, uint32_t& hi, uint32_t& mid) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 m = __floats2half2_rn((x - f.x) * kMidUp, (y - f.y) * kMidUp);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    mid = *reinterpret_cast<const uint32_t*>(&m);
}
// Two adjacent C fragments (16 x 8 each) as the A fragment of the 16 x 16 tile.
__device__ __forceinline__ void split_frag(const float (&c0)[4], const float (&c1)[4], uint32_t (&hi)[4], uint32_t (&mid)[4]) {
    split_f16x2(c0[0], c0[1], hi[0], mid[0]);
    split_f16x2(c0[2], c0[3], hi[1], mid[1]);
    split_f16x2(c1[0], c1[1], hi[2], mid[2]);
    split_f16x2(c1[2], c1[3], hi[3], mid[3]);
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// The largest of the lanes' values, none of them negative.
__device__ __forceinline__ float warp_most(float v) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v))); }

// One warp per (block, value head, sequence).
__global__ void __launch_bounds__(128) gdn_block_kernel(GdnBlock* blocks, const __half* qkv, const __half* bb, const __half* aa,
                                                        const float* A_log, const float* dt_bias, int rc, int hv, int hk) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float sh_l[4][kScanBlock][kScanBlock + 1];
    __shared__ float sh_lg[4][kScanBlock], sh_ik[4][kScanBlock], sh_iq[4][kScanBlock], sh_beta[4][kScanBlock];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int nblocks = (rc + kScanBlock - 1) / kScanBlock;
    const int blk = blockIdx.x * 4 + warp, h = blockIdx.y, b = blockIdx.z;
    const long long seq0 = static_cast<long long>(b) * rc;
    if (blk >= nblocks) return;  // (no barrier below spans warps)
    const int p0 = blk * kScanBlock, h_k = h / (hv / hk), channels = 2 * hk * 128 + hv * 128;
    GdnBlock& out = blocks[(static_cast<long long>(b) * hv + h) * nblocks + blk];

    // rows g and g + 8 of K and Q as A fragments; the same registers are the B fragments of K^T
    const __half *k_row[2], *q_row[2];
    bool live[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int p = p0 + g + 8 * r;
        live[r] = p < rc;
        q_row[r] = qkv + (seq0 + (live[r] ? p : p0)) * channels + h_k * 128;
        k_row[r] = q_row[r] + hk * 128;
    }
    // the largest |v| of eight values of rows 2u + lane / 16
    float v_most[kScanBlock / 2];
#pragma unroll
    for (int u = 0; u < kScanBlock / 2; ++u) {
        const int p = p0 + 2 * u + (lane >> 4);
        const uint4 v = *reinterpret_cast<const uint4*>(qkv + (seq0 + (p < rc ? p : p0)) * channels + 2 * hk * 128 + h * 128 + (lane & 15) * 8);
        const __half2* v2 = reinterpret_cast<const __half2*>(&v);
        const __half2 m = __hmax2(__hmax2(__habs2(v2[0]), __habs2(v2[1])), __hmax2(__habs2(v2[2]), __habs2(v2[3])));
        v_most[u] = fminf(fmaxf(__low2float(m), __high2float(m)), 65504.f);  // (an infinity takes only its own column along)
    }
    float kk[2][4] = {}, qk[2][4] = {}, k_sq[2] = {0.f, 0.f}, q_sq[2] = {0.f, 0.f};
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
        uint32_t ka[4], qa[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = i & 1, col = ks * 16 + (i >> 1) * 8 + 2 * t;
            ka[i] = live[r] ? *reinterpret_cast<const uint32_t*>(k_row[r] + col) : 0u;
            qa[i] = live[r] ? *reinterpret_cast<const uint32_t*>(q_row[r] + col) : 0u;
            const float2 kf = __half22float2(*reinterpret_cast<const __half2*>(&ka[i])), qf = __half22float2(*reinterpret_cast<const __half2*>(&qa[i]));
            k_sq[r] += kf.x * kf.x + kf.y * kf.y;
            q_sq[r] += qf.x * qf.x + qf.y * qf.y;
        }
        mma_f16(kk[0], ka, ka[0], ka[2]);
        mma_f16(kk[1], ka, ka[1], ka[3]);
        mma_f16(qk[0], qa, ka[0], ka[2]);
        mma_f16(qk[1], qa, ka[1], ka[3]);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
#pragma unroll
        for (int off = 1; off < 4; off <<= 1) {
            k_sq[r] += __shfl_xor_sync(0xffffffffu, k_sq[r], off);
            q_sq[r] += __shfl_xor_sync(0xffffffffu, q_sq[r], off);
        }
        if (t == 0) {
            sh_ik[warp][g + 8 * r] = 1.0f / sqrtf(k_sq[r] + 1e-6f);
            sh_iq[warp][g + 8 * r] = (1.0f / sqrtf(q_sq[r] + 1e-6f)) * 0.08838834764f;
        }
    }
    // log of the cumulative decay and beta; positions behind the end decay nothing and write nothing
    float lg = 0.f, beta = 0.f;
    if (lane < kScanBlock && p0 + lane < rc) {
        const long long row = (seq0 + p0 + lane);
        const float a_val = __half2float(aa[row * hv + h]) + dt_bias[h];
        const float softplus = (a_val > 20.0f) ? a_val : logf(1.0f + expf(a_val));
        lg = -expf(A_log[h]) * softplus;
        beta = 1.0f / (1.0f + expf(-__half2float(bb[row * hv + h])));
    }
    if (lane < kScanBlock) { sh_lg[warp][lane] = lg; sh_beta[warp][lane] = beta; }
    __syncwarp();
    // logarithms of G_i / G_j, summed from j + 1 on (a difference of prefix sums would lose what they have in common)
    const int j = lane & (kScanBlock - 1);
    float prefix = 0.f, suffix = 0.f;
    for (int i = 0; i <= j; ++i) prefix += sh_lg[warp][i];
    if (lane < kScanBlock) {
        for (int i = j + 1; i < kScanBlock; ++i) {
            suffix += sh_lg[warp][i];
            sh_l[warp][i][j] = suffix;
        }
        sh_l[warp][j][j] = 0.f;
    }
    __syncwarp();
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
        float ratio[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = g + 8 * (e >> 1), jj = nt * 8 + 2 * t + (e & 1);
            ratio[e] = jj <= i ? expf(sh_l[warp][i][jj]) : 0.f;
        }
        float pv[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = g + 8 * (e >> 1), jj = nt * 8 + 2 * t + (e & 1);
            const float ikj = sh_ik[warp][jj];
            sh_l[warp][i][jj] = jj < i ? sh_beta[warp][i] * ratio[e] * (kk[nt][e] * sh_ik[warp][i] * ikj) : 0.f;
            pv[e] = ratio[e] * (qk[nt][e] * sh_iq[warp][i] * ikj);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            uint32_t hi, mid;
            split_f16x2(pv[2 * r], pv[2 * r + 1], hi, mid);
            *reinterpret_cast<uint32_t*>(&out.p[0][g + 8 * r][nt * 8 + 2 * t]) = hi;
            *reinterpret_cast<uint32_t*>(&out.p[1][g + 8 * r][nt * 8 + 2 * t]) = mid;
        }
    }
    __syncwarp();
    // column j of the inverse by forward substitution, a lane per column
    float x[kScanBlock];
#pragma unroll
    for (int i = 0; i < kScanBlock; ++i) {
        float s0 = i == j ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
        for (int m = 0; m < i; ++m) {
            if (m & 1) s1 = fmaf(-sh_l[warp][i][m], x[m], s1);
            else s0 = fmaf(-sh_l[warp][i][m], x[m], s0);
        }
        x[i] = s0 + s1;
    }
    if (lane < kScanBlock) {
        const float bj = sh_beta[warp][j];
#pragma unroll
        for (int i = 0; i < kScanBlock; ++i) {
            const float v = i > j ? x[i] : 0.f;
            const __half hi = __float2half_rn(v);
            out.t[0][i][j] = hi;
            out.t[1][i][j] = __float2half_rn((v - __half2float(hi)) * kMidUp);
        }
        const float gj = expf(prefix);
        out.coef[j] = make_float4(bj * gj * sh_ik[warp][j], gj * sh_iq[warp][j], expf(suffix) * sh_ik[warp][j], bj);
        if (lane == 0) out.decay = expf(prefix + suffix);
    }
    // the largest beta |v|: sixteen lanes a row
    float most = 0.f;
#pragma unroll
    for (int u = 0; u < kScanBlock / 2; ++u) {
        const int i = 2 * u + (lane >> 4);
        most = fmaxf(most, sh_beta[warp][i] * v_most[u]);  // (beta is 0 behind the end)
    }
    most = warp_most(most);
    if (lane == 0) out.most = most;
    // Only now: CTAs of the scan that are placed between this kernel's end up two and three on one SM beside empty ones, and the
    // fullest SM sets the scan's time (128 tokens: 38 us for the three launches with the signal at the front, 25 with it here).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__global__ void __launch_bounds__(32 * kScanWarps) gdn_scan_kernel(float* raw, const __half* qkv, const GdnBlock* blocks, float* state,
                                                                   int rc, int hv, int hk, int zero_state) {
    griddep_prologue();
    __shared__ __align__(16) __half sh_q[2][kScanBlock][kScanPitch], sh_k[2][kScanBlock][kScanPitch];
    __shared__ __align__(16) __half sh_v[2][kScanBlock][kScanCols + 8];
    __shared__ __align__(16) GdnBlock sh_blk[2];
    const int slice = blockIdx.x % kScanSlices, h = blockIdx.x / kScanSlices, b = blockIdx.y;
    const long long seq0 = static_cast<long long>(b) * rc;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int nblocks = (rc + kScanBlock - 1) / kScanBlock;
    const int h_k = h / (hv / hk), channels = 2 * hk * 128 + hv * 128, value_dim = hv * 128;
    const int c0 = slice * kScanCols + warp * 16 + g;  // value columns of this thread: c0 and c0 + 8
    const GdnBlock* blk = blocks + (static_cast<long long>(b) * hv + h) * nblocks;
    float* S = state + (static_cast<long long>(b) * hv + h) * (128 * 128);

    // A block's q, k, v, matrices and factors: 16-byte pieces straight into shared memory, zeros behind the end.  (The small
    // operands were fetched to registers a block ahead before, but with 255 of them in use the compiler moved the loads down to
    // where they are needed: a trip to L2 in every block, 85 us against 67.)
    auto stage = [&](int n) {
        const int buf = n & 1;
#pragma unroll
        for (int u = 0; u < kScanBlock * 16 / (32 * kScanWarps); ++u) {
            const int idx = u * 32 * kScanWarps + tid, row = idx >> 4, c = (idx & 15) * 8, p = n * kScanBlock + row;
            const __half* cur = qkv + (seq0 + (p < rc ? p : n * kScanBlock)) * channels + h_k * 128 + c;
            const int bytes = p < rc ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(&sh_q[buf][row][c])), "l"(cur), "r"(bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(&sh_k[buf][row][c])), "l"(cur + hk * 128), "r"(bytes) : "memory");
        }
        constexpr int kVPieces = kScanCols / 8, kBlkPieces = static_cast<int>(sizeof(GdnBlock) / 16);
#pragma unroll
        for (int u = 0; u < (kScanBlock * kVPieces + 32 * kScanWarps - 1) / (32 * kScanWarps); ++u) {
            const int idx = u * 32 * kScanWarps + tid, row = idx / kVPieces, c = (idx % kVPieces) * 8, p = n * kScanBlock + row;
            const __half* cur = qkv + (seq0 + (p < rc ? p : n * kScanBlock)) * channels + 2 * hk * 128 + h * 128 + slice * kScanCols + c;
            if (row < kScanBlock)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(&sh_v[buf][row][c])), "l"(cur), "r"(p < rc ? 16 : 0) : "memory");
        }
#pragma unroll
        for (int u = 0; u < (kBlkPieces + 32 * kScanWarps - 1) / (32 * kScanWarps); ++u) {
            const int idx = u * 32 * kScanWarps + tid;
            if (idx < kBlkPieces)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&sh_blk[buf]) + idx * 16),
                             "l"(reinterpret_cast<const char*>(blk + n) + idx * 16) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0);

    float s[16][4];  // f S^T: s[n][e] = f S[8n + 2t + (e & 1)][c0 + 8 (e >> 1)]
    float f = 1.f, inv_f = 1.f;  // powers of two
    float most = blk[0].most;       // the largest of f |S| and f beta |v|

#pragma unroll
    for (int n = 0; n < 16; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            s[n][e] = zero_state ? 0.f : S[(8 * n + 2 * t + (e & 1)) * 128 + c0 + 8 * (e >> 1)];
            most = fmaxf(most, fabsf(s[n][e]));
        }
    }
    most = warp_most(most);
    // ldmatrix addresses: [token][state row] tiles, (token halves) x (row halves), plain and transposed
    const uint32_t lm_row = static_cast<uint32_t>(((lane >> 4) & 1) * 8 + (lane & 7)), lm_col = static_cast<uint32_t>(((lane >> 3) & 1) * 8);
    const uint32_t lt_row = static_cast<uint32_t>(((lane >> 3) & 1) * 8 + (lane & 7)), lt_col = static_cast<uint32_t>(((lane >> 4) & 1) * 8);

    for (int n = 0; n < nblocks; ++n) {
        const int buf = n & 1;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (n + 1 < nblocks) stage(n + 1);
        const GdnBlock& here = sh_blk[buf];
        if ((most > 2.0f && most < INFINITY) || (most < 0.0625f && most > 0.f)) {  // (the same for the warp)
            int step = 126 - static_cast<int>(__float_as_uint(most) >> 23);
            const int now = static_cast<int>(__float_as_uint(f) >> 23) - 127;  // (f stays within 2^-100 .. 2^100)
            step = now + step > 100 ? 100 - now : (now + step < -100 ? -100 - now : step);
            const float by = __uint_as_float(static_cast<uint32_t>(127 + step) << 23);
            f *= by;
            inv_f *= __uint_as_float(static_cast<uint32_t>(127 - step) << 23);
#pragma unroll
            for (int m = 0; m < 16; ++m) {
#pragma unroll
                for (int e = 0; e < 4; ++e) s[m][e] *= by;
            }
        }
        most = n + 1 < nblocks ? f * blk[n + 1].most : 0.f;
        float s_most[2] = {0.f, 0.f};

        // (K S0)^T and (Q S0)^T: 16 value columns x 16 tokens, contraction over the 128 state rows
        float ks[2][2][4] = {}, qs[2][2][4] = {};  // [hi, mid][token tile]
        const uint32_t k_base = smem_u32(&sh_k[buf][lm_row][lm_col]), q_base = smem_u32(&sh_q[buf][lm_row][lm_col]);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            uint32_t hi[4], mid[4], kb[4], qb[4];
            ldsm4(k_base + m * 32, kb);
            ldsm4(q_base + m * 32, qb);
            split_frag(s[2 * m], s[2 * m + 1], hi, mid);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                mma_f16(ks[0][nt], hi, kb[2 * nt], kb[2 * nt + 1]);
                mma_f16(qs[0][nt], hi, qb[2 * nt], qb[2 * nt + 1]);
                mma_f16(ks[1][nt], mid, kb[2 * nt], kb[2 * nt + 1]);
                mma_f16(qs[1][nt], mid, qb[2 * nt], qb[2 * nt + 1]);
            }
        }
        float v[2][4];  // f beta v of the thread's two columns, tokens 8 (i / 2) + 2t + i % 2
        float4 coef[4];
        uint32_t tm[2][2][2], pm[2][2][2];  // [hi, mid][i tile][j half]
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = 8 * (i >> 1) + 2 * t + (i & 1);
            coef[i] = here.coef[j];
            v[0][i] = f * coef[i].w * __half2float(sh_v[buf][j][warp * 16 + g]);
            v[1][i] = f * coef[i].w * __half2float(sh_v[buf][j][warp * 16 + g + 8]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int w = i >> 2, it = (i >> 1) & 1, jh = i & 1;
            tm[w][it][jh] = *reinterpret_cast<const uint32_t*>(&here.t[w][it * 8 + g][jh * 8 + 2 * t]);
            pm[w][it][jh] = *reinterpret_cast<const uint32_t*>(&here.p[w][it * 8 + g][jh * 8 + 2 * t]);
        }
        // f delta^T = (f diag(beta) (V - diag(G / |k|) K S0))^T T^T
        float delta[2][4] = {}, acc[2][4] = {}, u[2][4];
        float r[2][4];
        uint32_t ahi[4], amid[4];
        {
#pragma unroll
            for (int jt = 0; jt < 2; ++jt) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    r[jt][e] = v[e >> 1][jt * 2 + (e & 1)] - coef[jt * 2 + (e & 1)].x * (ks[0][jt][e] + kMidDown * ks[1][jt][e]);
            }
            split_frag(r[0], r[1], ahi, amid);
        }
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            mma_f16(delta[it], ahi, tm[0][it][0], tm[0][it][1]);
            mma_f16(acc[it], ahi, tm[1][it][0], tm[1][it][1]);
            mma_f16(acc[it], amid, tm[0][it][0], tm[0][it][1]);
        }
#pragma unroll
        for (int jt = 0; jt < 2; ++jt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                delta[jt][e] = r[jt][e] + (delta[jt][e] + kMidDown * acc[jt][e]);
                u[jt][e] = delta[jt][e] * coef[jt * 2 + (e & 1)].z;
                acc[jt][e] = 0.f;
            }
        }
        // O^T = diag(G / |q|) (Q S0)^T + delta^T P^T
        float od[2][4] = {};
        split_frag(delta[0], delta[1], ahi, amid);
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            mma_f16(od[it], ahi, pm[0][it][0], pm[0][it][1]);
            mma_f16(acc[it], ahi, pm[1][it][0], pm[1][it][1]);
            mma_f16(acc[it], amid, pm[0][it][0], pm[0][it][1]);
        }
        // S^T = G_15 S^T + (diag(G_15 / G_j / |k_j|) delta)^T K
        const float ge = here.decay;
        const uint32_t kt_base = smem_u32(&sh_k[buf][lt_row][lt_col]);
        split_frag(u[0], u[1], ahi, amid);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            uint32_t kb[4];
            ldsm4_trans(kt_base + m * 32, kb);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                float (&sn)[4] = s[2 * m + nt];
                float low[4] = {};
#pragma unroll
                for (int e = 0; e < 4; ++e) sn[e] *= ge;
                mma_f16(sn, ahi, kb[2 * nt], kb[2 * nt + 1]);
                mma_f16(low, amid, kb[2 * nt], kb[2 * nt + 1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    sn[e] = fmaf(low[e], kMidDown, sn[e]);
                    s_most[nt] = fmaxf(s_most[nt], fabsf(sn[e]));
                }
            }
        }
        most = warp_most(fmaxf(fmaxf(s_most[0], s_most[1]), most));
#pragma unroll
        for (int jt = 0; jt < 2; ++jt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int p = n * kScanBlock + 8 * jt + 2 * t + (e & 1);
                const float o = inv_f * (coef[jt * 2 + (e & 1)].y * (qs[0][jt][e] + kMidDown * qs[1][jt][e]) + (od[jt][e] + kMidDown * acc[jt][e]));
                if (p < rc) raw[((seq0 + p) * hv + h) * 128 + c0 + 8 * (e >> 1)] = o;
            }
        }
    }
#pragma unroll
    for (int n = 0; n < 16; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) S[(8 * n + 2 * t + (e & 1)) * 128 + c0 + 8 * (e >> 1)] = inv_f * s[n][e];
    }
}

// out = rmsnorm(raw) * w * silu(z) over the 128 values of a head: a warp per (row, head), memory bound (14 bytes a value moved,
// most of them still in L2).
__global__ void __launch_bounds__(256) gdn_norm_kernel(__half* out, const float* raw, const __half* z, const float* norm_w, long long heads) {
    const int lane = threadIdx.x & 31;
    const long long head = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5), at = head * 128 + 4 * lane;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    float w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = norm_w[4 * lane + i];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (head >= heads) return;
    const float4 x = *reinterpret_cast<const float4*>(raw + at);
    const __half2 z0 = *reinterpret_cast<const __half2*>(z + at), z1 = *reinterpret_cast<const __half2*>(z + at + 2);
    const float v[4] = {x.x, x.y, x.z, x.w}, g[4] = {__low2float(z0), __high2float(z0), __low2float(z1), __high2float(z1)};
    const float sq = warp_sum((v[0] * v[0] + v[1] * v[1]) + (v[2] * v[2] + v[3] * v[3]));
    const float inv_std = 1.0f / sqrtf(sq / 128.0f + 1e-6f);
    float y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = v[i] * inv_std * w[i] * silu(g[i]);
    *reinterpret_cast<__half2*>(out + at) = __floats2half2_rn(y[0], y[1]);
    *reinterpret_cast<__half2*>(out + at + 2) = __floats2half2_rn(y[2], y[3]);
}

// ------------------------------------------------------------------------------- speculative bookkeeping
struct AcceptRec {
    long long bonus;
    long long rejected;
    int num_accepted, num_rejected, num_resampled, num_remaining, has_rejected, pad;
};

// After acceptance: per sequence, publish the emitted tokens (accepted drafts then the bonus token),
// advance the context, remember how many recurrent updates to replay, pick the hidden row that feeds
// the next draft, and set the next step's first token.
__global__ void spec_commit_kernel(const AcceptRec* rec, const long long* draft_tokens, int k, int rows_per_seq,
                                   int* ctx, int* n_commit, long long* cur_tok, long long* emitted, int* emitted_n,
                                   __half* h_last, const __half* hidden_rows, int hidden) {
    griddep_prologue();
    const int b = blockIdx.x;
    const int na = rec[b].num_accepted;
    if (threadIdx.x == 0) {
        for (int i = 0; i < na; ++i) emitted[b * (k + 1) + i] = draft_tokens[b * k + i];
        emitted[b * (k + 1) + na] = rec[b].bonus;
        for (int i = na + 1; i < k + 1; ++i) emitted[b * (k + 1) + i] = -1;
        emitted_n[b] = na + 1;
        ctx[b] += na + 1;
        n_commit[b] = na + 1;
        cur_tok[b] = rec[b].bonus;
    }
    const __half* src = hidden_rows + (static_cast<long long>(b) * rows_per_seq + na) * hidden;
    for (int d = threadIdx.x; d < hidden; d += blockDim.x) h_last[static_cast<long long>(b) * hidden + d] = src[d];
}

// rows of the verify pass: row (b, 0) = current token, rows (b, 1..k) = draft tokens.  Signals its dependents only after its own
// wait: everything in front of it is complete before a launch of the verify pass starts, which reads the step before's context
// lengths, keys and states ahead of its own wait (mixers.h).
__global__ void build_verify_tokens_kernel(long long* out, const long long* cur_tok, const long long* draft, int k) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int b = blockIdx.x, i = threadIdx.x;
    if (i == 0) out[b * (k + 1)] = cur_tok[b];
    else if (i <= k) out[b * (k + 1) + i] = draft[b * k + i - 1];
}

__global__ void fill_int_kernel(int* p, int n, int v) {
    griddep_prologue();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

}  // namespace

#define XB_LAUNCH_OK() (cudaGetLastError() == cudaSuccess ? 0 : -1)

namespace {
// SMs of the current device.  (Asked of the runtime and kept: a norm may be the first call on a device, also under capture, where the
// library's own record of it cannot be set up.)
int sm_count() {
    static std::atomic<int> known[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    int n = known[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 148;
        known[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// As the kernel asks for vectors.
bool norm_aligned(const NormJob& j) {
    return ((reinterpret_cast<uintptr_t>(j.x) | reinterpret_cast<uintptr_t>(j.out) | reinterpret_cast<uintptr_t>(j.delta) |
             reinterpret_cast<uintptr_t>(j.table) | reinterpret_cast<uintptr_t>(j.w)) & 15) == 0;
}

template <bool TABLE>
void launch_norm(cudaStream_t s, dim3 grid, const NormJob& a, const NormJob& b, long long ld_out, int hidden, float eps, int perm_out) {
    const long long rows = static_cast<long long>(grid.x) * grid.y, sms = sm_count();  // (a block for every row of every job)
    const int warps_of_one = (hidden / 8 + 31) / 32, warps_of_two = (hidden / 8 + 63) / 64;
    const bool vectors = hidden % 8 == 0 && hidden <= 8 * 1024;
    // Rows that do not start on a vector's boundary go element by element: a thread for every eight of them, but no fewer than 256 (add and
    // norm of 32 x 512 with 64 threads 6.6 us, with 256 2.9).
    const int least = ld_out % 8 == 0 && norm_aligned(a) && (grid.y == 1 || norm_aligned(b)) ? 32 : 256;
    auto threads = [&](int warps) { return dim3(warps * 32 < least ? least : warps * 32); };
    const bool pairs = hidden > kNormNarrow && hidden <= kNormPairs &&
                       (rows > 6 * sms || (hidden > 4096 && rows > 3 * sms && rows <= 4 * sms));
    if (vectors && rows <= sms)
        launch_pdl(rmsnorm_kernel<TABLE, 1, true>, grid, threads(warps_of_one), 0, s, a, b, ld_out, hidden, eps, perm_out);
    else if (vectors && hidden <= kNormNarrow)
        launch_pdl(rmsnorm_kernel<TABLE, 1, false>, grid, threads(warps_of_one), 0, s, a, b, ld_out, hidden, eps, perm_out);
    else if (vectors && pairs)
        launch_pdl(rmsnorm_kernel<TABLE, 2, false>, grid, threads(warps_of_two), 0, s, a, b, ld_out, hidden, eps, perm_out);
    else
        launch_pdl(rmsnorm_kernel<TABLE, 4, false>, grid, dim3(256), 0, s, a, b, ld_out, hidden, eps, perm_out);
}
}  // namespace

int embed_norm_rows(cudaStream_t s, __half* out, __half* x, const void* table_bf16, const long long* tokens, const float* w, int rows,
                    int hidden, long long vocab, float eps, int perm_out) {
    NormJob j = {};
    j.out = out;
    j.x = x;
    j.w = w;
    j.table = static_cast<const uint16_t*>(table_bf16);
    j.tokens = tokens;
    j.vocab = vocab;
    launch_norm<true>(s, dim3(rows), j, j, static_cast<long long>(hidden), hidden, eps, perm_out);
    return XB_LAUNCH_OK();
}

int head_input_rows(cudaStream_t s, const HeadInput& h, int rows, int hidden, float eps, int perm_out) {
    NormJob e = {}, p = {};
    e.out = h.cat;
    e.w = h.embed_norm;
    e.table = static_cast<const uint16_t*>(h.table_bf16);
    e.tokens = h.tokens;
    e.vocab = h.vocab;
    e.token_copy = h.token_copy;
    e.token_ld = h.token_ld;
    e.pos_in = h.pos_in;
    e.pos_out = h.pos_out;
    e.pos_add = h.pos_add;
    p.out = h.cat + hidden;
    p.x = const_cast<__half*>(h.hidden_rows);
    p.w = h.hidden_norm;
    launch_norm<true>(s, dim3(rows, 2), e, p, 2LL * hidden, hidden, eps, perm_out);
    return XB_LAUNCH_OK();
}

int rmsnorm_rows(cudaStream_t s, __half* out, long long ld_out, const __half* in, const float* w, int rows, int hidden,
                 float eps, int perm_out) {
    NormJob j = {};
    j.out = out;
    j.x = const_cast<__half*>(in);
    j.w = w;
    launch_norm<false>(s, dim3(rows), j, j, ld_out, hidden, eps, perm_out);
    return XB_LAUNCH_OK();
}

int add_rmsnorm_rows(cudaStream_t s, __half* out, __half* x, const __half* delta, const float* w, int rows, int hidden,
                     float eps, int perm_out) {
    NormJob j = {};
    j.out = out;
    j.x = x;
    j.delta = delta;
    j.w = w;
    launch_norm<false>(s, dim3(rows), j, j, static_cast<long long>(hidden), hidden, eps, perm_out);
    return XB_LAUNCH_OK();
}

int attn_prep(cudaStream_t s, __half* q_out, __half* k_cache, __half* v_cache, const __half* q_gate, const __half* k_in,
              const __half* v_in, const float* q_norm_w, const float* k_norm_w, const int* ctx, int batch,
              int rows_per_seq, int hq, int hkv, long long max_seq, float eps, float rope_theta, int rope_dim) {
    return attn_prep_ex(s, q_out, k_cache, v_cache, q_gate, k_in, v_in, q_norm_w, k_norm_w, ctx, batch, rows_per_seq, hq, hkv,
                        max_seq, eps, rope_theta, rope_dim, 512, nullptr, 0, nullptr);
}

int attn_prep_ex(cudaStream_t s, __half* q_out, __half* k_cache, __half* v_cache, const __half* q_in, const __half* k_in,
                 const __half* v_in, const float* q_norm_w, const float* k_norm_w, const int* ctx, int batch,
                 int rows_per_seq, int hq, int hkv, long long max_seq, float eps, float rope_theta, int rope_dim,
                 int q_head_stride, const long long* positions, int ctx_base, __half* k_out) {
    const int rows = batch * rows_per_seq, slots = hq + 2 * hkv;
    // A block per head or a warp per head, in us: rotary embedding of 24 + 4 heads 8 rows 1.9 and 2.0, 32 rows 2.4 and 2.4, 77 rows 4.1 and
    // 3.1, 128 rows 5.7 and 3.3; cache write of 4 heads 32 rows 1.7 and 1.6, 512 rows 5.3 and 2.3.  With head norms a warp's own
    // sums are the longer chain (32 rows of 32 slots 3.6 and 5.6), and the block stays the faster until it is several waves.  So it does
    // for a single head a row, where seven warps of eight would have nothing to do (1100 rows 3.1 and 3.8, 4000 rows 6.6 and 7.2; of two
    // heads 4.6 and 3.8).
    const long long heads = static_cast<long long>(rows) * slots;
    if (heads > (q_norm_w || k_norm_w || slots == 1 ? 4096 : 1024))
        launch_pdl(heads > 4096 ? attn_prep_rows_kernel<true> : attn_prep_rows_kernel<false>, dim3(rows, (slots + 7) / 8), dim3(256), 0, s,
                   q_out, k_cache, v_cache, q_in, k_in, v_in, q_norm_w, k_norm_w, ctx, rows_per_seq, hq, hkv, max_seq, eps, logf(rope_theta),
                   rope_dim, q_head_stride, positions, ctx_base, k_out);
    else
        launch_pdl(attn_prep_kernel, dim3(rows, slots), dim3(256), 0, s, q_out, k_cache, v_cache, q_in, k_in, v_in, q_norm_w, k_norm_w, ctx,
                   rows_per_seq, hq, hkv, max_seq, eps, logf(rope_theta), rope_dim, q_head_stride, positions, ctx_base, k_out);
    return XB_LAUNCH_OK();
}

int conv1d_spec(cudaStream_t s, __half* out, const __half* in, const float* conv_w, float* state, float* pending,
                const int* n_commit, int batch, int rows_per_seq, int prev_rows, int channels, int nc_base, int early_state) {
    dim3 grid((channels + 255) / 256, batch);
    launch_pdl(conv1d_spec_kernel, dim3(grid), dim3(256), 0, s, out, in, conv_w, state, pending, n_commit, rows_per_seq, prev_rows, channels, nc_base, early_state);
    return XB_LAUNCH_OK();
}

int gdn_spec(cudaStream_t s, __half* out, const __half* qkv, const __half* z, const __half* b, const __half* a,
             const float* A_log, const float* dt_bias, const float* norm_w, float* state, float* pend_k, float* pend_d,
             float* pend_g, const int* n_commit, int batch, int rows_per_seq, int prev_rows, int hv, int hk, int nc_base,
             int early_state, int perm_out, int num_sms) {
    // more heads than SMs: several per SM, whose streams overlap each other (144 heads: 6.7 us with 512 threads a head and
    // 9.2 with 256; 192 heads: 13.5 and 9.4)
    const bool many = hv * batch > num_sms;
    const bool few_tokens = rows_per_seq <= 4;
    launch_pdl(many ? (few_tokens ? gdn_spec_kernel<2, 16, 4> : gdn_spec_kernel<2, 16, 8>)
                    : (few_tokens ? gdn_spec_kernel<4, 32, 4> : gdn_spec_kernel<4, 32, 8>),
               dim3(hv, batch), dim3(many ? 256 : 512), 0, s, out, qkv, z, b, a, A_log, dt_bias, norm_w, state, pend_k, pend_d, pend_g,
               n_commit, rows_per_seq, prev_rows, hv, hk, nc_base, early_state, perm_out);
    return XB_LAUNCH_OK();
}

int conv1d_chunk(cudaStream_t s, __half* out, const __half* in, const float* conv_w, float* state, int batch, int rc,
                 int channels) {
    if (rc <= 0) return 0;
    // Eight positions per thread; all of them when the output lies over the input (a position's inputs are its neighbours').
    const size_t bytes = static_cast<size_t>(batch) * rc * channels * sizeof(__half);
    const char *o = reinterpret_cast<const char*>(out), *i = reinterpret_cast<const char*>(in);
    const bool overlap = o < i + bytes && i < o + bytes;
    // One channel a thread is the shorter chain, which counts while a launch is no more than that: as long as its blocks are fewer than
    // kConvNarrowBlocks an SM (us a launch with four channels a thread and with one, blocks of the latter in brackets: 10240 channels, 1 row 2.46 and
    // 2.05 (80), 33 rows 3.79 and 3.48 (400), 48 rows 3.66 and 3.97 (480), 100 rows 4.7 and 5.6 (1040), 400 rows 8.1 and 11.4; 20480 channels, 16
    // rows 3.58 and 3.25 (320), 24 rows 3.58 and 3.99 (480); 4096 channels, 77 rows 3.56 and 3.15 (320), 100 rows 3.67 and 3.77 (416); 512 channels,
    // 400 rows 3.43 and 2.87 (200)), or with every position of a channel one after the other (in place, 509 x 10240 84 and 65).  More than 65535
    // blocks of 128 channels do not fit the grid's third dimension.
    const bool vec_ok = channels % 4 == 0 && ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(in)) & 7) == 0;
    const long long narrow_blocks = (channels + 127ll) / 128 * batch * ((rc + kAhead - 1) / kAhead);
    const bool vec = vec_ok && (channels > 65535 * 128 || (!overlap && narrow_blocks >= static_cast<long long>(kConvNarrowBlocks) * sm_count()));
    const int per_block = 128 * (vec ? 4 : 1);
    dim3 grid(overlap ? 1 : (rc + kAhead - 1) / kAhead, batch, (channels + per_block - 1) / per_block);
    launch_pdl(overlap ? (vec ? conv1d_chunk_kernel<4, 0> : conv1d_chunk_kernel<1, 0>) : (vec ? conv1d_chunk_kernel<4, kAhead> : conv1d_chunk_kernel<1, kAhead>),
               grid, dim3(128), 0, s, out, in, conv_w, state, rc, channels);
    return XB_LAUNCH_OK();
}

bool gdn_chunk_aligned(const void* out, const void* qkv, const void* z, const void* state) {
    return ((reinterpret_cast<uintptr_t>(qkv) & 15) | (reinterpret_cast<uintptr_t>(state) & 15) |
            ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(z)) & 3)) == 0;
}

size_t gdn_chunk_scratch_bytes(int batch, int rc, int hv) {
    const size_t heads = static_cast<size_t>(batch) * hv;
    return heads * rc * 128 * sizeof(float) + heads * ((rc + kScanBlock - 1) / kScanBlock) * sizeof(GdnBlock);  // outputs, blocks
}

int gdn_chunk(cudaStream_t s, __half* out, const __half* qkv, const __half* z, const __half* b, const __half* a,
              const float* A_log, const float* dt_bias, const float* norm_w, float* state, int batch, int rc, int hv, int hk,
              void* scratch, int num_sms, int zero_state) {
    if (rc <= kGdnWalkRows) {
        // As many CTAs as four a SM are: shared memory that keeps a fifth out, since the whole clusters would otherwise be packed on
        // half of the SMs (48 heads, 1 and 16 tokens: 6.0 and 13.1 us against 7.6 and 18.7; 96 heads 10.9 and 24.2 against 8.1 and 20.0).
        const size_t spread = hv * kGdnSlices * batch <= 4 * num_sms ? 20 * 1024 : 0;
        launch_pdl(gdn_walk_kernel, dim3(hv * kGdnSlices, batch), dim3(kGdnThreads), spread, s, out, qkv, z, b, a, A_log, dt_bias, norm_w,
                   state, rc, hv, hk, zero_state);
        return XB_LAUNCH_OK();
    }
    const long long heads = static_cast<long long>(batch) * rc * hv;
    float* raw = static_cast<float*>(scratch);
    GdnBlock* blocks = reinterpret_cast<GdnBlock*>(raw + heads * 128);
    const int nblocks = (rc + kScanBlock - 1) / kScanBlock;
    launch_pdl(gdn_block_kernel, dim3((nblocks + 3) / 4, hv, batch), dim3(128), 0, s, blocks, qkv, b, a, A_log, dt_bias, rc, hv, hk);
    launch_pdl(gdn_scan_kernel, dim3(hv * kScanSlices, batch), dim3(32 * kScanWarps), 0, s, raw, qkv, static_cast<const GdnBlock*>(blocks),
               state, rc, hv, hk, zero_state);
    launch_pdl(gdn_norm_kernel, dim3(static_cast<unsigned>((heads + 7) / 8)), dim3(256), 0, s, out, static_cast<const float*>(raw), z, norm_w, heads);
    return XB_LAUNCH_OK();
}

int spec_commit(cudaStream_t s, const void* accept_records, const long long* draft_tokens, int batch, int k,
                int rows_per_seq, int* ctx, int* n_commit, long long* cur_tok, long long* emitted, int* emitted_n,
                __half* h_last, const __half* hidden_rows, int hidden) {
    launch_pdl(spec_commit_kernel, dim3(batch), dim3(256), 0, s, static_cast<const AcceptRec*>(accept_records), draft_tokens, k, rows_per_seq,
                                             ctx, n_commit, cur_tok, emitted, emitted_n, h_last, hidden_rows, hidden);
    return XB_LAUNCH_OK();
}

int build_verify_tokens(cudaStream_t s, long long* out, const long long* cur_tok, const long long* draft, int batch,
                        int k) {
    launch_pdl(build_verify_tokens_kernel, dim3(batch), dim3(32), 0, s, out, cur_tok, draft, k);
    return XB_LAUNCH_OK();
}

int fill_int(cudaStream_t s, int* p, int n, int v) {
    launch_pdl(fill_int_kernel, dim3((n + 127) / 128), dim3(128), 0, s, p, n, v);
    return XB_LAUNCH_OK();
}

}  // namespace xb
