// Causal GQA attention over the KV cache on tcgen05: prompts and prefill chunks in tiles of up to 128 query rows, and the
// few rows of a decode or verify pass.
//
// Stands where the reference runs ops::sdpa_causal_cached (src/ops/attention.h:89-113, called from
// src/targets/qwen3_8/forward.cpp:229-262, 402-554).
//
// The G = Hq / Hkv query heads that share a KV head attend to the same keys, so the rows of a tile are (position, head of
// the group) pairs: up to floor(128 / G) positions of one sequence and one KV head.  Per 64 keys of a tile:
//   S = Q K^T     M = 128 rows, N = 64 keys, K = 256 dims, both operands from shared memory, S double-buffered in tensor memory;
//   P = exp2(..)  a thread per row: running maximum (raised only when a row exceeds it by 2^8, so that the accumulator is
//                 rarely rescaled: the conditional rescaling published with FlashAttention-4), fp32 sums, fp16 probabilities back
//                 into tensor memory.  (Raised at once, 512 rows behind 7680 keys take 149 us instead of 129; the error against 64
//                 bits, 2.9e-4 with the output's fp16 rounding, would be 2.8e-4);
//   O += P V      M = 128, N = 256 dims, K = 64 keys, A from tensor memory, V as it lies in the cache (its 256 dims are
//                 contiguous: an MN-major operand), O in 256 tensor-memory columns.
// K and V blocks of 32 KB arrive by TMA, a warp each: three slots of keys and two of values beside 64 KB of queries, three and
// three where the queries are at most 32 rows and take 16 KB.
//
// (sequence, tile) x 64-key blocks are cut evenly over groups of Hkv CTAs, one per KV head and together one per SM, on the
// device, from the context lengths that lie there: a CTA takes a contiguous range of (tile, block) units.  What covers a whole
// tile is written out, the two ends of a range as fp32 partials for attn_tile_combine_kernel.  The CTAs of a group walk the
// same keys in step: in the cache the heads of a key lie
// side by side.
//
// Bounds.  Prefill: per block the tensor core needs 128 * 64 * 256 * 4 flop = 1024 clocks at its full rate, the exponentials
// 512; measured 2500 (8192 keys, 512 rows: 130 us, 770 TFLOP/s; 4.9 ms five rows a launch), the S product at N = 64 being
// bound by its shared-memory reads.  Decode (24 of the 128 rows in use): 64 KB of cache per block are 2900 clocks of an SM's
// share of HBM, so the padded rows cost nothing; 269 MB of cache take 56 us in the step (41 at the measured copy rate, 47 at
// the 5.8 TB/s that a longer context settles at).  (Pulling the blocks into L2 ahead in 32 KB runs of all heads made it slower, 60 to 70 us.)
//
// Every wait is bounded (WaitState); one that runs out sets the device status word and the CTA leaves through its normal exit.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <mutex>

#include "launch.cuh"
#include "mixers.h"
#include "ptx_sm100.cuh"
#include "w4a16.h"

namespace xb {
namespace {

constexpr int kTileRows = 128, kTileKeys = 64, kDim = 256, kDimBlocks = kDim / 64;
constexpr int kSoftmaxThreads = 128, kTileThreads = kSoftmaxThreads + 96;
constexpr int kKWarp = 4, kVWarp = 5, kMmaWarp = 6;  // two TMA warps: keys (and queries), values
constexpr int kKvBytes = kTileKeys * kDim * 2;
constexpr int kKSlots = 3;
constexpr int tile_v_slots(int rows) { return rows <= 32 ? 3 : 2; }
// Bytes of a 64-dim block of the queries.  At 32 rows the MMA, which always takes 128, reads on into what lies behind: rows of
// S that nobody looks at.
constexpr int tile_q_block(int rows) { return (rows <= 32 ? 32 : kTileRows) * 128; }
// tensor memory columns
constexpr uint32_t kColO = 0, kColS = 256, kColP = 384, kTileTmemCols = 512;
constexpr float kLazyRescale = 8.0f;  // in base-2 units: probabilities stay below 2^8

struct TileCtrl {
    uint64_t q_full, q_empty, o_free, k_full[kKSlots], k_empty[kKSlots], v_full[3], v_empty[3];
    uint64_t s_full[2], s_free[2], p_ready[2], pv_done[2];
    uint32_t tmem_base;
    WaitState ws;
};
constexpr size_t tile_smem_bytes(int rows) {
    return 1024 + kDimBlocks * tile_q_block(rows) + (kKSlots + tile_v_slots(rows)) * kKvBytes + sizeof(TileCtrl);
}
static_assert(tile_smem_bytes(32) <= 227 * 1024 && tile_smem_bytes(kTileRows) <= 227 * 1024, "shared memory");

struct TileShape {          // what both kernels need to find their work
    const int* ctx;         // keys in front of each sequence's first row; null: ctx_base
    int ctx_base;
    int rows_per_seq, hq, hkv, group, tile_pos, tiles, items;  // items = batch * tiles, tiles fastest
    long long max_seq;
};
struct TileParams {
    CUtensorMap q_map, k_map, v_map;
    TileShape sh;
    __half* out;
    const __half* q_gate;   // [rows][hq][512], the gate in the upper 256; null: none
    int perm_out, out_vec;
    int early;              // keys below ctx, and ctx itself, do not come from the launch in front of this one
    float scale2;           // softmax scale * log2 e
    float *part_o, *part_ml;  // [CTA][2][row][256], [CTA][2][row][max, sum]
    int2* table;            // [items] first and last group at work on every item
    long long wait_limit;
    int withhold;           // test hook: the queries are never requested
    int* status;
};

__device__ __forceinline__ void umma_ss_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}"
        :
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const void* map, uint32_t bar, int x, int y, int z, int w, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1, {%3, %4, %5, %6}], [%2], %7;"
        :
        : "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w), "l"(policy)
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        :
        : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
// Bounded waits of a whole warp: all of its lanes go on, or all leave.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile WaitState* ws) {
    return __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity, ws));
}
__device__ __forceinline__ bool warp_wait_parked(uint64_t* bar, uint32_t parity, volatile WaitState* ws) {
    return __all_sync(0xffffffffu, mbar_wait_parked(smem_u32(bar), parity, ws));
}
__device__ __forceinline__ float exp2_ftz(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// Eight finished values of a head as fp16: rounded, gated, in the order the caller wants.
__device__ __forceinline__ uint4 finish8(const float* v, const __half* gate, bool perm) {
    uint4 o;
    if (gate) {
        // rounding point: the reference's SDPA writes fp16, the gate then multiplies in fp32
        const uint4 g4 = *reinterpret_cast<const uint4*>(gate);
        const uint32_t gw[4] = {g4.x, g4.y, g4.z, g4.w};
        float r[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 g = __half22float2(*reinterpret_cast<const __half2*>(&gw[j]));
            r[2 * j] = __half2float(__float2half_rn(v[2 * j])) * (1.0f / (1.0f + expf(-g.x)));
            r[2 * j + 1] = __half2float(__float2half_rn(v[2 * j + 1])) * (1.0f / (1.0f + expf(-g.y)));
        }
        o = make_uint4(pack_half2(r[0], r[1]), pack_half2(r[2], r[3]), pack_half2(r[4], r[5]), pack_half2(r[6], r[7]));
    } else {
        o = make_uint4(pack_half2(v[0], v[1]), pack_half2(v[2], v[3]), pack_half2(v[4], v[5]), pack_half2(v[6], v[7]));
    }
    if (perm)  // (h0 h1 | h2 h3 | h4 h5 | h6 h7) -> (h0 h4 | h1 h5 | h2 h6 | h3 h7)
        o = make_uint4(__byte_perm(o.x, o.z, 0x5410), __byte_perm(o.x, o.z, 0x7632), __byte_perm(o.y, o.w, 0x5410), __byte_perm(o.y, o.w, 0x7632));
    return o;
}

__device__ __forceinline__ void store8(__half* dst, const uint4& v, int vec) {
    if (vec) {
        *reinterpret_cast<uint4*>(dst) = v;
    } else {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) dst[j] = __ushort_as_half(static_cast<unsigned short>(w[j >> 1] >> (16 * (j & 1))));
    }
}

// Four lanes' four pieces each, transposed: lane q's t[k] becomes what t[q] of lane k of the four was.
__device__ __forceinline__ uint4 shfl_xor4(const uint4& v, int mask) {
    return make_uint4(__shfl_xor_sync(0xffffffffu, v.x, mask), __shfl_xor_sync(0xffffffffu, v.y, mask), __shfl_xor_sync(0xffffffffu, v.z, mask),
                      __shfl_xor_sync(0xffffffffu, v.w, mask));
}
__device__ __forceinline__ uint4 pick4(bool first, const uint4& a, const uint4& b) {
    return make_uint4(first ? a.x : b.x, first ? a.y : b.y, first ? a.z : b.z, first ? a.w : b.w);
}
__device__ __forceinline__ void transpose4(uint4 (&t)[4], int lane) {
    const bool b1 = lane & 2, b0 = lane & 1;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const uint4 got = shfl_xor4(pick4(b1, t[j], t[j + 2]), 2);
        t[j] = pick4(b1, got, t[j]);
        t[j + 2] = pick4(b1, t[j + 2], got);
    }
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
        const uint4 got = shfl_xor4(pick4(b0, t[j], t[j + 1]), 1);
        t[j] = pick4(b0, got, t[j]);
        t[j + 1] = pick4(b0, t[j + 1], got);
    }
}

// Keys in front of item e's first row, and its number of 64-key blocks (at least one).
__device__ __forceinline__ int item_ctx(const TileShape& sh, int e) { return sh.ctx ? __ldg(sh.ctx + e / sh.tiles) : sh.ctx_base; }
__device__ __forceinline__ int item_blocks(const TileShape& sh, int e) {
    const int end = (e % sh.tiles + 1) * sh.tile_pos;
    long long keys = static_cast<long long>(item_ctx(sh, e)) + (end < sh.rows_per_seq ? end : sh.rows_per_seq);
    if (keys > sh.max_seq) keys = sh.max_seq;
    return static_cast<int>((keys + kTileKeys - 1) / kTileKeys);
}
__device__ __forceinline__ int range_begin(int group, int total, int groups) { return static_cast<int>(static_cast<long long>(group) * total / groups); }
// The group whose range holds unit u: the largest c with floor(c total / groups) <= u.
__device__ __forceinline__ int unit_owner(int u, int total, int groups) {
    return static_cast<int>((static_cast<long long>(u + 1) * groups - 1) / total);
}

// A group's walk through its units, a run of blocks of one item at a time.
struct TileWalk {
    int item, off, u, u_end, total, groups;  // next item, next block of it, next unit
    int kb0, n, blocks;                    // the current run
    // Every lane of a warp calls it.  BY_ITEM: a group to every item, none cut (whole_items).
    template <bool BY_ITEM>
    __device__ void start(const TileShape& sh, int group, int most_groups) {
        const int lane = threadIdx.x & 31;
        total = 0;
        if constexpr (BY_ITEM) {
            groups = sh.items;
            item = group;
            off = u = 0;
            u_end = group < groups ? item_blocks(sh, group) : 0;
            return;
        }
        for (int e0 = 0; e0 < sh.items; e0 += 32) {
            const int mine = e0 + lane < sh.items ? item_blocks(sh, e0 + lane) : 0;
            total += __reduce_add_sync(0xffffffffu, mine);
        }
        // Below two blocks a CTA, the partials cost more than the additional CTAs bring.
        groups = total / 2 < 1 ? 1 : (total / 2 < most_groups ? total / 2 : most_groups);
        item = off = 0;
        u = group < groups ? range_begin(group, total, groups) : total;
        u_end = group < groups ? range_begin(group + 1, total, groups) : total;
        int before = 0;
        for (int e0 = 0; e0 < sh.items && u < u_end; e0 += 32) {
            const int mine = e0 + lane < sh.items ? item_blocks(sh, e0 + lane) : 0;
            int sum = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int o = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += o;
            }
            const int chunk = __shfl_sync(0xffffffffu, sum, 31);
            if (u < before + chunk) {
                const unsigned past = __ballot_sync(0xffffffffu, before + sum > u);
                const int first = __ffs(past) - 1;
                item = e0 + first;
                off = u - before - __shfl_sync(0xffffffffu, sum - mine, first);
                break;
            }
            before += chunk;
        }
    }
    __device__ bool next(const TileShape& sh) {
        if (u >= u_end) return false;
        blocks = item_blocks(sh, item);
        kb0 = off;
        n = blocks - off < u_end - u ? blocks - off : u_end - u;
        return true;
    }
    __device__ void advance() {
        u += n;
        ++item;
        off = 0;
    }
    __device__ bool whole() const { return kb0 == 0 && n == blocks; }
};

// BY_ITEM: whole_items.  FOUR: parts are stored by four lanes a row.  Both are compiled apart from the form of a step's rows, which is slower by
// the mere presence of either (8 x 8192 keys: 56.6 us, 58.6 beside FOUR, 60.3 beside both).
template <bool BY_ITEM, bool FOUR>
__global__ void __launch_bounds__(kTileThreads, 1) attn_tile_kernel(const __grid_constant__ TileParams p) {
    extern __shared__ uint8_t tile_smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tile_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const TileShape& sh = p.sh;
    const int rows = sh.group * sh.tile_pos, live_warps = (rows + 31) / 32, v_slots = tile_v_slots(rows), q_block = tile_q_block(rows);
    uint8_t* q_smem = smem;                          // [dim block][rows][128 B]
    uint8_t* k_smem = q_smem + kDimBlocks * q_block; // [slot][dim block][64 keys][128 B]
    uint8_t* v_smem = k_smem + kKSlots * kKvBytes;
    TileCtrl* ctrl = reinterpret_cast<TileCtrl*>(v_smem + v_slots * kKvBytes);
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    volatile WaitState* ws = &ctrl->ws;
    griddep_launch_dependents();

    if (tid == 0) {
        mbar_init(smem_u32(&ctrl->q_full), 1);
        mbar_init(smem_u32(&ctrl->q_empty), 1);
        mbar_init(smem_u32(&ctrl->o_free), live_warps);
        for (int i = 0; i < 3; ++i) {
            mbar_init(smem_u32(&ctrl->k_full[i]), 1);
            mbar_init(smem_u32(&ctrl->k_empty[i]), 1);
            mbar_init(smem_u32(&ctrl->v_full[i]), 1);
            mbar_init(smem_u32(&ctrl->v_empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&ctrl->s_full[i]), 1);
            mbar_init(smem_u32(&ctrl->s_free[i]), live_warps);
            mbar_init(smem_u32(&ctrl->p_ready[i]), live_warps);
            mbar_init(smem_u32(&ctrl->pv_done[i]), 1);
        }
        ctrl->ws.abort_flag = 0;
        ctrl->ws.dep_ready = 0;
        ctrl->ws.limit = p.wait_limit;
        mbar_fence_init();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(smem_u32(&ctrl->tmem_base), kTileTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = ctrl->tmem_base;
    if (!p.early) griddep_wait();
    TileWalk walk;
    const int kvh = static_cast<int>(blockIdx.x) % sh.hkv;
    walk.start<BY_ITEM>(sh, static_cast<int>(blockIdx.x) / sh.hkv, static_cast<int>(gridDim.x) / sh.hkv);
    const int units = walk.u_end - walk.u;

    if (warp == kKWarp || warp == kVWarp) {
        // ------------------------------------------------------------------ TMA producers (whole warp waits, one lane issues)
        const bool keys = warp == kKWarp;
        const bool leader = elect_one_sync();
        const CUtensorMap* map = keys ? &p.k_map : &p.v_map;
        if (leader) {
            tma_prefetch_desc(map);
            if (keys) tma_prefetch_desc(&p.q_map);
        }
        // keys and values are read once by a decode pass, by every tile of a prompt
        const uint64_t pol_q = l2_policy_evict_first(), pol_kv = sh.tiles == 1 ? l2_policy_evict_first() : l2_policy_evict_last();
        uint64_t *full = keys ? ctrl->k_full : ctrl->v_full, *empty = keys ? ctrl->k_empty : ctrl->v_empty;
        const uint32_t ring = smem_u32(keys ? k_smem : v_smem);
        const int slots = keys ? kKSlots : v_slots;
        auto load = [&](int slot, int block, int item) {
            if (leader) {
                const int b = item / sh.tiles;
                const uint32_t bar = smem_u32(&full[slot]);
                mbar_arrive_expect_tx(bar, kKvBytes);
                for (int d = 0; d < kDimBlocks; ++d)
                    tma_load_3d(ring + slot * kKvBytes + d * (kTileKeys * 128), map, bar, kvh * kDim + d * 64, block * kTileKeys, b, pol_kv);
            }
            __syncwarp();  // (or the other lanes wait for the next slot before this one's load is issued)
        };
        int i = 0, ahead = 0, nq = 0, slot = 0;
        uint32_t parity = 1;  // under which a slot's first use passes at once
        bool ok = true;
        if (p.early) {
            // the first blocks while the launch in front of this one, which writes the newest keys and the queries, finishes
            if (walk.next(sh)) {
                const int old_blocks = item_ctx(sh, walk.item) / kTileKeys;
                for (; ahead < slots && ahead < walk.n && walk.kb0 + ahead < old_blocks; ++ahead) load(ahead, walk.kb0 + ahead, walk.item);
            }
            griddep_wait();
        }
        if (leader && keys) ws->dep_ready = 1;
        __syncwarp();
        for (int run = 0; ok && walk.next(sh); ++run) {
            for (int j = 0; j < walk.n && ok; ++j) {
                if (i >= ahead) {
                    ok = warp_wait_parked(&empty[slot], parity, ws);
                    if (!ok) break;
                    load(slot, walk.kb0 + j, walk.item);
                }
                ++i;
                if (++slot == slots) { slot = 0; parity ^= 1u; }
                if (j == 0 && keys) {
                    ok = run == 0 || warp_wait_parked(&ctrl->q_empty, (run & 1u) ^ 1u, ws);
                    if (!ok) break;
                    if (leader && !p.withhold) {
                        const int b = walk.item / sh.tiles;
                        const uint32_t bar = smem_u32(&ctrl->q_full);
                        mbar_arrive_expect_tx(bar, static_cast<uint32_t>(rows) * kDim * 2);
                        for (int d = 0; d < kDimBlocks; ++d)
                            tma_load_4d(smem_u32(q_smem) + d * q_block, &p.q_map, bar, d * 64, kvh * sh.group, walk.item % sh.tiles * sh.tile_pos, b, pol_q);
                    }
                    __syncwarp();
                    nq += !p.withhold;
                }
            }
            walk.advance();
        }
        if (ws->abort_flag) {
            // give the copies still in flight a bounded chance to land before the CTA exits
            const long long t0 = clock64();
            const int loaded = i > ahead ? i : ahead;
            for (int c = 0; c < slots && c < loaded; ++c) {
                const int k = loaded - 1 - c;
                while (!mbar_try_wait(smem_u32(&full[k % slots]), (k / slots) & 1u) && clock64() - t0 < p.wait_limit / 8) {
                }
            }
            while (nq > 0 && !mbar_try_wait(smem_u32(&ctrl->q_full), (nq - 1) & 1u) && clock64() - t0 < p.wait_limit / 8) {
            }
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuer: S of block i, then O of block i - 1
        const bool leader = elect_one_sync();
        if (p.early) griddep_wait();
        constexpr uint32_t idesc_s = umma_idesc_f16_f32(kTileRows, kTileKeys);
        constexpr uint32_t idesc_o = umma_idesc_f16_f32(kTileRows, kDim) | (1u << 16);  // B is MN-major
        // 128-byte swizzle, 8-row groups 1024 bytes apart, descriptor version 1.  MN-major (V): 64-dim chunks 8 KB apart.
        constexpr uint32_t desc_hi = ((1024u >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
        constexpr uint32_t lo_k = 1u << 16, lo_v = static_cast<uint32_t>((kTileKeys * 128) >> 4) << 16;
        const uint32_t q_lo = (smem_u32(q_smem) >> 4) & 0x3FFFu, k_lo = (smem_u32(k_smem) >> 4) & 0x3FFFu, v_lo = (smem_u32(v_smem) >> 4) & 0x3FFFu;
        auto desc = [&](uint32_t lo) { return (static_cast<uint64_t>(desc_hi) << 32) | lo; };
        uint32_t k_slot = 0, k_phase = 0, v_slot = 0, v_phase = 0;
        auto issue_s = [&](int i, bool last_of_run) {
            const uint32_t buf = static_cast<uint32_t>(i & 1), slot = k_slot;
            if (!warp_wait_parked(&ctrl->k_full[slot], k_phase, ws)) return false;
            if (++k_slot == kKSlots) { k_slot = 0; k_phase ^= 1u; }
            if (i >= 2 && !warp_wait_parked(&ctrl->s_free[buf], ((i >> 1) & 1u) ^ 1u, ws)) return false;
            tc_fence_after_sync();
            if (leader) {
#pragma unroll
                for (int k = 0; k < kDim / 16; ++k) {
                    const uint32_t a = q_lo + (((k >> 2) * q_block + (k & 3) * 32) >> 4);
                    const uint32_t c = k_lo + ((slot * kKvBytes + (k >> 2) * (kTileKeys * 128) + (k & 3) * 32) >> 4);
                    umma_ss_f16(tmem + kColS + buf * kTileKeys, desc(lo_k | a), desc(lo_k | c), idesc_s, k > 0 ? 1u : 0u);
                }
                umma_commit(smem_u32(&ctrl->s_full[buf]));
                umma_commit(smem_u32(&ctrl->k_empty[slot]));
                if (last_of_run) umma_commit(smem_u32(&ctrl->q_empty));
            }
            __syncwarp();
            return true;
        };
        // `run` >= 0: the block is the first of that run and overwrites O, which the run before must have been read from
        auto issue_o = [&](int i, int run) {
            const uint32_t buf = static_cast<uint32_t>(i & 1), slot = v_slot;
            if (!warp_wait_parked(&ctrl->v_full[slot], v_phase, ws)) return false;
            if (++v_slot == static_cast<uint32_t>(v_slots)) { v_slot = 0; v_phase ^= 1u; }
            if (!warp_wait_parked(&ctrl->p_ready[buf], (i >> 1) & 1u, ws)) return false;
            if (run > 0 && !warp_wait_parked(&ctrl->o_free, (run & 1u) ^ 1u, ws)) return false;
            tc_fence_after_sync();
            if (leader) {
#pragma unroll
                for (int k = 0; k < kTileKeys / 16; ++k)
                    umma_ts_f16(tmem + kColO, tmem + kColP + buf * (kTileKeys / 2) + k * 8,
                                desc(lo_v | (v_lo + ((slot * kKvBytes + k * 16 * 128) >> 4))), idesc_o, (run < 0 || k > 0) ? 1u : 0u);
                umma_commit(smem_u32(&ctrl->pv_done[buf]));
                umma_commit(smem_u32(&ctrl->v_empty[slot]));
            }
            __syncwarp();
            return true;
        };
        bool ok = true;
        int i = 0, prev_run = -1;  // what issue_o wants to know of block i - 1
        for (int run = 0; ok && walk.next(sh); ++run) {
            for (int j = 0; j < walk.n && ok; ++j, ++i) {
                // (a new run's S waits for its queries: the previous run's last product goes first)
                if (j == 0) ok = (i == 0 || issue_o(i - 1, prev_run)) && warp_wait_parked(&ctrl->q_full, run & 1u, ws);
                ok = ok && issue_s(i, j + 1 == walk.n);
                if (j > 0) ok = ok && issue_o(i - 1, prev_run);
                prev_run = j == 0 ? run : -1;
            }
            walk.advance();
        }
        if (ok && units > 0) issue_o(units - 1, prev_run);
    } else if (warp < live_warps) {
        // ------------------------------------------------------------------ softmax and output: one thread per row
        if (p.early) griddep_wait();
        const int r = tid, pr = r / sh.group, head_in_group = r % sh.group;
        const uint32_t lanes = static_cast<uint32_t>(warp * 32) << 16;
        bool ok = true;
        int i = 0;
        while (ok && walk.next(sh)) {
            const int item = walk.item, b = item / sh.tiles, pos = item % sh.tiles * sh.tile_pos + pr;
            const bool valid = r < rows && pos < sh.rows_per_seq;
            long long lim = static_cast<long long>(item_ctx(sh, item)) + pos + 1;
            if (lim > sh.max_seq) lim = sh.max_seq;
            const int limit = valid ? static_cast<int>(lim) : 0x7FFFFFFF;
            float m = -INFINITY, l = 0.f;
            for (int j = 0; j < walk.n; ++j, ++i) {
                const uint32_t buf = static_cast<uint32_t>(i & 1);
                if (!warp_wait(&ctrl->s_full[buf], (i >> 1) & 1u, ws)) { ok = false; break; }
                tc_fence_after_sync();
                uint32_t raw[kTileKeys];
                tmem_ld32(tmem + lanes + kColS + buf * kTileKeys, raw);
                tmem_ld32(tmem + lanes + kColS + buf * kTileKeys + 32, raw + 32);
                tmem_wait_ld();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ctrl->s_free[buf]));
                const int key0 = (walk.kb0 + j) * kTileKeys;
                if (__any_sync(0xffffffffu, key0 + kTileKeys > limit)) {
#pragma unroll
                    for (int c = 0; c < kTileKeys; ++c)
                        if (key0 + c >= limit) raw[c] = 0xFF800000u;  // -inf
                }
                float mx0 = __uint_as_float(raw[0]), mx1 = __uint_as_float(raw[1]), mx2 = __uint_as_float(raw[2]), mx3 = __uint_as_float(raw[3]);
#pragma unroll
                for (int c = 4; c < kTileKeys; c += 4) {
                    mx0 = fmaxf(mx0, __uint_as_float(raw[c]));
                    mx1 = fmaxf(mx1, __uint_as_float(raw[c + 1]));
                    mx2 = fmaxf(mx2, __uint_as_float(raw[c + 2]));
                    mx3 = fmaxf(mx3, __uint_as_float(raw[c + 3]));
                }
                const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * p.scale2;
                // Each row by its own scores: what its neighbours hold, or the rows of S behind the last, which are products of whatever
                // lies in shared memory there, must not show in its rounding.
                const bool raise = valid && (mx > m + kLazyRescale || (m == -INFINITY && mx > m));
                if (__any_sync(0xffffffffu, raise)) {
                    const float alpha = !raise ? 1.f : (m == -INFINITY ? 0.f : exp2_ftz(m - mx));
                    l *= alpha;
                    if (raise) m = mx;
                    if (j > 0) {
                        // O holds the blocks before this one once their products are done
                        if (!warp_wait(&ctrl->pv_done[buf ^ 1u], ((i - 1) >> 1) & 1u, ws)) { ok = false; break; }
                        tc_fence_after_sync();
#pragma unroll 1
                        for (int c = 0; c < kDim; c += 32) {
                            uint32_t o[32];
                            tmem_ld32(tmem + lanes + kColO + c, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
                            tmem_st32(tmem + lanes + kColO + c, o);
                        }
                        tmem_wait_st();
                    }
                }
                const float base = m == -INFINITY ? 0.f : m;
                uint32_t pk[kTileKeys / 2];
                float l0 = 0.f, l1 = 0.f;
#pragma unroll
                for (int c = 0; c < kTileKeys; c += 2) {
                    const float e0 = exp2_ftz(fmaf(__uint_as_float(raw[c]), p.scale2, -base)), e1 = exp2_ftz(fmaf(__uint_as_float(raw[c + 1]), p.scale2, -base));
                    l0 += e0;
                    l1 += e1;
                    pk[c / 2] = pack_half2(e0, e1);
                }
                l += l0 + l1;
                // the buffer's previous probabilities have been multiplied
                if (i >= 2 && !warp_wait(&ctrl->pv_done[buf], ((i >> 1) & 1u) ^ 1u, ws)) { ok = false; break; }
                tmem_st32(tmem + lanes + kColP + buf * (kTileKeys / 2), pk);
                tmem_wait_st();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ctrl->p_ready[buf]));
            }
            ok = ok && mbar_wait(smem_u32(&ctrl->pv_done[(i - 1) & 1]), ((i - 1) >> 1) & 1u, ws);
            if (!ok) break;
            tc_fence_after_sync();
            const bool whole = BY_ITEM || walk.whole();
            const size_t slot = (static_cast<size_t>(blockIdx.x) * 2 + (walk.kb0 > 0 ? 0 : 1)) * rows + r;
            const long long at = (static_cast<long long>(b) * sh.rows_per_seq + pos) * sh.hq + kvh * sh.group + head_in_group;
            const float inv = whole ? 1.0f / (l > 0.f ? l : 1.0f) : 1.0f;
            // A part of a tile of many rows is stored by four lanes a row, sixteen bytes each: a thread's own row piece by piece, every store is 32
            // lines of memory and half a sector of each (24 heads, us: 512 rows behind 1536 50.3 -> 44.1, 77 behind 2000 30.8 -> 24.8).  Few rows
            // do not pay for the shuffles (1 row behind 1023 10.6 and 11.3, 8 rows of 48 queries 13.8 and 13.5), finished fp16 rows, whose
            // stores are half as many, neither (77 rows 15.8 and 19.3).
            if (FOUR && !whole) {
                const int quad = lane & ~3, q = lane & 3;
                const uint32_t live = __ballot_sync(0xffffffffu, valid) >> quad;
#pragma unroll 1
                for (int c = 0; c < kDim; c += 32) {
                    uint32_t o[32];
                    tmem_ld32(tmem + lanes + kColO + c, o);
                    tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 32; e += 16) {
                        uint4 t[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) t[k] = make_uint4(o[e + 4 * k], o[e + 4 * k + 1], o[e + 4 * k + 2], o[e + 4 * k + 3]);
                        transpose4(t, lane);
                        float* dst = p.part_o + (slot - q) * kDim + c + e + 4 * q;  // (rows follow one another)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (live >> k & 1u) __stcg(reinterpret_cast<uint4*>(dst + k * kDim), t[k]);
                    }
                }
            } else {
#pragma unroll 1
                for (int c = 0; c < kDim; c += 32) {
                    uint32_t o[32];
                    tmem_ld32(tmem + lanes + kColO + c, o);
                    tmem_wait_ld();
                    if (valid) {
                        float v[32];
#pragma unroll
                        for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(o[e]) * inv;
                        if (whole) {
                            __half* dst = p.out + at * kDim + c;
                            const __half* gate = p.q_gate ? p.q_gate + at * 512 + 256 + c : nullptr;
#pragma unroll
                            for (int e = 0; e < 4; ++e) store8(dst + 8 * e, finish8(v + 8 * e, gate ? gate + 8 * e : nullptr, p.perm_out != 0), p.out_vec);
                        } else {
                            float4* dst = reinterpret_cast<float4*>(p.part_o + slot * kDim + c);
#pragma unroll
                            for (int e = 0; e < 8; ++e) __stcg(dst + e, make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]));
                        }
                    }
                    __syncwarp();
                }
            }
            if (!whole && valid) *reinterpret_cast<float2*>(p.part_ml + slot * 2) = make_float2(m, l);
            if (!BY_ITEM && tid == 0 && kvh == 0 && walk.kb0 == 0)
                p.table[item] = make_int2(static_cast<int>(blockIdx.x) / sh.hkv, unit_owner(walk.u + walk.blocks - 1, walk.total, walk.groups));
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctrl->o_free));
            walk.advance();
        }
    } else if (p.early) {
        griddep_wait();
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before_sync();
    __syncthreads();
    if (tid == 0 && ctrl->ws.abort_flag && p.status) atomicExch(p.status, kStatusWaitTimeout);
    if (warp == kMmaWarp) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTileTmemCols);
    }
}

// Merges the parts of the items that were cut.  A warp takes every kWarpsPerRow-th part of a row, eight dims per lane; grid
// (items * Hkv, row blocks).  What the table says is kept inside the `groups` of the launch in front: one that gave up has not
// written all of it.  A row of few long sequences has up to one part per group (37 at one sequence): eight warps, a row
// a block (8192 keys, one row: 4 us, 8 with a warp a row).  Otherwise there are a few parts and many rows: a warp each.
template <int kWarpsPerRow>
__global__ void __launch_bounds__(256, 4) attn_tile_combine_kernel(__half* out, const float* part_o, const float* part_ml, const int2* table,
                                                                   const __half* q_gate, const TileShape sh, int groups, int perm_out, int out_vec) {
    griddep_prologue();
    constexpr int kBatch = 4;  // parts whose loads are in flight together
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = warp % kWarpsPerRow;
    const int item = blockIdx.x / sh.hkv, kvh = blockIdx.x % sh.hkv, rows = sh.group * sh.tile_pos;
    const int r = blockIdx.y * (8 / kWarpsPerRow) + warp / kWarpsPerRow;
    const int2 who = table[item];
    const int b = item / sh.tiles, pos = item % sh.tiles * sh.tile_pos + r / sh.group;
    const long long at = (static_cast<long long>(b) * sh.rows_per_seq + pos) * sh.hq + kvh * sh.group + r % sh.group;
    const bool gated = q_gate && r < rows && pos < sh.rows_per_seq && sub == 0;
    uint4 gate = make_uint4(0, 0, 0, 0);  // (asked for here: its way from memory is the parts')
    if (gated) gate = __ldg(reinterpret_cast<const uint4*>(q_gate + at * 512 + 256 + lane * 8));
    const int c0 = min(max(who.x, 0), groups - 1), c1 = min(max(who.y, c0), groups - 1);
    if (c0 == c1 || r >= rows || pos >= sh.rows_per_seq) return;  // (the same for all warps of a row)
    auto slot = [&](int c) { return ((static_cast<size_t>(c) * sh.hkv + kvh) * 2 + (c == c0 ? 1 : 0)) * rows + r; };
    float m = -INFINITY, l = 0.f, acc[8] = {};
    for (int c = c0 + sub; c <= c1; c += kBatch * kWarpsPerRow) {
        float2 ml[kBatch];
        float4 v[kBatch][2];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            ml[i] = make_float2(-INFINITY, 0.f);
            const int ci = c + i * kWarpsPerRow;
            if (ci <= c1) {
                ml[i] = __ldcg(reinterpret_cast<const float2*>(part_ml + slot(ci) * 2));
                const float4* src = reinterpret_cast<const float4*>(part_o + slot(ci) * kDim + lane * 8);
                v[i][0] = __ldcg(src);
                v[i][1] = __ldcg(src + 1);
            }
        }
        float top = m;
#pragma unroll
        for (int i = 0; i < kBatch; ++i) top = fmaxf(top, ml[i].x);
        const float w0 = m == -INFINITY ? 0.f : exp2_ftz(m - top);
        m = top;
        l *= w0;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] *= w0;
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            if (ml[i].x == -INFINITY) continue;
            const float w = exp2_ftz(ml[i].x - m);
            l += ml[i].y * w;
            acc[0] += v[i][0].x * w; acc[1] += v[i][0].y * w; acc[2] += v[i][0].z * w; acc[3] += v[i][0].w * w;
            acc[4] += v[i][1].x * w; acc[5] += v[i][1].y * w; acc[6] += v[i][1].z * w; acc[7] += v[i][1].w * w;
        }
    }
    if constexpr (kWarpsPerRow > 1) {
        static_assert(kWarpsPerRow == 8, "a row is a block");
        __shared__ float2 sh_ml[8];
        __shared__ __align__(16) float sh_acc[8][kDim];
        if (lane == 0) sh_ml[warp] = make_float2(m, l);
        *reinterpret_cast<float4*>(&sh_acc[warp][lane * 8]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        *reinterpret_cast<float4*>(&sh_acc[warp][lane * 8 + 4]) = make_float4(acc[4], acc[5], acc[6], acc[7]);
        __syncthreads();
        if (warp > 0) return;
        float w[8];
#pragma unroll
        for (int i = 1; i < 8; ++i) m = fmaxf(m, sh_ml[i].x);
        l = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            w[i] = sh_ml[i].x == -INFINITY ? 0.f : exp2_ftz(sh_ml[i].x - m);
            l += sh_ml[i].y * w[i];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            acc[j] = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[j] += sh_acc[i][lane * 8 + j] * w[i];
        }
    }
    const float inv = 1.0f / (l > 0.f ? l : 1.0f);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] *= inv;
    store8(out + at * kDim + lane * 8, finish8(acc, gated ? reinterpret_cast<const __half*>(&gate) : nullptr, perm_out != 0), out_vec);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn tile_encode_fn() {
    static EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<EncodeTiledFn>(sym);
    }();
    return fn;
}
bool encode_half(CUtensorMap* map, const __half* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return tile_encode_fn() &&
           tile_encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, static_cast<cuuint32_t>(rank), const_cast<__half*>(base), dims, strides, box,
                            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One CTA per SM, in whole groups of one per KV head.
int tile_ctas(int hkv, int num_sms) { return (num_sms / hkv > 0 ? num_sms / hkv : 1) * hkv; }
struct TileDims { int tile_pos, tiles, rows; long long items; };
TileDims tile_dims(int batch, int rows_per_seq, int hq, int hkv) {
    TileDims d;
    const int group = hq / hkv;
    d.tiles = (rows_per_seq + kTileRows / group - 1) / (kTileRows / group);
    d.tile_pos = (rows_per_seq + d.tiles - 1) / d.tiles;  // evenly filled
    d.rows = d.tile_pos * group;
    d.items = static_cast<long long>(batch) * d.tiles;
    return d;
}

}  // namespace

namespace {
// Whether every item is better left whole, with a group of CTAs for each.  Cut evenly, a group has two blocks or more, of one item or of two
// (which it then reads out one after the other), and the parts are merged by another launch: with several tiles a sequence that costs
// as much as kCutBlocks more blocks of the largest item, with one, which few groups share, kOneTileBlocks blocks are as long as two and the merge.
// 24 heads, us cut and whole: 77 rows behind none 15.4 and 8.4, behind 400 18.7 and 15.6, behind 600 19.1 and 19.7; 128 behind none 17.4 and 8.9;
// 512 behind none 27.0 and 17.1, behind 256 26.8 and 22.1; 2 rows behind 126 10.5 and 8.3, 1 behind 200 10.2 and 10.4, 4 behind 380 10.5 and 12.6.
// Where groups are many for the blocks, the even share is met without groups that read two parts out, and a cut costs less: kFreeCutBlocks.
// Twelve head layouts, whole / cut, mean over 16 to 24 calls: less than half a block a group, 7 blocks in the largest item 0.90 to 0.95, 8
// blocks 1.08 to 1.18 (1 head, 512 rows behind none 15.3 and 12.5 us; 32 / 1 heads, 16 rows behind 496 15.5 and 12.5), 9 blocks 1.02 to 1.09; more
// blocks a group, 8 blocks 0.87 to 0.96, 9 0.88 to 0.90, 10 0.95 to 1.15.
constexpr long long kCutBlocks = 7, kFreeCutBlocks = 5, kOneTileBlocks = 3;
bool whole_items(const AttnTiles& a, const TileDims& d, int groups) {
    if (a.ctx || d.items > groups) return false;  // (only the device knows the number of keys)
    long long most = 0, total = 0;
    for (int t = 0; t < d.tiles; ++t) {
        const long long end = static_cast<long long>(t + 1) * d.tile_pos;
        most = (a.ctx_base + (end < a.rows_per_seq ? end : a.rows_per_seq) + kTileKeys - 1) / kTileKeys;
        total += most * a.batch;
    }
    if (d.tiles == 1) return most <= kOneTileBlocks;
    return most <= (total > 2 * groups ? total / groups : 2) + (2 * total < groups ? kFreeCutBlocks : kCutBlocks);
}
}  // namespace

// Enough for every launch of at most `rows_per_seq` rows (tiles of fewer rows may each hold more of them: 128 positions are
// 7 tiles of 19, 59 are 3 of 20).
size_t attn_tile_scratch_bytes(int batch, int rows_per_seq, int hq, int hkv, int num_sms) {
    const int group = hq / hkv, most_pos = kTileRows / group < rows_per_seq ? kTileRows / group : rows_per_seq;
    const TileDims d = tile_dims(batch, rows_per_seq, hq, hkv);
    return static_cast<size_t>(tile_ctas(hkv, num_sms)) * 2 * (most_pos * group) * (kDim + 2) * sizeof(float) + static_cast<size_t>(d.items) * sizeof(int2);
}

int attn_tiles(cudaStream_t s, const AttnTiles& a, int num_sms, int* status) {
    TileParams p;
    memset(&p, 0, sizeof(p));
    const int group = a.hq / a.hkv;
    const TileDims d = tile_dims(a.batch, a.rows_per_seq, a.hq, a.hkv);
    if (d.items * a.hkv > (1 << 24)) return -2;
    {
        const cuuint64_t head = kDim * 2, pos = head * a.hq;
        const cuuint64_t dims[4] = {kDim, static_cast<cuuint64_t>(a.hq), static_cast<cuuint64_t>(a.rows_per_seq), static_cast<cuuint64_t>(a.batch)};
        const cuuint64_t strides[3] = {head, pos, pos * a.rows_per_seq};
        const cuuint32_t box[4] = {64, static_cast<cuuint32_t>(group), static_cast<cuuint32_t>(d.tile_pos), 1};
        if (!encode_half(&p.q_map, a.q, 4, dims, strides, box)) return -2;
    }
    {
        const cuuint64_t row = static_cast<cuuint64_t>(a.hkv) * kDim * 2;
        const cuuint64_t dims[3] = {static_cast<cuuint64_t>(a.hkv) * kDim, static_cast<cuuint64_t>(a.cache_rows), static_cast<cuuint64_t>(a.batch)};
        const cuuint64_t strides[2] = {row, row * static_cast<cuuint64_t>(a.cache_stride)};
        const cuuint32_t box[3] = {64, kTileKeys, 1};
        if (!encode_half(&p.k_map, a.k_cache, 3, dims, strides, box) || !encode_half(&p.v_map, a.v_cache, 3, dims, strides, box)) return -2;
    }
    p.sh.ctx = a.ctx;
    p.sh.ctx_base = a.ctx_base;
    p.sh.rows_per_seq = a.rows_per_seq;
    p.sh.hq = a.hq;
    p.sh.hkv = a.hkv;
    p.sh.group = group;
    p.sh.tile_pos = d.tile_pos;
    p.sh.tiles = d.tiles;
    p.sh.items = static_cast<int>(d.items);
    p.sh.max_seq = a.cache_rows;
    p.out = a.out;
    p.q_gate = a.q_gate;
    p.perm_out = a.perm_out;
    p.out_vec = (reinterpret_cast<uintptr_t>(a.out) & 15) == 0;
    p.early = a.early;
    p.scale2 = a.scale * 1.4426950408889634f;
    p.part_o = a.scratch;
    const int ctas = tile_ctas(a.hkv, num_sms);
    const bool by_item = whole_items(a, d, ctas / a.hkv);
    p.part_ml = a.scratch + static_cast<size_t>(ctas) * 2 * d.rows * kDim;
    p.table = reinterpret_cast<int2*>(p.part_ml + static_cast<size_t>(ctas) * 2 * d.rows * 2);
    p.wait_limit = tc_wait_limit();
    p.withhold = tc_x_stage_limit() >= 0;
    p.status = status;
    {
        static bool configured[64];
        static std::mutex mu;
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
        std::lock_guard<std::mutex> lock(mu);
        if (!configured[dev]) {
            for (auto* f : {attn_tile_kernel<false, false>, attn_tile_kernel<false, true>, attn_tile_kernel<true, false>})
                if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return -1;
            configured[dev] = true;
        }
    }
    auto* kernel = by_item ? attn_tile_kernel<true, false> : d.rows > 32 ? attn_tile_kernel<false, true> : attn_tile_kernel<false, false>;
    if (launch_pdl(kernel, dim3(ctas), dim3(kTileThreads), tile_smem_bytes(d.rows), s, p) != cudaSuccess) return -1;
    // (nothing was cut, or every item is a single block)
    if (by_item || (!a.ctx && static_cast<long long>(a.ctx_base) + a.rows_per_seq <= kTileKeys)) return 0;
    const bool wide = d.tiles == 1 && ctas >= 8 * a.batch * a.hkv;  // eight parts a row
    if (launch_pdl(wide ? attn_tile_combine_kernel<8> : attn_tile_combine_kernel<1>, dim3(p.sh.items * a.hkv, wide ? d.rows : (d.rows + 7) / 8),
                   dim3(256), 0, s, a.out, static_cast<const float*>(p.part_o), static_cast<const float*>(p.part_ml),
                   static_cast<const int2*>(p.table), a.q_gate, p.sh, ctas / a.hkv, a.perm_out, p.out_vec) != cudaSuccess)
        return -1;
    return 0;
}

}  // namespace xb
