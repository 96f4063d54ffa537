// INT4-G128 W4A16 GEMM for many activation rows (prompts, prefill chunks): Y[M,N] = X[M,K] * W^T (+ bias), M > 32.
//
// Replaces, for M = hundreds of rows, what the reference runs its prefill through: the same ops::linear_int4 /
// linear_int4_fused / mlp_gate_up_swiglu_int4 entry points (src/ops/linear.h:30-139), called with
// M = chunk length from forward_prefill_chunk (src/targets/qwen3_8/forward.cpp:402-554), where the reference
// repeats its GEMV row by row.  At M = 512 the contraction is compute-bound (2*M*N*K flops against N*K/2 bytes:
// ~2000 flop per weight byte), so this kernel is built around the tensor pipe:
//
//   * a pair of CTAs (tcgen05 cta_group::2) owns 256 weight rows (the MMA's M, 128 per CTA) x up to 256 activation rows
//     (its N, of which each CTA loads half: one CTA alone would have to pull 64 KB of activations through L2 per 128-k
//     group, 18 TB/s over the chip at full tensor rate);
//   * the int4 values go into the MMA as exact fp16 integers.  One 128-k group accumulates into one of two
//     tensor-memory tiles of 256 columns (four of 128 up to 128 rows), and while the tensor core works on the next group eight warps read the finished one back
//     and fold it into fp32 registers with the group's scale: acc += d * scale, the reference's own association
//     (src/ops/linear.cpp:239-287).  So every product is exact and every weight costs one MMA (the form before this one
//     put scale * weight into the MMA as a high and a low fp16 operand, two MMAs per k step, because it kept one
//     accumulator over all of K: 113 us at M = 512, K = 5120, N = 17408);
//   * both operands from shared memory: the activations land by TMA in the canonical 128-byte-swizzled K-major layout,
//     the packed weights land raw (64 bytes per row and group) and four warps, one thread per weight row, unpack them
//     into the same layout (up to 128 rows eight, four to every other group);
//   * the work of one launch - all tiles of all its projections x K / 128 groups - is dealt to one pair per two SMs, whole
//     tiles or, where that leaves the last wave too empty, cut evenly.  A tile that straddles a cut is finished by the CTA
//     that arrives last, which adds the others' fp32 partials in pair order (the result does not depend on who is last).
//
// Every wait is bounded (WaitState); a wait that runs out sets the device status word and the CTA leaves through
// its normal exit, releasing its tensor memory.

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <mutex>

#include "launch.cuh"
#include "ptx_sm100.cuh"
#include "silu.cuh"
#include "w4a16.h"

namespace xb {
namespace {

constexpr int kGemmFoldThreads = 256;    // two per weight row: each folds half of the tile's activation columns
constexpr int kGemmUnpackThreads = 128;  // one per weight row
constexpr int kGemmThreads = kGemmFoldThreads + kGemmUnpackThreads + 128;  // + a warpgroup with the two TMA warps and the MMA warp
constexpr int kGemmUnpackWarp0 = 8, kGemmXWarp = 12, kGemmMmaWarp = 13, kGemmWWarp = 14, kGemmUnpackWarp1 = 16;
// Sets of unpacking warps, which take the groups in turn.  A set needs 1100 clocks a group (600 of work, the rest two waits and the
// fences); at more than 128 rows the MMAs take as long.  Up to 128 rows a second
// set brings gate/up 5120 x 17408 from 49.7 to 46.9 us at 77 rows and from 52.2 to 48.0 at 128, 5120 x 14336 at 128 from 26.7 to 24.2.
constexpr int gemm_unpack_sets(int nc) { return nc <= 2 ? 2 : 1; }
constexpr int gemm_threads(int nc) { return kGemmThreads + (gemm_unpack_sets(nc) - 1) * kGemmUnpackThreads; }
constexpr int kGemmTileN = 128;   // weight rows of one CTA of a pair (gate/up: 64 of each)
constexpr int kGemmTileM = 256;   // most activation rows per tile (the MMA's N)
constexpr int kSwizzleK = 64;     // k of one 128-byte swizzle row of fp16
// Operand ring: a slot holds a whole 128-k group of unpacked weights and of activations.  The MMA warp's own loop - waits, issue
// and commits, each a hundred clocks or two - is what every stage goes through, and with 64-k slots it took longer than the
// tensor core: at M = 512 900 TFLOP/s with three waits a slot (weights and activations apart), 1120 with one, 1150 to
// 1280 with its instructions predicated and its two waits side by side (umma_ss_f16_pair, the MMA warp).
// Accumulator tiles: tiles of at most 128 rows have four, the larger ones two (all of tensor memory).
constexpr int kOpSlotsMax = 4, kDBufsMax = 4, kWSlotsMax = 8;
constexpr int kWSlotBytes = kGemmTileN * 64;                    // 8 KB of packed weights: one group
constexpr int kAHalfBytes = kGemmTileN * kSwizzleK * 2;         // 16 KB: 64 k of unpacked weights
constexpr int kASlotBytes = 2 * kAHalfBytes;
constexpr int kGemmTmemCols = 512;
constexpr int kGemmMaxProj = 4;
// Register split of the launch's 512 x 128, or 640 x 96: the fold keeps 128, or 64, sums per thread.
constexpr int kUnpackRegs = 64, kCtrlRegs = 32;
constexpr int gemm_fold_regs(int nc) { return nc <= 2 ? 144 : 208; }
constexpr int gemm_split_regs(int nc) { return gemm_fold_regs(nc) * 256 + kUnpackRegs * 128 * gemm_unpack_sets(nc) + kCtrlRegs * 128; }
static_assert(gemm_split_regs(4) <= 512 * 128 && gemm_split_regs(2) <= 640 * 96, "register split");

struct GemmCtrl {
    uint64_t w_full[kWSlotsMax], w_empty[kWSlotsMax];
    uint64_t op_full[kOpSlotsMax], op_empty[kOpSlotsMax];  // full: the pair's unpack warps and the activations' bytes
    uint64_t d_full[kDBufsMax], d_empty[kDBufsMax];
    uint32_t tmem_base;
    int last_arrival;
    WaitState ws;
};

// [control] [alignment slack] [A ring] [X ring: slots x 2 x tile_m / 2 x 128 bytes] [W ring]
constexpr int kGemmSmemBytes = 227 * 1024;
constexpr int kGemmSmemFixed = 1024 + static_cast<int>(sizeof(GemmCtrl));
constexpr int gemm_slots_bytes(int tile_m, int slots) { return slots * (kASlotBytes + tile_m * 2 * kSwizzleK); }
constexpr int gemm_op_slots(int tile_m) {
    return kGemmSmemFixed + gemm_slots_bytes(tile_m, 4) + 3 * kWSlotBytes <= kGemmSmemBytes ? 4 : 3;
}
// (the packed weights come from HBM, a microsecond and more away: their ring takes the rest)
constexpr int gemm_w_slots(int tile_m) {
    const int n = (kGemmSmemBytes - kGemmSmemFixed - gemm_slots_bytes(tile_m, gemm_op_slots(tile_m))) / kWSlotBytes;
    return n < kWSlotsMax ? n : kWSlotsMax;
}
constexpr int gemm_d_bufs(int tile_m) { return tile_m > 128 ? 2 : kDBufsMax; }
static_assert(gemm_w_slots(kGemmTileM) >= 3 && gemm_w_slots(128) >= 3, "shared memory");
// Sets of unpacking warps that take the groups in turn keep to slots of their own: the rings' lengths are multiples of their number.
// Otherwise a set would come to a slot that the other one used last, and a wait for a parity that tells its own last use from the next
// would be let through by a use that lies between them, before the bytes have landed.
constexpr bool gemm_sets_keep_their_slots() {
    for (int tile_m = 32; tile_m <= kGemmTileM; tile_m += 32) {
        const int sets = gemm_unpack_sets((tile_m + 63) / 64);
        if (gemm_op_slots(tile_m) % sets || gemm_w_slots(tile_m) % sets) return false;
    }
    return true;
}
static_assert(gemm_sets_keep_their_slots(), "ring lengths");

struct GemmProj {
    const __half* scales[2];  // gate/up: of both
    const float* bias;
    void* y;
    long long ldy;
    int n;           // output features
    int tile0;       // index of its first tile in the launch
};

struct GemmParams {
    CUtensorMap w_map[kGemmMaxProj];  // packed weights of each projection (gate/up: 0 = gate, 1 = up)
    CUtensorMap x_map;
    GemmProj proj[kGemmMaxProj];
    int num_proj;
    int m;           // activation rows
    int tile_m;      // activation rows per tile, a multiple of 32
    int w_slots;     // slots of the packed-weight ring
    int m_tiles;
    int groups;      // k / 128
    int scales_vec;  // every row of scales starts on a 16-byte boundary
    long long units;     // tiles * groups
    int pairs;           // CTA pairs of the launch
    int whole_tiles;     // cut between tiles only
    int swiglu;      // a CTA's rows: gate and up of the same 64 features, sixteen and sixteen; y = silu(gate) * up
    long long wait_limit;
    int* status;
    int x_stage_limit;  // test hook: activation stages (of a CTA) from this index on are never requested (-1: off)
    float* partials;    // [CTA][2][column / 4][fold thread][4]: fp32 sums of the tiles a CTA holds a part of
    int* counters;      // [CTA]: groups of the tile that starts in that pair's range and ends behind it, added up so far
};

// (This and the commit are executed by a whole warp under uniform control flow; the lane with `issue` set issues.  Inside `if (leader)`
// the descriptors were moved to uniform registers for every instruction: the eight of a group took 500 clocks, and 400 this way.)
// D[tmem] (+)= A[smem descriptor] * B[smem descriptor], kind::f16, on a CTA pair: A and D rows 0-127 in the even CTA,
// 128-255 in the odd one; B rows half and half, each CTA's at the descriptor's offset.  Issued by one thread of the even CTA.
__device__ __forceinline__ void umma_ss_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate, uint32_t issue) {
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}"
        :
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(issue)
        : "memory");
}
// Arrives on the mbarrier at this offset in both CTAs of the pair when every MMA issued so far has completed.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar, uint32_t issue) {
    asm volatile(
        "{\n\t"
        ".reg .pred q;\n\t"
        "setp.ne.b32 q, %2, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t"
        "}" ::"r"(bar),
        "h"(static_cast<uint16_t>(3)), "r"(issue)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// A tiled load into this CTA whose bytes are counted on a barrier of either CTA of the pair (a shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void* map, uint32_t cluster_bar, int x, int y, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1, {%3, %4}], [%2], %5;"
        :
        : "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(cluster_bar), "r"(x), "r"(y), "l"(policy)
        : "memory");
}
// (Release at CTA scope, and the waits acquire at CTA scope: what the arriving warps publish is their own SM's shared and
// tensor memory, fenced for that SM's tensor core; a release at cluster scope costs the arriving warp half a microsecond.)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// Barrier of the fold threads that also tells all of them whether any of them has given up: they leave together.
__device__ __forceinline__ bool fold_barrier_or(bool pred) {
    uint32_t r;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.b32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t"
        "}"
        : "=r"(r)
        : "r"(pred ? 1u : 0u), "n"(kGemmFoldThreads)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void fold_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kGemmFoldThreads) : "memory"); }

__device__ __forceinline__ void store_out(float* y, float v) { *y = v; }
__device__ __forceinline__ void store_out(__half* y, float v) { *y = __float2half_rn(v); }

// Scales of the groups g .. g + 7 of one weight row (g a multiple of 8; zero behind the last), and on to the next one.  `vec`:
// the row starts on a 16-byte boundary and has a multiple of eight of them; a caller's scales may lie anywhere.
__device__ __forceinline__ uint4 load_scales(const unsigned short* sp, int g, int groups, int vec) {
    uint4 q = make_uint4(0, 0, 0, 0);
    if (g >= groups) return q;
    if (vec) return __ldg(reinterpret_cast<const uint4*>(sp + g));
    uint32_t h[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) h[j] = g + j < groups ? __ldg(sp + g + j) : 0u;
    return make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
}
__device__ __forceinline__ void shift_scales(uint4& q) {
    q.x = __funnelshift_r(q.x, q.y, 16);
    q.y = __funnelshift_r(q.y, q.z, 16);
    q.z = __funnelshift_r(q.z, q.w, 16);
    q.w >>= 16;
}

// First unit of pair c: units cut evenly, or whole tiles only.
__device__ __forceinline__ long long unit_begin(const GemmParams& p, long long c) {
    if (p.whole_tiles) {
        const long long tiles = p.units / p.groups;
        return c * tiles / p.pairs * p.groups;
    }
    return c * p.units / p.pairs;
}
// The pair whose range holds unit u.
__device__ __forceinline__ int unit_owner(const GemmParams& p, long long u) {
    int c = static_cast<int>(u * p.pairs / p.units);
    while (c + 1 < p.pairs && unit_begin(p, c + 1) <= u) ++c;
    while (c > 0 && unit_begin(p, c) > u) --c;
    return c;
}
__device__ __forceinline__ int proj_of_tile(const GemmParams& p, int tile) {
    int i = 0;
    while (i + 1 < p.num_proj && tile >= p.proj[i + 1].tile0) ++i;
    return i;
}

// NC: 32-column reads a fold thread makes of an accumulator tile, ceil(tile_m / 64).
template <int NC, typename OutT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(gemm_threads(NC), 1) w4a16_gemm_kernel(const __grid_constant__ GemmParams p) {
    extern __shared__ uint8_t gemm_smem_raw[];
    // (the control block first: its addresses are then constants, and the fold, which needs every register, holds none of them)
    GemmCtrl* ctrl = reinterpret_cast<GemmCtrl*>(gemm_smem_raw);
    // the swizzled operand tiles want 1024-byte alignment
    uint8_t* a_ring = gemm_smem_raw + (((smem_u32(gemm_smem_raw) + sizeof(GemmCtrl) + 1023u) & ~1023u) - smem_u32(gemm_smem_raw));
    constexpr int d_bufs = gemm_d_bufs(NC * 64), d_shift = d_bufs == 2 ? 1 : 2, d_cols = kGemmTmemCols / d_bufs;
    const int op_slots = gemm_op_slots(p.tile_m);
    uint8_t* x_ring = a_ring + op_slots * kASlotBytes;
    const uint32_t x_half_bytes = static_cast<uint32_t>(p.tile_m) * kSwizzleK;  // 64 k of this CTA's half of the rows
    uint8_t* w_ring = x_ring + op_slots * 2 * x_half_bytes;
    const int w_slots = p.w_slots;

    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int lane = tid & 31;
    const uint32_t rank = cluster_ctarank();  // the even CTA issues the pair's MMAs
    volatile WaitState* ws = &ctrl->ws;
    griddep_launch_dependents();

    if (tid == 0) {
        for (int i = 0; i < w_slots; ++i) { mbar_init(smem_u32(&ctrl->w_full[i]), 1); mbar_init(smem_u32(&ctrl->w_empty[i]), kGemmUnpackThreads / 32); }
        for (int i = 0; i < op_slots; ++i) {
            mbar_init(smem_u32(&ctrl->op_full[i]), 2 * kGemmUnpackThreads / 32 + 1);
            mbar_init(smem_u32(&ctrl->op_empty[i]), 1);
        }
        for (int i = 0; i < d_bufs; ++i) { mbar_init(smem_u32(&ctrl->d_full[i]), 1); mbar_init(smem_u32(&ctrl->d_empty[i]), 2 * kGemmFoldThreads / 32); }
        ctrl->ws.abort_flag = 0;
        ctrl->ws.dep_ready = 0;
        ctrl->ws.limit = p.wait_limit;
        mbar_fence_init();
    }
    if (warp == kGemmMmaWarp) tmem_alloc_pair(smem_u32(&ctrl->tmem_base), kGemmTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();  // the other CTA's barriers are initialised too
    tc_fence_after_sync();
    const uint32_t tmem_base = *const_cast<volatile uint32_t*>(&ctrl->tmem_base);

    // this pair's units (tile, 128-k group), tile-major; ring slots and phases count from its first unit
    const int pair = static_cast<int>(blockIdx.x >> 1);
    const long long u0 = unit_begin(p, pair), u1 = unit_begin(p, static_cast<long long>(pair) + 1);
    const int U = static_cast<int>(u1 - u0);
    const int first_tile = static_cast<int>(u0 / p.groups), first_group = static_cast<int>(u0 - static_cast<long long>(first_tile) * p.groups);

    constexpr int kSets = gemm_unpack_sets(NC);
    if (warp >= kGemmXWarp && warp < kGemmUnpackWarp1) {
        setmaxnreg_dec<kCtrlRegs>();
        if (warp == kGemmWWarp) {
            // -------------------------------------------------------------- TMA: packed weights (whole warp waits, one lane issues)
            // They do not depend on the kernel in front of this one.  (Both TMA warps find a tile's coordinates once per tile: with the
            // projection, the divisions and the address of its map worked out per stage, 500 clocks each, they held everybody up.)
            const bool leader = elect_one_sync();
            if (leader)
                for (int i = 0; i < (p.swiglu ? 2 : p.num_proj); ++i) tma_prefetch_desc(&p.w_map[i]);
            const uint64_t pol_w = l2_policy_evict_first();
            const uint32_t ring = smem_u32(w_ring), full0 = smem_u32(&ctrl->w_full[0]), empty0 = smem_u32(&ctrl->w_empty[0]);
            int slot = 0, n = 0, group = first_group;
            uint32_t phase = 1;  // parity under which a slot's first use passes at once
            bool ok = true;
            for (int tile = first_tile; n < U && ok; ++tile) {
                const int pr = proj_of_tile(p, tile), nt = (tile - p.proj[pr].tile0) / p.m_tiles * 2 + static_cast<int>(rank);
                const CUtensorMap *map0 = &p.w_map[p.swiglu ? 0 : pr], *map1 = &p.w_map[1];
                const int y = nt * (p.swiglu ? 64 : kGemmTileN), end = U - n < p.groups - group ? group + (U - n) : p.groups;
                for (; group < end; ++group, ++n) {
                    const uint32_t full = full0 + slot * 8, dst = ring + slot * kWSlotBytes;
                    ok = mbar_wait_parked(empty0 + slot * 8, phase, ws);
                    if (!ok) break;
                    if (leader) {
                        mbar_arrive_expect_tx(full, kWSlotBytes);
                        tma_load_2d(dst, map0, full, group * 64, y, pol_w);
                        if (p.swiglu) tma_load_2d(dst + kWSlotBytes / 2, map1, full, group * 64, y, pol_w);
                    }
                    __syncwarp();  // (or the other lanes wait for the next slot before this one's load is issued)
                    if (++slot == w_slots) { slot = 0; phase ^= 1u; }
                }
                group = 0;
            }
            if (ws->abort_flag) {
                // give the copies still in flight a bounded chance to land before the CTA exits
                const long long t0 = clock64();
                for (int i = 0; i < w_slots && i < n; ++i) {
                    const int k = n - 1 - i;
                    while (!mbar_try_wait(smem_u32(&ctrl->w_full[k % w_slots]), (k / w_slots) & 1u) && clock64() - t0 < p.wait_limit / 8) {
                    }
                }
            }
            __syncwarp();
        } else if (warp == kGemmXWarp) {
            // -------------------------------------------------------------- TMA: activations
            const bool leader = elect_one_sync();
            if (leader) tma_prefetch_desc(&p.x_map);
            const uint64_t pol_x = l2_policy_evict_last();
            const int SX = (p.x_stage_limit >= 0 && p.x_stage_limit < U) ? p.x_stage_limit : U;
            const uint32_t ring = smem_u32(x_ring), full0 = smem_u32(&ctrl->op_full[0]), empty0 = smem_u32(&ctrl->op_empty[0]);
            // both halves of the rows are counted on the even CTA's barrier, where the MMAs are issued
            const uint32_t pair_full0 = mapa_shared_cluster(full0, 0);
            griddep_wait();
            if (leader) ws->dep_ready = 1;
            int nx = 0, slot = 0, k0 = first_group * 128;
            uint32_t phase = 1;
            bool ok = true;
            for (int tile = first_tile; nx < SX && ok; ++tile) {
                const int m0 = (tile - p.proj[proj_of_tile(p, tile)].tile0) % p.m_tiles * p.tile_m + static_cast<int>(rank) * (p.tile_m >> 1);
                for (; k0 < p.groups * 128 && nx < SX; k0 += 128, ++nx) {
                    ok = mbar_wait_parked(empty0 + slot * 8, phase, ws);
                    if (!ok) break;
                    if (leader) {
                        if (rank == 0) mbar_arrive_expect_tx(full0 + slot * 8, 4 * x_half_bytes);
                        tma_load_2d_pair(ring + slot * 2 * x_half_bytes, &p.x_map, pair_full0 + slot * 8, k0, m0, pol_x);
                        tma_load_2d_pair(ring + slot * 2 * x_half_bytes + x_half_bytes, &p.x_map, pair_full0 + slot * 8, k0 + kSwizzleK, m0, pol_x);
                    }
                    __syncwarp();
                    if (++slot == op_slots) { slot = 0; phase ^= 1u; }
                }
                k0 = 0;
            }
            if (ws->abort_flag) {
                const long long t0 = clock64();
                for (int i = 0; i < op_slots && i < nx; ++i) {
                    const int k = nx - 1 - i;
                    while (!mbar_try_wait(smem_u32(&ctrl->op_full[k % op_slots]), (k / op_slots) & 1u) && clock64() - t0 < p.wait_limit / 8) {
                    }
                }
            }
            __syncwarp();
        } else if (warp == kGemmMmaWarp && rank == 0) {
            // -------------------------------------------------------------- MMA issuer of the pair
            const bool leader = elect_one_sync();
            const uint32_t idesc = umma_idesc_f16_f32(256, 0) | (static_cast<uint32_t>(p.tile_m >> 3) << 17);
            // K-major, 128-byte swizzle: rows of 64 k, 8-row groups 1024 bytes apart; descriptor version 1
            constexpr uint32_t desc_hi = ((1024u >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
            constexpr uint32_t desc_lo_const = 1u << 16;
            const uint32_t a_lo0 = (smem_u32(a_ring) >> 4) & 0x3FFFu;
            const uint32_t x_lo0 = (smem_u32(x_ring) >> 4) & 0x3FFFu;
            bool ok = true;
            uint32_t slot = 0, phase = 0;
            for (int i = 0; i < U && ok; ++i) {
                const uint32_t buf = static_cast<uint32_t>(i & (d_bufs - 1));
                // (both asked before either answer is looked at: an answer takes a hundred clocks, also where there is nothing to wait for)
                const uint32_t d_bar = smem_u32(&ctrl->d_empty[buf]), d_phase = ((i >> d_shift) & 1u) ^ 1u, op_bar = smem_u32(&ctrl->op_full[slot]);
                const bool d_ready = mbar_try_wait(d_bar, d_phase), op_ready = mbar_try_wait(op_bar, phase);  // (an unused tile is ready)
                ok = (d_ready || mbar_wait_parked(d_bar, d_phase, ws)) && (op_ready || mbar_wait_parked(op_bar, phase, ws));
                if (!ok) break;
                tc_fence_after_sync();
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t alo = desc_lo_const | (a_lo0 + ((slot * kASlotBytes + (k >> 2) * kAHalfBytes + (k & 3) * 32) >> 4));
                    const uint32_t xlo = desc_lo_const | (x_lo0 + ((slot * 2 * x_half_bytes + (k >> 2) * x_half_bytes + (k & 3) * 32) >> 4));
                    umma_ss_f16_pair(tmem_base + buf * d_cols, (static_cast<uint64_t>(desc_hi) << 32) | alo,
                                     (static_cast<uint64_t>(desc_hi) << 32) | xlo, idesc, k > 0 ? 1u : 0u, leader);
                }
                umma_commit_pair(smem_u32(&ctrl->op_empty[slot]), leader);
                umma_commit_pair(smem_u32(&ctrl->d_full[buf]), leader);
                __syncwarp();
                if (++slot == static_cast<uint32_t>(op_slots)) { slot = 0; phase ^= 1u; }
            }
        }
    } else if (warp >= kGemmUnpackWarp0) {
        // ------------------------------------------------------------------ unpack: one thread per weight row of the tile
        setmaxnreg_dec<kUnpackRegs>();
        const int r = tid & (kGemmUnpackThreads - 1), set = warp >= kGemmUnpackWarp1 ? 1 : 0;
        // raw rows of 64 bytes under the 64-byte swizzle: 16-byte chunk c of row r sits at chunk c ^ ((r >> 1) & 3)
        const uint32_t w_row = static_cast<uint32_t>(r) * 64, w_sw = static_cast<uint32_t>((r >> 1) & 3);
        // gate/up: the raw tile is 64 rows of each, the operand sixteen and sixteen, so that a feature's two sums meet in one warp
        const int ra = p.swiglu ? ((r & 48) << 1) + ((r >> 6) << 4) + (r & 15) : r;
        const uint32_t a_row = static_cast<uint32_t>((ra >> 3) * 1024 + (ra & 7) * 128), a_sw = static_cast<uint32_t>(ra & 7);
        int wslot = set, aslot = set;  // (a set's own slots: gemm_sets_keep_their_slots)
        uint32_t w_phase = 0, a_phase = 1;
        for (int i = set; i < U; i += kSets) {
            const uint32_t w_bar = smem_u32(&ctrl->w_full[wslot]), a_bar = smem_u32(&ctrl->op_empty[aslot]);
            const bool w_ready = mbar_try_wait(w_bar, w_phase), a_ready = mbar_try_wait(a_bar, a_phase);  // (as in the MMA warp)
            if (!w_ready && !mbar_wait(w_bar, w_phase, ws)) break;
            const uint32_t wsrc = smem_u32(w_ring) + wslot * kWSlotBytes + w_row;
            uint4 v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] = lds128(wsrc + ((static_cast<uint32_t>(c) ^ w_sw) << 4));
            if (!a_ready && !mbar_wait(a_bar, a_phase, ws)) break;
            const uint32_t adst = smem_u32(a_ring) + aslot * kASlotBytes + a_row;
#pragma unroll
            for (int w = 0; w < 16; ++w) {
                const uint4& vw = v[w >> 2];
                uint32_t q[4];
                dequant_word((w & 3) == 0 ? vw.x : (w & 3) == 1 ? vw.y : (w & 3) == 2 ? vw.z : vw.w, q);  // (k0,k4) (k1,k5) (k2,k6) (k3,k7)
                uint4 o;
                o.x = prmt(q[0], q[1], 0x5410u);  // (k0,k1)
                o.y = prmt(q[2], q[3], 0x5410u);  // (k2,k3)
                o.z = prmt(q[0], q[1], 0x7632u);  // (k4,k5)
                o.w = prmt(q[2], q[3], 0x7632u);  // (k6,k7)
                sts128(adst + (w >> 3) * kAHalfBytes + ((static_cast<uint32_t>(w & 7) ^ a_sw) << 4), o);
            }
            fence_proxy_async_smem();  // the tensor core reads this tile through the async proxy
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_cluster(mapa_shared_cluster(smem_u32(&ctrl->op_full[aslot]), 0));
                mbar_arrive(smem_u32(&ctrl->w_empty[wslot]));
            }
            if ((aslot += kSets) >= op_slots) { aslot -= op_slots; a_phase ^= 1u; }
            if ((wslot += kSets) >= w_slots) { wslot -= w_slots; w_phase ^= 1u; }
        }
    } else {
        // ------------------------------------------------------------------ fold, then write: two threads per weight row
        setmaxnreg_inc<gemm_fold_regs(NC)>();
        const int r = tid & 127, ch = tid >> 7;          // tile row, column half
        const int half_cols = p.tile_m >> 1;             // a multiple of 16
        const uint32_t d_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(ch * half_cols);
        const bool up_row = p.swiglu && (r & 16);
        float acc[NC * 32];
        int i = 0, tile = first_tile, group = first_group;
        bool dead = false;
        while (i < U) {
            // one tile, or the part of it that lies in this pair's range
            const int pr = proj_of_tile(p, tile);
            const GemmProj& pj = p.proj[pr];
            const int rel = tile - pj.tile0, nt = rel / p.m_tiles * 2 + static_cast<int>(rank), m0 = (rel % p.m_tiles) * p.tile_m;
            const int row = p.swiglu ? nt * 64 + ((r & 96) >> 1) + (r & 15) : nt * kGemmTileN + r;
            const bool valid = row < pj.n;
            const unsigned short* sp = reinterpret_cast<const unsigned short*>(pj.scales[up_row ? 1 : 0]) +
                                       static_cast<long long>(valid ? row : 0) * p.groups;
            const int seg_begin = group, seg_end = (U - i < p.groups - group) ? group + (U - i) : p.groups;
#pragma unroll
            for (int j = 0; j < NC * 32; ++j) acc[j] = 0.f;
            // scales eight groups at a time, a block of eight ahead of its use (one group ahead, their latency is the loop's)
            uint4 q_cur = load_scales(sp, seg_begin & ~7, p.groups, p.scales_vec), q_next = load_scales(sp, (seg_begin & ~7) + 8, p.groups, p.scales_vec);
            for (int j = 0; j < (seg_begin & 7); ++j) shift_scales(q_cur);
            for (; group < seg_end; ++group, ++i) {
                const float sc = __half2float(__ushort_as_half(static_cast<unsigned short>(q_cur.x & 0xFFFFu)));
                shift_scales(q_cur);
                if ((group & 7) == 7) {
                    q_cur = q_next;
                    q_next = load_scales(sp, group + 9, p.groups, p.scales_vec);
                }
                const uint32_t buf = static_cast<uint32_t>(i & (d_bufs - 1));
                if (dead || !mbar_wait_parked(smem_u32(&ctrl->d_full[buf]), (i >> d_shift) & 1u, ws)) { dead = true; continue; }
                tc_fence_after_sync();
                const uint32_t src = d_addr + buf * d_cols;
                // 32 columns a read (one tcgen05.ld; with two of 16 the whole kernel is 20 % slower at M = 512).  A tile of
                // fewer columns reads on into columns that are allocated and not used.
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    // (always true; without a branch between them the compiler sets up a read beside the additions of the one before it,
                    // runs out of registers and keeps launch-wide values in memory, which costs every warp of the CTA: 12 % at M = 512)
                    if (NC < 4 || c * 32 < half_cols) {
                        uint32_t d[32];
                        tmem_ld32(src + c * 32, d);
                        tmem_wait_ld();
                        if (c == NC - 1) {  // the last read of this group: the MMA warp may have the columns
                            tc_fence_before_sync();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_cluster(mapa_shared_cluster(smem_u32(&ctrl->d_empty[buf]), 0));
                        }
#pragma unroll
                        for (int j = 0; j < 32; ++j) acc[c * 32 + j] = fmaf(__uint_as_float(d[j]), sc, acc[c * 32 + j]);
                    }
                }
            }
            if (fold_barrier_or(dead || ws->abort_flag != 0)) break;

            // ------------------------------------------------------------ a straddling tile: the last CTA to arrive finishes it
            int c_first = 0, c_last = 0;
            const bool split = seg_begin > 0 || seg_end < p.groups;
            if (split) {
                const long long tu = static_cast<long long>(tile) * p.groups;
                c_first = unit_owner(p, tu);
                c_last = unit_owner(p, tu + p.groups - 1);
                const size_t slot_floats = static_cast<size_t>(kGemmTileN) * kGemmTileM;
                int* counter = p.counters + c_first * 2 + rank;
                const int n = seg_end - seg_begin;
                // A tile cut once: the second pair met its part at the start of its range, long ago.  If it has indeed arrived, this
                // one's sums stay in registers (writing them, the fence behind it and reading them back took 3 us of 42 at N = 5120,
                // M = 512).
                bool kept = false;
                if (pair == c_first && c_last == c_first + 1) {
                    if (tid == 0) {
                        const bool last = atomicAdd(counter, 0) + n == p.groups;
                        if (last) *counter = 0;  // as the next launch expects it
                        ctrl->last_arrival = last ? 1 : 0;
                        __threadfence();
                    }
                    fold_barrier();
                    kept = ctrl->last_arrival != 0;
                    fold_barrier();
                }
                if (!kept) {
                    float4* mine = reinterpret_cast<float4*>(p.partials + (static_cast<size_t>(blockIdx.x) * 2 + (seg_begin > 0 ? 0 : 1)) * slot_floats) + tid;
#pragma unroll
                    for (int j = 0; j < NC * 32; j += 4)
                        if (j < half_cols) __stcg(mine + j / 4 * kGemmFoldThreads, make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]));
                    __threadfence();
                    fold_barrier();
                    if (tid == 0) {
                        const bool last = atomicAdd(counter, n) + n == p.groups;
                        if (last) *counter = 0;
                        ctrl->last_arrival = last ? 1 : 0;
                        __threadfence();
                    }
                    fold_barrier();
                }
                if (ctrl->last_arrival) {
                    // The parts are added in pair order, whoever is last; this pair's own comes back from memory too, which leaves
                    // the registers free to request a whole part, or half of one, at once.  (Sixteen columns at a time, each a
                    // trip to L2, cost 8 us a part: N = 5120, M = 256 took 43 us and takes 34.)
                    __threadfence();
                    const float* base = p.partials + static_cast<size_t>(rank) * 2 * slot_floats + tid * 4;
                    if (!kept) {
                        // a contributor's part of this tile: slot 1 if the tile starts in its range, else slot 0
                        const float4* src = reinterpret_cast<const float4*>(base + static_cast<size_t>(c_first) * 4 * slot_floats + slot_floats);
#pragma unroll
                        for (int j = 0; j < NC * 32; j += 4) {
                            if (j < half_cols) {
                                const float4 t = __ldcg(src + j / 4 * kGemmFoldThreads);
                                acc[j] = t.x;
                                acc[j + 1] = t.y;
                                acc[j + 2] = t.z;
                                acc[j + 3] = t.w;
                            }
                        }
                    }
#pragma unroll 1
                    for (int o = c_first + 1; o <= c_last; ++o) {
                        const float4* src = reinterpret_cast<const float4*>(base + static_cast<size_t>(o) * 4 * slot_floats);
#pragma unroll
                        for (int c = 0; c < NC * 32; c += 64) {
                            if (c < half_cols) {
                                float4 t[16];
#pragma unroll
                                for (int j = 0; j < 16; ++j)
                                    if (c + j * 4 < NC * 32) t[j] = __ldcg(src + (c / 4 + j) * kGemmFoldThreads);
#pragma unroll
                                for (int j = 0; j < 16; ++j) {
                                    if (c + j * 4 >= NC * 32) continue;
                                    acc[c + j * 4] += t[j].x;
                                    acc[c + j * 4 + 1] += t[j].y;
                                    acc[c + j * 4 + 2] += t[j].z;
                                    acc[c + j * 4 + 3] += t[j].w;
                                }
                            }
                        }
                    }
                }
            }
            if (!split || ctrl->last_arrival) {
                const float bias = (valid && pj.bias && !p.swiglu) ? pj.bias[row] : 0.f;
#pragma unroll
                for (int c = 0; c < NC * 2; ++c) {
                    if (c * 16 < half_cols) {
                        const int mc = m0 + ch * half_cols + c * 16;
                        OutT* out = static_cast<OutT*>(pj.y) + static_cast<long long>(mc) * pj.ldy + row;
                        if (!p.swiglu) {
                            const int live = valid ? p.m - mc : 0;
#pragma unroll
                            for (int j = 0; j < 16; ++j, out += pj.ldy)
                                if (j < live) store_out(out, acc[c * 16 + j] + bias);
                        } else {
                            // Gate and up of one feature sit sixteen lanes apart, which trade halves of the 16 columns: the gate
                            // lane finishes columns 0-7, the up lane 8-15.  (Through shared memory, with two barriers per 16
                            // columns, the trade took 4 us a tile.)
                            float y[8];  // (all of them before the first store: inside its condition each would wait for the last)
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const float a = acc[c * 16 + j], b = acc[c * 16 + 8 + j];
                                const float theirs = __shfl_xor_sync(0xffffffffu, up_row ? a : b, 16);
                                const float g = up_row ? theirs : a, u = up_row ? b : theirs;
                                // (With the compiler's division, which has a branch, the eight came one after the other: 1500 clocks per 16
                                // columns, 12000 between two tiles of 256 rows.)
                                y[j] = silu(g) * u;
                            }
                            if (up_row) out += 8 * pj.ldy;
                            const int live = valid ? p.m - mc - (up_row ? 8 : 0) : 0;
#pragma unroll
                            for (int j = 0; j < 8; ++j, out += pj.ldy)
                                if (j < live) store_out(out, y[j]);
                        }
                    }
                }
            }
            if (group == p.groups) { group = 0; ++tile; }
        }
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();  // the pair's MMAs read both CTAs' shared memory, and each arrives on the other's barriers
    uint32_t t;  // (again, rather than through the fold)
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    if (t == 0 && ctrl->ws.abort_flag && p.status) atomicExch(p.status, kStatusWaitTimeout);
    if (t >> 5 == kGemmMmaWarp) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc_pair(*const_cast<volatile uint32_t*>(&ctrl->tmem_base), kGemmTmemCols);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn gemm_encode_fn() {
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

// packed weights [n rows][k/2 bytes]: boxes of `rows` rows x 64 bytes (one 128-k group), 64-byte swizzled so that the
// unpacking threads - one per row - read their 16-byte chunks without bank conflicts
bool encode_gemm_w(CUtensorMap* map, const uint8_t* w, long long n, long long k, int rows) {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k / 2), static_cast<cuuint64_t>(n)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k / 2)};
    const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(rows)};
    const cuuint32_t estr[2] = {1, 1};
    return gemm_encode_fn() &&
           gemm_encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(w), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// activations [m rows][k] fp16: boxes of tile_m / 2 rows (each CTA of a pair loads half) x 64 k, 128-byte swizzled (the
// MMA's K-major operand layout)
bool encode_gemm_x(CUtensorMap* map, const __half* x, long long m, long long k, int tile_m) {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(m)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k) * 2};
    const cuuint32_t box[2] = {kSwizzleK, static_cast<cuuint32_t>(tile_m / 2)};
    const cuuint32_t estr[2] = {1, 1};
    return gemm_encode_fn() &&
           gemm_encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(x), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NC, typename OutT>
cudaError_t gemm_configure_and_launch(const GemmParams& p, dim3 grid, cudaStream_t stream) {
    static bool configured[64];
    static std::mutex mu;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!configured[dev]) {
            // the register re-split draws on what the block was launched with: a request above that would wait forever
            cudaFuncAttributes a;
            e = cudaFuncGetAttributes(&a, w4a16_gemm_kernel<NC, OutT>);
            if (e != cudaSuccess) return e;
            if (a.numRegs * gemm_threads(NC) < gemm_split_regs(NC)) return cudaErrorLaunchOutOfResources;
            e = cudaFuncSetAttribute(w4a16_gemm_kernel<NC, OutT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmemBytes);
            if (e != cudaSuccess) return e;
            configured[dev] = true;
        }
    }
    return launch_pdl(w4a16_gemm_kernel<NC, OutT>, grid, dim3(gemm_threads(NC)), kGemmSmemBytes, stream, p);
}

template <typename OutT>
cudaError_t gemm_configure_and_launch(const GemmParams& p, dim3 grid, cudaStream_t stream) {
    switch ((p.tile_m + 63) / 64) {
        case 1: return gemm_configure_and_launch<1, OutT>(p, grid, stream);
        case 2: return gemm_configure_and_launch<2, OutT>(p, grid, stream);
        case 3: return gemm_configure_and_launch<3, OutT>(p, grid, stream);
        default: return gemm_configure_and_launch<4, OutT>(p, grid, stream);
    }
}

}  // namespace

bool gemm_eligible(const void* x, const TcProj* proj, int num, bool swiglu, long long m, long long k, int group_size) {
    if (m <= 32 || group_size != 128 || k < 128 || (k % 128) != 0) return false;
    if (reinterpret_cast<uintptr_t>(x) & 15) return false;
    const int cnt = swiglu ? 2 : num;
    if (cnt < 1 || cnt > 4) return false;
    for (int i = 0; i < cnt; ++i)
        if ((reinterpret_cast<uintptr_t>(proj[i].w) & 15) || proj[i].n < 1 || proj[i].push) return false;
    if (swiglu && proj[0].n != proj[1].n) return false;
    return true;
}

namespace {

// How a launch's tiles are dealt to the CTA pairs.  One pair per two SMs.  Cutting tiles evens the pairs' work out and costs the
// exchange of partial sums, about as much as kCutCost groups; a small problem takes fewer pairs (below eight groups each, the
// pipeline's fill dominates).
constexpr long long kCutCost = 16;
struct GemmDeal {
    long long tiles, units, pairs;
    bool whole_tiles;
};
GemmDeal gemm_deal(const TcProj* proj, int num, bool swiglu, long long m, long long k, int num_sms, bool may_cut) {
    GemmDeal d;
    const long long groups = k / 128, m_tiles = (m + kGemmTileM - 1) / kGemmTileM, rows = swiglu ? kGemmTileN : 2 * kGemmTileN;  // of a pair
    d.tiles = 0;
    for (int i = 0; i < (swiglu ? 1 : num); ++i) d.tiles += (proj[i].n + rows - 1) / rows * m_tiles;
    d.units = d.tiles * groups;
    const long long max_pairs = num_sms / 2, whole = (d.tiles + max_pairs - 1) / max_pairs * groups;
    long long cut_pairs = d.units / 8;
    if (cut_pairs < 1) cut_pairs = 1;
    if (cut_pairs > max_pairs) cut_pairs = max_pairs;
    d.whole_tiles = !may_cut || whole <= (d.units + cut_pairs - 1) / cut_pairs + kCutCost;
    d.pairs = !d.whole_tiles ? cut_pairs : (d.tiles < max_pairs ? d.tiles : max_pairs);
    return d;
}

}  // namespace

// The kernel as it was when the routes of 33 to 64 rows were drawn (c_api.cu), up to 30 % slower than now: 5.8 us a tile of a pair (fill,
// read-out and stores) and 0.53 us a group; a cut costs kCutCost groups, or six where it falls on equal parts of every tile.  It was
// within 6 % of most of 18 shapes at 33 .. 64 rows, and off by more for the narrowest (5120 x 2048 and narrower: within 3 us) and
// for few tiles in many parts (16384 x 1024: 21 us, modelled 13).
double gemm_modelled_us(const TcProj* proj, int num, bool swiglu, long long m, long long k, int num_sms) {
    const GemmDeal d = gemm_deal(proj, num, swiglu, m, k, num_sms, true);
    const long long groups = k / 128;
    if (d.whole_tiles) {
        const long long tiles = (d.tiles + d.pairs - 1) / d.pairs;
        return 5.8 * static_cast<double>(tiles) + 0.53 * static_cast<double>(tiles * groups);
    }
    const bool even = d.units % d.pairs == 0 && groups % (d.units / d.pairs) == 0;
    return 5.8 + 0.53 * (static_cast<double>(d.units) / static_cast<double>(d.pairs) + (even ? 6.0 : static_cast<double>(kCutCost)));
}

size_t gemm_partial_bytes(int num_sms) {
    return static_cast<size_t>(num_sms) * 2 * kGemmTileN * kGemmTileM * sizeof(float);
}

// One launch for all projections that share X.  Returns 0, -1 on a launch error, -2 when the problem cannot be
// described to the kernel.
int gemm_launch(cudaStream_t stream, const void* x, const TcProj* proj, int num, bool swiglu, bool out_f32, long long m,
                long long k, int* status, long long wait_limit, int x_stage_limit, int num_sms, float* partials, int* counters) {
    GemmParams p;
    memset(&p, 0, sizeof(p));
    // rows per tile: as few tiles as 256 rows allow, evenly filled, in steps of 32 (a fold thread reads 16 columns at a time)
    p.m_tiles = static_cast<int>((m + kGemmTileM - 1) / kGemmTileM);
    p.tile_m = static_cast<int>(((m + p.m_tiles - 1) / p.m_tiles + 31) / 32 * 32);
    p.w_slots = gemm_w_slots(p.tile_m);
    p.groups = static_cast<int>(k / 128);
    long long tiles = 0;
    if (swiglu) {
        if (!encode_gemm_w(&p.w_map[0], proj[0].w, proj[0].n, k, 64) || !encode_gemm_w(&p.w_map[1], proj[1].w, proj[1].n, k, 64)) return -2;
        p.proj[0].scales[1] = static_cast<const __half*>(proj[1].scales);
    }
    p.num_proj = swiglu ? 1 : num;
    p.scales_vec = p.groups % 8 == 0;  // (one flag a launch: read for every projection it cost the kernel 1 to 2 %)
    for (int i = 0; i < p.num_proj; ++i) {
        const TcProj& a = proj[i];
        if (!swiglu && !encode_gemm_w(&p.w_map[i], a.w, a.n, k, kGemmTileN)) return -2;
        p.proj[i].scales[0] = static_cast<const __half*>(a.scales);
        p.proj[i].bias = a.bias;
        p.proj[i].y = a.y;
        p.proj[i].ldy = a.ldy > 0 ? a.ldy : a.n;
        p.proj[i].n = static_cast<int>(a.n);
        if (((reinterpret_cast<uintptr_t>(a.scales) | reinterpret_cast<uintptr_t>(p.proj[i].scales[1])) & 15) != 0) p.scales_vec = 0;
        p.proj[i].tile0 = static_cast<int>(tiles);
        const int rows = swiglu ? kGemmTileN : 2 * kGemmTileN;  // of a pair
        tiles += (a.n + rows - 1) / rows * p.m_tiles;
    }
    const GemmDeal deal = gemm_deal(proj, num, swiglu, m, k, num_sms, partials != nullptr);
    if (deal.tiles > (1 << 30)) return -2;
    if (!encode_gemm_x(&p.x_map, static_cast<const __half*>(x), m, k, p.tile_m)) return -2;
    p.m = static_cast<int>(m);
    p.units = deal.units;
    p.swiglu = swiglu ? 1 : 0;
    p.wait_limit = wait_limit;
    p.x_stage_limit = x_stage_limit;
    p.status = status;
    p.partials = partials;
    p.counters = counters;
    p.whole_tiles = deal.whole_tiles ? 1 : 0;
    p.pairs = static_cast<int>(deal.pairs);
    const dim3 grid(static_cast<unsigned>(2 * deal.pairs));
    const cudaError_t e = out_f32 ? gemm_configure_and_launch<float>(p, grid, stream) : gemm_configure_and_launch<__half>(p, grid, stream);
    return e == cudaSuccess ? 0 : -1;
}

}  // namespace xb
