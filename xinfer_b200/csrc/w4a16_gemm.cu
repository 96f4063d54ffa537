// INT4-G128 W4A16 GEMM for many activation rows (prompts, prefill chunks): Y[M,N] = X[M,K] * W^T (+ bias), M > 32.
//
// Replaces, for M = hundreds of rows, what the reference runs its prefill through: the same ops::linear_int4 /
// linear_int4_fused / mlp_gate_up_swiglu_int4 entry points (src/ops/linear.h:30-139), called with
// M = chunk length from forward_prefill_chunk (src/targets/qwen3_8/forward.cpp:402-554), where the reference
// repeats its GEMV row by row.  At M = 512 the contraction is compute-bound (2*M*N*K flops against N*K/2 bytes:
// ~2000 flop per weight byte), so this kernel is built around the tensor pipe:
//
//   * a pair of CTAs (tcgen05 cta_group::2) owns 256 weight rows (the MMA's M, 128 per CTA) x up to 256 activation rows
//     (of which each CTA loads half: one CTA alone would have to pull 64 KB of activations through L2 per 128-k group, 18 TB/s
//     over the chip at full tensor rate);
//   * the int4 values go into the MMA as exact fp16 integers.  One 128-k group accumulates into a tensor-memory tile of up to 192
//     columns (above 192 activation rows two such tiles of half the rows each, one after the other).  There are two or three, and while
//     the tensor core works on the next one eight warps read the finished one back and fold it into fp32 registers with the group's
//     scale: acc += d * scale, the reference's own association (src/ops/linear.cpp:239-287).  So every product is exact and every weight
//     costs one MMA;
//   * the weights are the operand in tensor memory, the activations the one in shared memory.  Activations land by TMA in the
//     canonical 128-byte-swizzled K-major layout; the packed weights land raw (64 bytes per row and group) and four warps, one
//     thread per weight row, unpack them into their lanes of tensor memory (up to 128 rows eight, four to every other group).
//     With both operands in shared memory its bandwidth was the pace: of 128 bytes a clock, a CTA's group moved 8 KB of packed
//     weights in and out, 32 KB of unpacked ones in and out, and its half of the activations in and out, 900 clocks at 96 rows
//     (measured: 860 a group, the MMAs of it 384) and 1270 at 256 (1215; 1024).  The unpacked weights were 512 of either.
//     What is the pace now: up to 128 rows issue slots, 70 % of which are taken, most of all on the scheduler that the MMA warp shares
//     with two fold and two unpacking warps (700 to 900 clocks a group); at 256 rows the MMAs, at the clock that the power limit
//     leaves (720 to 780 ns a group: 1.6 to 1.7 PFLOP/s, what the library's GEMM reaches in a burst).  Gate/up 5120 x 17408, one GPU
//     in turn: 77 rows 45.0 -> 40.7 us, 96 44.5 -> 43.2, 160 56.4 -> 53.2, 352 115.8 -> 108.1, 512 141.5 -> 138.6;
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
constexpr int kGemmTileN = 128;   // weight rows of one CTA of a pair (gate/up: 64 of each)
constexpr int kGemmTileM = 256;   // most activation rows per tile
constexpr int kSwizzleK = 64;     // k of one 128-byte swizzle row of fp16
// Shapes of a kernel: H accumulator tiles per group of C times 16 columns (the MMA's N).  Up to 192 activation rows are one accumulator
// tile, of which tensor memory has room for two beside two slots of unpacked weights, up to 128 rows for three; more rows are two tiles of
// half of them each.  The rows are a multiple of 16 * H, so that the rows of an accumulator tile that each CTA holds are whole 8-row
// swizzle atoms.
constexpr int kGemmTmemCols = 512, kASlotCols = 64, kDBufsMax = 3;
constexpr int gemm_halves(int tile_m) { return tile_m > 192 ? 2 : 1; }
constexpr int gemm_d_bufs(int c) { return c <= 8 ? 3 : 2; }
constexpr int gemm_a_slots(int c) { return gemm_d_bufs(c) * c * 16 + 4 * kASlotCols <= kGemmTmemCols ? 4 : 2; }  // (at the end of it)
// Up to 80 rows the two fold threads of a row take the groups in turn (kInTurn), all columns of each, and add their sums up when the tile, or the
// part of it, is done; with more, sums for all columns do not fit the registers and each takes half of the columns of every group.  So they do
// on tiles of up to kHalvesGroups groups too, where what they trade at the end is the larger part (us in turn and in halves: 640 x 20000, 64 rows
// 11.1 and 9.9, 77 rows 11.9 and 10.6; 1024 x 25000, 64 rows 13.4 and 12.4, 77 rows 14.5 and 13.3; 512 x 10000, 48 rows 5.8 in halves; but gate/up
// 5120 x 17408, 48 rows 37.1 and 38.7, 77 rows 40.8 and 41.8).  Two or three groups in turn, the products of the second thread's first group
// rounded by themselves, have a tenth larger error against 64 bits than in sequence; with more it is smaller, 0.84 of it at 16 groups and 0.77
// at 40, which is why tiles of 9 to 24 groups stay in turn although some are faster in halves (2048 x 5632, 64 rows 10.2 and 9.7).
constexpr bool gemm_may_fold_in_turn(int h, int c) { return h == 1 && c <= 5; }
constexpr int kHalvesGroups = 8;
// Sets of unpacking warps, which take the groups in turn.  Up to 128 rows the MMAs of a group take up to 512 clocks, less than a set needs.
constexpr int gemm_unpack_sets(int h, int c) { return h == 1 && c <= 8 ? 2 : 1; }
constexpr int gemm_threads(int h, int c) { return kGemmThreads + (gemm_unpack_sets(h, c) - 1) * kGemmUnpackThreads; }
// Shared memory: a slot of either ring holds a whole 128-k group.
constexpr int kXSlotsMax = 8, kWSlotsMax = 12, kASlotsMax = 4;
constexpr int kWSlotBytes = kGemmTileN * 64;                    // 8 KB of packed weights: one group
constexpr int kGemmMaxProj = 4;
constexpr long long kOthersWait = 12000;  // clocks
// Register split of the launch's 512 x 128, or 640 x 96: the fold keeps up to 128, or 96, sums per thread.
constexpr int kCtrlRegs = 32, kUnpackRegs = 64;
constexpr int gemm_fold_regs(int h, int c) { return gemm_unpack_sets(h, c) == 2 ? 160 : 208; }
constexpr int gemm_split_regs(int h, int c) { return gemm_fold_regs(h, c) * 256 + kUnpackRegs * 128 * gemm_unpack_sets(h, c) + kCtrlRegs * 128; }
static_assert(gemm_split_regs(2, 8) <= 512 * 128 && gemm_split_regs(1, 12) <= 512 * 128 && gemm_split_regs(1, 8) <= 640 * 96, "register split");

struct GemmCtrl {
    uint64_t w_full[kWSlotsMax], w_empty[kWSlotsMax];
    uint64_t x_full[kXSlotsMax];  // the activations' bytes, both CTAs'
    // A group's MMAs are done: its accumulator tile (the second one of two) may be read, its slots of weights and activations be filled
    // again.  One commit for all three: the ring has the length of the activations' and those who wait look up the group they wait for.
    uint64_t done[kXSlotsMax], half_done[kXSlotsMax];
    uint64_t a_full[kASlotsMax];  // the pair's unpacking warps
    uint64_t d_empty[kDBufsMax];
    uint32_t tmem_base;
    WaitState ws;
};

// [control] [alignment slack] [X ring] [W ring] [sums that the two fold threads of a row trade]
constexpr int kGemmSmemBytes = 227 * 1024;
constexpr int kGemmSmemFixed = 1024 + static_cast<int>(sizeof(GemmCtrl));
constexpr int gemm_x_slots(int h, int c) { return h * c <= 8 ? 8 : 4; }
constexpr int gemm_x_half_bytes(int h, int c) { return h * c * 8 * 2 * kSwizzleK; }  // 64 k of a CTA's half of the rows
constexpr int gemm_trade_bytes(int h, int c) { return gemm_may_fold_in_turn(h, c) ? kGemmFoldThreads * c * 8 * 4 : 0; }
// (the packed weights come from HBM, a microsecond and more away: their ring takes the rest)
constexpr int gemm_w_slots(int h, int c) {
    const int n = (kGemmSmemBytes - kGemmSmemFixed - gemm_x_slots(h, c) * 2 * gemm_x_half_bytes(h, c) - gemm_trade_bytes(h, c)) / kWSlotBytes & ~1;
    return n < kWSlotsMax ? n : kWSlotsMax;
}
// Who waits for a phase of a barrier by its parity must have seen the phase before it end, and the phase after it must not end before he
// has looked.  Sets of unpacking warps that take the groups in turn come to every slot of the packed weights, and to every entry of
// `done`, by themselves if the rings' lengths are multiples of their number; no group's MMAs are issued before those of the group that
// lies as many before as there are accumulator tiles, or slots of unpacked weights, have been seen done: the ring is no shorter.
constexpr bool gemm_rings_keep_in_step() {
    for (int tile_m = 16; tile_m <= kGemmTileM; tile_m += 16 * gemm_halves(tile_m + 1)) {
        const int h = gemm_halves(tile_m), c = tile_m / h / 16, sets = gemm_unpack_sets(h, c);
        const int x = gemm_x_slots(h, c), w = gemm_w_slots(h, c), a = gemm_a_slots(c), d = gemm_d_bufs(c);
        if (x % sets || w % sets || a % sets || x < d || x < a || x > kXSlotsMax || a > kASlotsMax || d > kDBufsMax || w < 8) return false;
        if (d * c * 16 + a * kASlotCols > kGemmTmemCols) return false;
    }
    return true;
}
static_assert(gemm_rings_keep_in_step(), "ring lengths");

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
    int tile_m;      // activation rows per tile, a multiple of 16 up to 192 and of 32 above
    int pair_stores; // two neighbouring features of every output lie in one aligned word (fp16)
    int m_tiles;
    int groups;      // k / 128
    int scales_vec;  // every row of scales starts on a 16-byte boundary
    long long units;     // tiles * groups
    int pairs;           // CTA pairs of the launch
    long long deal_quot; // what is dealt to each pair: whole tiles (deal_size groups) or single groups, the remainder spread evenly
    int deal_rem, deal_size;
    long long wait_limit;
    int* status;
    int x_stage_limit;  // test hook: activation stages (of a CTA) from this index on are never requested (-1: off)
    float* partials;    // [CTA][2][column / 4][fold thread][4]: fp32 sums of the tiles a CTA holds a part of
    int* counters;      // [CTA][fold warp]: groups of the tile that starts in that pair's range and ends behind it, added up so far
};

// (This and the commit are executed by a whole warp under uniform control flow; the lane with `issue` set issues.  Inside `if (leader)`
// the descriptors were moved to uniform registers for every instruction: the eight of a group took 500 clocks, and 400 this way.)
// D[tmem] (+)= A[tmem] * B[smem descriptor], kind::f16, on a CTA pair: A and D rows 0-127 in the even CTA's tensor memory,
// 128-255 in the odd one's; B rows half and half, each CTA's at the descriptor's offset.  Issued by one thread of the even CTA.
__device__ __forceinline__ void umma_ts_f16_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate, uint32_t issue) {
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}"
        :
        : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(issue)
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
// `live` (of at most eight) activation rows of one output feature, from `y` on.  Neighbouring lanes trade four of their eight, so that each
// stores two features of four rows: half the stores, each of four bytes.  `pairs`: such words are aligned, and neighbouring lanes agree
// about `live`.  All lanes call.
template <typename OutT>
__device__ __forceinline__ void store_rows(OutT* y, long long ldy, const float* v, int live, bool pairs, int lane) {
    if constexpr (sizeof(OutT) == 2) {
        const bool odd = lane & 1;
        uint32_t h[4], even_f[2], odd_f[2];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __half2 t = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
            h[j] = *reinterpret_cast<const uint32_t*>(&t);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t theirs = __shfl_xor_sync(0xffffffffu, odd ? h[2 * j] : h[2 * j + 1], 1), mine = odd ? h[2 * j + 1] : h[2 * j];
            even_f[j] = odd ? theirs : mine;
            odd_f[j] = odd ? mine : theirs;
        }
        if (pairs && live >= 8) {
            OutT* out = odd ? y - 1 + 2 * ldy : y;
#pragma unroll
            for (int j = 0; j < 2; ++j, out += 4 * ldy) {
                *reinterpret_cast<uint32_t*>(out) = prmt(even_f[j], odd_f[j], 0x5410u);
                *reinterpret_cast<uint32_t*>(out + ldy) = prmt(even_f[j], odd_f[j], 0x7632u);
            }
            return;
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j, y += ldy)
        if (j < live) store_out(y, v[j]);
}

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
__device__ __forceinline__ void next_word(uint4& q) {
    q.x = q.y;
    q.y = q.z;
    q.z = q.w;
}
__device__ __forceinline__ void shift_scales(uint4& q) {
    q.x = __funnelshift_r(q.x, q.y, 16);
    q.y = __funnelshift_r(q.y, q.z, 16);
    q.z = __funnelshift_r(q.z, q.w, 16);
    q.w >>= 16;
}

// First unit of pair c: floor(c * tiles / pairs) tiles on, or floor(c * units / pairs) units (the division by host, but for its remainder).
__device__ __forceinline__ long long unit_begin(const GemmParams& p, int c) { return (c * p.deal_quot + c * p.deal_rem / p.pairs) * p.deal_size; }
__device__ __forceinline__ int proj_of_tile(const GemmParams& p, int tile) {
    int i = 0;
    while (i + 1 < p.num_proj && tile >= p.proj[i + 1].tile0) ++i;
    return i;
}

// Eight packed int4 (k0 in the lowest nibble) -> (k0,k1) (k2,k3) (k4,k5) (k6,k7) as fp16 pairs.  As dequant_word, but each byte is first
// copied into both halves of a register, its low nibble used of the one and its high nibble of the other, which leaves them in k order.
// (Volatile: the words of a group are to be ready in registers when its slot of tensor memory becomes free.)
__device__ __forceinline__ void dequant_word_in_order(uint32_t w, uint32_t* q) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
        asm volatile(
            "{\n\t"
            ".reg .b32 t;\n\t"
            "prmt.b32 t, %1, 0, %2;\n\t"
            "lop3.b32 t, t, 0x00F0000F, %3, 0x6A;\n\t"
            "sub.f16x2 %0, t, %3;\n\t"
            "}"
            : "=r"(q[j])
            : "r"(w), "r"(0x4040u | static_cast<uint32_t>(j * 0x101)), "r"(0x54806408u));
}

__device__ __forceinline__ int load_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void add4(float* acc, const float4& t) {
    acc[0] += t.x;
    acc[1] += t.y;
    acc[2] += t.z;
    acc[3] += t.w;
}
// f(Step<0>()) ... f(Step<N - 1>()): a loop whose index is a constant.
template <int I>
struct Step { static constexpr int value = I; };
template <int N, int I = 0, typename F>
__device__ __forceinline__ void for_steps(F&& f) {
    if constexpr (I < N) {
        f(Step<I>());
        for_steps<N, I + 1>(f);
    }
}

// H accumulator tiles a group of C times 16 columns each.  kInTurn: see gemm_may_fold_in_turn.  kSwiglu: a CTA's rows are gate and up of the
// same 64 features, sixteen and sixteen; y = silu(gate) * up.
template <int H, int C, bool kInTurn, typename OutT, bool kSwiglu>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(gemm_threads(H, C), 1) w4a16_gemm_kernel(const __grid_constant__ GemmParams p) {
    extern __shared__ uint8_t gemm_smem_raw[];
    // (the control block first: its addresses are then constants, and the fold, which needs every register, holds none of them)
    GemmCtrl* ctrl = reinterpret_cast<GemmCtrl*>(gemm_smem_raw);
    // the swizzled operand tiles want 1024-byte alignment
    uint8_t* x_ring = gemm_smem_raw + (((smem_u32(gemm_smem_raw) + sizeof(GemmCtrl) + 1023u) & ~1023u) - smem_u32(gemm_smem_raw));
    constexpr int acc_cols = C * 16, half_cols = C * 8, tile_m = H * acc_cols;
    constexpr int x_slots = gemm_x_slots(H, C), x_shift = x_slots == 8 ? 3 : 2, w_slots = gemm_w_slots(H, C), a_slots = gemm_a_slots(C);
    constexpr int d_bufs = gemm_d_bufs(C);
    constexpr uint32_t x_half_bytes = gemm_x_half_bytes(H, C);
    uint8_t* w_ring = x_ring + x_slots * 2 * x_half_bytes;

    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int lane = tid & 31;
    const uint32_t rank = cluster_ctarank();  // the even CTA issues the pair's MMAs
    volatile WaitState* ws = &ctrl->ws;
    griddep_launch_dependents();

    if (tid == 0) {
        for (int i = 0; i < w_slots; ++i) { mbar_init(smem_u32(&ctrl->w_full[i]), 1); mbar_init(smem_u32(&ctrl->w_empty[i]), kGemmUnpackThreads / 32); }
        for (int i = 0; i < x_slots; ++i) {
            mbar_init(smem_u32(&ctrl->x_full[i]), 1);
            mbar_init(smem_u32(&ctrl->done[i]), 1);
            mbar_init(smem_u32(&ctrl->half_done[i]), 1);
        }
        for (int i = 0; i < a_slots; ++i) mbar_init(smem_u32(&ctrl->a_full[i]), 2 * kGemmUnpackThreads / 32);
        for (int i = 0; i < d_bufs; ++i) mbar_init(smem_u32(&ctrl->d_empty[i]), 2 * kGemmFoldThreads / 32 / (kInTurn ? 2 : 1));
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
    const long long u0 = unit_begin(p, pair), u1 = unit_begin(p, pair + 1);
    const int U = static_cast<int>(u1 - u0);
    const int first_tile = static_cast<int>(u0 / p.groups), first_group = static_cast<int>(u0 - static_cast<long long>(first_tile) * p.groups);

    constexpr int kSets = gemm_unpack_sets(H, C);
    const uint32_t a_base = tmem_base + kGemmTmemCols - static_cast<uint32_t>(a_slots * kASlotCols);
    if (warp >= kGemmXWarp && warp < kGemmUnpackWarp1) {
        setmaxnreg_dec<kCtrlRegs>();
        if (warp == kGemmWWarp) {
            // -------------------------------------------------------------- TMA: packed weights (whole warp waits, one lane issues)
            // They do not depend on the kernel in front of this one.  (Both TMA warps find a tile's coordinates once per tile: with the
            // projection, the divisions and the address of its map worked out per stage, 500 clocks each, they held everybody up.)
            const bool leader = elect_one_sync();
            if (leader)
                for (int i = 0; i < (kSwiglu ? 2 : p.num_proj); ++i) tma_prefetch_desc(&p.w_map[i]);
            const uint64_t pol_w = l2_policy_evict_first();
            const uint32_t ring = smem_u32(w_ring), full0 = smem_u32(&ctrl->w_full[0]), empty0 = smem_u32(&ctrl->w_empty[0]);
            int slot = 0, n = 0, group = first_group;
            uint32_t phase = 1;  // parity under which a slot's first use passes at once
            bool ok = true;
            for (int tile = first_tile; n < U && ok; ++tile) {
                const int pr = proj_of_tile(p, tile), nt = (tile - p.proj[pr].tile0) / p.m_tiles * 2 + static_cast<int>(rank);
                const CUtensorMap *map0 = &p.w_map[kSwiglu ? 0 : pr], *map1 = &p.w_map[1];
                const int y = nt * (kSwiglu ? 64 : kGemmTileN), end = U - n < p.groups - group ? group + (U - n) : p.groups;
                for (; group < end; ++group, ++n) {
                    const uint32_t full = full0 + slot * 8, dst = ring + slot * kWSlotBytes;
                    ok = mbar_wait_parked(empty0 + slot * 8, phase, ws);
                    // (all CTAs start together: without a pause the first group would come back interleaved with the whole ring of every CTA)
                    if (n == 3) ok = ok && mbar_wait_parked(full0, 0, ws);
                    if (!ok) break;
                    if (leader) {
                        mbar_arrive_expect_tx(full, kWSlotBytes);
                        tma_load_2d(dst, map0, full, group * 64, y, pol_w);
                        if (kSwiglu) tma_load_2d(dst + kWSlotBytes / 2, map1, full, group * 64, y, pol_w);
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
            const uint32_t ring = smem_u32(x_ring), full0 = smem_u32(&ctrl->x_full[0]), empty0 = smem_u32(&ctrl->done[0]);
            // both halves of the rows are counted on the even CTA's barrier, where the MMAs are issued
            const uint32_t pair_full0 = mapa_shared_cluster(full0, 0);
            griddep_wait();
            if (leader) ws->dep_ready = 1;
            int nx = 0, slot = 0, k0 = first_group * 128;
            uint32_t phase = 1;
            bool ok = true;
            for (int tile = first_tile; nx < SX && ok; ++tile) {
                const int m0 = (tile - p.proj[proj_of_tile(p, tile)].tile0) % p.m_tiles * tile_m + static_cast<int>(rank) * (tile_m >> 1);
                for (; k0 < p.groups * 128 && nx < SX; k0 += 128, ++nx) {
                    ok = mbar_wait_parked(empty0 + slot * 8, phase, ws);
                    if (!ok) break;
                    if (leader) {
                        if (rank == 0) mbar_arrive_expect_tx(full0 + slot * 8, tile_m * 256u);
                        tma_load_2d_pair(ring + slot * 2 * x_half_bytes, &p.x_map, pair_full0 + slot * 8, k0, m0, pol_x);
                        tma_load_2d_pair(ring + slot * 2 * x_half_bytes + x_half_bytes, &p.x_map, pair_full0 + slot * 8, k0 + kSwizzleK, m0, pol_x);
                    }
                    __syncwarp();
                    if (++slot == x_slots) { slot = 0; phase ^= 1u; }
                }
                k0 = 0;
            }
            if (ws->abort_flag) {
                const long long t0 = clock64();
                for (int i = 0; i < x_slots && i < nx; ++i) {
                    const int k = nx - 1 - i;
                    while (!mbar_try_wait(smem_u32(&ctrl->x_full[k % x_slots]), (k / x_slots) & 1u) && clock64() - t0 < p.wait_limit / 8) {
                    }
                }
            }
            __syncwarp();
        } else if (warp == kGemmMmaWarp && rank == 0) {
            // -------------------------------------------------------------- MMA issuer of the pair
            const bool leader = elect_one_sync();
            const uint32_t idesc = umma_idesc_f16_f32(256, 0) | (static_cast<uint32_t>(acc_cols >> 3) << 17);
            // K-major, 128-byte swizzle: rows of 64 k, 8-row groups 1024 bytes apart; descriptor version 1
            constexpr uint32_t desc_hi = ((1024u >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
            constexpr uint32_t desc_lo_const = 1u << 16;
            const uint32_t x_lo0 = (smem_u32(x_ring) >> 4) & 0x3FFFu;
            // (Barriers are asked in the middle of the group before, all before any answer is looked at: an answer takes a hundred clocks, also
            // where there is nothing to wait for, and the tensor core has little more than that to do when a group's last MMA is issued.)
            const uint32_t x_bar0 = smem_u32(&ctrl->x_full[0]), a_bar0 = smem_u32(&ctrl->a_full[0]), d_bar0 = smem_u32(&ctrl->d_empty[0]);
            bool ok = true, x_ready = false, a_ready = false, d_ready = true;  // (an unused accumulator tile is ready)
            uint32_t xslot = 0, x_phase = 0, aslot = 0, a_phase = 0, buf = 0, d_phase = 1;
            for (int i = 0; i < U && ok; ++i) {
                const uint32_t x_now = x_lo0 + xslot * (2 * x_half_bytes >> 4), a_now = a_base + aslot * kASlotCols;
                ok = (x_ready || mbar_wait_parked(x_bar0 + xslot * 8, x_phase, ws)) && (a_ready || mbar_wait_parked(a_bar0 + aslot * 8, a_phase, ws));
                const uint32_t done_bar = smem_u32(&ctrl->done[0]) + xslot * 8, half_bar = smem_u32(&ctrl->half_done[0]) + xslot * 8;
                if (++xslot == static_cast<uint32_t>(x_slots)) { xslot = 0; x_phase ^= 1u; }
                if (++aslot == static_cast<uint32_t>(a_slots)) { aslot = 0; a_phase ^= 1u; }
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    ok = ok && (d_ready || mbar_wait_parked(d_bar0 + buf * 8, d_phase, ws));
                    if (!ok) break;
                    tc_fence_after_sync();
                    const uint32_t d_now = tmem_base + buf * acc_cols;
                    const uint32_t b_now = desc_lo_const | (x_now + (h ? static_cast<uint32_t>(acc_cols) * 64 >> 4 : 0u));
                    if (++buf == d_bufs) { buf = 0; d_phase ^= 1u; }
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        if (k == 4) {
                            d_ready = mbar_test_wait(d_bar0 + buf * 8, d_phase);
                            if (h == H - 1) {
                                x_ready = mbar_test_wait(x_bar0 + xslot * 8, x_phase);
                                a_ready = mbar_test_wait(a_bar0 + aslot * 8, a_phase);
                            }
                        }
                        umma_ts_f16_pair(d_now, a_now + k * 8, (static_cast<uint64_t>(desc_hi) << 32) | (b_now + ((k >> 2) * x_half_bytes + (k & 3) * 32 >> 4)),
                                         idesc, k > 0 ? 1u : 0u, leader);
                    }
                    umma_commit_pair(h == H - 1 ? done_bar : half_bar, leader);
                    __syncwarp();
                }
            }
        }
    } else if (warp >= kGemmUnpackWarp0) {
        // ------------------------------------------------------------------ unpack: one thread per weight row of the tile
        setmaxnreg_dec<kUnpackRegs>();
        const int r = tid & (kGemmUnpackThreads - 1), set = warp >= kGemmUnpackWarp1 ? 1 : 0;
        // gate/up: the raw tile is 64 rows of each, the operand sixteen and sixteen, so that a feature's two sums meet in one warp
        const int rr = kSwiglu ? ((r >> 5) << 4) + (r & 15) + ((r & 16) << 2) : r;
        // raw rows of 64 bytes under the 64-byte swizzle: 16-byte chunk c of row rr sits at chunk c ^ ((rr >> 1) & 3)
        const uint32_t w_row = smem_u32(w_ring) + static_cast<uint32_t>(rr) * 64, w_sw = static_cast<uint32_t>((rr >> 1) & 3);
        const uint32_t a_row = a_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        int wslot = set;  // (a set's own slots: gemm_rings_keep_in_step)
        uint32_t w_phase = 0;
        constexpr int kAhead = 8;  // of a group's sixteen words, those unpacked before its slot is asked for
        for (int i = set; i < U; i += kSets) {
            // the slot's last user: the group a_slots before this one
            const int last = i - a_slots;
            const uint32_t w_bar = smem_u32(&ctrl->w_full[wslot]), a_bar = smem_u32(&ctrl->done[last & (x_slots - 1)]);
            const uint32_t a_phase = static_cast<uint32_t>(last >> x_shift) & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(w_bar, w_phase, ws))) break;
            const uint32_t wsrc = w_row + wslot * kWSlotBytes;
            uint4 v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] = lds128(wsrc + ((static_cast<uint32_t>(c) ^ w_sw) << 4));
            const uint32_t adst = a_row + static_cast<uint32_t>(i & (a_slots - 1)) * kASlotCols;
            uint32_t q[kAhead * 4];
#pragma unroll
            for (int w = 0; w < kAhead; ++w) {
                const uint4& vw = v[w >> 2];
                dequant_word_in_order((w & 3) == 0 ? vw.x : (w & 3) == 1 ? vw.y : (w & 3) == 2 ? vw.z : vw.w, q + w * 4);
            }
            if (!__all_sync(0xffffffffu, last < 0 || mbar_wait(a_bar, a_phase, ws))) break;  // (tcgen05.st wants the whole warp)
            tc_fence_after_sync();
#pragma unroll
            for (int w = 0; w < kAhead; w += 2) tmem_st8(adst + w * 4, q + w * 4);
#pragma unroll
            for (int w = kAhead; w < 16; w += 2) {
                uint32_t t[8];
                const uint4& vw = v[w >> 2];
                dequant_word_in_order((w & 2) ? vw.z : vw.x, t);
                dequant_word_in_order((w & 2) ? vw.w : vw.y, t + 4);
                tmem_st8(adst + w * 4, t);
            }
            if (lane == 0) mbar_arrive(smem_u32(&ctrl->w_empty[wslot]));
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(mapa_shared_cluster(smem_u32(&ctrl->a_full[i & (a_slots - 1)]), 0));
            if ((wslot += kSets) >= w_slots) { wslot -= w_slots; w_phase ^= 1u; }
        }
    } else {
        // ------------------------------------------------------------------ fold, then write: two threads per weight row
        setmaxnreg_inc<gemm_fold_regs(H, C)>();
        const int r = tid & 127, ch = tid >> 7;  // tile row, and which of the row's two threads
        const uint32_t d_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + (kInTurn ? 0u : static_cast<uint32_t>(ch * half_cols));
        const uint32_t d_empty0 = mapa_shared_cluster(smem_u32(&ctrl->d_empty[0]), 0);
        const bool up_row = kSwiglu && (r & 16);
        // (accumulator tile h holds, of each CTA's activation rows, those from h * half_cols on: a thread's columns are rows in sequence)
        constexpr int kCols = kInTurn || H == 2 ? half_cols : (half_cols + 15) / 16 * 16;  // of an accumulator tile, as they are written
        float acc[kInTurn ? acc_cols : H * kCols];
        uint32_t buf = kInTurn ? static_cast<uint32_t>(ch) : 0u;
        int i = 0, tile = first_tile, group = first_group;
        bool dead = false;
        auto wait_tile = [&](int n, int h) {  // (tcgen05.ld wants the whole warp)
            const uint32_t bar = smem_u32(h == H - 1 ? &ctrl->done[0] : &ctrl->half_done[0]) + static_cast<uint32_t>(n & (x_slots - 1)) * 8;
            dead = !__all_sync(0xffffffffu, !dead && mbar_wait_parked(bar, static_cast<uint32_t>(n >> x_shift) & 1u, ws));
            if (!dead) tc_fence_after_sync();
            return !dead;
        };
        auto release_tile = [&]() {  // the MMA warp may have the columns
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(d_empty0 + buf * 8);
        };
        while (i < U) {
            // one tile, or the part of it that lies in this pair's range
            const int pr = proj_of_tile(p, tile);
            const GemmProj& pj = p.proj[pr];
            const int rel = tile - pj.tile0, nt = rel / p.m_tiles * 2 + static_cast<int>(rank), m0 = (rel % p.m_tiles) * tile_m;
            const int row = kSwiglu ? nt * 64 + ((r & 96) >> 1) + (r & 15) : nt * kGemmTileN + r;
            const bool valid = row < pj.n;
            const unsigned short* sp = reinterpret_cast<const unsigned short*>(pj.scales[up_row ? 1 : 0]) +
                                       static_cast<long long>(valid ? row : 0) * p.groups;
            const int seg_begin = group, seg_end = (U - i < p.groups - group) ? group + (U - i) : p.groups;
#pragma unroll
            for (int j = 0; j < static_cast<int>(sizeof(acc) / sizeof(acc[0])); ++j) acc[j] = 0.f;
            // Scales eight groups at a time, a block of eight ahead of its use (one group ahead, their latency is the loop's).
            // One read of tensor memory is in flight while the one before it is added up, and a tile is handed back before its last columns
            // are added: the slowest fold warp of the pair, which shares its scheduler with the MMA warp, is the pace.
            if constexpr (kInTurn) {
                static_assert(gemm_may_fold_in_turn(H, C), "columns");
                const int n0 = i + ((i ^ ch) & 1), g0 = group + (n0 - i);  // this thread's first group
                uint4 q_cur = load_scales(sp, g0 & ~7, p.groups, p.scales_vec), q_next = load_scales(sp, (g0 & ~7) + 8, p.groups, p.scales_vec);
                const uint32_t pick = g0 & 1 ? 0x4432u : 0x4410u;  // its scales lie in the same half of every word
                for (int j = 0; j < (g0 & 7) >> 1; ++j) next_word(q_cur);
                constexpr int kOdd = C == 4 ? 32 : 16, kSteps = C <= 4 ? 2 : 3;  // 32 and 16, 32 and 32, or 32, 16 and 32 columns
                uint32_t d0[32], d1[kOdd];
                auto read = [&](auto step) {
                    constexpr int t = decltype(step)::value, c = t / 2 * 48 + (t & 1) * 32;
                    if constexpr (!(t & 1)) tmem_ld32(d_addr + buf * acc_cols + c, d0);
                    else if constexpr (kOdd == 32) tmem_ld32(d_addr + buf * acc_cols + c, d1);
                    else tmem_ld16(d_addr + buf * acc_cols + c, d1);
                };
                for (int g = g0, n = n0; g < seg_end; g += 2, n += 2) {
                    const float sc = __half2float(__ushort_as_half(static_cast<unsigned short>(prmt(q_cur.x, 0u, pick))));
                    next_word(q_cur);
                    if ((g & 6) == 6) {
                        q_cur = q_next;
                        q_next = load_scales(sp, (g & ~7) + 16, p.groups, p.scales_vec);
                    }
                    if (!wait_tile(n, 0)) break;
                    read(Step<0>());
                    for_steps<kSteps>([&](auto step) {
                        constexpr int t = decltype(step)::value, c = t / 2 * 48 + (t & 1) * 32, width = t & 1 ? kOdd : 32;
                        tmem_wait_ld();
                        if constexpr (t + 1 < kSteps) read(Step<t + 1>());
                        else release_tile();
#pragma unroll
                        for (int j = 0; j < width; j += 2) {
                            if constexpr (t & 1) fma_pair(acc[c + j], acc[c + j + 1], d1[j], d1[j + 1], sc);
                            else fma_pair(acc[c + j], acc[c + j + 1], d0[j], d0[j + 1], sc);
                        }
                    });
                    buf = buf == 0 ? d_bufs - 1 : buf - 1;  // two further
                }
                i += seg_end - group;
                group = seg_end;
            } else {
                uint4 q_cur = load_scales(sp, seg_begin & ~7, p.groups, p.scales_vec), q_next = load_scales(sp, (seg_begin & ~7) + 8, p.groups, p.scales_vec);
                for (int j = 0; j < (seg_begin & 7); ++j) shift_scales(q_cur);
                constexpr int kRead = H == 1 ? 32 : 16, kReads = (kCols + kRead - 1) / kRead, kSteps = H * kReads;
                constexpr bool kAcross = kSteps % 2 == 0;  // (else the two buffers would change places from group to group)
                uint32_t d[2][kRead];
                auto read = [&](auto step) {
                    constexpr int t = decltype(step)::value, c = t % kReads * kRead;
                    // (One tile of fewer columns reads on into columns that are allocated and not used.  Two of 112 do not, the fold being the pace:
                    // 5120 x 14336 at 448 rows 58.0 -> 57.5 us, 5120 x 2048 22.3 -> 22.0.)
                    if constexpr (kRead == 32 && kCols - c >= 32) tmem_ld32(d_addr + buf * acc_cols + c, d[t & 1]);
                    else if constexpr (kCols - c < 16) tmem_ld8(d_addr + buf * acc_cols + c, d[t & 1]);
                    else tmem_ld16(d_addr + buf * acc_cols + c, d[t & 1]);
                };
                if (wait_tile(i, 0)) {
                    read(Step<0>());
                    for (; group < seg_end && !dead; ++group, ++i) {
                        const float sc = __half2float(__ushort_as_half(static_cast<unsigned short>(q_cur.x & 0xFFFFu)));
                        shift_scales(q_cur);
                        if ((group & 7) == 7) {
                            q_cur = q_next;
                            q_next = load_scales(sp, group + 9, p.groups, p.scales_vec);
                        }
                        for_steps<kSteps>([&](auto step) {
                            constexpr int t = decltype(step)::value, h = t / kReads, c = t % kReads * kRead;
                            tmem_wait_ld();
                            if constexpr (t % kReads < kReads - 1) {
                                read(Step<t + 1>());
                            } else {
                                release_tile();
                                buf = buf == d_bufs - 1 ? 0 : buf + 1;
                                if (t < kSteps - 1 || (kAcross && group + 1 < seg_end)) {
                                    if (wait_tile(t < kSteps - 1 ? i : i + 1, (h + 1) % H)) read(Step<(t + 1) % kSteps>());
                                }
                            }
#pragma unroll
                            for (int j = 0; j < kRead && c + j < kCols; j += 2)
                                fma_pair(acc[h * kCols + c + j], acc[h * kCols + c + j + 1], d[t & 1][j], d[t & 1][j + 1], sc);
                            if constexpr (!kAcross && t == kSteps - 1) {
                                if (group + 1 < seg_end && wait_tile(i + 1, 0)) read(Step<0>());
                            }
                        });
                    }
                }
            }
            if (fold_barrier_or(dead || ws->abort_flag != 0)) break;

            if constexpr (kInTurn) {
                // The row's other thread has the other groups' sums: each passes half of its columns on and finishes the other half.  (The
                // barrier above: the trade of the tile before has been read.)
                float4* trade = reinterpret_cast<float4*>(w_ring + w_slots * kWSlotBytes);
#pragma unroll
                for (int j = 0; j < half_cols; j += 4) {
                    const int k = half_cols + j;
                    trade[j / 4 * kGemmFoldThreads + tid] = make_float4(ch ? acc[j] : acc[k], ch ? acc[j + 1] : acc[k + 1], ch ? acc[j + 2] : acc[k + 2],
                                                                        ch ? acc[j + 3] : acc[k + 3]);
                }
                fold_barrier();
#pragma unroll
                for (int j = 0; j < half_cols; j += 4) {
                    const int k = half_cols + j;
                    const float4 t = trade[j / 4 * kGemmFoldThreads + (tid ^ 128)];
                    acc[j] = (ch ? acc[k] : acc[j]) + t.x;
                    acc[j + 1] = (ch ? acc[k + 1] : acc[j + 1]) + t.y;
                    acc[j + 2] = (ch ? acc[k + 2] : acc[j + 2]) + t.z;
                    acc[j + 3] = (ch ? acc[k + 3] : acc[j + 3]) + t.w;
                }
            }

            // ------------------------------------------------------------ a straddling tile: the last CTA to arrive finishes it
            const bool split = seg_begin > 0 || seg_end < p.groups;
            bool last = true;
            if (split) {
                const long long tu = static_cast<long long>(tile) * p.groups;
                int c_first = pair, c_last = pair;
                if (seg_begin > 0)
                    do --c_first;
                    while (unit_begin(p, c_first) > tu);
                if (seg_end < p.groups)
                    do ++c_last;
                    while (unit_begin(p, c_last + 1) < tu + p.groups);
                const size_t slot_floats = static_cast<size_t>(kGemmTileN) * kGemmTileM;
                // (every fold warp exchanges its own rows and columns with the same warp of the others, without the CTA's other warps)
                int* counter = p.counters + (c_first * 2 + static_cast<int>(rank)) * (kGemmFoldThreads / 32) + warp;
                const int n = seg_end - seg_begin;
                // The pair in whose range a tile starts comes to it last of all it does, after an exchange more than the pairs with one part
                // only: the others have mostly arrived or are about to, and then its sums stay in registers.  Writing them, with the fence behind
                // it, takes 3.5 us at 256 rows, and so it does for the others, who may be at it: a wait of less than that is lost where all
                // parts end together.  5120 x 1024 (five equal parts a tile), us without a wait / 3000 / 12000 clocks: 77 rows 12.6 / 13.5 / 12.6,
                // 128 rows 14.8 / 16.0 / 14.8, 256 21.3 / 22.5 / 21.3; 17408 x 5120, 128 rows 30.2 / 29.8 / 29.8, 448 67.1 / 66.4 / 66.2.
                last = false;
                if (seg_begin == 0) {
                    // (the whole warp asks: a loop of one lane's own costs the epilogue registers)
                    const long long t0 = clock64();
                    int have;
                    do have = load_acquire(counter);
                    while (__any_sync(0xffffffffu, have + n != p.groups && clock64() - t0 < kOthersWait));
                    last = __all_sync(0xffffffffu, have + n == p.groups);
                    if (last && lane == 0) *counter = 0;  // as the next launch expects it
                }
                if (!last) {
                    float4* mine = reinterpret_cast<float4*>(p.partials + (static_cast<size_t>(blockIdx.x) * 2 + (seg_begin > 0 ? 0 : 1)) * slot_floats) + tid;
#pragma unroll
                    for (int j = 0; j < H * kCols; j += 4)
                        __stcg(mine + j / 4 * kGemmFoldThreads, make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]));
                    __threadfence();
                    __syncwarp();
                    int have = 0;
                    if (lane == 0) {
                        have = atomicAdd(counter, n);
                        if (have + n == p.groups) *counter = 0;
                    }
                    last = __any_sync(0xffffffffu, lane == 0 && have + n == p.groups);
                }
                if (last) {
                    // The parts are added in pair order, whoever is last: those in front of this pair's own, it, those behind.
                    __threadfence();
                    const float* base = p.partials + static_cast<size_t>(rank) * 2 * slot_floats + tid * 4;
                    auto part = [&](int o) {  // a contributor's part of this tile: slot 1 if the tile starts in its range, else slot 0
                        return reinterpret_cast<const float4*>(base + static_cast<size_t>(o) * 4 * slot_floats + (o == c_first ? slot_floats : 0));
                    };
                    constexpr int kParts = H * kCols / 4, kBatch = 12;
                    if (c_first < pair) {
#pragma unroll
                        for (int c = 0; c < kParts; c += kBatch) {
                            float4 t[kBatch];
#pragma unroll
                            for (int j = 0; j < kBatch; ++j)
                                if (c + j < kParts) t[j] = __ldcg(part(c_first) + (c + j) * kGemmFoldThreads);
#pragma unroll 1
                            for (int o = c_first + 1; o < pair; ++o) {
#pragma unroll
                                for (int j = 0; j < kBatch; ++j)
                                    if (c + j < kParts) {
                                        const float4 u = __ldcg(part(o) + (c + j) * kGemmFoldThreads);
                                        t[j].x += u.x;
                                        t[j].y += u.y;
                                        t[j].z += u.z;
                                        t[j].w += u.w;
                                    }
                            }
#pragma unroll
                            for (int j = 0; j < kBatch; ++j)
                                if (c + j < kParts) add4(acc + (c + j) * 4, t[j]);
                        }
                    }
#pragma unroll 1
                    for (int o = pair + 1; o <= c_last; ++o) {
#pragma unroll
                        for (int c = 0; c < kParts; c += kBatch) {
                            float4 t[kBatch];
#pragma unroll
                            for (int j = 0; j < kBatch; ++j)
                                if (c + j < kParts) t[j] = __ldcg(part(o) + (c + j) * kGemmFoldThreads);
#pragma unroll
                            for (int j = 0; j < kBatch; ++j)
                                if (c + j < kParts) add4(acc + (c + j) * 4, t[j]);
                        }
                    }
                }
            }
            if (last) {
                const float bias = (valid && pj.bias && !kSwiglu) ? pj.bias[row] : 0.f;
#pragma unroll
                for (int c = 0; c < H * ((kCols + 15) / 16); ++c) {
                    constexpr int kBlocks = (kCols + 15) / 16;
                    const int col = c % kBlocks * 16, at = c / kBlocks * kCols + col;  // of its accumulator tile, in `acc`
                    if (col < half_cols) {
                        const int mc = m0 + ch * (tile_m >> 1) + c / kBlocks * half_cols + col;
                        const int rows = p.m - mc < half_cols - col ? p.m - mc : half_cols - col;
                        OutT* out = static_cast<OutT*>(pj.y) + static_cast<long long>(mc) * pj.ldy + row;
                        if (!kSwiglu) {
#pragma unroll
                            for (int b = 0; b < 16; b += 8) {
                                float y[8];
#pragma unroll
                                for (int j = 0; j < 8; ++j) y[j] = at + b + j < H * kCols ? acc[at + b + j] + bias : 0.f;
                                if (b < half_cols - col) store_rows(out, pj.ldy, y, valid ? rows - b : 0, p.pair_stores, lane);
                                out += 8 * pj.ldy;
                            }
                        } else {
                            // Gate and up of one feature sit sixteen lanes apart, which trade halves of the 16 columns: the gate
                            // lane finishes columns 0-7, the up lane 8-15.  (Through shared memory, with two barriers per 16
                            // columns, the trade took 4 us a tile.)
                            float y[8];  // (all of them before the first store: inside its condition each would wait for the last)
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const float a = acc[at + j], b = at + 8 + j < H * kCols ? acc[at + 8 + j] : 0.f;
                                const float theirs = __shfl_xor_sync(0xffffffffu, up_row ? a : b, 16);
                                const float g = up_row ? theirs : a, u = up_row ? b : theirs;
                                // (With the compiler's division, which has a branch, the eight came one after the other: 1500 clocks per 16
                                // columns, 12000 between two tiles of 256 rows.)
                                y[j] = silu(g) * u;
                            }
                            if (up_row) out += 8 * pj.ldy;
                            store_rows(out, pj.ldy, y, valid ? rows - (up_row ? 8 : 0) : 0, p.pair_stores, lane);
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

template <int H, int C, bool kInTurn, typename OutT, bool kSwiglu>
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
            e = cudaFuncGetAttributes(&a, w4a16_gemm_kernel<H, C, kInTurn, OutT, kSwiglu>);
            if (e != cudaSuccess) return e;
            if (a.numRegs * gemm_threads(H, C) < gemm_split_regs(H, C)) return cudaErrorLaunchOutOfResources;
            e = cudaFuncSetAttribute(w4a16_gemm_kernel<H, C, kInTurn, OutT, kSwiglu>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmemBytes);
            if (e != cudaSuccess) return e;
            configured[dev] = true;
        }
    }
    return launch_pdl(w4a16_gemm_kernel<H, C, kInTurn, OutT, kSwiglu>, grid, dim3(gemm_threads(H, C)), kGemmSmemBytes, stream, p);
}

template <typename OutT, bool kSwiglu>
cudaError_t gemm_configure_and_launch(const GemmParams& p, dim3 grid, cudaStream_t stream) {
    const bool in_turn = p.groups > kHalvesGroups;
    switch (p.tile_m) {
        case 48: return in_turn ? gemm_configure_and_launch<1, 3, true, OutT, kSwiglu>(p, grid, stream) : gemm_configure_and_launch<1, 3, false, OutT, kSwiglu>(p, grid, stream);
        case 64: return in_turn ? gemm_configure_and_launch<1, 4, true, OutT, kSwiglu>(p, grid, stream) : gemm_configure_and_launch<1, 4, false, OutT, kSwiglu>(p, grid, stream);
        case 80: return in_turn ? gemm_configure_and_launch<1, 5, true, OutT, kSwiglu>(p, grid, stream) : gemm_configure_and_launch<1, 5, false, OutT, kSwiglu>(p, grid, stream);
        case 96: return gemm_configure_and_launch<1, 6, false, OutT, kSwiglu>(p, grid, stream);
        case 112: return gemm_configure_and_launch<1, 7, false, OutT, kSwiglu>(p, grid, stream);
        case 128: return gemm_configure_and_launch<1, 8, false, OutT, kSwiglu>(p, grid, stream);
        case 144: return gemm_configure_and_launch<1, 9, false, OutT, kSwiglu>(p, grid, stream);
        case 160: return gemm_configure_and_launch<1, 10, false, OutT, kSwiglu>(p, grid, stream);
        case 176: return gemm_configure_and_launch<1, 11, false, OutT, kSwiglu>(p, grid, stream);
        case 192: return gemm_configure_and_launch<1, 12, false, OutT, kSwiglu>(p, grid, stream);
        case 224: return gemm_configure_and_launch<2, 7, false, OutT, kSwiglu>(p, grid, stream);
        case 256: return gemm_configure_and_launch<2, 8, false, OutT, kSwiglu>(p, grid, stream);
        default: return cudaErrorInvalidValue;  // (33 rows and more, in the steps of gemm_launch: none)
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
// exchange of partial sums, about as much as kCutCost groups (with 12, 8 or 4 in its place 14336 x 5120 is cut up to 256 rows and takes
// 35.7 -> 37 to 40 us there, and nothing else gains; of the exchange's 12 us at 512 rows, 4 are writing the part met first, 4 reading
// the others' two, 2 the outputs); a small problem takes fewer pairs (below eight groups each, the pipeline's fill dominates).
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

// The kernel as it was when the routes of 33 to 64 rows were drawn (c_api.cu), not as it is: 5.8 us a tile of a pair (fill, read-out and
// stores) and 0.53 us a group; a cut costs kCutCost groups, or six where it falls on equal parts of every tile.  Then it was within 6 % of
// most of 18 shapes at 33 .. 64 rows; now it is 40 to 46 % too long for the larger ones (gate/up 5120 x 17408 at 33 rows 54 modelled, 37
// measured; 17408 x 5120 34 and 24).
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
    // rows per tile: as few tiles as 256 rows allow, evenly filled, in steps of what the accumulator tiles' halves need
    p.m_tiles = static_cast<int>((m + kGemmTileM - 1) / kGemmTileM);
    const int rows = static_cast<int>((m + p.m_tiles - 1) / p.m_tiles), step = 16 * gemm_halves(rows);
    p.tile_m = (rows + step - 1) / step * step;
    p.groups = static_cast<int>(k / 128);
    long long tiles = 0;
    if (swiglu) {
        if (!encode_gemm_w(&p.w_map[0], proj[0].w, proj[0].n, k, 64) || !encode_gemm_w(&p.w_map[1], proj[1].w, proj[1].n, k, 64)) return -2;
        p.proj[0].scales[1] = static_cast<const __half*>(proj[1].scales);
    }
    p.num_proj = swiglu ? 1 : num;
    p.pair_stores = out_f32 ? 0 : 1;
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
        if ((reinterpret_cast<uintptr_t>(a.y) & 3) || (p.proj[i].ldy & 1) || (a.n & 1)) p.pair_stores = 0;
        p.proj[i].tile0 = static_cast<int>(tiles);
        const int rows = swiglu ? kGemmTileN : 2 * kGemmTileN;  // of a pair
        tiles += (a.n + rows - 1) / rows * p.m_tiles;
    }
    const GemmDeal deal = gemm_deal(proj, num, swiglu, m, k, num_sms, partials != nullptr);
    if (deal.tiles > (1 << 30)) return -2;
    if (!encode_gemm_x(&p.x_map, static_cast<const __half*>(x), m, k, p.tile_m)) return -2;
    p.m = static_cast<int>(m);
    p.units = deal.units;
    p.wait_limit = wait_limit;
    p.x_stage_limit = x_stage_limit;
    p.status = status;
    p.partials = partials;
    p.counters = counters;
    p.pairs = static_cast<int>(deal.pairs);
    const long long dealt = deal.whole_tiles ? deal.tiles : deal.units;
    p.deal_quot = dealt / deal.pairs;
    p.deal_rem = static_cast<int>(dealt % deal.pairs);
    p.deal_size = deal.whole_tiles ? p.groups : 1;
    const dim3 grid(static_cast<unsigned>(2 * deal.pairs));
    if (swiglu && out_f32) return -2;  // (fp16 activations give fp16 results there)
    const cudaError_t e = swiglu    ? gemm_configure_and_launch<__half, true>(p, grid, stream)
                          : out_f32 ? gemm_configure_and_launch<float, false>(p, grid, stream)
                                    : gemm_configure_and_launch<__half, false>(p, grid, stream);
    return e == cudaSuccess ? 0 : -1;
}

}  // namespace xb
