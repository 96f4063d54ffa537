// W4A16 linear with fp32 activations (the reference's "reference and oracle testing" overloads, src/ops/linear.h:30-139) on the
// tensor cores without losing a bit of them: an fp32 value is the exact sum of three bf16 values (24 bits of significand, 8 each,
// by truncation; bf16 has fp32's exponent range), the int4 weights are exact in bf16, and each 128-k group accumulates in fp32
// before acc += dot * scale, the reference's association (src/ops/linear.cpp:239-287).
//
// A warp takes units of (32 weight rows, one 128-k group, 8 activation rows): mma.sync m16n8k16, the weights as A and the three
// parts of x as three B operands.  The contraction index may be taken in any order, so a thread's A fragments are the sixteen
// bytes it loads from its rows and its B fragments the 128 bytes it loads from its activation row: nothing goes through shared
// memory but the sums.  K is cut over the warps of a CTA and over the CTAs of a cluster, which adds up in rank order
// (deterministic) through distributed shared memory.  mma.sync, not tcgen05: at these sizes the work is a few hundred
// instructions per warp, and the time is the latency of one launch and two round trips to memory.
//
// 8 x 5120 x 1024: 5.7 us, where one warp per two weight rows on the CUDA cores took 28 (a serial chain of 5120 fused
// multiply-adds over conversions per row and lane).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx_sm100.cuh"
#include "silu.cuh"
#include "w4a16.h"

namespace xb {
namespace {

constexpr int kF32Warps = 8, kF32Threads = kF32Warps * 32, kF32Rows = 32, kF32Cols = 8, kF32MaxProj = 4, kF32MaxCluster = 8;
constexpr int kF32Pitch = kF32Cols + 1;

struct F32Proj {
    float* y;
    const uint8_t* w;
    const unsigned short* scales;
    const float* bias;
    long long n, ldy, tile0;
};
struct F32Params {
    F32Proj proj[kF32MaxProj];  // gate/up: 0 = gate, 1 = up; a tile is 16 rows of each
    int num, swiglu, cluster, groups;
    long long m, k;
    const float* x;
};

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// nibbles i and i + 4 of a word as bf16: (128 + (q + 8)) - 136, where the sign bit's flip adds the 8
__device__ __forceinline__ uint32_t unpack_pair(uint32_t w, int i) {
    const uint32_t v = lop3_6a(w >> (4 * i), 0x000F000Fu, 0x43084308u);
    uint32_t d;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(v), "r"(0x3F803F80u), "r"(0xC308C308u));
    return d;
}
// (a, b) as three pairs of bf16, by truncation: exact (of an infinity the second part is NaN; see plain_dot)
__device__ __forceinline__ void split_bf16(float a, float b, uint32_t (&p)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        p[i] = prmt(__float_as_uint(a), __float_as_uint(b), 0x7632u);
        if (i < 2) {
            a -= __uint_as_float(__float_as_uint(a) & 0xFFFF0000u);
            b -= __uint_as_float(__float_as_uint(b) & 0xFFFF0000u);
        }
    }
}

// One output without the split.  Taken for sums that came out as NaN: an infinite activation has parts inf, NaN, NaN, where its
// products are infinities unless the weight is zero.  (A select in the split that keeps the second part zero costs 0.5 of the 4.3 us
// of a 1 x 5120 x 1024 call, this 0.1.)
__device__ __noinline__ float plain_dot(const float* x, const uint8_t* w, const unsigned short* scales, int groups) {
    float acc = 0.f;
    for (int gr = 0; gr < groups; ++gr) {
        float dot = 0.f;
        for (int i = 0; i < 64; ++i) {
            const int b = w[gr * 64LL + i];
            dot = fmaf(x[gr * 128LL + 2 * i], static_cast<float>(((b & 15) ^ 8) - 8), dot);
            dot = fmaf(x[gr * 128LL + 2 * i + 1], static_cast<float>(((b >> 4) ^ 8) - 8), dot);
        }
        acc = fmaf(dot, __half2float(__ushort_as_half(scales[gr])), acc);
    }
    return acc;
}

__global__ void __launch_bounds__(kF32Threads, 2) w4a16_f32_kernel(const __grid_constant__ F32Params p) {
    __shared__ float red[kF32Warps][kF32Rows][kF32Pitch];
    __shared__ float parts[kF32MaxCluster][kF32Threads];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int rank = static_cast<int>(cluster_ctarank());
    const long long tile = blockIdx.x / p.cluster, m0 = static_cast<long long>(blockIdx.y) * kF32Cols;
    griddep_launch_dependents();

    int pi = 0;
    if (!p.swiglu)
        while (pi + 1 < p.num && tile >= p.proj[pi + 1].tile0) ++pi;
    const long long base = (tile - p.proj[pi].tile0) * (p.swiglu ? 16 : kF32Rows);
    // rows g and g + 8 of the tile's two halves (past the end: the last row, whose sums nobody writes)
    const uint8_t* w_row[4];
    const unsigned short* s_row[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const F32Proj& pj = p.proj[p.swiglu ? i >> 1 : pi];
        long long row = base + (p.swiglu ? 0 : (i >> 1) * 16) + (i & 1) * 8 + g;
        if (row >= pj.n) row = pj.n - 1;
        w_row[i] = pj.w + row * (p.k / 2) + t * 16;
        s_row[i] = pj.scales + row * p.groups;
    }
    const bool live = m0 + g < p.m;
    const float* x_row = p.x + (live ? m0 + g : 0) * p.k + t * 32;

    float acc[2][4] = {};
    uint4 w[4];
    float4 x[8];
    unsigned short sc[4];
    const int step = kF32Warps * p.cluster;
    auto load_w = [&](int gr) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w[i] = __ldg(reinterpret_cast<const uint4*>(w_row[i] + gr * 64));
            sc[i] = __ldg(s_row[i] + gr);
        }
    };
    auto load_x = [&](int gr) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            x[i] = live ? *reinterpret_cast<const float4*>(x_row + static_cast<long long>(gr) * 128 + i * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    int gr = rank * kF32Warps + warp;
    if (gr < p.groups) load_w(gr);  // (the weights do not come from the launch in front of this one)
    griddep_wait();
    for (; gr < p.groups; gr += step) {
        load_x(gr);
        uint32_t words[4][4];
        float scale[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            words[i][0] = w[i].x; words[i][1] = w[i].y; words[i][2] = w[i].z; words[i][3] = w[i].w;
            scale[i] = __half2float(__ushort_as_half(sc[i]));
        }
        if (gr + step < p.groups) load_w(gr + step);
        // The leading part's products in two sums, and the other two's.  The tensor core's additions truncate: in one sum, activations
        // whose magnitudes spread over e^3 came out 1.6 times as far from 64 bits as a chain of fused multiply-adds, now 1.1 times
        // (like magnitudes: 0.65 times).  A sum for every MMA: 0.8 times, but 6.0 us instead of 5.7 at 8 x 5120 x 1024.
        float d[2][3][4] = {};
#pragma unroll
        for (int j = 0; j < 8; ++j) {  // 16 k: nibbles i, i + 4 and i + 1, i + 5 of word j / 2
            const int c = j >> 1, i = 2 * (j & 1);
            uint32_t b0[3], b1[3];
            const float4 lo = x[2 * c], hi = x[2 * c + 1];
            split_bf16(i ? lo.z : lo.x, i ? hi.z : hi.x, b0);
            split_bf16(i ? lo.w : lo.y, i ? hi.w : hi.y, b1);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t a[4] = {unpack_pair(words[2 * h][c], i), unpack_pair(words[2 * h + 1][c], i), unpack_pair(words[2 * h][c], i + 1),
                                       unpack_pair(words[2 * h + 1][c], i + 1)};
#pragma unroll
                for (int q = 0; q < 3; ++q) mma_bf16(d[h][q > 0 ? 2 : j & 1], a, b0[q], b1[q]);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[h][e] = fmaf(d[h][2][e] + (d[h][1][e] + d[h][0][e]), scale[2 * h + (e >> 1)], acc[h][e]);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int e = 0; e < 4; ++e) red[warp][h * 16 + (e >> 1) * 8 + g][2 * t + (e & 1)] = acc[h][e];
    }
    __syncthreads();
    const int row = tid & 31, col = tid >> 5;
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kF32Warps; ++i) sum += red[i][row][col];
    if (p.cluster > 1) {
        cluster_sync_all();  // (rank 0 has started)
        st_shared_cluster_f32(mapa_shared_cluster(smem_u32(&parts[rank][tid]), 0), sum);
        cluster_sync_all();
        if (rank > 0) return;
        sum = 0.f;
        for (int r = 0; r < p.cluster; ++r) sum += parts[r][tid];
    }
    if (sum != sum && m0 + col < p.m) {
        const F32Proj& pj = p.proj[p.swiglu ? row >> 4 : pi];
        const long long r = base + (p.swiglu ? row & 15 : row);
        if (r < pj.n) sum = plain_dot(p.x + (m0 + col) * p.k, pj.w + r * (p.k / 2), pj.scales + r * p.groups, p.groups);
    }
    if (p.swiglu) {
        parts[0][tid] = sum;  // (this thread's own slot; the others' sums of it are in)
        __syncthreads();
        if (row >= 16) return;
        sum = silu(sum) * parts[0][tid + 16];
    }
    const F32Proj& pj = p.proj[pi];
    if (base + row < pj.n && m0 + col < p.m) {
        if (pj.bias && !p.swiglu) sum += pj.bias[base + row];
        pj.y[(m0 + col) * pj.ldy + base + row] = sum;
    }
}

}  // namespace

bool f32_eligible(const void* x, const TcProj* proj, int num, bool swiglu, long long m, long long k, int group_size) {
    const int cnt = swiglu ? 2 : num;
    if (group_size != 128 || k < 128 || k % 128 != 0 || k > (1ll << 30) || cnt < 1 || cnt > kF32MaxProj) return false;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (m + kF32Cols - 1) / kF32Cols > 65535) return false;
    for (int i = 0; i < cnt; ++i)
        if (reinterpret_cast<uintptr_t>(proj[i].w) & 15) return false;
    return true;
}

int f32_launch(cudaStream_t stream, const void* x, const TcProj* proj, int num, bool swiglu, long long m, long long k, int num_sms) {
    F32Params p{};
    p.num = swiglu ? 2 : num;
    p.swiglu = swiglu ? 1 : 0;
    p.m = m;
    p.k = k;
    p.groups = static_cast<int>(k / 128);
    p.x = static_cast<const float*>(x);
    long long tiles = 0;
    for (int i = 0; i < p.num; ++i) {
        const TcProj& a = proj[i];
        p.proj[i] = F32Proj{static_cast<float*>(a.y), a.w, static_cast<const unsigned short*>(a.scales), a.bias, a.n, a.ldy > 0 ? a.ldy : a.n, tiles};
        if (swiglu) {
            if (i == 0) tiles = (a.n + 15) / 16;
            else p.proj[i].tile0 = 0;
        } else {
            tiles += (a.n + kF32Rows - 1) / kF32Rows;
        }
    }
    const long long cols = (m + kF32Cols - 1) / kF32Cols;
    // Two CTAs fit an SM.  Few tiles are cut over K, as long as every warp gets a group.
    long long cluster = 2LL * num_sms / (tiles * cols);
    if (cluster > (p.groups + kF32Warps - 1) / kF32Warps) cluster = (p.groups + kF32Warps - 1) / kF32Warps;
    cluster = cluster < 1 ? 1 : (cluster < kF32MaxCluster ? cluster : kF32MaxCluster);
    p.cluster = static_cast<int>(cluster);
    if (tiles * cluster > 0x7FFFFFFF) return -2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles * cluster), static_cast<unsigned>(cols));
    cfg.blockDim = dim3(kF32Threads);
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = static_cast<unsigned>(cluster);
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, w4a16_f32_kernel, p) == cudaSuccess ? 0 : -1;
}

}  // namespace xb
