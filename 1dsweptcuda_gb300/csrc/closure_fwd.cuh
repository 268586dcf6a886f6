// Forward pass of the KS closure network, and the coarse KS step fused with it.
//
// A tile is 128 consecutive rows of layer 2 of one domain, a row per thread:
//   us[j] = u[x0 - 6 + j],        j < 136
//   a1[r] : position x0 - 4 + r,  r < 132
//   z2[p] : position x0 - 2 + p,  p < 128  (needs a1[p .. p+4])
//   out q : position x0 + q       (needs z2[q .. q+4])
// so 124 of its rows are outputs, or all 128 where the domain has 128 cells: its
// rows then wrap onto themselves.
//
// Layer 2 (128 x 32 outputs, K = 5 taps x 32 channels) is ten tcgen05.mma of
// 128 x 32 x 16, issued by one thread, FP32 sums in TMEM.  Both operands lie in
// shared memory without swizzle as planes of 8 channels, 16 bytes per row, so the
// rows shifted by a tap are the same planes 16 bytes on: the im2col is a start
// address.  Layer 1 writes a plane per warp (consecutive lanes 16 bytes apart);
// the epilogue reads a row of 32 sums per thread, so its tap sums need no
// shuffles.  The arithmetic runs on channel pairs (f32x2).
//
// What bounds it: shared memory and latency.  A cell takes 64 tanh (16 per clock
// and SM) and the MMAs read each row of a1 ten times, but with one tile at a time
// most of shared memory's cycles went into the epilogue's weights, 32 lanes x 16
// bytes a read although all lanes read the same.  So a block takes NT = 2 tiles
// at a time where there are enough (the rule is at the launch), each weight read
// serving both.  At 1024 domains of 1024 cells a step takes 102.5 us with
// mma.sync, 54 us with one tile, 48.5 us with two (FP32 pipe 41 % busy, SFU 32 %,
// tensor core 32 %, issue slots 49 %, shared memory 54 %); 4, 6 blocks per SM instead of 5:
// 49.1, 49.9 us.  Blocks take their tiles in a stride of the grid, so weights and
// TMEM are set up once per block, before the wait for the launch before it, and
// the next tiles' inputs are fetched behind the work.
//
// The GELUs are kept doubled, 2 gelu(x) = x + x tanh(...), and the next layer's
// weights halved: powers of two, exact in BF16 and FP32.
#pragma once

#include <cuda_bf16.h>

#include "engine.cuh"

namespace sw {
namespace cl {

constexpr int FWD_THREADS = 128, FWD_BLOCKS = 5;  // blocks per SM
constexpr int FWD_OUT = 124;                      // outputs per tile of a domain of more than 128 cells
constexpr int FWD_PLANE = 136 * 16;               // bytes of one a1 plane (132 rows used)

// The parameters in the layout of shared memory (k_pack_weights), halved as above.
struct alignas(16) FwdWeights {
    __nv_bfloat16 w2[KW][4][CH][8];  // [t][plane of input channels][o][i % 8]
    float2 w1[CH / 2][KW + 1];       // channel pairs: taps 0..4, bias
    float2 w3[CH / 2][KW + 1];       // channel pairs: layer 2's bias, taps 0..4
    float b3, scale, pad[2];
};
static_assert(sizeof(FwdWeights) % 16 == 0, "copied in 16-byte words");

template <int NT>
struct alignas(128) FwdSmem {
    FwdWeights w;
    unsigned char a1[NT][4 * FWD_PLANE];
    float us[NT][136];
    float pred[NT][128];    // KS predictor on x0-2 .. x0+125
    float p3[NT][KW][128];  // p3[t][r] = sum_i w3[i][t] gelu(z2[r][i])
    uint64_t bar;
    uint32_t tmem;
};

__global__ void k_pack_weights(const float *__restrict__ theta, FwdWeights *__restrict__ w) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < CH * CH * KW) {  // theta's w2 is [o][i][t]
        const int o = k / (CH * KW), i = (k / KW) % CH, t = k % KW;
        w->w2[t][i >> 3][o][i & 7] = __float2bfloat16_rn(0.5f * bf16r(theta[OW2 + k]));
    }
    if (k < CH) {
        float *w1 = &w->w1[k >> 1][0].x + (k & 1), *w3 = &w->w3[k >> 1][0].x + (k & 1);
        for (int t = 0; t < KW; ++t) {
            w1[2 * t] = bf16r(theta[OW1 + k * KW + t]);
            w3[2 * (t + 1)] = 0.5f * bf16r(theta[OW3 + k * KW + t]);
        }
        w1[2 * KW] = theta[OB1 + k];
        w3[0] = theta[OB2 + k];
    }
    if (k == 0) {
        w->b3 = theta[OB3];
        w->scale = theta[OSCALE];
        w->pad[0] = w->pad[1] = 0.0f;
    }
}

// Twice the GELU of both components: x + x tanh(x (c + c a x^2)).
__device__ __forceinline__ float2 gelu2_doubled(float2 x) {
    const float2 inner = __ffma2_rn(f2(kGeluC * kGeluA), __fmul2_rn(x, x), f2(kGeluC));
    const float2 arg = __fmul2_rn(x, inner);
    return __ffma2_rn(x, make_float2(tanh_sfu(arg.x), tanh_sfu(arg.y)), x);
}

// ---- tcgen05
// Operand descriptor: K-major without swizzle, 8-row groups 128 bytes apart, planes `plane` bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t plane) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(plane >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) |
           ((uint64_t)1 << 46);
}
// FP32 sums, BF16 operands, both K-major, M = 128, N = 32.
constexpr uint32_t kUmmaIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(CH >> 3) << 17) | ((128u >> 4) << 24);
__device__ __forceinline__ void umma(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(kUmmaIdesc), "r"(accumulate)
        : "memory");
}
// 16 consecutive columns of the thread's row.
__device__ __forceinline__ void tmem_load16(float (&v)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
          "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tcgen05_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Wait for the phase of the given parity, bounded like bulk_wait.
__device__ __forceinline__ bool umma_wait(uint64_t *bar, unsigned parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (uint64_t polls = 0; !mbar_try_wait(bar, parity); ++polls)
        if (global_ns() - t0 > kBulkWaitNs || polls > kBulkWaitNs / 16) return false;
    return true;
}

// STEP: out = classic KS step(u) + scale net(u); else out = scale net(u).  Domains of n cells, tiles_per_dom tiles
// of n_out outputs each (the last of a domain fewer); a block takes NT tiles at a time.  A wait that runs out sets
// *status (pinned host memory).
template <bool STEP, int NT>
__global__ void __launch_bounds__(FWD_THREADS, FWD_BLOCKS)
    k_forward(const FwdWeights *__restrict__ weights, const Params<float> pk, const float *u, float *out,
              const int64_t n, const uint32_t tiles_per_dom, const uint32_t n_tiles, const int n_out, int *status) {
    __shared__ FwdSmem<NT> s;
    constexpr uint32_t TMEM_COLS = 32 * NT;  // the blocks that fit an SM's shared memory use at most 384 of its 512
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(weights);
        uint4 *dst = reinterpret_cast<uint4 *>(&s.w);
        for (int k = tid; k < (int)(sizeof(FwdWeights) / 16); k += FWD_THREADS) dst[k] = src[k];
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s.tmem)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) mbar_init(&s.bar, 1);
    tcgen05_before_sync();
    __syncthreads();
    tcgen05_after_sync();
    const uint32_t tmem = s.tmem;
    wait_for_previous_launch();

    // the next tiles' inputs (positions x0 - 6 + tid and, for 8 threads, x0 + 122 + tid; n >= 128), and their
    // place: row[h] the domain's first cell, at[h] this thread's output in the domain
    float next[NT], next_hi[NT];
    int64_t row[NT], at[NT], next_row[NT], next_at[NT];
    auto fetch = [&](uint32_t first) {
#pragma unroll
        for (int h = 0; h < NT; ++h) {
            const uint32_t tile = min(first + h, n_tiles - 1);  // past the last: its inputs again, its outputs dropped
            const uint32_t dom = tile / tiles_per_dom;
            next_row[h] = (int64_t)dom * n;
            next_at[h] = (int64_t)(tile - dom * tiles_per_dom) * n_out + tid;
            int64_t x = next_at[h] - 6;
            x += x < 0 ? n : 0;
            x -= x >= n ? n : 0;
            next[h] = u[next_row[h] + x];
            if (tid < 8) {
                x = next_at[h] + 122;
                x -= x >= n ? n : 0;
                next_hi[h] = u[next_row[h] + x];
            }
            if (first + h >= n_tiles) next_at[h] = n;
        }
    };
    const uint32_t stride = gridDim.x * NT;
    if (blockIdx.x * NT < n_tiles) fetch(blockIdx.x * NT);
    unsigned parity = 0;
    for (uint32_t first = blockIdx.x * NT; first < n_tiles; first += stride) {
#pragma unroll
        for (int h = 0; h < NT; ++h) {
            s.us[h][tid] = next[h];
            if (tid < 8) s.us[h][128 + tid] = next_hi[h];
            row[h] = next_row[h];
            at[h] = next_at[h];
        }
        __syncthreads();
        if (n_tiles - first > stride) fetch(first + stride);  // arrives behind this tile's work
        // layer 1: a warp takes 8 channels (one plane) of all rows
        {
            float2 w[4][KW + 1];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float4 *p = reinterpret_cast<const float4 *>(s.w.w1[warp * 4 + c]);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float4 v = p[k];
                    w[c][2 * k] = make_float2(v.x, v.y);
                    w[c][2 * k + 1] = make_float2(v.z, v.w);
                }
            }
#pragma unroll 1
            for (int k = 0; k < 4 * NT; ++k) {
                const int h = k >> 2, r = (k & 3) * 32 + lane;
                float2 x[KW];
#pragma unroll
                for (int t = 0; t < KW; ++t) x[t] = f2(s.us[h][r + t]);
                __nv_bfloat162 a[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float2 z = w[c][KW];
#pragma unroll
                    for (int t = 0; t < KW; ++t) z = __ffma2_rn(w[c][t], x[t], z);
                    a[c] = __float22bfloat162_rn(gelu2_doubled(z));
                }
                *reinterpret_cast<uint4 *>(s.a1[h] + warp * FWD_PLANE + r * 16) = *reinterpret_cast<const uint4 *>(a);
            }
            if (lane < 16 * NT) {  // rows 128 .. 131, a channel pair per lane
                const int h = lane >> 4, r = 128 + ((lane >> 2) & 3), c = lane & 3;
                const float2 *wc = s.w.w1[warp * 4 + c];
                float2 z = wc[KW];
#pragma unroll
                for (int t = 0; t < KW; ++t) z = __ffma2_rn(wc[t], f2(s.us[h][r + t]), z);
                *reinterpret_cast<__nv_bfloat162 *>(s.a1[h] + warp * FWD_PLANE + r * 16 + c * 4) =
                    __float22bfloat162_rn(gelu2_doubled(z));
            }
        }
        if constexpr (STEP) {
#pragma unroll
            for (int h = 0; h < NT; ++h) {
                const float *c = &s.us[h][tid + 4];
                s.pred[h][tid] = ks_predict(pk, c[-2], c[-1], c[0], c[1], c[2]);
            }
        }
        fence_smem_for_bulk();  // a1 and the weights are read by the tensor core's copy path
        tcgen05_before_sync();
        __syncthreads();
        if (tid == 0) {
            tcgen05_after_sync();
#pragma unroll
            for (int h = 0; h < NT; ++h) {
                const uint64_t da = umma_desc(smem_addr(s.a1[h]), FWD_PLANE), db = umma_desc(smem_addr(s.w.w2), CH * 16);
#pragma unroll
                for (int k = 0; k < 2 * KW; ++k) {  // tap k / 2, input channels 16 (k % 2) on: offsets in 16 bytes
                    const int t = k >> 1, c = k & 1;
                    umma(tmem + 32 * h, da + t + c * (2 * FWD_PLANE / 16), db + t * (4 * CH) + c * (2 * CH), k > 0);
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(&s.bar))
                         : "memory");
        }
        __syncwarp();
        float v[NT];
#pragma unroll
        for (int h = 0; h < NT; ++h) {
            v[h] = 0.0f;
            if constexpr (STEP) {  // a domain of 128 cells wraps onto its own predictors
                const float *p = s.pred[h];
                v[h] = ks_correct(pk, s.us[h][tid + 6], p[tid], p[(tid + 1) & 127], p[(tid + 2) & 127], p[(tid + 3) & 127],
                                  p[(tid + 4) & 127]);
            }
        }
        const bool done = __all_sync(0xffffffffu, umma_wait(&s.bar, parity));
        if (done) {
            tcgen05_after_sync();
            float2 sum[NT][KW];
#pragma unroll
            for (int h = 0; h < NT; ++h)
#pragma unroll
                for (int t = 0; t < KW; ++t) sum[h][t] = f2(0.0f);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float z[NT][16];
#pragma unroll
                for (int h = 0; h < NT; ++h) tmem_load16(z[h], tmem + ((uint32_t)warp << 21) + 32 * h + 16 * half);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 *p = reinterpret_cast<const float4 *>(s.w.w3[half * 8 + c]);
                    const float4 p0 = p[0], p1 = p[1], p2 = p[2];
#pragma unroll
                    for (int h = 0; h < NT; ++h) {
                        const float2 g =
                            gelu2_doubled(__fadd2_rn(make_float2(z[h][2 * c], z[h][2 * c + 1]), make_float2(p0.x, p0.y)));
                        sum[h][0] = __ffma2_rn(make_float2(p0.z, p0.w), g, sum[h][0]);
                        sum[h][1] = __ffma2_rn(make_float2(p1.x, p1.y), g, sum[h][1]);
                        sum[h][2] = __ffma2_rn(make_float2(p1.z, p1.w), g, sum[h][2]);
                        sum[h][3] = __ffma2_rn(make_float2(p2.x, p2.y), g, sum[h][3]);
                        sum[h][4] = __ffma2_rn(make_float2(p2.z, p2.w), g, sum[h][4]);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < NT; ++h)
#pragma unroll
                for (int t = 0; t < KW; ++t) s.p3[h][t][tid] = sum[h][t].x + sum[h][t].y;
        }
        if (__syncthreads_or(!done)) {
            if (tid == 0) *(volatile int *)status = 1;
            umma_wait(&s.bar, parity);  // once more, bounded: the MMAs write this block's TMEM
            break;
        }
        parity ^= 1;
#pragma unroll
        for (int h = 0; h < NT; ++h) {
            if (tid < n_out && at[h] < n) {
                float d = 0.0f;
#pragma unroll
                for (int t = 0; t < KW; ++t) d += s.p3[h][t][(tid + t) & 127];
                d = s.w.scale * (d + s.w.b3);
                out[row[h] + at[h]] = STEP ? v[h] + d : d;
            }
        }
    }
    tcgen05_before_sync();
    __syncthreads();
    if (warp == 0) {
        tcgen05_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

// The plain coarse KS step: four cells per thread, a warp per 128 cells, each thread forming the eight predictors its
// cells need from 12 values (neighbouring lanes share them through L1): no barriers, no shared memory.
constexpr int PLAIN_THREADS = 256;
__global__ void __launch_bounds__(PLAIN_THREADS)
    k_plain_step(const Params<float> pk, const float *u, float *out, const int64_t n, const uint32_t warps_per_dom,
                 const uint32_t n_warps) {
    wait_for_previous_launch();
    const uint32_t wid = blockIdx.x * (PLAIN_THREADS / 32) + (threadIdx.x >> 5);
    if (wid >= n_warps) return;
    const uint32_t dom = wid / warps_per_dom;
    const int64_t x = (int64_t)(wid - dom * warps_per_dom) * 128 + 4 * (threadIdx.x & 31);
    const float *ud = u + (int64_t)dom * n;
    const int64_t xs[3] = {x == 0 ? n - 4 : x - 4, x, x + 4 == n ? 0 : x + 4};
    float v[12], pr[8];
#pragma unroll
    for (int i = 0; i < 12; ++i) v[i] = ud[xs[i >> 2] + (i & 3)];
#pragma unroll
    for (int i = 0; i < 8; ++i) pr[i] = ks_predict(pk, v[i], v[i + 1], v[i + 2], v[i + 3], v[i + 4]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        out[(int64_t)dom * n + x + i] = ks_correct(pk, v[i + 4], pr[i], pr[i + 1], pr[i + 2], pr[i + 3], pr[i + 4]);
}

}  // namespace cl
}  // namespace sw
