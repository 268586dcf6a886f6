// KS closure network: a 3-layer 1D convolution (1 -> 32 -> 32 -> 1 channels,
// kernel 5, GELU, circular padding per domain) that corrects a coarse KS step.
// Parameters are FP32 masters rounded to BF16 for the forward pass.  The
// 32 -> 32 layer -- 94 % of the work -- runs on the tensor cores
// (tcgen05.mma in the forward pass, mma.sync.m16n8k16 in the backward pass; BF16
// operands, FP32 accumulation); the 1 -> 32 and 32 -> 1 layers run in FP32 on the
// CUDA cores with the BF16-rounded weights.  oracle/closure.py restates the same arithmetic.
//
// The forward pass alone (inference, the coarse step) is closure_fwd.cuh; this
// file has the backward pass, training and the certified adaptive run.
//
// Tiles of the backward pass: a block takes TOUT = 128 consecutive outputs of one domain.  In
// tile coordinates (x0 = first output):
//   us[j] = u[x0 - 6 + j],        j < 152
//   a1[r] : position x0 - 4 + r,  r < 148  (z1 = w1 * us[r .. r+4] + b1)
//   z2[p] : position x0 - 2 + p,  p < 144  (needs a1[p .. p+4]; p < 132 used)
//   d[q]  : position x0 + q,      q < 128  (needs a2[q .. q+4])
// The im2col of layer 2 is free: the A fragment of tap t is the a1 rows
// shifted by t.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <vector>

#include "ctx.h"
#include "launch.cuh"
#include "stencils.cuh"
#include "sw_internal.h"

namespace sw {
namespace cl {

constexpr int CH = 32, KW = 5;
static_assert(CH == 32, "layer 1 maps one warp lane to each channel");
constexpr int TOUT = 128;
constexpr int NU = TOUT + 24;   // 152 input cells
constexpr int NA1 = TOUT + 20;  // 148 a1 rows
constexpr int NZ2 = 144;        // 9 m-tiles of 16 rows
constexpr int NA2 = TOUT + 4;   // 132 a2 rows used
constexpr int LDB = 40;         // bf16 row stride (80 B: conflict-free fragment reads)
constexpr int LDF = 33;         // fp32 row stride
constexpr int THREADS = 256;
// parameter offsets (flat FP32 vector); the last value is the output scale s
// (delta = s * net(u)), fixed by the caller and left alone by training
constexpr int OW1 = 0, OB1 = 160, OW2 = 192, OB2 = 5312, OW3 = 5344, OB3 = 5504, OSCALE = 5505;
constexpr int NTRAIN = 5505, NPARAM = 5506;

// GELU in its tanh form (Hendrycks & Gimpel, "Gaussian Error Linear Units",
// 2016): gelu(x) = x/2 (1 + tanh(c (x + a x^3))), c = sqrt(2/pi), a = 0.044715,
// with tanh from the SFU's tanh.approx.f32 (relative error below 2^-10.7):
// a handful of instructions where the erf form took a long polynomial, and
// the step is bound by instruction issue.  oracle/closure.py restates the same
// function (with an exact tanh).
constexpr float kGeluC = 0.79788456080286536f, kGeluA = 0.044715f;
__device__ __forceinline__ float tanh_sfu(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float gelu(float x) {  // x/2 + (x/2) t
    const float t = tanh_sfu((kGeluC * x) * fmaf(kGeluA, x * x, 1.0f));
    const float hx = 0.5f * x;
    return fmaf(hx, t, hx);
}
__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float gelu_grad(float x) {
    const float x2 = x * x;
    const float t = tanh_sfu(kGeluC * x * fmaf(kGeluA, x2, 1.0f));
    return fmaf(0.5f * x * (1.0f - t * t), kGeluC * fmaf(3.0f * kGeluA, x2, 1.0f), 0.5f * (1.0f + t));
}
__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
}  // namespace cl
}  // namespace sw

#include "closure_fwd.cuh"

namespace sw {
namespace cl {

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// D = A * B + D, m16n8k16, A row-major BF16, B column-major BF16, FP32 accumulate
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Four (two) 8 x 8 BF16 matrices into fragments, lane l giving the address of row l % 8 of matrix l / 8; T: transposed.
template <bool T>
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const __nv_bfloat16 *row) {
    if constexpr (T)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(smem_addr(row))
                     : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(smem_addr(row))
                     : "memory");
}
__device__ __forceinline__ void ldm2_t(uint32_t (&r)[2], const __nv_bfloat16 *row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1])
                 : "r"(smem_addr(row))
                 : "memory");
}

// Shared memory of a tile.
constexpr int LDT = NZ2 + 8;  // dzT's row stride: 304 bytes, conflict-free fragment reads
struct Smem {
    alignas(16) __nv_bfloat16 a1[NA1 * LDB];     // layer-1 activations (an MMA operand)
    alignas(16) __nv_bfloat16 w2[KW * CH * LDB]; // w2[t][o][i], i contiguous (an MMA operand)
    alignas(16) __nv_bfloat16 dzT[CH * LDT];     // dz2 as [o][p], p contiguous, for dW2
    alignas(16) __nv_bfloat16 dzP[LDT * LDB];    // dz2 as [4 + p][o], 4 zero rows in front, for da1
    alignas(16) float w3[KW * CH];               // [t][i]
    float w1[CH * KW], b1[CH], b2[CH];
    float us[NU + 8];                            // the last 8 pad the last warp's window
    float dd[4 + LDT + 8];                       // dL/ddelta of output q at 4 + q, zeros around it
    float part[2][TOUT];                         // layer 3: the two channel halves' sums
    float a2[NA2 * LDF];                         // layer-2 activations gelu(z2)
    float z2[NA2 * LDF];                         // layer-2 pre-activations
    float z1[NA1 * LDF];                         // layer-1 pre-activations, then dz1
};

// The tile's inputs (periodic within the domain).
__device__ void load_tile(Smem &s, const float *__restrict__ u, int64_t n, int64_t x0) {
    for (int j = threadIdx.x; j < NU; j += blockDim.x) {
        int64_t q = x0 - 6 + j;
        q %= n;
        if (q < 0) q += n;
        s.us[j] = u[q];
    }
}
__device__ void load_weights(Smem &s, const float *__restrict__ theta) {
    for (int k = threadIdx.x; k < CH * KW; k += blockDim.x) {
        s.w1[k] = bf16r(theta[OW1 + k]);
        s.w3[(k % KW) * CH + k / KW] = bf16r(theta[OW3 + k]);
    }
    for (int i = threadIdx.x; i < CH; i += blockDim.x) {
        s.b1[i] = theta[OB1 + i];
        s.b2[i] = theta[OB2 + i];
    }
    // w2 flat is [o][i][t]; smem is [t][o][i]
    for (int k = threadIdx.x; k < CH * CH * KW; k += blockDim.x) {
        const int o = k / (CH * KW), i = (k / KW) % CH, t = k % KW;
        s.w2[(t * CH + o) * LDB + i] = __float2bfloat16_rn(theta[OW2 + k]);
    }
}

// Layers 1 and 2 of the forward pass: a1 (BF16), a2 = gelu(z2) (FP32) and the
// pre-activations z1, z2 for the backward pass.  Requires load_tile and a barrier first.
__device__ void forward_12(Smem &s) {
    {
        // lane = output channel o; each warp a contiguous run of rows, with o's
        // five weights and a sliding window of five inputs in registers (one
        // shared load per row; the FMA chain is the same, tap 0 first)
        const int o = threadIdx.x & 31, nw = blockDim.x >> 5;
        const int per = (NA1 + nw - 1) / nw, r0 = (threadIdx.x >> 5) * per;
        const int r1 = min(r0 + per, NA1);
        float w[KW], u[KW];
#pragma unroll
        for (int t = 0; t < KW; ++t) w[t] = s.w1[o * KW + t];
        const float b = s.b1[o];
        int r = r0;
        if (r < r1) {
#pragma unroll
            for (int t = 0; t < KW - 1; ++t) u[t + 1] = s.us[r + t];
        }
        for (; r < r1; ++r) {
#pragma unroll
            for (int t = 0; t < KW - 1; ++t) u[t] = u[t + 1];
            u[KW - 1] = s.us[r + KW - 1];
            float z = b;
#pragma unroll
            for (int t = 0; t < KW; ++t) z = fmaf(w[t], u[t], z);
            s.z1[r * LDF + o] = z;
            s.a1[r * LDB + o] = __float2bfloat16_rn(gelu(z));
        }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    for (int m = warp; m < NZ2 / 16; m += blockDim.x >> 5) {
        const int p0 = m * 16;
        float acc[4][4] = {};
#pragma unroll
        for (int t = 0; t < KW; ++t) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // rows beyond NA1 are only reached for p >= NA2 (discarded rows): clamp the read
                uint32_t a[4], b[4];
                ldm4<false>(a, &s.a1[min(p0 + t + (lane & 15), NA1 - 1) * LDB + 16 * h + (lane >> 4) * 8]);
#pragma unroll
                for (int nt = 0; nt < 4; nt += 2) {
                    ldm4<false>(b, &s.w2[(t * CH + (nt + (lane >> 4)) * 8 + (lane & 7)) * LDB + 16 * h + ((lane >> 3) & 1) * 8]);
                    mma_bf16(acc[nt], a[0], a[1], a[2], a[3], b[0], b[1]);
                    mma_bf16(acc[nt + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
                }
            }
        }
        const int r0 = p0 + g, r1 = p0 + g + 8;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const int o = nt * 8 + 2 * q;
            if (r0 < NA2) {
                const float z0 = acc[nt][0] + s.b2[o], z1 = acc[nt][1] + s.b2[o + 1];
                s.z2[r0 * LDF + o] = z0;
                s.z2[r0 * LDF + o + 1] = z1;
                s.a2[r0 * LDF + o] = gelu(z0);
                s.a2[r0 * LDF + o + 1] = gelu(z1);
            }
            if (r1 < NA2) {
                const float z2 = acc[nt][2] + s.b2[o], z3 = acc[nt][3] + s.b2[o + 1];
                s.z2[r1 * LDF + o] = z2;
                s.z2[r1 * LDF + o + 1] = z3;
                s.a2[r1 * LDF + o] = gelu(z2);
                s.a2[r1 * LDF + o + 1] = gelu(z3);
            }
        }
    }
    __syncthreads();
}

// Loss and parameter gradients (forward + backward), summed over the tiles a
// block visits into its row of `partial` ([gridDim.x][NPARAM + 1], last = loss).
// The loss is on the scaled defect: L = wpt * sum (net(u) - target / s)^2,
// wpt = 1 / (points in the batch), s the output scale.
//
// Bound by latency: a tile is a chain of eight short phases, 512 tiles (a minibatch
// of 64 x 1024) on 152 SMs.  So the small layers' sums run with a lane per channel,
// each warp on its own rows with a sliding window, and stay in registers from tile
// to tile (sums over all rows by a few threads, through shared memory, took half of
// the tile); fragments are loaded with ldmatrix, transposed where the operand lies
// the other way; and a block's 100 KB of shared memory lets two share an SM.
__global__ void __launch_bounds__(THREADS, 2) k_grad(const float *__restrict__ theta, const float *__restrict__ u,
                                                     const float *__restrict__ target, const int64_t *__restrict__ rows,
                                                     float *__restrict__ partial, int64_t n, int64_t tiles_per_dom,
                                                     int64_t n_tiles, float scale) {
    extern __shared__ __align__(16) unsigned char raw[];
    Smem &s = *reinterpret_cast<Smem *>(raw);
    constexpr int NW = THREADS / 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, q4 = lane & 3;
    load_weights(s, theta);
    for (int i = tid; i < 4 + LDT + 8; i += THREADS) s.dd[i] = 0.0f;
    if (tid < 8) s.us[NU + tid] = 0.0f;
    for (int i = tid; i < 4 * LDB; i += THREADS) s.dzP[i] = __float2bfloat16_rn(0.0f);
    const float b3 = theta[OB3], out_scale = theta[OSCALE];
    __syncthreads();
    float w3[KW];  // channel `lane`
#pragma unroll
    for (int t = 0; t < KW; ++t) w3[t] = s.w3[t * CH + lane];
    // this thread's sums: dW2 of output channels 16 (warp / 4) on and columns (t, i) of n-tiles 5 (warp % 4) on;
    // channel `lane`'s dW1, db1, dW3, db2 over its warp's rows; db3 and the loss over its outputs
    float accw[5][4] = {}, dw1[KW] = {}, dw3[KW] = {}, db1 = 0.0f, db2 = 0.0f, db3 = 0.0f, loss = 0.0f;

    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const int64_t b = tile / tiles_per_dom, x0 = (tile % tiles_per_dom) * TOUT;
        const int64_t dom = rows ? rows[b] : b;  // minibatch row -> sample
        load_tile(s, u + dom * n, n, x0);
        const float want = tid < TOUT ? target[dom * n + x0 + tid] : 0.0f;
        __syncthreads();
        forward_12(s);
        {  // layer 3, half of the channels per thread
            const int q = tid & (TOUT - 1), i0 = (tid / TOUT) * (CH / 2);
            float d = 0.0f;
#pragma unroll
            for (int t = 0; t < KW; ++t)
#pragma unroll
                for (int i = 0; i < CH / 2; i += 4) {
                    const float4 w = *reinterpret_cast<const float4 *>(&s.w3[t * CH + i0 + i]);
                    const float *a = &s.a2[(q + t) * LDF + i0 + i];
                    d = fmaf(w.x, a[0], d);
                    d = fmaf(w.y, a[1], d);
                    d = fmaf(w.z, a[2], d);
                    d = fmaf(w.w, a[3], d);
                }
            s.part[tid / TOUT][q] = d;
        }
        __syncthreads();
        if (tid < TOUT) {
            const float e = (s.part[0][tid] + s.part[1][tid] + b3) - want / out_scale;
            const float g = 2.0f * scale * e;
            s.dd[4 + tid] = g;
            loss += scale * e * e;
            db3 += g;
        }
        __syncthreads();
        {  // dz2[p][o] = (sum_t w3[o][t] dd[p - t]) * gelu'(z2[p][o]), p < NA2, zero beyond; dW3, db2
            constexpr int PER = 20;  // rows per warp (even: they are stored in pairs)
            const int p0 = warp * PER, p1 = min(p0 + PER, LDT);
            float w[KW];  // w[t] = dd[p - t]
#pragma unroll
            for (int t = 0; t < KW - 1; ++t) w[t] = s.dd[p0 + 3 - t];
            for (int p = p0; p < p1; p += 2) {
                __nv_bfloat16 z[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
#pragma unroll
                    for (int t = KW - 1; t > 0; --t) w[t] = w[t - 1];
                    w[0] = s.dd[p + k + 4];
                    float v = 0.0f;
                    if (p + k < NA2) {
                        float da = 0.0f;
                        const float a = s.a2[(p + k) * LDF + lane];
#pragma unroll
                        for (int t = 0; t < KW; ++t) {
                            da = fmaf(w3[t], w[t], da);
                            dw3[t] = fmaf(w[t], a, dw3[t]);
                        }
                        v = da * gelu_grad(s.z2[(p + k) * LDF + lane]);
                    }
                    z[k] = __float2bfloat16_rn(v);
                    db2 += __bfloat162float(z[k]);
                    if (p + k + 4 < LDT) s.dzP[(p + k + 4) * LDB + lane] = z[k];
                }
                *reinterpret_cast<uint32_t *>(&s.dzT[lane * LDT + p]) = pack2(z[0], z[1]);
            }
        }
        __syncthreads();
        // dW2[o][(t,i)] += sum_p dz2[p][o] a1[p + t][i]: M = o (2 tiles), N = (t, i) (20 tiles), K = p (9 steps);
        // rows past NA1 meet dz2 = 0
        for (int ks = 0; ks < NZ2 / 16; ++ks) {
            uint32_t a[4], f[2];
            ldm4<false>(a, &s.dzT[((warp >> 2) * 16 + (lane & 15)) * LDT + ks * 16 + (lane >> 4) * 8]);
#pragma unroll
            for (int slot = 0; slot < 5; ++slot) {
                const int nn = (warp & 3) * 5 + slot, t = nn / 4, i0 = (nn % 4) * 8;
                ldm2_t(f, &s.a1[min(ks * 16 + t + (lane & 15), NA1 - 1) * LDB + i0]);
                mma_bf16(accw[slot], a[0], a[1], a[2], a[3], f[0], f[1]);
            }
        }
        // da1[r][i] = sum_{t,o} w2[o][i][t] dz2[r - t][o]: M = r (10 tiles of 16 over NA1), N = i (4), K = (t, o) (10)
        // then dz1 = da1 * gelu'(z1)
        for (int m = warp; m < (NA1 + 15) / 16; m += NW) {
            const int r0 = m * 16;
            float acc[4][4] = {};
#pragma unroll
            for (int t = 0; t < KW; ++t) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    // A[r][o] = dz2[r - t][o] = dzP[r - t + 4][o]; rows beyond NA1 are discarded: clamp the read
                    uint32_t a[4], f[4];
                    ldm4<false>(a, &s.dzP[min(r0 + (lane & 15) - t + 4, LDT - 1) * LDB + 16 * h + (lane >> 4) * 8]);
#pragma unroll
                    for (int nt = 0; nt < 4; nt += 2) {
                        ldm4<true>(f, &s.w2[(t * CH + 16 * h + (lane & 15)) * LDB + (nt + (lane >> 4)) * 8]);
                        mma_bf16(acc[nt], a[0], a[1], a[2], a[3], f[0], f[1]);
                        mma_bf16(acc[nt + 1], a[0], a[1], a[2], a[3], f[2], f[3]);
                    }
                }
            }
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int r = r0 + gq + (e >= 2 ? 8 : 0), i = nt * 8 + 2 * q4 + (e & 1);
                    if (r < NA1) s.z1[r * LDF + i] = acc[nt][e] * gelu_grad(s.z1[r * LDF + i]);  // dz1 in place
                }
            }
        }
        __syncthreads();
        {  // dW1, db1
            constexpr int PER = (NA1 + NW - 1) / NW;
            const int r0 = warp * PER, r1 = min(r0 + PER, NA1);
            float w[KW];  // w[t] = us[r + t]
#pragma unroll
            for (int t = 0; t < KW - 1; ++t) w[t + 1] = s.us[r0 + t];
            for (int r = r0; r < r1; ++r) {
#pragma unroll
                for (int t = 0; t < KW - 1; ++t) w[t] = w[t + 1];
                w[KW - 1] = s.us[r + KW - 1];
                const float z = s.z1[r * LDF + lane];
#pragma unroll
                for (int t = 0; t < KW; ++t) dw1[t] = fmaf(z, w[t], dw1[t]);
                db1 += z;
            }
        }
        __syncthreads();
    }
    float *row = partial + (int64_t)blockIdx.x * (NPARAM + 1);
    // dW2 (flat w2 is [o][i][t])
#pragma unroll
    for (int slot = 0; slot < 5; ++slot) {
        const int nn = (warp & 3) * 5 + slot, t = nn / 4, i0 = (nn % 4) * 8;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int o = (warp >> 2) * 16 + gq + (e >= 2 ? 8 : 0), i = i0 + 2 * q4 + (e & 1);
            row[OW2 + (o * CH + i) * KW + t] = accw[slot][e];
        }
    }
    // the other sums over the warps: red[value][warp][lane], values dW1 x 5, db1, dW3 x 5, db2, db3, loss
    constexpr int NV = 2 * (KW + 1) + 2;
    static_assert(NV * THREADS <= NA1 * LDF, "the reduction takes z1's place");
    float *red = s.z1;
#pragma unroll
    for (int t = 0; t < KW; ++t) {
        red[t * THREADS + tid] = dw1[t];
        red[(KW + 1 + t) * THREADS + tid] = dw3[t];
    }
    red[KW * THREADS + tid] = db1;
    red[(2 * KW + 1) * THREADS + tid] = db2;
    red[(2 * KW + 2) * THREADS + tid] = db3;
    red[(2 * KW + 3) * THREADS + tid] = loss;
    __syncthreads();
    for (int v = warp; v < NV; v += NW) {
        float a = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; ++w) a += red[v * THREADS + w * 32 + lane];
        if (v >= 2 * (KW + 1)) {
#pragma unroll
            for (int off = 16; off; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
            if (lane == 0) row[v == 2 * (KW + 1) ? OB3 : NPARAM] = a;
        } else {
            const int t = v % (KW + 1);
            row[v <= KW ? (t < KW ? OW1 + lane * KW + t : OB1 + lane) : (t < KW ? OW3 + lane * KW + t : OB2 + lane)] = a;
        }
    }
    if (tid == 0) row[OSCALE] = 0.0f;  // not trained
}

// Sum the blocks' rows: out[j] = sum_b partial[b][j], j < NPARAM + 1.  A block takes 32 values, each warp every eighth
// row (one thread per value, 304 rows in a chain, took 16 us).
constexpr int REDUCE_WARPS = 8;
__global__ void __launch_bounds__(32 * REDUCE_WARPS) k_reduce(const float *__restrict__ partial, int rows,
                                                              float *__restrict__ out) {
    __shared__ float sums[REDUCE_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j = blockIdx.x * 32 + lane;
    float a = 0.0f;
    if (j < NPARAM + 1) {
#pragma unroll 8
        for (int b = warp; b < rows; b += REDUCE_WARPS) a += partial[(int64_t)b * (NPARAM + 1) + j];
    }
    sums[warp][lane] = a;
    __syncthreads();
    if (warp || j >= NPARAM + 1) return;
    a = 0.0f;
#pragma unroll
    for (int w = 0; w < REDUCE_WARPS; ++w) a += sums[w][lane];
    out[j] = a;
}

// Adam on the FP32 master parameters.
__global__ void k_adam(float *__restrict__ theta, const float *__restrict__ grad, float *__restrict__ m,
                       float *__restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= NTRAIN) return;
    const float gj = grad[j];
    const float mj = b1 * m[j] + (1.0f - b1) * gj;
    const float vj = b2 * v[j] + (1.0f - b2) * gj * gj;
    m[j] = mj;
    v[j] = vj;
    theta[j] -= lr * (mj / c1) / (sqrtf(vj / c2) + eps);
}

// Cell averages of `factor` fine cells: coarse[d][j] = mean(fine[d][factor j .. factor j + factor - 1]).
__global__ void k_coarse_grain(const double *__restrict__ fine, float *__restrict__ coarse, int64_t n_coarse_total,
                               int factor) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_coarse_total) return;
    double a = 0.0;
    for (int k = 0; k < factor; ++k) a += fine[j * factor + k];
    coarse[j] = (float)(a / factor);
}

// Rows idx[0..m) of the (domains x n) array src into the (m x n) array dst.
template <typename T>
__global__ void k_gather_rows(const T *__restrict__ src, const int32_t *__restrict__ idx, int64_t n,
                              T *__restrict__ dst) {
    const T *a = src + (int64_t)idx[blockIdx.x] * n;
    T *b = dst + (int64_t)blockIdx.x * n;
    for (int64_t j = threadIdx.x; j < n; j += blockDim.x) b[j] = a[j];
}

// out[d] = ||a_d - b_d|| / ||b_d|| (FP64 sums) for the m rows of b; a's row d is
// row rows[d] of a when rows is given, else row d.  One block per row.
__global__ void __launch_bounds__(256) k_rel_l2(const float *__restrict__ a, const int32_t *__restrict__ rows,
                                                const float *__restrict__ b, int64_t n, double *__restrict__ out) {
    const float *x = a + (int64_t)(rows ? rows[blockIdx.x] : (int)blockIdx.x) * n;
    const float *y = b + (int64_t)blockIdx.x * n;
    double s1 = 0.0, s2 = 0.0;
    for (int64_t j = threadIdx.x; j < n; j += blockDim.x) {
        const double d = (double)x[j] - (double)y[j];
        s1 += d * d;
        s2 += (double)y[j] * (double)y[j];
    }
    __shared__ double r1[256], r2[256];
    r1[threadIdx.x] = s1;
    r2[threadIdx.x] = s2;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if ((int)threadIdx.x < k) {
            r1[threadIdx.x] += r1[threadIdx.x + k];
            r2[threadIdx.x] += r2[threadIdx.x + k];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = sqrt(r1[0] / r2[0]);
}

constexpr size_t smem_bytes() { return sizeof(Smem); }

}  // namespace cl
}  // namespace sw

using namespace sw;

namespace {

int closure_check(sw_ctx *ctx, int32_t n_dom, int64_t n) {
    if (!ctx || n_dom < 1 || n < cl::TOUT || n % cl::TOUT) return SW_ERR_SIZE;
    return SW_OK;
}

// The kernels' shared-memory limits, once per device (the attribute belongs to
// the current device): a bit per device 0..63, set again on every call above.
cudaError_t allow_smem() {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = (dev >= 0 && dev < 64) ? (uint64_t(1) << dev) : 0;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    e = cudaFuncSetAttribute(cl::k_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cl::smem_bytes());
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
}

// The closure calls run on the context's stream, a non-blocking one: order
// them after the work already queued on the legacy default stream (where a
// torch caller's default-stream copies of their inputs are).
int after_legacy(sw_ctx *ctx) {
    SW_CUDA(ctx, cudaEventRecord(ctx->e0, cudaStreamLegacy));
    SW_CUDA(ctx, cudaStreamWaitEvent(ctx->stream, ctx->e0, 0));
    return SW_OK;
}

// Stage theta for the forward kernels (stream-ordered before them).
int stage_weights(sw_ctx *ctx, const float *theta) {
    if (!ctx->d_fwd) SW_CUDA(ctx, cudaMalloc(&ctx->d_fwd, sizeof(cl::FwdWeights)));
    if (!ctx->h_fwd_status) {
        SW_CUDA(ctx, cudaMallocHost(&ctx->h_fwd_status, sizeof(int)));
        *ctx->h_fwd_status = 0;
    }
    cl::k_pack_weights<<<(cl::CH * cl::CH * cl::KW + 255) / 256, 256, 0, ctx->stream>>>(
        theta, static_cast<cl::FwdWeights *>(ctx->d_fwd));
    SW_CUDA(ctx, cudaGetLastError());
    return SW_OK;
}

// One forward launch over n_dom domains of n cells.  Dependent launches read the staged weights before they wait for
// the launch before them, so the first launch after stage_weights is an ordinary one.
template <bool STEP, int NT>
cudaError_t launch_forward_tiles(sw_ctx *ctx, bool dependent, int sms, const Params<float> &p, const float *u, float *out,
                                 int64_t n, uint32_t per_dom, uint32_t tiles, int n_out) {
    const unsigned grid = std::min<unsigned>((tiles + NT - 1) / NT, (unsigned)(sms * cl::FWD_BLOCKS));
    const cl::FwdWeights *w = static_cast<const cl::FwdWeights *>(ctx->d_fwd);
    if (dependent)
        return launch_dependent(cl::k_forward<STEP, NT>, grid, cl::FWD_THREADS, 0, ctx->stream, w, p, u, out, n, per_dom,
                                tiles, n_out, ctx->h_fwd_status);
    cl::k_forward<STEP, NT><<<grid, cl::FWD_THREADS, 0, ctx->stream>>>(w, p, u, out, n, per_dom, tiles, n_out,
                                                                        ctx->h_fwd_status);
    return cudaGetLastError();
}
template <bool STEP>
cudaError_t launch_forward(sw_ctx *ctx, bool dependent, const Params<float> &p, const float *u, float *out, int32_t n_dom,
                           int64_t n) {
    const int n_out = n == 128 ? 128 : cl::FWD_OUT;
    const uint32_t per_dom = (uint32_t)((n + n_out - 1) / n_out), tiles = per_dom * (uint32_t)n_dom;
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    if (e != cudaSuccess) return e;
    // Two tiles at a time share each weight read, one at a time spreads a small step over more blocks: us per step at
    // 16, 48, 64, 256, 1024 domains of 1024 cells (9 tiles each) one 4.6, 6.7, 7.7, 17.5, 54; two 5.7, 7.1, 7.2, 15.8, 49
    if (tiles > 3u * (uint32_t)sms)
        return launch_forward_tiles<STEP, 2>(ctx, dependent, sms, p, u, out, n, per_dom, tiles, n_out);
    return launch_forward_tiles<STEP, 1>(ctx, dependent, sms, p, u, out, n, per_dom, tiles, n_out);
}

// After the forward launches have completed.
int forward_status(sw_ctx *ctx) {
    if (!ctx->h_fwd_status || !*(volatile int *)ctx->h_fwd_status) return SW_OK;
    *ctx->h_fwd_status = 0;
    return fail(ctx, SW_ERR_TIMEOUT, "closure kernel: a tensor-core wait ran out");
}

}  // namespace

extern "C" {

int sw_closure_infer(sw_ctx *ctx, const float *theta, const float *u, float *delta, int32_t n_dom, int64_t n) {
    int rc = closure_check(ctx, n_dom, n);
    if (rc) return rc;
    if (!theta || !u || !delta) return SW_ERR_ARG;
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    if ((rc = after_legacy(ctx)) != SW_OK) return rc;
    if ((rc = stage_weights(ctx, theta))) return rc;
    SW_CUDA(ctx, launch_forward<false>(ctx, false, Params<float>{}, u, delta, n_dom, n));
    SW_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return forward_status(ctx);
}

}  // extern "C"

namespace {
// The coarse steps of sw_closure_step, enqueued on ctx's stream without
// waiting for them (ctx->d_work is their second row buffer).
int closure_enqueue(sw_ctx *ctx, const sw_config *coarse, const float *theta, float *u, int32_t n_dom, int64_t n,
                    int64_t n_steps, int32_t use_closure) {
    int rc = closure_check(ctx, n_dom, n);
    if (rc) return rc;
    if (!coarse || !u || (use_closure && !theta)) return SW_ERR_ARG;
    if (coarse->problem != SW_KS || coarse->precision != 4) return fail(ctx, SW_ERR_UNSUPPORTED, "closure steps KS FP32");
    if (coarse->flags != 0) return fail(ctx, SW_ERR_UNSUPPORTED, "closure steps take no sw_config.flags");
    sw_config c = *coarse;
    c.nx = n;
    sw_constants k;
    sw_constants_of(&c, &k);
    const Params<float> p = make_params<float>(c, k);
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    if ((rc = after_legacy(ctx)) != SW_OK) return rc;
    SW_CUDA(ctx, grow_dev(&ctx->d_work, &ctx->n_work, sizeof(float) * (size_t)n * n_dom));
    float *alt = static_cast<float *>(ctx->d_work), *cur = u;
    if (use_closure && (rc = stage_weights(ctx, theta))) return rc;
    const uint32_t warps_per_dom = (uint32_t)(n / 128), warps = warps_per_dom * (uint32_t)n_dom;
    constexpr uint32_t per_block = cl::PLAIN_THREADS / 32;
    for (int64_t i = 0; i < n_steps; ++i) {
        if (use_closure)
            SW_CUDA(ctx, launch_forward<true>(ctx, i > 0, p, cur, alt, n_dom, n));
        else
            SW_CUDA(ctx, launch_dependent(cl::k_plain_step, (warps + per_block - 1) / per_block, cl::PLAIN_THREADS, 0,
                                          ctx->stream, p, cur, alt, n, warps_per_dom, warps));
        std::swap(cur, alt);
    }
    SW_CUDA(ctx, cudaGetLastError());
    if (cur != u) SW_CUDA(ctx, cudaMemcpyAsync(u, cur, sizeof(float) * (size_t)n * n_dom, cudaMemcpyDeviceToDevice,
                                               ctx->stream));
    return SW_OK;
}
}  // namespace

extern "C" {

int sw_closure_step(sw_ctx *ctx, const sw_config *coarse, const float *theta, float *u, int32_t n_dom, int64_t n,
                    int64_t n_steps, int32_t use_closure, sw_result *out) {
    if (!ctx) return SW_ERR_ARG;
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    SW_CUDA(ctx, cudaEventRecord(ctx->k0, ctx->stream));
    const int rc = closure_enqueue(ctx, coarse, theta, u, n_dom, n, n_steps, use_closure);
    if (rc) return rc;
    SW_CUDA(ctx, cudaEventRecord(ctx->k1, ctx->stream));
    SW_CUDA(ctx, cudaEventSynchronize(ctx->k1));
    if (const int st = forward_status(ctx)) return st;
    if (out) {
        float ms = 0;
        cudaEventElapsedTime(&ms, ctx->k0, ctx->k1);
        std::memset(out, 0, sizeof(*out));
        out->n_steps = n_steps;
        out->t_final = n_steps * coarse->dt;
        out->kernel_ms = out->elapsed_ms = ms;
        out->launches = n_steps;
    }
    return SW_OK;
}

int sw_closure_grad(sw_ctx *ctx, const float *theta, const float *u, const float *target, const int64_t *rows,
                    int32_t n_dom, int64_t n, float *grad_and_loss) {
    int rc = closure_check(ctx, n_dom, n);
    if (rc) return rc;
    if (!theta || !u || !target || !grad_and_loss) return SW_ERR_ARG;
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    if ((rc = after_legacy(ctx)) != SW_OK) return rc;
    SW_CUDA(ctx, allow_smem());
    const int64_t tiles_per = n / cl::TOUT, n_tiles = tiles_per * n_dom;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    const int64_t grid = std::min<int64_t>(n_tiles, (int64_t)sms * 2);
    SW_CUDA(ctx, grow_dev(&ctx->d_io, &ctx->n_io, sizeof(float) * (size_t)grid * (cl::NPARAM + 1)));
    float *partial = static_cast<float *>(ctx->d_io);
    const float scale = 1.0f / (float)((double)n_dom * n);
    cl::k_grad<<<(unsigned)grid, cl::THREADS, cl::smem_bytes(), ctx->stream>>>(theta, u, target, rows, partial, n,
                                                                                tiles_per, n_tiles, scale);
    SW_CUDA(ctx, cudaGetLastError());
    cl::k_reduce<<<(cl::NPARAM + 1 + 31) / 32, 32 * cl::REDUCE_WARPS, 0, ctx->stream>>>(partial, (int)grid, grad_and_loss);
    SW_CUDA(ctx, cudaGetLastError());
    SW_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return SW_OK;
}

int sw_closure_adam(sw_ctx *ctx, float *theta, const float *grad, float *m, float *v, int32_t step, float lr) {
    if (!ctx || !theta || !grad || !m || !v || step < 1) return SW_ERR_ARG;
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    const int rc = after_legacy(ctx);
    if (rc) return rc;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - std::pow(b1, (float)step), c2 = 1.0f - std::pow(b2, (float)step);
    cl::k_adam<<<(cl::NTRAIN + 255) / 256, 256, 0, ctx->stream>>>(theta, grad, m, v, lr, b1, b2, 1e-8f, c1, c2);
    SW_CUDA(ctx, cudaGetLastError());
    return SW_OK;
}

int sw_closure_train(sw_ctx *ctx, float *theta, const float *inputs, const float *targets, int64_t n_samples,
                     int64_t n, int32_t batch, int32_t steps, float lr, uint64_t seed, float *loss_host) {
    int rc = closure_check(ctx, batch, n);
    if (rc) return rc;
    if (!theta || !inputs || !targets || n_samples < 1 || steps < 0) return SW_ERR_ARG;
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    if ((rc = after_legacy(ctx)) != SW_OK) return rc;
    // Adam moments and a gradient row live in one allocation owned by this call
    float *buf = nullptr;
    int64_t *rows = nullptr;
    SW_CUDA(ctx, cudaMalloc(&buf, sizeof(float) * (3 * cl::NPARAM + 2)));
    cudaError_t e = cudaMalloc(&rows, sizeof(int64_t) * (size_t)batch);
    if (e != cudaSuccess) {
        cudaFree(buf);
        return cuda_fail(ctx, e, "cudaMalloc rows");
    }
    float *m = buf, *v = buf + cl::NPARAM, *grad = buf + 2 * cl::NPARAM;
    cudaMemsetAsync(buf, 0, sizeof(float) * 2 * cl::NPARAM, ctx->stream);
    std::vector<int64_t> host_rows((size_t)batch);
    uint64_t st = seed ? seed : 0x9E3779B97F4A7C15ull;
    for (int32_t s = 0; s < steps && rc == SW_OK; ++s) {
        for (auto &r : host_rows) {  // splitmix64 draws of the minibatch rows
            st += 0x9E3779B97F4A7C15ull;
            uint64_t z = st;
            z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
            z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
            r = (int64_t)((z ^ (z >> 31)) % (uint64_t)n_samples);
        }
        e = cudaMemcpyAsync(rows, host_rows.data(), sizeof(int64_t) * batch, cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) { rc = cuda_fail(ctx, e, "rows"); break; }
        rc = sw_closure_grad(ctx, theta, inputs, targets, rows, batch, n, grad);
        if (rc) break;
        if (loss_host) {
            e = cudaMemcpy(&loss_host[s], grad + cl::NPARAM, sizeof(float), cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) { rc = cuda_fail(ctx, e, "loss"); break; }
        }
        rc = sw_closure_adam(ctx, theta, grad, m, v, s + 1, lr);
    }
    cudaStreamSynchronize(ctx->stream);
    cudaFree(rows);
    cudaFree(buf);
    return rc;
}

// Closure steps the ensemble runs in the first segment before the judge has
// picked a variant.  At 1024 domains eight take 0.42 ms; the judge's first segment
// alone takes 0.20 ms for 8 coarse steps, 0.36 for 16, 1.05 for 50, longer beside
// them.  More steps gain where the closure is picked and cost where the plain step
// is.  ms for a run of one segment, 4, 8, 12, 16, 24 steps ahead: closure picked, 15
// steps 1.41, 1.37, 1.32, 1.27, 1.26, 50 steps 3.83, 3.74, 3.60, 3.56, 3.38; plain
// picked, 10 steps 0.71, 0.84, 0.94, 0.94, 0.94, 50 steps 1.74, 1.89, 1.93, 2.10, 2.29.
constexpr int64_t kSpeculativeSteps = 8;

int sw_closure_adaptive(sw_ctx *ctx, sw_ctx *judge, const sw_config *coarse, const sw_config *fine,
                        const float *theta, const double *fine0, int32_t n_dom, int64_t n_fine, int32_t factor,
                        int64_t coarse_steps, int64_t segment, double tau, int32_t shadow_every,
                        int32_t shadow_offset, float *u_out, sw_adaptive_info *info, double *log_out,
                        int32_t log_cap) {
    if (!ctx || !judge || judge == ctx || !coarse || !fine || !fine0 || !u_out || !info) return SW_ERR_ARG;
    if (factor < 1 || n_fine % factor || shadow_every < 1 || shadow_offset < 0 || shadow_offset >= shadow_every ||
        segment < 1 || coarse_steps < 0 || !(tau >= 0))
        return SW_ERR_ARG;
    if (judge->device != ctx->device) return fail(ctx, SW_ERR_ARG, "the judge context must be on the run's device");
    const int64_t n = n_fine / factor;
    int rc = closure_check(ctx, n_dom, n);
    if (rc) return rc;
    std::vector<int32_t> idx;
    for (int32_t d = shadow_offset; d < n_dom; d += shadow_every) idx.push_back(d);
    if (idx.empty()) return fail(ctx, SW_ERR_ARG, "the judge's sample is empty");
    const int32_t m = (int32_t)idx.size();
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    // run context scratch: the sample's coarse rows for each variant and the reference (m x n
    // floats each), the ensemble's state kept at the start of the first segment, errors,
    // indices (each at a 256-byte boundary)
    const size_t fb = sizeof(float) * (size_t)m * n, fbr = (fb + 255) & ~(size_t)255;
    const size_t ub = sizeof(float) * (size_t)n_dom * n, ubr = (ub + 255) & ~(size_t)255;
    SW_CUDA(ctx, grow_dev(&ctx->d_judge, &ctx->n_judge,
                          3 * fbr + ubr + 4 * sizeof(double) * m + sizeof(int32_t) * m + 64));
    // the coarse runs' second row buffer, sized for the ensemble before any run is enqueued
    SW_CUDA(ctx, grow_dev(&ctx->d_work, &ctx->n_work, ub));
    char *scratch = static_cast<char *>(ctx->d_judge);
    float *samp = reinterpret_cast<float *>(scratch), *samp2 = reinterpret_cast<float *>(scratch + fbr);
    float *ref = reinterpret_cast<float *>(scratch + 2 * fbr);
    float *u_kept = reinterpret_cast<float *>(scratch + 3 * fbr);
    double *err = reinterpret_cast<double *>(scratch + 3 * fbr + ubr);  // [2][m]
    int32_t *idx_d = reinterpret_cast<int32_t *>(err + 2 * m);
    SW_CUDA(ctx, grow_dev(&judge->d_judge, &judge->n_judge, sizeof(double) * (size_t)m * n_fine));
    double *shadow = static_cast<double *>(judge->d_judge);
    SW_CUDA(ctx, cudaMemcpy(idx_d, idx.data(), sizeof(int32_t) * m, cudaMemcpyHostToDevice));
    if ((rc = after_legacy(ctx)) != SW_OK) return rc;
    cudaStream_t s = ctx->stream;
    cl::k_gather_rows<double><<<m, 256, 0, s>>>(fine0, idx_d, n_fine, shadow);
    SW_CUDA(ctx, cudaGetLastError());
    SW_CUDA(ctx, cudaStreamSynchronize(s));
    if ((rc = sw_coarse_grain(ctx, fine0, u_out, (int64_t)n_dom * n, factor))) return rc;
    std::memset(info, 0, sizeof(*info));
    info->n_shadow = m;
    std::vector<int64_t> nx_s((size_t)m, n_fine);
    std::vector<double> h_err(2 * (size_t)m);
    sw_config fc = *fine;
    fc.time_mode = SW_TIME_STEPS;
    auto rel = [&](const float *a, const int32_t *rows, int slot) -> int {
        cl::k_rel_l2<<<m, 256, 0, s>>>(a, rows, ref, n, err + (size_t)slot * m);
        SW_CUDA(ctx, cudaGetLastError());
        return SW_OK;
    };
    auto stats = [&](int slot, double *mean, double *mx) {
        double a = 0.0, b = 0.0;
        for (int32_t d = 0; d < m; ++d) {
            a += h_err[(size_t)slot * m + d];
            b = std::max(b, h_err[(size_t)slot * m + d]);
        }
        *mean = a / m;
        *mx = b;
    };
    int64_t done = 0;
    int pick = -1;  // 0 plain, 1 closure
    double prev = 0.0;
    int32_t nlog = 0;
    while (done < coarse_steps) {
        const int64_t k = std::min(segment, coarse_steps - done);
        // Enqueued first, in this order on the run's stream: the sample's runs (both
        // variants in the first segment, later the variant the ensemble does not run),
        // then the ensemble's run of the pick.  The judge's segment runs meanwhile on its
        // own context, and the segment takes as long as the longer of the two.  The first
        // segment's pick is not known yet: the ensemble starts the closure for the first
        // kSpeculativeSteps steps (about the judge's time), its state at the segment's
        // start kept, then continues it, or runs the plain step from the kept state
        // should the sample pick that.  The results are those of running the pick alone.
        cl::k_gather_rows<float><<<m, 256, 0, s>>>(u_out, idx_d, n, samp);
        SW_CUDA(ctx, cudaGetLastError());
        int64_t started = 0;  // closure steps the ensemble ran ahead of the first pick
        if (pick < 0) {
            SW_CUDA(ctx, cudaMemcpyAsync(samp2, samp, fb, cudaMemcpyDeviceToDevice, s));
            if ((rc = closure_enqueue(ctx, coarse, theta, samp, m, n, k, 0))) return rc;
            if ((rc = closure_enqueue(ctx, coarse, theta, samp2, m, n, k, 1))) return rc;
            SW_CUDA(ctx, cudaMemcpyAsync(u_kept, u_out, ub, cudaMemcpyDeviceToDevice, s));
            started = std::min(k, kSpeculativeSteps);
            if ((rc = closure_enqueue(ctx, coarse, theta, u_out, n_dom, n, started, 1))) return rc;
        } else {
            if ((rc = closure_enqueue(ctx, coarse, theta, samp, m, n, k, 1 - pick))) return rc;
            if ((rc = closure_enqueue(ctx, coarse, theta, u_out, n_dom, n, k, pick))) return rc;
        }
        fc.n_steps = k * factor;
        if ((rc = sw_run_batch_device(judge, &fc, m, nx_s.data(), shadow, nullptr, nullptr))) return rc;
        if ((rc = sw_coarse_grain(judge, shadow, ref, (int64_t)m * n, factor))) return rc;
        int cur_slot, alt_slot;
        if (pick < 0) {  // first segment: the better variant on the sample runs the ensemble
            if ((rc = rel(samp, nullptr, 0))) return rc;
            if ((rc = rel(samp2, nullptr, 1))) return rc;
            SW_CUDA(ctx, cudaMemcpyAsync(h_err.data(), err, sizeof(double) * 2 * m, cudaMemcpyDeviceToHost, s));
            SW_CUDA(ctx, cudaStreamSynchronize(s));
            if ((rc = forward_status(ctx))) return rc;
            double m0, m1, x0, x1;
            stats(0, &m0, &x0);
            stats(1, &m1, &x1);
            pick = (m1 < m0) ? 1 : 0;
            if (pick == 0) {  // the plain step, from the kept state
                SW_CUDA(ctx, cudaMemcpyAsync(u_out, u_kept, ub, cudaMemcpyDeviceToDevice, s));
                if ((rc = sw_closure_step(ctx, coarse, theta, u_out, n_dom, n, k, 0, nullptr))) return rc;
            } else if (k > started) {  // the rest of the closure's segment
                if ((rc = sw_closure_step(ctx, coarse, theta, u_out, n_dom, n, k - started, 1, nullptr))) return rc;
            }
            cur_slot = pick;
            alt_slot = 1 - pick;
        } else {  // the ensemble ran the pick, the sample the other variant
            if ((rc = rel(u_out, idx_d, 0))) return rc;
            if ((rc = rel(samp, nullptr, 1))) return rc;
            SW_CUDA(ctx, cudaMemcpyAsync(h_err.data(), err, sizeof(double) * 2 * m, cudaMemcpyDeviceToHost, s));
            SW_CUDA(ctx, cudaStreamSynchronize(s));
            if ((rc = forward_status(ctx))) return rc;
            cur_slot = 0;
            alt_slot = 1;
        }
        double e, emax, eo, eomax;
        stats(cur_slot, &e, &emax);  // the certificate: the sample's mean relative L2 error
        stats(alt_slot, &eo, &eomax);
        done += k;
        if (log_out && nlog < log_cap) {
            double *row = log_out + 4 * (size_t)nlog;
            row[0] = (double)done;
            row[1] = pick;
            row[2] = e;
            row[3] = eo;
            ++nlog;
        }
        const double left = (double)(coarse_steps - done) / (double)k;  // segments still to run
        if (e > tau || e + std::max(e - prev, 0.0) * left > tau) {
            info->fallback = 1;
            break;
        }
        if (pick == 1) ++info->closure_segments;
        else ++info->plain_segments;
        info->shadow_mean_rel_l2 = e;
        info->shadow_max_rel_l2 = emax;
        prev = e;
        if (eo < e) pick = 1 - pick;
    }
    info->n_log = nlog;
    if (info->fallback) {  // every domain by the fine solver from fine0: the answer is the fine solution
        const size_t bytes = sizeof(double) * (size_t)n_dom * n_fine;
        SW_CUDA(ctx, grow_dev(&ctx->d_state, &ctx->n_state, bytes));
        SW_CUDA(ctx, cudaMemcpyAsync(ctx->d_state, fine0, bytes, cudaMemcpyDeviceToDevice, s));
        SW_CUDA(ctx, cudaStreamSynchronize(s));
        std::vector<int64_t> nx_all((size_t)n_dom, n_fine);
        fc.n_steps = coarse_steps * factor;
        if ((rc = sw_run_batch_device(ctx, &fc, n_dom, nx_all.data(), ctx->d_state, nullptr, nullptr))) return rc;
        if ((rc = sw_coarse_grain(ctx, static_cast<const double *>(ctx->d_state), u_out, (int64_t)n_dom * n, factor)))
            return rc;
    }
    return SW_OK;
}

int sw_coarse_grain(sw_ctx *ctx, const double *fine, float *coarse, int64_t n_coarse_total, int32_t factor) {
    if (!ctx || !fine || !coarse || n_coarse_total < 1 || factor < 1) return SW_ERR_ARG;
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    const int rc = after_legacy(ctx);
    if (rc) return rc;
    cl::k_coarse_grain<<<(unsigned)((n_coarse_total + 255) / 256), 256, 0, ctx->stream>>>(fine, coarse,
                                                                                            n_coarse_total, factor);
    SW_CUDA(ctx, cudaGetLastError());
    SW_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return SW_OK;
}

}  // extern "C"
