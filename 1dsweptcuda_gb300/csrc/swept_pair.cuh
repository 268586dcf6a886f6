// FP32 KS swept passes with two tiles per block, one in each half of the f32x2
// instructions.
//
// The four-cells-per-thread path (tile_span4) is bound by instruction issue: 82 %
// of the issue slots, with the FMA pipe at 48 %.  An f32x2 instruction does
// the arithmetic of two cells in one issue slot, but pairing a cell with its
// neighbour needs the operands re-paired for every shift of the stencil
// (measured slower than scalar code).  Pairing cell x of one tile with cell x of
// another does not: every shift moves whole pairs.  So the tiles 2b and 2b + 1
// of a pass share a block, their rows interleaved in shared memory as (tile A,
// tile B) pairs, and each thread updates four positions of both.
//
//  * Levels are taken two at a time (predictor, corrector) with one thread
//    mapping: the thread keeps its four u and u* in registers from one to the
//    other and reads only its two neighbours' values on each side: 10 16-byte shared
//    accesses for the two levels, where re-reading whole windows takes 14.
//  * Position pairs (4k, 4k + 1) and (4k + 2, 4k + 3) lie in two planes, so that
//    the 16-byte accesses of consecutive threads are 16 bytes apart: no bank
//    conflicts.
//  * The live range is packed onto the lowest threads as in tile_span4.
//
// Measured at 2^22 cells, 2048 steps, against one tile per block (tile_span4; at
// 128 cells k_swept_ks_warp): tile 1024 5.82e11 -> 7.65e11 cell-updates/s, 512
// 5.43e11 -> 7.27e11, 256 3.88e11 -> 5.12e11, 128 3.00e11 -> 4.96e11 (2^24 cells, tile
// 1024: 8.47e11).  The FMA pipe is now 63 % busy (an f32x2 instruction takes it
// two cycles), the issue slots 56 %; idle warps of the narrow levels hold most of
// the rest of the occupancy.
//
// Slots, modes, level ranges and arithmetic are those of swept_tile, so the
// results are the same bit for bit; sums a - b are formed as fma(b, -1, a) and
// products as fma(a, b, -0.0) (see ml2), the same single roundings.
#pragma once

#include <cuda_runtime.h>

#include "engine.cuh"

SW_KERNELS_BEGIN

#ifndef SW_KS_DIVIDE_TU
// One tile of a pair: its domain's state (at the domain's first cell), its two
// slots, its first cell and the domain's length.
struct PairTile {
    float *state, *sl, *sr;
    int64_t base, nx;
};
__device__ __forceinline__ PairTile pair_tile(float *state, float *slots, int W, int phase, int64_t t, int64_t nx) {
    const int64_t nhalf = nx / (W >> 1), hl = (2 * t + phase) % nhalf, hr = (hl + 1 == nhalf) ? 0 : hl + 1;
    return PairTile{state, slots + hl * W, slots + hr * W, t * W + (int64_t)phase * (W >> 1), nx};
}

// Rows of a pair: position x of row r, -4 <= x < W + 4, in float2 units.
__host__ __device__ constexpr int pair_plane(int W) { return (W + 8) / 2; }
__host__ __device__ constexpr size_t pair_smem_bytes(int W) { return sizeof(float2) * 4 * (size_t)pair_plane(W); }
__device__ __forceinline__ int pair_at(int PS, int row, int x) {
    const int q = (x + 4) >> 1;
    return (2 * row + (q & 1)) * PS + (q & ~1) + (x & 1);
}
// The position pairs (4k - 4, 4k - 3), plane 0, and (4k - 2, 4k - 1), plane 1.
__device__ __forceinline__ void pair_load(const float2 *plane, int k, float2 &a, float2 &b) {
    const float4 v = *reinterpret_cast<const float4 *>(plane + 2 * k);
    a = make_float2(v.x, v.y);
    b = make_float2(v.z, v.w);
}
__device__ __forceinline__ void pair_store(float2 *plane, int k, float2 a, float2 b) {
    *reinterpret_cast<float4 *>(plane + 2 * k) = make_float4(a.x, a.y, b.x, b.y);
}

// Right-hand sides of four positions from the window w[0..7] around them.
template <bool POW2>
__device__ __forceinline__ void ks_rhs_pairs(const Params<float> &p, const float2 (&w)[8], float2 (&rhs)[4]) {
    const float2 nz = dup2(p.nz);
    float2 sq[6];  // squares of w[1..6]
#pragma unroll
    for (int i = 0; i < 6; ++i) sq[i] = __ffma2_rn(w[i + 1], w[i + 1], nz);
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // ks_rhs_sq
        const float2 ll = w[i], l = w[i + 1], c = w[i + 2], r = w[i + 3], rr = w[i + 4];
        const float2 conv = __ffma2_rn(sq[i], dup2(-1.0f), sq[i + 2]);
        const float2 sec = __ffma2_rn(dup2(-2.0f), c, __fadd2_rn(l, r));
        const float2 f1 = __fadd2_rn(__ffma2_rn(dup2(-4.0f), l, ll), __ffma2_rn(dup2(6.0f), c, nz));
        const float2 fourth = __fadd2_rn(__ffma2_rn(dup2(-4.0f), r, f1), rr);
        if constexpr (POW2) {
            rhs[i] = __ffma2_rn(fourth, dup2(p.d4), __ffma2_rn(conv, dup2(p.c4), __ffma2_rn(sec, dup2(p.d2), nz)));
        } else {
            const float2 s = __fadd2_rn(__ffma2_rn(conv, dup2(p.c4), nz), __ffma2_rn(sec, dup2(p.d2), nz));
            rhs[i] = __fadd2_rn(s, __ffma2_rn(fourth, dup2(p.d4), nz));
        }
    }
}

// Two levels: the predictor on [lo1, hi1) (row 0 -> row 1), then, unless LAST, the
// corrector on [lo2, hi2) (row 1 -> row 0), in n groups of four positions from
// base, C groups (thread, thread + block, ...) per thread.  All ranges are even.  DOWN: positions outside the
// predictor's range hold imported u* in row 1.
template <int C, bool POW2, bool DOWN, bool LAST>
__device__ __forceinline__ void ks_pair_levels(const Params<float> &p, float2 *rows, int PS, int base, int n, int lo1,
                                               int hi1, int lo2, int hi2) {
    float2 *u0 = rows, *u1 = rows + PS, *s0 = rows + 2 * PS, *s1 = rows + 3 * PS;
    float2 u[C][4], s[C][4];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const int g = (int)threadIdx.x + c * (int)blockDim.x, x0 = base + 4 * g, k = (base >> 2) + g + 1;
        if (g < n) {
            float2 w[8], rhs[4];
            pair_load(u1, k - 1, w[0], w[1]);
            pair_load(u0, k, w[2], w[3]);
            pair_load(u1, k, w[4], w[5]);
            pair_load(u0, k + 1, w[6], w[7]);
            ks_rhs_pairs<POW2>(p, w, rhs);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                u[c][i] = w[i + 2];
                s[c][i] = __ffma2_rn(__ffma2_rn(dup2(p.dth), rhs[i], dup2(p.nz)), dup2(-1.0f), u[c][i]);
            }
            if (x0 >= lo1 && x0 + 2 <= hi1) pair_store(s0, k, s[c][0], s[c][1]);
            else if (DOWN) pair_load(s0, k, s[c][0], s[c][1]);
            if (x0 + 2 >= lo1 && x0 + 4 <= hi1) pair_store(s1, k, s[c][2], s[c][3]);
            else if (DOWN) pair_load(s1, k, s[c][2], s[c][3]);
        }
    }
    __syncthreads();
    if constexpr (!LAST) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int g = (int)threadIdx.x + c * (int)blockDim.x, x0 = base + 4 * g, k = (base >> 2) + g + 1;
            if (g < n) {
                float2 w[8], rhs[4];
                pair_load(s1, k - 1, w[0], w[1]);
                w[2] = s[c][0], w[3] = s[c][1], w[4] = s[c][2], w[5] = s[c][3];
                pair_load(s0, k + 1, w[6], w[7]);
                ks_rhs_pairs<POW2>(p, w, rhs);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    u[c][i] = __fadd2_rn(u[c][i], __ffma2_rn(dup2(-p.dt), rhs[i], dup2(p.nz)));
                if (x0 >= lo2 && x0 + 2 <= hi2) pair_store(u0, k, u[c][0], u[c][1]);
                if (x0 + 2 >= lo2 && x0 + 4 <= hi2) pair_store(u1, k, u[c][2], u[c][3]);
            }
        }
        __syncthreads();
    }
}

template <int MODE, int C, bool POW2>
__device__ __forceinline__ void ks_pair_block(const Params<float> &p, const PairTile &A, const PairTile &B, float2 *rows,
                                              const int W) {
    constexpr int R = 2;
    const int PS = pair_plane(W), h = W >> 1, H = W / (2 * R);
    for (int i = threadIdx.x; i < W; i += blockDim.x) {
        if constexpr (MODE == MODE_UP) {
            rows[pair_at(PS, 0, i)] = make_float2(A.state[A.base + i], B.state[B.base + i]);
        } else if (i < h) {
            rows[pair_at(PS, 0, i)] = make_float2(A.sl[i], B.sl[i]);
            rows[pair_at(PS, 1, i - R)] = make_float2(A.sl[h + i], B.sl[h + i]);
        } else {
            rows[pair_at(PS, 0, i)] = make_float2(A.sr[i - h], B.sr[i - h]);
            rows[pair_at(PS, 1, i + R)] = make_float2(A.sr[i], B.sr[i]);
        }
    }
    __syncthreads();
    if constexpr (MODE != MODE_UP) {
        for (int j = 1; j < H; j += 2)
            ks_pair_levels<C, POW2, true, false>(p, rows, PS, h - 2 * j - 2, j + 1, h - 2 * j, h + 2 * j, h - 2 * j - 2,
                                              h + 2 * j + 2);
    }
    if constexpr (MODE == MODE_DOWN) {
        for (int i = threadIdx.x; i < W; i += blockDim.x) {
            const float2 v = rows[pair_at(PS, 0, i)];
            A.state[wrap_pos(A.base + i, A.nx)] = v.x;
            B.state[wrap_pos(B.base + i, B.nx)] = v.y;
        }
    } else {
        int u = 1;
        for (; u + 1 < H; u += 2)
            ks_pair_levels<C, POW2, false, false>(p, rows, PS, 2 * u - 2, W / 4 - u + 1, 2 * u, W - 2 * u, 2 * u + 2,
                                               W - 2 * u - 2);
        ks_pair_levels<C, POW2, false, true>(p, rows, PS, 2 * u - 2, W / 4 - u + 1, 2 * u, W - 2 * u, 0, 0);  // u = H - 1
        for (int i = threadIdx.x; i < W; i += blockDim.x) {
            const float2 v = rows[pair_at(PS, 0, i)];
            if (i < h) {
                const float2 s = rows[pair_at(PS, 1, i + R)];
                A.sl[i] = v.x, B.sl[i] = v.y;
                A.sl[h + i] = s.x, B.sl[h + i] = s.y;
            } else {
                const float2 s = rows[pair_at(PS, 1, i - R)];
                A.sr[i - h] = v.x, B.sr[i - h] = v.y;
                A.sr[i] = s.x, B.sr[i] = s.y;
            }
        }
    }
}

// Tiles 2b and 2b + 1 of one domain (ntile tiles launched; the last block of an
// odd count runs its tile in both halves, both storing the same values).
template <int MODE, int C, bool POW2>
__global__ void __launch_bounds__(256 / C, (C == 2 ? 8 : 5))
    k_swept_ks_pair(const Params<float> p, float *state, float *slots, const int W, const int phase, const int64_t ntile) {
    extern __shared__ __align__(16) unsigned char sw_smem[];
    wait_for_previous_launch();
    const int64_t t0 = 2 * (int64_t)blockIdx.x, t1 = t0 + 1 < ntile ? t0 + 1 : t0;
    ks_pair_block<MODE, C, POW2>(p, pair_tile(state, slots, W, phase, t0, p.nx), pair_tile(state, slots, W, phase, t1, p.nx),
                              reinterpret_cast<float2 *>(sw_smem), W);
}
// The same over an ensemble's tiles; a pair may belong to two domains (KS is
// periodic: a level never looks at a cell's place in its domain).
template <int MODE, int C, bool POW2>
__global__ void __launch_bounds__(256 / C, (C == 2 ? 8 : 5))
    k_swept_ks_pair_batch(const Params<float> p, float *state, float *slots, const BatchDev b, const int W, const int phase) {
    extern __shared__ __align__(16) unsigned char sw_smem[];
    wait_for_previous_launch();
    const int64_t g0 = 2 * (int64_t)blockIdx.x, g1 = g0 + 1 < b.n_tiles ? g0 + 1 : g0;
    auto tile = [&](int64_t g) {
        const int d = b.tile_dom[g / b.split];
        const int64_t off = b.off[d];
        return pair_tile(state + off, slots + 2 * off, W, phase, g - b.tile0[d] * b.split, b.off[d + 1] - off);
    };
    ks_pair_block<MODE, C, POW2>(p, tile(g0), tile(g1), reinterpret_cast<float2 *>(sw_smem), W);
}

// Whether a pass over ntile tiles of width W pairs them (0: no), and the
// position groups per thread.  Below one tile per SM a pair halves the SMs at
// work (1024 cells: 0.82 against 0.78 ms for 1024 steps at 152 tiles, 0.82
// against 0.91 at 304; between three and four tiles per SM the two are within
// 2 %, and pairs win from there on).  128-cell tiles run in one warp's registers
// without barriers (k_swept_ks_warp) and lose to pairs only where those fill the
// SMs (equal at 8 tiles per SM, 1.25x at 16, 1.65x at 2^15 tiles); 160-cell tiles,
// whose second warp has 8 threads, are 4 % faster grouped at 8192 tiles.  Two groups
// per thread keep more of a block's warps at work as a triangle narrows, and
// half as many warps per block let more blocks share an SM: 3 to 6 % faster
// from 768 cells up where there is a full wave of such blocks (8 per SM),
// slower below (1.07 against 0.82 ms at 304 tiles) and on narrower tiles.
inline int pair_chunks(int W, int64_t ntile) {
    int dev = 0, sms = 0;
    if ((W != 128 && W < 192) || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    if (ntile <= (W == 128 ? 8 : 1) * (int64_t)sms) return 0;
    return W >= 768 && W % 256 == 0 && ntile >= 16 * (int64_t)sms ? 2 : 1;
}

template <int MODE, int C>
inline cudaError_t launch_ks_pair_mode(const Params<float> &p, float *st, float *sl, int W, int phase, int64_t ntile, cudaStream_t s) {
    const unsigned grid = (unsigned)((ntile + 1) / 2);
    const size_t smem = pair_smem_bytes(W);
    if (p.ks_form == KS_POW2) return launch_dependent(k_swept_ks_pair<MODE, C, true>, grid, W / 4 / C, smem, s, p, st, sl, W, phase, ntile);
    return launch_dependent(k_swept_ks_pair<MODE, C, false>, grid, W / 4 / C, smem, s, p, st, sl, W, phase, ntile);
}
template <int C>
inline cudaError_t launch_ks_pair(const Params<float> &p, int mode, int phase, float *st, float *sl, int64_t nx, int W,
                                  cudaStream_t s) {
    switch (mode) {
    case MODE_UP: return launch_ks_pair_mode<MODE_UP, C>(p, st, sl, W, phase, nx / W, s);
    case MODE_DIAMOND: return launch_ks_pair_mode<MODE_DIAMOND, C>(p, st, sl, W, phase, nx / W, s);
    default: return launch_ks_pair_mode<MODE_DOWN, C>(p, st, sl, W, phase, nx / W, s);
    }
}
template <int MODE, int C>
inline cudaError_t launch_ks_pair_batch_mode(const Params<float> &p, float *st, float *sl, const BatchDev &b, int W, int phase,
                                      cudaStream_t s) {
    const unsigned grid = (unsigned)((b.n_tiles + 1) / 2);
    const size_t smem = pair_smem_bytes(W);
    if (p.ks_form == KS_POW2) return launch_dependent(k_swept_ks_pair_batch<MODE, C, true>, grid, W / 4 / C, smem, s, p, st, sl, b, W, phase);
    return launch_dependent(k_swept_ks_pair_batch<MODE, C, false>, grid, W / 4 / C, smem, s, p, st, sl, b, W, phase);
}
template <int C>
inline cudaError_t launch_ks_pair_batch(const Params<float> &p, int mode, int phase, float *st, float *sl,
                                        const BatchDev &b, int W, cudaStream_t s) {
    switch (mode) {
    case MODE_UP: return launch_ks_pair_batch_mode<MODE_UP, C>(p, st, sl, b, W, phase, s);
    case MODE_DIAMOND: return launch_ks_pair_batch_mode<MODE_DIAMOND, C>(p, st, sl, b, W, phase, s);
    default: return launch_ks_pair_batch_mode<MODE_DOWN, C>(p, st, sl, b, W, phase, s);
    }
}
#endif  // SW_KS_DIVIDE_TU

SW_KERNELS_END
