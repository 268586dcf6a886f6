// FP32 Heat swept passes, four levels per exchange through shared memory.
//
// The four-cells-per-thread path (tile_span4) was bound by shared memory: per level
// and four cells, two 16-byte reads and four 4-byte writes a quarter of whose banks
// collide, 24 cycles a warp for 16 FP32 instructions.  Here a thread takes eight
// cells and reads them with four more on each side (four 16-byte reads), and computes
// four levels in registers, the outer cells' again as its neighbours do (44 updates
// for 32); then it writes eight values: 24 cycles a warp for 1024 updates.  2^22 cells,
// tile 1024, 4096 steps: 11.76 -> 6.48 ms; now bound by instruction issue (11 FP32
// instructions for 8 needed, the part of a triangle that its warps overhang, two
// barriers per four levels).
//
//  * Quads of cells alternate between two planes, so that the 16-byte accesses of
//    consecutive threads are 16 bytes apart.
//  * Row 0 is rewritten in place, between two barriers.  A round's range starts and
//    ends at a multiple of four cells, so which cells of a thread lie outside a level
//    is known from which of a few places the thread has; every thread runs the same
//    instructions, and only the assignments (down part: imported values stay) or the
//    stores (up part: a cell keeps its last even and odd level) of the threads at
//    the edges differ.  (Tested per cell and level instead, most warps hold an edge and
//    ran 3.5 times as long.)
//  * An insulated end mirrors a neighbour; only the warp whose windows hold one tests for it.
//  * The live range is packed onto the lowest threads as in tile_span4.
//
// Slots, modes, level ranges and arithmetic (heat_step) are those of swept_tile, so
// the results are the same bit for bit.
#pragma once

#include <cuda_runtime.h>

#include "engine.cuh"

SW_KERNELS_BEGIN

// Rows: position x of row r, -8 <= x < W + 8; quad q = (x + 8) / 4 in plane q % 2.
__host__ __device__ constexpr int heat_plane(int W) { return (W + 16) >> 1; }  // floats per plane
__host__ __device__ constexpr size_t heat_smem_bytes(int W) { return sizeof(float) * 4 * (size_t)heat_plane(W); }
__device__ __forceinline__ int heat_at(int PS, int row, int x) {
    const int q = (x + 8) >> 2;
    return (2 * row + (q & 1)) * PS + (q >> 1) * 4 + (x & 3);
}
// The 16 cells from x0 - 4 on, x0 a multiple of 8 (k = x0 / 8 + 1: plane 0's quad of x0).
__device__ __forceinline__ void heat_window(const float *row, int PS, int k, float (&w)[16]) {
    load4(row + PS + 4 * (k - 1), w);
    load4(row + 4 * k, w + 4);
    load4(row + PS + 4 * k, w + 8);
    load4(row + 4 * (k + 1), w + 12);
}
__device__ __forceinline__ void heat_put(float *row, int PS, int k, const float (&w)[16]) {
    *reinterpret_cast<float4 *>(row + 4 * k) = make_float4(w[4], w[5], w[6], w[7]);
    *reinterpret_cast<float4 *>(row + PS + 4 * k) = make_float4(w[8], w[9], w[10], w[11]);
}

// heat_step at window cell i; ENDS: insulated ends at window cells `first` and `last`.
template <bool ENDS>
__device__ __forceinline__ float heat_cell(const Params<float> &p, const float (&w)[16], int i, int first, int last) {
    float l = w[i - 1], r = w[i + 1];
    if constexpr (ENDS) {
        if (i == first) l = r;
        if (i == last) r = l;
    }
    return heat_step(p, l, w[i], r);
}

// Levels j + 1 .. j + 4 of the down part, level l on [h - l, h + l), at the thread's cells x0 .. x0 + 7: the fourth in w.
// ODD: j is 4 (else 0) mod 8.
template <bool ODD, bool ENDS>
__device__ __forceinline__ void heat_down_cells(const Params<float> &p, const float *rows, int PS, int h, int j, int x0,
                                                int first, int last, float (&w)[16]) {
    const int k = (x0 >> 3) + 1;
    // The thread's place.  j = 0 mod 8: its last (first) four cells enter in this round (L0, R0); or its first (last)
    // cells entered in the last round, and two imported cells of row 1 lie in its window (L1, R1).  j = 4 mod 8: its
    // first (last) four cells enter (L0, R0).
    const bool L0 = x0 == (ODD ? h - j - 4 : h - j - 8), R0 = x0 == (ODD ? h + j - 4 : h + j);
    const bool L1 = !ODD && x0 == h - j, R1 = !ODD && x0 == h + j - 8;
    constexpr int E = ODD ? 6 : 10;  // L0: window cells 1 .. E lie outside level 1; one fewer in each level after it
    float o[16];
    heat_window(rows, PS, k, w);
    if (L0 || L1 || R0 || R1) heat_window(rows + 2 * PS, PS, k, o);
#pragma unroll
    for (int i = 1; i < 15; ++i) {
        const float v = heat_cell<ENDS>(p, w, i, first, last);
        if (!((i <= E && L0) || (15 - i <= E && R0) || (i <= 2 && L1) || (15 - i <= 2 && R1))) o[i] = v;
    }
#pragma unroll
    for (int i = 2; i < 14; ++i) {
        const float v = heat_cell<ENDS>(p, o, i, first, last);
        if (!((i <= E - 1 && L0) || (15 - i <= E - 1 && R0))) w[i] = v;
    }
#pragma unroll
    for (int i = 3; i < 13; ++i) {
        const float v = heat_cell<ENDS>(p, w, i, first, last);
        if (!((i <= E - 2 && L0) || (15 - i <= E - 2 && R0))) o[i] = v;
    }
#pragma unroll
    for (int i = 4; i < 12; ++i) {
        const float v = heat_cell<ENDS>(p, o, i, first, last);
        if (!((i <= E - 3 && L0) || (15 - i <= E - 3 && R0))) w[i] = v;
    }
}

// Whether the warp's windows from x0 - 4 on hold an insulated end (window cells first, last).
__device__ __forceinline__ bool heat_warp_ends(bool live, int first, int last) {
    return __any_sync(0xffffffffu, live && ((unsigned)first < 16u || (unsigned)last < 16u));
}

template <bool ODD, bool ENDS>
__device__ __forceinline__ void heat_down(const Params<float> &p, float *rows, int PS, int h, int j, Ends e) {
    const int base = (h - j - 4) & ~7, n = (h + j + 4 - base + 7) >> 3, x0 = base + 8 * (int)threadIdx.x;
    const bool live = (int)threadIdx.x < n;
    const int first = e.first - x0 + 4, last = e.last - x0 + 4;
    float w[16];
    if (ENDS && heat_warp_ends(live, first, last)) {
        if (live) heat_down_cells<ODD, true>(p, rows, PS, h, j, x0, first, last, w);
    } else if (live) {
        heat_down_cells<ODD, false>(p, rows, PS, h, j, x0, first, last, w);
    }
    __syncthreads();
    if (live) heat_put(rows, PS, (x0 >> 3) + 1, w);  // row 1 is read only at imported cells
    __syncthreads();
}

// Levels m + 1 .. m + 4 of the up part, level l on [l, W - l), at the thread's cells: into a, b, c and w.
template <bool ENDS>
__device__ __forceinline__ void heat_up_cells(const Params<float> &p, const float *rows, int PS, int x0, int first, int last,
                                              float (&a)[16], float (&b)[16], float (&c)[16], float (&w)[16]) {
    heat_window(rows, PS, (x0 >> 3) + 1, w);
#pragma unroll
    for (int i = 1; i < 15; ++i) a[i] = heat_cell<ENDS>(p, w, i, first, last);
#pragma unroll
    for (int i = 2; i < 14; ++i) b[i] = heat_cell<ENDS>(p, a, i, first, last);
#pragma unroll
    for (int i = 3; i < 13; ++i) c[i] = heat_cell<ENDS>(p, b, i, first, last);
#pragma unroll
    for (int i = 4; i < 12; ++i) w[i] = heat_cell<ENDS>(p, c, i, first, last);
}

template <bool ENDS>
__device__ __forceinline__ void heat_up(const Params<float> &p, float *rows, int PS, int W, int m, Ends e) {
    const int base = (m + 1) & ~7, n = (W - m - 1 - base + 7) >> 3, x0 = base + 8 * (int)threadIdx.x, k = (x0 >> 3) + 1;
    const bool live = (int)threadIdx.x < n;
    const int first = e.first - x0 + 4, last = e.last - x0 + 4;
    float w[16], a[16], b[16], c[16];
    if (ENDS && heat_warp_ends(live, first, last)) {
        if (live) heat_up_cells<true>(p, rows, PS, x0, first, last, a, b, c, w);
    } else if (live) {
        heat_up_cells<false>(p, rows, PS, x0, first, last, a, b, c, w);
    }
    __syncthreads();
    if (live) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {  // the quad of cells x .. x + 3
            const int x = x0 + 4 * q, i = 4 + 4 * q;
            float *r0 = rows + q * PS + 4 * k, *r1 = r0 + 2 * PS;
            if (x >= m + 4 && x + 4 <= W - m - 4) {
                *reinterpret_cast<float4 *>(r0) = make_float4(w[i], w[i + 1], w[i + 2], w[i + 3]);
                if (x == m + 4) r1[0] = c[i];  // the last odd level of cell m + 4
                if (x + 4 == W - m - 4) r1[3] = c[i + 3];
            } else if (x == m) {  // cell m + l leaves after level m + l
                r1[1] = a[i + 1], r1[2] = a[i + 2], r1[3] = c[i + 3];
                r0[2] = b[i + 2], r0[3] = b[i + 3];
            } else if (x + 4 == W - m) {
                r1[2] = a[i + 2], r1[1] = a[i + 1], r1[0] = c[i];
                r0[1] = b[i + 1], r0[0] = b[i];
            }
        }
    }
    __syncthreads();
}

template <bool ENDS>
__device__ __forceinline__ void heat_tile_down(const Params<float> &p, float *rows, int PS, int W, Ends e) {
    const int h = W >> 1;  // a multiple of 16
    for (int j = 0; j < h; j += 8) {
        heat_down<false, ENDS>(p, rows, PS, h, j, e);
        heat_down<true, ENDS>(p, rows, PS, h, j + 4, e);
    }
}
template <bool ENDS>
__device__ __forceinline__ void heat_tile_up(const Params<float> &p, float *rows, int PS, int W, Ends e) {
    for (int m = 0; m < W / 2; m += 4) heat_up<ENDS>(p, rows, PS, W, m, e);  // the last round's fourth level is empty
}

constexpr int kHeatMaxTile = 1024;
template <int MODE>
__global__ void __launch_bounds__(kHeatMaxTile / 8, 8)
    k_swept_heat4(const Params<float> p, float *state, float *slots, const int W, const int phase) {
    extern __shared__ __align__(16) unsigned char sw_smem[];
    float *rows = reinterpret_cast<float *>(sw_smem);
    wait_for_previous_launch();
    const int PS = heat_plane(W), h = W >> 1;
    const int64_t nx = p.nx, t = blockIdx.x, nhalf = nx / h, base = t * W + (int64_t)phase * h;
    const int64_t hl = (2 * t + phase) % nhalf, hr = (hl + 1 == nhalf) ? 0 : hl + 1;
    float *sl = slots + hl * W, *sr = slots + hr * W;
    for (int i = threadIdx.x; i < W; i += blockDim.x) {  // as tile_import_at
        if constexpr (MODE == MODE_UP) {
            rows[heat_at(PS, 0, i)] = state[base + i];
        } else if (i < h) {
            rows[heat_at(PS, 0, i)] = sl[i];
            rows[heat_at(PS, 1, i - 1)] = sl[h + i];
        } else {
            rows[heat_at(PS, 0, i)] = sr[i - h];
            rows[heat_at(PS, 1, i + 1)] = sr[i];
        }
    }
    __syncthreads();
    // The tile with the insulated ends runs loops of its own: their tests' registers would spill in the others'
    // (2^22 cells, tile 1024: 7.50 against 6.48 ms for 4096 steps).
    const Ends e = tile_ends(base, nx, W, 1);
    const bool ends = p.bc != SW_BC_PERIODIC && (e.first >= -1 || e.last >= -1);
    if constexpr (MODE != MODE_UP) {
        if (ends) heat_tile_down<true>(p, rows, PS, W, e);
        else heat_tile_down<false>(p, rows, PS, W, e);
    }
    if constexpr (MODE == MODE_DOWN) {
        for (int i = threadIdx.x; i < W; i += blockDim.x) state[wrap_pos(base + i, nx)] = rows[heat_at(PS, 0, i)];
    } else {
        if (ends) heat_tile_up<true>(p, rows, PS, W, e);
        else heat_tile_up<false>(p, rows, PS, W, e);
        for (int i = threadIdx.x; i < W; i += blockDim.x) {  // as tile_export_at
            const float v = rows[heat_at(PS, 0, i)];
            if (i < h) {
                sl[i] = v;
                sl[h + i] = rows[heat_at(PS, 1, i + 1)];
            } else {
                sr[i - h] = v;
                sr[i] = rows[heat_at(PS, 1, i - 1)];
            }
        }
    }
}

// Tiles of whole warps (W / 8 threads), and 192 to 224 cells in one warp; below 768 cells where the pass has two tiles
// per SM.  us for W cells per tile, insulated ends, 4 cycles (2 at 2^20 cells and above), tile_span4 -> here: 2^22 cells
// 192 877 -> 609, 256 922 -> 621, 512 1637 -> 1117, 768 2320 -> 1284, 1024 2971 -> 1619 (1.30e12 -> 2.36e12
// cell-updates/s); 2^18 cells 192 223 -> 216, 256 287 -> 238, 512 402 -> 386, 1024 731 -> 677; 2^12 cells 192 176 -> 181,
// 256 209 -> 217, 512 345 -> 349, 768 506 -> 484, 1024 668 -> 615.  Narrower tiles (equal at 128 and 64, 0.8x at 32) keep
// tile_span4, and so do the widths above 256 that leave a part-empty warp.  Of those only the narrow ones on 2^18 cells
// lose here (288 to 416 cells, 0.91x to 0.95x); us, tile_span4 -> here, 4 cycles at 2^18 cells, 2 at 2^20 and 2^22: 384
// 313 -> 340, 394 -> 353, 1294 -> 1090; 640 463 -> 438, 583 -> 429, 1997 -> 1189; 896 624 -> 575, 787 -> 484, 2654 ->
// 1525.  The line is not at that crossover yet.
inline bool heat4_tiles(int W, int64_t ntile) {
    if (W > kHeatMaxTile || (W % 256 != 0 && (W < 192 || W > 256))) return false;
    return W >= 768 || !few_tiles(ntile);
}

inline cudaError_t launch_swept_heat4(const Params<float> &p, int mode, int phase, float *st, float *sl, int64_t nx, int W,
                                      cudaStream_t s) {
    const unsigned grid = (unsigned)(nx / W);
    const unsigned block = (unsigned)(W / 8 + 31) & ~31u;  // whole warps
    const size_t smem = heat_smem_bytes(W);
    switch (mode) {
    case MODE_UP: return launch_dependent(k_swept_heat4<MODE_UP>, grid, block, smem, s, p, st, sl, W, phase);
    case MODE_DIAMOND: return launch_dependent(k_swept_heat4<MODE_DIAMOND>, grid, block, smem, s, p, st, sl, W, phase);
    default: return launch_dependent(k_swept_heat4<MODE_DOWN>, grid, block, smem, s, p, st, sl, W, phase);
    }
}

SW_KERNELS_END
