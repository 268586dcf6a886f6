// Internal interface between the C ABI (api.cu) and the per-problem kernel
// translation units (k_heat.cu, k_ks.cu, k_euler.cu).  Not installed.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/swept1d.h"

namespace sw {

// Kernel parameters: every constant of every scheme, in the run's precision.
// Passed by value (constant bank), so a launch never reads a __constant__
// symbol that another context might be rewriting.
template <typename T>
struct Params {
    T fo, fo2;                 // Heat: fourier, 1 - 2 fourier
    T c4, d2, d4, dt, dth;     // KS: 1/(4dx), 1/dx^2, 1/dx^4, dt, dt/2
    T gam, mgam, dtdx;         // Euler
    T bd[6];                   // Euler boundary states (rho, rho u, E) left, right
    int64_t nx;
    int bc;                    // SW_BC_MIRROR / PERIODIC / DIRICHLET
    int ks_form;               // KS: how c4, d2, d4 enter the right-hand side (enum KsForm)
    int d2_e;                  // KS_POW2: d2 = 2^d2_e
    T nz;                      // -0.0, the addend that makes an fma a plain product (paired FP32 path)
    int *status;               // device word a kernel sets when a bounded wait runs out (may be null)
};

// KS right-hand-side forms.  KS_POW2: c4, d2, d4 are exact powers of two, so
// their products fold into fused multiply-adds without changing a bit;
// KS_DIVIDE: c4, d2, d4 are the divisors 4dx, dx^2, dx^4 (SW_FLAG_KS_DIVIDE).
enum KsForm { KS_MULTIPLY = 0, KS_POW2 = 1, KS_DIVIDE = 2 };

// Device tables of an ensemble (see sw_run_batch): domain d holds cells
// [off[d], off[d+1]), its slots are the same range times two, its flags
// [2*tile0[d], ...); tile_dom maps a global tile of width W to its domain.
struct BatchDev {
    const int32_t *tile_dom;
    const int64_t *off;      // n_dom + 1 cell offsets
    const int64_t *tile0;    // first global tile of each domain
    const int32_t *blk_dom;  // domain of the first cell of each kClassicBlock-cell classic block
    int64_t n_tiles;
    int64_t n_cells;
    int32_t n_dom;
    int32_t group;  // the largest of 1, 2, 4 that divides every domain's tile count
    int32_t vec4;   // every domain length is a multiple of 4
    int32_t split;  // the launch's tiles are 1/split of the tables' (tail_tile)
};
constexpr int kClassicBlock = 256;  // threads (= cells) per block of the ensemble classic kernel

// Swept launch modes.
enum SweptMode { MODE_UP = 0, MODE_DIAMOND = 1, MODE_DOWN = 2 };

// Per (problem, precision) kernel table.  `params` points at a Params<T>
// of the table's precision.
struct Ops {
    int problem;
    int prec;        // 4 or 8
    int R;           // stencil radius per sub-step
    int S;           // sub-steps per time step
    int C;           // state components per cell on the host (1 or 3)
    size_t cell;     // bytes per cell in device layout
    int max_threads; // largest threads per block a swept kernel is built for
    // one classic sub-step (sub 0: predictor / heat step, 1: corrector)
    cudaError_t (*classic)(const void *params, const void *in, void *out, int sub, int64_t nx, int block,
                           cudaStream_t s);
    // one swept launch over all tiles of width W at `phase` (0 aligned, 1 shifted by W/2);
    // `threads` per block, 0 (or out of range) = the default for W
    cudaError_t (*swept)(const void *params, int mode, int phase, void *state, void *slots, int64_t nx, int W,
                         int threads, cudaStream_t s);
    // persistent swept variant: up-triangle, n_diamonds diamonds and the down-triangle in
    // one cooperative launch with per-half-tile phase flags; *status set non-zero on timeout.
    cudaError_t (*persistent)(const void *params, void *state, void *slots, unsigned *flags, int *status,
                              int64_t nx, int W, int threads, int64_t n_diamonds, cudaStream_t s);
    // Euler host layout (3 per cell) <-> device layout (4 per cell); null for Heat/KS
    cudaError_t (*pack)(const void *in3, void *out4, int64_t nx, cudaStream_t s);
    cudaError_t (*unpack)(const void *in4, void *out3, int64_t nx, cudaStream_t s);
    // dynamic shared memory a swept block of width W needs
    size_t (*swept_smem)(int W);
    // ensembles: `batch` points at a BatchDev (device tables), `threads` per block (0 = the default for W)
    cudaError_t (*batch_swept)(const void *params, int mode, int phase, void *state, void *slots, const void *batch,
                               int W, int threads, cudaStream_t s);
    cudaError_t (*batch_classic)(const void *params, const void *in, void *out, int sub, const void *batch, int block,
                                 cudaStream_t s);
    cudaError_t (*batch_persistent)(const void *params, void *state, void *slots, const void *batch, unsigned *flags,
                                    int *status, int W, int threads, int64_t n_diamonds, cudaStream_t s);
};

// The tile width of one more swept cycle (an up- and a down-triangle, two
// launches) that takes up to `rem` time steps left over after a run's whole
// cycles of width W, or 0: classic steps, S launches each, for the rest.  A width
// that divides W divides every domain of the run, and every (cell, sub-step)
// value is the same whatever tile it is computed in.
// A narrow cycle beats its classic steps where those are bound by launches and
// memory: us per step at 2^20 and 2^22 cells, cycle against classic: Heat FP32 128
// cells 1.5 and 4.8 against 1.8 and 5.0, 512 cells 0.9 and 3.1; KS FP32 128 cells
// 3.0 and 9.3 against 4.1 and 10.9, 512 cells 1.9 and 6.1; Heat FP64 128 cells 6.3
// and 24 against 7.3 and 25.  64 cells lose there (Heat FP32 2.8 and 10), but not
// on small domains (4096 cells: 0.8 against 1.7).  Euler takes none: the steps left
// over ran 0.4x to 1.0x as fast in narrow cycles, FP32 and FP64, 2^10 to 2^20 cells,
// tiles 128 to 1024.  FP64 KS takes none either: on large domains it is bound by
// arithmetic, which classic wastes none of (2^20 cells, tile 256, 31 steps: 1608 us
// against 1565).  On small ones launches bound it as they do the others, and narrow
// cycles would be the faster ones: 31 steps of tile 256 at 2^12 cells 141 against 173,
// 127 of tile 1024 585 against 1258, at 2^18 cells 2013 against 2162.
inline int tail_tile(const Ops &ops, bool divide, int W, int64_t cells, int64_t rem) {
    if (divide || ops.problem == SW_EULER || (ops.problem == SW_KS && ops.prec == 8)) return 0;
    const int least = cells <= ((int64_t)1 << 18) ? 64 : 128;
    for (int k = 2; W / k >= least; ++k)
        if (W % (32 * k) == 0 && W / k / (2 * ops.R * ops.S) <= rem) return W / k;
    return 0;
}

// The hybrid variant's host tile (host_tile.cu): the wrapping phase-1 tile of
// a domain computed on the CPU from its two slots (sl: the last half-tile's,
// sr: the first's); MODE_DIAMOND writes the slots back, MODE_DOWN the state's
// first and last half-tiles.  params: a Params<float or double>.
int host_tile_run(int problem, int prec, const void *params, int mode, void *sl, void *sr, void *state_first,
                  void *state_last, int W);

const Ops *heat_ops(int prec);
const Ops *ks_ops(int prec);
const Ops *ks_divide_ops(int prec);  // SW_FLAG_KS_DIVIDE (k_ks_div.cu)
const Ops *euler_ops(int prec);

inline const Ops *ops_for(int problem, int prec, int flags) {
    switch (problem) {
    case SW_HEAT: return heat_ops(prec);
    case SW_KS: return (flags & SW_FLAG_KS_DIVIDE) ? ks_divide_ops(prec) : ks_ops(prec);
    case SW_EULER: return euler_ops(prec);
    default: return nullptr;
    }
}

}  // namespace sw
