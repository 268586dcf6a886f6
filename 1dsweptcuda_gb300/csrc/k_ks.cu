// KS kernels (reference: KS1D_SweptShared.cu:111-394), float and double instances.
#include "engine.cuh"
#include "persistent.cuh"
#include "swept_pair.cuh"

namespace sw {
namespace {
// FP32 with four cells per thread runs two tiles per block where pair_chunks
// says so (swept_pair.cuh), everything else the kernels of engine.cuh and
// persistent.cuh.
template <typename T>
cudaError_t launch_swept_ks(const void *vp, int mode, int phase, void *state, void *slots, int64_t nx, int W, int threads,
                            cudaStream_t s) {
#ifndef SW_KS_DIVIDE_TU
    if constexpr (sizeof(T) == 4) {
        const int c = swept_threads_for<SW_KS, T>(W, threads) * 4 == W ? pair_chunks(W, nx / W) : 0;
        const Params<T> &p = *static_cast<const Params<T> *>(vp);
        T *st = static_cast<T *>(state), *sl = static_cast<T *>(slots);
        if (c == 1) return launch_ks_pair<1>(p, mode, phase, st, sl, nx, W, s);
        if (c == 2) return launch_ks_pair<2>(p, mode, phase, st, sl, nx, W, s);
    }
#endif
    return launch_swept<SW_KS, T>(vp, mode, phase, state, slots, nx, W, threads, s);
}
template <typename T>
cudaError_t launch_swept_ks_batch(const void *vp, int mode, int phase, void *state, void *slots, const void *bt, int W,
                                  int threads, cudaStream_t s) {
#ifndef SW_KS_DIVIDE_TU
    if constexpr (sizeof(T) == 4) {
        const BatchDev &b = *static_cast<const BatchDev *>(bt);
        const int c = swept_threads_for<SW_KS, T>(W, threads) * 4 == W ? pair_chunks(W, b.n_tiles) : 0;
        const Params<T> &p = *static_cast<const Params<T> *>(vp);
        T *st = static_cast<T *>(state), *sl = static_cast<T *>(slots);
        if (c == 1) return launch_ks_pair_batch<1>(p, mode, phase, st, sl, b, W, s);
        if (c == 2) return launch_ks_pair_batch<2>(p, mode, phase, st, sl, b, W, s);
    }
#endif
    return launch_swept_batch<SW_KS, T>(vp, mode, phase, state, slots, bt, W, threads, s);
}
template <typename T>
Ops make_ops() {
    using Sc = Scheme<SW_KS, T>;
    Ops o{};
    o.problem = SW_KS;
    o.prec = (int)sizeof(T);
    o.R = Sc::R;
    o.S = Sc::S;
    o.C = 1;
    o.cell = sizeof(typename Sc::G);
    o.max_threads = Sc::MAXT;
    o.classic = launch_classic<SW_KS, T>;
    o.swept = launch_swept_ks<T>;
    o.persistent = launch_persistent<SW_KS, T>;
    o.pack = nullptr;
    o.unpack = nullptr;
    o.swept_smem = smem_of<SW_KS, T>;
    o.batch_swept = launch_swept_ks_batch<T>;
    o.batch_classic = launch_classic_batch<SW_KS, T>;
    o.batch_persistent = launch_persistent_batch<SW_KS, T>;
    return o;
}
}  // namespace

#ifdef SW_KS_DIVIDE_TU
const Ops *ks_divide_ops(int prec) {
#else
const Ops *ks_ops(int prec) {
#endif
    static const Ops f = make_ops<float>();
    static const Ops d = make_ops<double>();
    return prec == 4 ? &f : (prec == 8 ? &d : nullptr);
}
}  // namespace sw
