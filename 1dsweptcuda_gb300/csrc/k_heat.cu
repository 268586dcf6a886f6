// HEAT kernels (reference: Heat1D_SweptShared.cu:121-408), float and double instances.
#include "engine.cuh"
#include "persistent.cuh"
#include "swept_heat.cuh"

namespace sw {
namespace {
// FP32 with four cells per thread takes four levels per exchange where heat4_tiles says so (swept_heat.cuh).
template <typename T>
cudaError_t launch_swept_heat(const void *vp, int mode, int phase, void *state, void *slots, int64_t nx, int W, int threads,
                              cudaStream_t s) {
    if constexpr (sizeof(T) == 4) {
        if (heat4_tiles(W, nx / W) && swept_threads_for<SW_HEAT, T>(W, threads) * 4 == W)
            return launch_swept_heat4(*static_cast<const Params<float> *>(vp), mode, phase, static_cast<float *>(state),
                                      static_cast<float *>(slots), nx, W, s);
    }
    return launch_swept<SW_HEAT, T>(vp, mode, phase, state, slots, nx, W, threads, s);
}
template <typename T>
Ops make_ops() {
    using Sc = Scheme<SW_HEAT, T>;
    Ops o{};
    o.problem = SW_HEAT;
    o.prec = (int)sizeof(T);
    o.R = Sc::R;
    o.S = Sc::S;
    o.C = 1;
    o.cell = sizeof(typename Sc::G);
    o.max_threads = Sc::MAXT;
    o.classic = launch_classic<SW_HEAT, T>;
    o.swept = launch_swept_heat<T>;
    o.persistent = launch_persistent<SW_HEAT, T>;
    o.pack = nullptr;
    o.unpack = nullptr;
    o.swept_smem = smem_of<SW_HEAT, T>;
    o.batch_swept = launch_swept_batch<SW_HEAT, T>;
    o.batch_classic = launch_classic_batch<SW_HEAT, T>;
    o.batch_persistent = launch_persistent_batch<SW_HEAT, T>;
    return o;
}
}  // namespace

const Ops *heat_ops(int prec) {
    static const Ops f = make_ops<float>();
    static const Ops d = make_ops<double>();
    return prec == 4 ? &f : (prec == 8 ? &d : nullptr);
}
}  // namespace sw
