// fast_served.cu - the FAST_FP32 kernels of a queue of many instances.
#include "fast_kernel.cuh"

namespace dsmc {
namespace {

template <int kT, int kB, int kMode>
constexpr ServedKernel served() { return fast_kernel<kT, kB, kMode, 1, FastArgsT<float>, float>; }

template <int kT, int kB>
ServedKernel by_mode(int mode) {
    return mode == 2 ? served<kT, kB, 2>() : mode == 1 ? served<kT, kB, 1>() : served<kT, kB, 0>();
}

}  // namespace

// Register budgets: 0: 256 x 2 (128 registers a thread), 1: 256 x 3 (80), 2: 128 x 3 (168),
// 3: 128 x 2 (255), 4: 128 x 4 (128), 5: 128 x 5 (96). The lean loops (modes 1 and 2) exist for
// budgets 0, 2, 4 and 5; elsewhere the general loop runs.
ServedKernel served_kernel(int variant, int mode) {
    switch (variant) {
        case 1: return served<256, 3, 0>();
        case 2: return by_mode<128, 3>(mode);
        case 3: return served<128, 2, 0>();
        case 4: return by_mode<128, 4>(mode);
        case 5: return by_mode<128, 5>(mode);
        default: return by_mode<256, 2>(mode);
    }
}

}  // namespace dsmc
