// fast_one64.cu - the FAST_FP64 kernels of a solve of one instance.
#include "fast_kernel.cuh"

namespace dsmc {
namespace {

template <int kB, int kMode, int kUnroll = 1>
constexpr OneKernel<double> one() { return fast_kernel<128, kB, kMode, kUnroll, OneArgsT<double>, double>; }

template <int kB>
OneKernel<double> by_mode(int mode) {
    return mode == 1 ? one<kB, 1>() : mode == 2 ? one<kB, 2>() : one<kB, 0>();
}

}  // namespace

OneKernel<double> one_kernel64(int blocks_per_sm, int mode, long long lanes_per_sm) {
    if (lanes_per_sm <= kSparsePerSm && mode == 1) return one<4, 1, kSparseUnroll>();
    if (blocks_per_sm == 5) return one<5, 1>();   // the lean loop only
    return blocks_per_sm == 3 ? by_mode<3>(mode) : by_mode<4>(mode);
}

}  // namespace dsmc
