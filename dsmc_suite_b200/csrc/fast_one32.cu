// fast_one32.cu - the FAST_FP32 kernels of a solve of one instance, and the fed-state FP32 push.
#include "dsmc_kernels.h"
#include "fast_kernel.cuh"

namespace dsmc {
namespace {

template <int kB, int kMode>
constexpr OneKernel<float> one() { return fast_kernel<128, kB, kMode, 1, OneArgsT<float>, float>; }

template <int kB>
OneKernel<float> by_mode(int mode) {
    switch (mode) {
        case 1: return one<kB, 1>();
        case 2: return one<kB, 2>();
        case 4: return one<kB, 4>();
        case 5: return one<kB, 5>();
        default: return one<kB, 0>();
    }
}

// Fed-state FP32 push (dsmc_push_host with FAST_FP32).
__global__ void push_fp32_kernel(const dsmc_params p, long long n, int nsteps, double *pos,
                                 double *vel, int *status, int *taken) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Hot h;
    const double s[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
    const double v[3] = {vel[3 * i], vel[3 * i + 1], vel[3 * i + 2]};
    set_pos(h, s);
    set_vel(h, v);
    const double R0 = sqrt(s[0] * s[0] + s[1] * s[1] + s[2] * s[2]);
    const double g0 = p.GM / (R0 * R0 * R0);
    for (int k = 0; k < 3; k++) h.oa[k] = -static_cast<float>(g0 * s[k] * p.dt_step);
    const float GM = static_cast<float>(p.GM * p.dt_step), dt = static_cast<float>(p.dt_step);
    const float c1 = static_cast<float>(1.5 * p.dt_step);
    const float c2 = static_cast<float>(p.dt_step / 6.0);
    const float rl2 = static_cast<float>(p.Radii * p.Radii);
    const float re2 = static_cast<float>(p.max_height * p.max_height);
    PosT<float> q;
    start_pos(h, q);
    int st = 0, k = 0;
    for (; k < nsteps && st == 0; k++) {
        float d[3];
        gravity(q, GM);
        verlet_step(h, q, dt, c1, c2, d);
        st = q.r2 <= rl2 ? 1 : (q.r2 >= re2 ? 2 : 0);
    }
    double so[3], vo[3];
    get_pos(h, so);
    get_vel(h, vo);
    for (int j = 0; j < 3; j++) { pos[3 * i + j] = so[j]; vel[3 * i + j] = vo[j]; }
    status[i] = st;
    taken[i] = k;
}

}  // namespace

// Which loop (see fast_kernel and warp_kernel for both sides' times): the warp's step loop for few
// lanes per SM, in every mode that has one, and for the bulk where hops are long (ballistic config
// model) or events are most of the work (reference model); elsewhere the free-running lanes.
OneKernel<float> one_kernel32(int blocks_per_sm, int mode, bool long_hops, long long lanes_per_sm) {
    if (lanes_per_sm <= kSparsePerSm) {
        if (mode == 1) return lanes_per_sm <= kTinyPerSm ? warp_kernel<128, 4, 1, 12> : warp_kernel<128, 4, 1, 8>;
        if (mode == 2) return warp_kernel<128, 4, 2, 12>;
        if (mode == 3) return warp_kernel<128, 4, 3, 8>;
        if (mode == 5) return warp_kernel<128, 4, 5, 12>;
    }
    if (mode == 3) return blocks_per_sm == 5 ? warp_kernel<128, 5, 3, 8> : warp_kernel<128, 4, 3, 8>;
    if (mode == 1 && long_hops) return blocks_per_sm == 5 ? warp_kernel<128, 5, 1, 8> : warp_kernel<128, 4, 1, 8>;
    return blocks_per_sm == 5 ? by_mode<5>(mode) : by_mode<4>(mode);
}

cudaError_t launch_push_fp32(const dsmc_params &p, long long n, int nsteps, double *pos,
                             double *vel, int *status, int *taken, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    push_fp32_kernel<<<static_cast<unsigned>((n + 127) / 128), 128, 0, stream>>>(p, n, nsteps, pos, vel,
                                                                                status, taken);
    return cudaGetLastError();
}

}  // namespace dsmc
