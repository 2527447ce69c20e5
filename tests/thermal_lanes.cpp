// Host build of the thermal kernels (csrc/kernel_thermal.cu up to its launcher, as thermal_lanes.inc).
// Each lane of one warp is a fiber that runs until the next warp-wide call before the next lane
// starts: an order that CUDA allows, and the one in which a missing synchronisation shows.
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <vector>

#define __device__
#define __global__
#define __shared__
#define __forceinline__ inline
using std::max;
using std::min;
struct Dim { int x; };
static Dim threadIdx, blockIdx, blockDim;

namespace {
constexpr int kLanes = 32;
ucontext_t lane_ctx[kLanes], main_ctx;
double slot[kLanes];
bool running[kLanes];

void meet() { swapcontext(&lane_ctx[threadIdx.x], &main_ctx); }   // back once every lane has come

double gather(double v, int src) {
    slot[threadIdx.x] = v;
    meet();
    const double r = slot[src];
    meet();
    return r;
}
}  // namespace

static int __clz(int v) { return __builtin_clz(static_cast<unsigned>(v)); }
static void __syncwarp() { meet(); }
static void __syncthreads() { meet(); }   // one warp a block here
static double __shfl_sync(unsigned, double v, int src, int width) {
    return gather(v, (threadIdx.x & ~(width - 1)) + (src & (width - 1)));
}
static bool __any_sync(unsigned, bool b) {
    slot[threadIdx.x] = b;
    meet();
    bool r = false;
    for (double x : slot) r = r || x != 0.0;
    meet();
    return r;
}

#include "thermal_lanes.inc"

namespace dsmc {
namespace {
double thermal_smem[1 << 14];
ThermalArgs the_args;
bool the_shared;

void lane_main() {
    if (the_shared) thermal_shared_kernel<8>(the_args);
    else thermal_column_kernel(the_args);
    running[threadIdx.x] = false;
    swapcontext(&lane_ctx[threadIdx.x], &main_ctx);
}
}  // namespace
}  // namespace dsmc

// Surface temperatures of ncol <= 32 columns of h depths, by one warp: 8 lanes a column on shared
// profiles (4 columns a block), or one lane a column. reverse: the last lane runs first.
extern "C" int thermal_lanes(int shared, int reverse, int ncol, int h, int n_sub, double R, double k_over_dr,
                             double a_last, const double *p, const double *LH, const double *consts,
                             const double *flux, const double *T_init, const double *cp, const double *piv,
                             const double *rcp, double *T_surface) {
    using namespace dsmc;
    const int cols = shared ? kLanes / 8 : kLanes;
    if (shared && h * (3 + 2 * cols) > (1 << 14)) return -1;
    std::vector<double> q(static_cast<size_t>(h) * ncol), d(q.size());
    ThermalArgs &a = the_args;
    a.ncol = ncol; a.h = h; a.n_sub = n_sub;
    a.R = R; a.k_over_dr = k_over_dr; a.a_last = a_last;
    std::copy(p, p + 5, a.p);
    std::copy(LH, LH + 5, a.LH);
    a.tran_p = consts[0]; a.tran_LH = consts[1]; a.mmol = consts[2];
    a.flux = flux; a.T_init = T_init; a.cp = cp; a.piv = piv; a.rcp = rcp;
    a.qT = q.data(); a.dp = d.data(); a.T_surface = T_surface;
    the_shared = shared != 0;
    std::vector<char> stack(kLanes << 16);
    blockDim.x = kLanes;
    for (blockIdx.x = 0; blockIdx.x * cols < ncol; blockIdx.x++) {
        for (int l = 0; l < kLanes; l++) {
            getcontext(&lane_ctx[l]);
            lane_ctx[l].uc_stack.ss_sp = stack.data() + (static_cast<size_t>(l) << 16);
            lane_ctx[l].uc_stack.ss_size = 1 << 16;
            lane_ctx[l].uc_link = nullptr;
            makecontext(&lane_ctx[l], lane_main, 0);
            running[l] = true;
        }
        for (bool any = true; any;) {
            any = false;
            for (int k = 0; k < kLanes; k++) {
                const int l = reverse ? kLanes - 1 - k : k;
                if (!running[l]) continue;
                threadIdx.x = l;
                swapcontext(&main_ctx, &lane_ctx[l]);
                any = any || running[l];
            }
        }
    }
    return 0;
}
