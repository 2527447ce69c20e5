// kernel_thermal.cu - the thermal model that feeds the DSMC phases (src/thermal/thermal_model.c
// of the reference), eight lanes or one thread per surface column. Compiled with -fmad=false: the
// column arithmetic follows the reference's FP64 operation order, so the Crank-Nicolson steps and the
// Thomas sweeps are bit-identical to the CPU's; only CUDA's log10 / pow / sqrt inside the surface
// energy balance may round differently in the last place from glibc's.
//
// Per column (td, fd), each of n_sub time steps (thermal_model.c:196-254):
//   1. surface temperature by bisection of the energy balance
//        F + k/dr T_1 - k/dr T - sigma T^4 - L(T) sqrt(m / (2 pi k_B T)) p(T) = 0
//      on [50, 300] K, the upper end growing x5 while both ends have one sign, until the bracket
//      is within 0.01 K (at most 30 iterations);
//   2. one implicit (Crank-Nicolson) diffusion step with the surface fixed and a zero-flux
//      bottom, by the Thomas algorithm.
// The coefficients of the tridiagonal system are the same for every column and step, so the
// forward-sweep terms that depend on them alone (c'_i, the pivots and their reciprocals) come from
// the host.
//
// The work is one chain per column: 467 dependent right-hand sides down, 467 substitutions up and
// about 17 balance evaluations per step, for 2,592 columns on 148 SMs, so latency is all there is.
// A column is worked by a group of kGroup = 8 lanes on a profile in shared memory:
//   - the sweeps run on every lane of the group alike (nothing to divide), reading a block of
//     depths ahead, with the pivot division as a multiplication by the host's reciprocal and two
//     corrections (divide below): 7 dependent operations a depth;
//   - the bisection evaluates the 7 midpoints of its next three halvings at once, one a lane, and
//     then takes the same three decisions one after the other.
// On the 36 x 72 grid (467 depths, 5 steps) 0.28 ms, against 1.21 ms for one thread per column on
// device memory that read each depth when the chain reached it and divided. Grids of more or
// deeper columns than run side by side that way (shared_cols) keep their profiles
// [depth][column] in device memory, one thread each, so that the threads of a warp read and write
// each depth together; the same read-ahead and division took 180 x 360 columns of 1044 depths
// from 5.8 to 2.5 ms.
#include "dsmc_kernels.h"

#include <cmath>

namespace dsmc {
namespace {

struct ThermalArgs {
    int ncol, h, n_sub;
    double R, k_over_dr, a_last;     // CN weight, k/dr, lower coefficient of the bottom row
    double p[5], LH[5], tran_p, tran_LH, mmol;
    const double *flux;              // [ncol] absorbed flux |F|
    const double *T_init;            // [ncol] initial column temperature
    const double *cp, *piv, *rcp;    // [h] c'_i, pivots b_i - a_i c'_(i-1), reciprocals of the pivots
    double *qT, *dp;                 // [h][ncol] profiles and forward-sweep d'_i (device-memory kernel)
    double *T_surface;               // [ncol]
};

// n / b, correctly rounded, from y = 1 / b correctly rounded: two corrections by the exact
// remainder, the second of which rounds the exact quotient (P. Markstein, IBM J. Res. Dev. 34,
// 1990; no overflow or underflow at these temperatures and pivots).
__device__ __forceinline__ double divide(double n, double b, double y) {
    double q = n * y;
    q = fma(fma(-b, q, n), y, q);
    return fma(fma(-b, q, n), y, q);
}

__device__ double surface_balance(const ThermalArgs &a, double T, double F, double oT) {
    const double log10_p = a.p[0] / T + a.p[1] + a.p[2] * T + a.p[3] * T * T + a.p[4] * log10(T);
    const double pres = a.tran_p * pow(10.0, log10_p);
    const double LH = a.tran_LH * (a.LH[0] / T + a.LH[1] + a.LH[2] * T + a.LH[3] * T * T +
                                   a.LH[4] * log10(T));
    constexpr double kSigma = 5.6704e-8, kKB = 1.38e-23, kPi = 3.14159265358979323846;
    const double sublim = LH * sqrt(a.mmol / (2.0 * kPi * kKB * T)) * pres;
    return F + a.k_over_dr * oT - a.k_over_dr * T - kSigma * T * T * T * T - sublim;
}

// Surface temperature by bisection, worked by the kGroup lanes that share a column (all lanes of
// the warp call it). Every lane of a group returns the same value.
template <int kGroup>
__device__ double surface_temperature(const ThermalArgs &a, double F, double oT) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & (kGroup - 1);
    auto from = [&](double v, int src) { return kGroup > 1 ? __shfl_sync(kAll, v, src, kGroup) : v; };
    double T0 = 50.0, T1 = 300.0, f0, f1;
    if (kGroup > 1) {
        const double f = surface_balance(a, lane & 1 ? T1 : T0, F, oT);
        f0 = from(f, 0);
        f1 = from(f, 1);
    } else {
        f0 = surface_balance(a, T0, F, oT);
        f1 = surface_balance(a, T1, F, oT);
    }
    int m = 0;
    bool done = false;
    while (__any_sync(kAll, !done)) {
        if (!done && (m >= 30 || T1 >= 10000.0)) done = true;
        const bool widen = f0 * f1 > 0;
        // node `lane` (1 to kGroup - 1) of the tree of the next halvings: 1 halves (T0, T1), 2n
        // the lower and 2n + 1 the upper part that n leaves
        double lo = T0, hi = T1;
        const int node = kGroup > 1 && lane ? lane : 1;
        for (int bit = 30 - __clz(node); bit >= 0; bit--) {
            const double mid = (lo + hi) / 2.0;
            if (node >> bit & 1) lo = mid;
            else hi = mid;
        }
        const double T = widen ? T1 * 5.0 : (lo + hi) / 2.0;
        const double f = surface_balance(a, T, F, oT);
        bool walk = !done;
        int cur = 1;
        do {   // at most log2(kGroup) decisions on the values at hand, the reference's order
            const double T2 = from(T, kGroup > 1 ? cur : 0), f2 = from(f, kGroup > 1 ? cur : 0);
            if (walk) {
                if (m >= 30 || T1 >= 10000.0) {
                    walk = false;
                } else if (widen) {
                    T1 = T2;
                    f1 = f2;
                    m++;
                    walk = false;
                } else if (f0 * f1 > 0) {
                    walk = false;
                } else {
                    const bool upper = !(f0 * f2 <= 0);
                    if (upper) { T0 = T2; f0 = f2; }
                    else { T1 = T2; f1 = f2; }
                    m++;
                    if (fabs(T0 - T1) <= 0.01) { done = true; walk = false; }
                    cur = 2 * cur + (upper ? 1 : 0);
                }
            }
            cur = cur < kGroup ? cur : kGroup;   // kGroup: the tree is used up
            if (cur == kGroup) { walk = false; cur = kGroup > 1 ? 1 : 0; }
        } while (__any_sync(kAll, walk));
    }
    return (T0 + T1) / 2.0;
}

// One implicit step of a column with its profile in q and scratch d, element i at [i * n]. kGroup lanes
// (all of the warp's groups together) work on one q and d: the step overwrites the old profile once
// every lane has read it, and the next step reads the new one once every lane has written it.
template <int kGroup>
__device__ __forceinline__ void diffuse(const ThermalArgs &a, const double *cp, const double *piv,
                                        const double *rcp, double *q, double *d, long long n, double Ts) {
    constexpr int kAhead = 8;   // depths read before the chain needs them
    const int h = a.h;
    const double R = a.R, w0 = 1.0 - 2.0 * R;
    // forward sweep with the right-hand side built on the fly from the old profile:
    // d_0 = Ts (row 0 is the identity), d_i = R T_(i-1) + (1 - 2R) T_i + R T_(i+1), d_(h-1) = 0
    double prev_old = Ts, cur_old = q[n];   // the old T_0 is replaced by Ts first
    double dprev = Ts;                      // d'_0 = d_0 / b_0 with b_0 = 1
    d[0] = dprev;
    for (int i = 1; i < h - 1; i += kAhead) {
        double old[kAhead], b[kAhead], y[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
            const int k = min(i + j, h - 2);
            old[j] = q[(k + 1) * n];
            b[j] = piv[k];
            y[j] = rcp[k];
        }
#pragma unroll
        for (int j = 0; j < kAhead; j++)
            if (i + j < h - 1) {
                const double rhs = R * prev_old + w0 * cur_old + R * old[j];
                dprev = divide(rhs - (-R) * dprev, b[j], y[j]);
                d[(i + j) * n] = dprev;
                prev_old = cur_old;
                cur_old = old[j];
            }
    }
    dprev = divide(0.0 - a.a_last * dprev, piv[h - 1], rcp[h - 1]);
    if (kGroup > 1) __syncwarp();
    // back substitution, overwriting the profile
    double x = dprev;
    q[(h - 1) * n] = x;
    for (int i = h - 2; i >= 0; i -= kAhead) {
        double di[kAhead], c[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
            const int k = max(i - j, 0);
            di[j] = d[k * n];
            c[j] = cp[k];
        }
#pragma unroll
        for (int j = 0; j < kAhead; j++)
            if (i - j >= 0) {
                x = di[j] - c[j] * x;
                q[(i - j) * n] = x;
            }
    }
    if (kGroup > 1) __syncwarp();
}

// Columns in device memory, one thread each.
__global__ void thermal_column_kernel(const ThermalArgs a) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = min(col, a.ncol - 1);   // the lanes past the end repeat the last column
    const bool mine = col < a.ncol;
    const long long n = a.ncol;
    double *qT = a.qT + c, *dp = a.dp + c;
    const double F = a.flux[c];
    if (mine)
        for (int d = 0; d < a.h; d++) qT[d * n] = a.T_init[c];
    for (int step = 0; step < a.n_sub; step++) {
        const double Ts = surface_temperature<1>(a, F, mine ? qT[n] : a.T_init[c]);
        if (mine) diffuse<1>(a, a.cp, a.piv, a.rcp, qT, dp, n, Ts);
    }
    if (mine) a.T_surface[c] = qT[0];
}

extern __shared__ double thermal_smem[];

// Columns in shared memory, kGroup lanes each: [cp | piv | rcp] of h, then the profiles and d' of
// the block's columns, [h][columns]. Every lane of a group reads and writes the whole column, all the
// same values; the warp meets wherever one lane would write what another has still to read.
template <int kGroup>
__global__ void thermal_shared_kernel(const ThermalArgs a) {
    const int h = a.h, cols = blockDim.x / kGroup, own = threadIdx.x / kGroup;
    double *cp = thermal_smem, *piv = cp + h, *rcp = piv + h;
    double *q = rcp + h + own, *d = q + static_cast<long long>(h) * cols;
    for (int i = threadIdx.x; i < h; i += blockDim.x) {
        cp[i] = a.cp[i];
        piv[i] = a.piv[i];
        rcp[i] = a.rcp[i];
    }
    __syncthreads();
    const int col = blockIdx.x * cols + own;
    const int c = min(col, a.ncol - 1);   // the groups past the end repeat the last column
    const double F = a.flux[c], T_init = a.T_init[c];
    for (int i = 0; i < h; i++) q[i * cols] = T_init;
    __syncwarp();
    for (int step = 0; step < a.n_sub; step++)
        diffuse<kGroup>(a, cp, piv, rcp, q, d, cols, surface_temperature<kGroup>(a, F, q[cols]));
    if (col < a.ncol && threadIdx.x % kGroup == 0) a.T_surface[c] = q[0];
}

constexpr int kGroup = 8;

constexpr size_t kSharedPerSm = 227 * 1024;   // of an SM, and of a block at most

size_t shared_bytes(int h, int cols) { return static_cast<size_t>(h) * (3 + 2 * cols) * sizeof(double); }

// Columns per block of the shared-memory kernel (8, or 4 where the depth leaves no room for more),
// or 0 for the device-memory kernel. The line lies where the blocks no longer run side by side: a
// second wave doubles a time that is all latency. 2,592 columns of 467 depths (3 blocks of 8 per
// SM): 0.28 ms against 0.53 ms in device memory; 5,184 (1.5 waves) 0.51 against 0.52 ms; 8,640 of
// 763 depths and 8 steps (7 waves) 4.2 against 1.4 ms; 2,592 of 1401 (2 waves) 1.7 against 1.4 ms.
int shared_cols(int h, int ncol, int num_sms) {
    for (int cols = 8; cols >= 4; cols /= 2) {
        const long long per_sm = static_cast<long long>(kSharedPerSm / (shared_bytes(h, cols) + 1024));
        if ((ncol + cols - 1) / cols <= per_sm * num_sms) return cols;
    }
    return 0;
}

}  // namespace

cudaError_t launch_thermal(const ThermalSetup &s, const double *flux, const double *T_init,
                           const double *cp, const double *piv, const double *rcp, double *qT,
                           double *dp, double *T_surface, int num_sms, cudaStream_t stream) {
    ThermalArgs a{};
    a.ncol = s.ncol;
    a.h = s.h;
    a.n_sub = s.n_sub;
    a.R = s.R;
    a.k_over_dr = s.k_over_dr;
    a.a_last = s.a_last;
    for (int k = 0; k < 5; k++) {
        a.p[k] = s.p[k];
        a.LH[k] = s.LH[k];
    }
    a.tran_p = s.tran_p;
    a.tran_LH = s.tran_LH;
    a.mmol = s.mmol;
    a.flux = flux;
    a.T_init = T_init;
    a.cp = cp;
    a.piv = piv;
    a.rcp = rcp;
    a.qT = qT;
    a.dp = dp;
    a.T_surface = T_surface;
    const int cols = shared_cols(s.h, s.ncol, num_sms);
    if (cols) {
        // the limit belongs to the function, which other threads launch too: always the largest
        const cudaError_t e = cudaFuncSetAttribute(thermal_shared_kernel<kGroup>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(kSharedPerSm));
        if (e != cudaSuccess) return e;
        const size_t smem = shared_bytes(s.h, cols);
        thermal_shared_kernel<kGroup><<<(s.ncol + cols - 1) / cols, cols * kGroup, smem, stream>>>(a);
        return cudaGetLastError();
    }
    const int block = 32;
    thermal_column_kernel<<<(s.ncol + block - 1) / block, block, 0, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace dsmc
