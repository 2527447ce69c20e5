// fast_kernel.cuh - the step-loop kernel of the FAST paths: resident particle slots, a device work
// queue, cell tracking by comparisons against register-cached cell bounds, and per-cell register
// accumulation of the fixed-point deposits. Two precisions share this code: FAST_FP32 pushes in
// FP32 with two-sum compensated position and velocity; FAST_FP64 runs the same loop on double
// state and FP64 boundary tables without compensation, so the pair isolates what the precision
// buys.
//
// Per step the hot loop does one gravity evaluation (one rsqrt), the reference's Verlet variant
// (src/common/integrator.c:21-44) with the position and velocity sums kept as (hi, lo) float
// pairs (FP32) or doubles (FP64), an in-cell test against the eight bounds of the current cell
// held in registers (no asin, atan2, log or table load), photolysis as a running product
// re-anchored to W0 * 2^(-c * n_day) (one ex2), and the deposit into the register accumulator of
// the current cell, flushed with one 64-bit atomic when the particle leaves the cell. Rare events
// (cell change, launch, landing, collision, end of life) leave the loop for code that reads the
// boundary tables and the cold per-particle fields.
//
// Two loops share the pieces: fast_kernel, whose lanes run free of one another, and warp_kernel,
// whose lanes step together.
//
// Included by the translation units that instantiate it (fast_served.cu, fast_one32.cu,
// fast_one64.cu), one per family of kernels so that they compile side by side.
#pragma once

#include "fast_engine.h"

#include <type_traits>

namespace dsmc {
namespace {

constexpr float kPiF = 3.14159265358979f;

template <typename R>
constexpr bool is_f64() { return std::is_same<R, double>::value; }

// Packed FP32 pairs (sm_100a's two-value FP32 instructions): one issue slot works on two values,
// and each half rounds as the scalar instruction does, so packing changes no result. The step
// loop is bound by issue slots (77 % issue-active with the FMA pipe half busy), which is why it
// packs: the Verlet update takes 32 instructions instead of 49. Written as PTX because the
// operands must flush subnormals like the rest of this translation unit (-ftz=true).
struct F2 { float x, y; };

#define DSMC_F2_OP2(name, op)                                                                    \
    __device__ __forceinline__ F2 name(F2 a, F2 b) {                                              \
        F2 r;                                                                                     \
        asm("{\n.reg .b64 a, b, r;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\n" op               \
            " r, a, b;\nmov.b64 {%0, %1}, r;\n}"                                                  \
            : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                     \
        return r;                                                                                 \
    }
DSMC_F2_OP2(add2, "add.rn.ftz.f32x2")
DSMC_F2_OP2(sub2, "sub.rn.ftz.f32x2")
DSMC_F2_OP2(mul2, "mul.rn.ftz.f32x2")
#undef DSMC_F2_OP2

__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("{\n.reg .b64 a, b, c, r;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\n"
        "fma.rn.ftz.f32x2 r, a, b, c;\nmov.b64 {%0, %1}, r;\n}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}

// Compensated accumulation hi + lo += b of two components (Dekker's fast two-sum): exact when
// |hi| >= |b|, which holds for position and velocity components except in the few steps where a
// component passes through zero, whose error is then at most ulp(b) (< 1e-4 m or 1e-7 m/s here).
__device__ __forceinline__ void accumulate2(float &hx, float &hy, float &lx, float &ly, F2 b) {
    const F2 hi{hx, hy}, t = add2(hi, b);
    const F2 lo = add2(F2{lx, ly}, sub2(b, sub2(t, hi)));
    hx = t.x; hy = t.y;
    lx = lo.x; ly = lo.y;
}

// Philox4x32-10 block of the generator's current counter, with the ten rounds kept as a loop: the
// same words as Philox::next in a fraction of its code. The config model's collision loop takes it in
// its event paths (launch, start, collision), which run on single lanes: there it cuts ptxas' spill
// stores (96 registers: 628 to 336 B in the served queue, 184 to 92 B in a solve of one instance) and
// measured 7 % faster on the 1e7-particle collisional phase 2; the lean and general loops measured
// 1-3 % slower with it and keep the unrolled rounds.
__device__ __forceinline__ void philox_next_rolled(Philox &r) {
    uint32_t c0 = r.pid, c1 = r.event, c2 = r.inst, c3 = 0u, a = r.k0, b = r.k1;
#pragma unroll 1
    for (int k = 0; k < 10; k++) {
        const uint32_t lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
        const uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
        c0 = hi1 ^ c1 ^ a;
        c1 = lo1;
        c2 = hi0 ^ c3 ^ b;
        c3 = lo0;
        a += 0x9E3779B9u;
        b += 0xBB67AE85u;
    }
    r.w[0] = c0; r.w[1] = c1; r.w[2] = c2; r.w[3] = c3;
    r.event++;
}

// kRoll: the collision loop's choice of the rolled rounds (same random words either way).
template <bool kRoll>
__device__ __forceinline__ void philox_next(Philox &r) {
    if (kRoll) philox_next_rolled(r);
    else r.next();
}

// u in (0, 1]: 24 random bits plus half a step, so u is never 0. From 2^23 on the half is rounded away
// (ties to even), and the top word gives exactly 1: a launch that draws it (1 in 2^24, of either of its
// two) takes log(1 - u) = -infinity and has an infinite speed; see drift_nowhere.
__device__ __forceinline__ float unit_open(uint32_t w) {
    return (static_cast<float>(w >> 8) + 0.5f) * (1.0f / 16777216.0f);
}

// Features of the step loops (kMode). 0: everything, chosen at run time. The lean loops compile
// out what their instances do not use; each gives an instance the same results as loop 0.
// 1 config model, ballistic; 2 config model with collisions; 3 reference model, ballistic;
// 4 config model with speed histograms; 5 reference model with collisions.
template <int kMode>
struct Mode {
    static constexpr bool kAny = kMode == 0;
    static constexpr bool kCfg = kMode == 1 || kMode == 2 || kMode == 4;
    static constexpr bool kRef = kMode == 3 || kMode == 5;
    static constexpr bool kCol = kMode == 2 || kMode == 5;
    static constexpr bool kHist = kMode == 4;
    static constexpr bool kRoll = kMode == 2;
    __device__ static bool ref(const dsmc_params &p) {
        return kRef || (kAny && p.model == DSMC_MODEL_REFERENCE);
    }
};

// Register-resident state of the particle a thread pushes. The cold fields (particle id, Philox
// event counter, collision count, freeze waiting time) stay in the slot arrays.
template <typename R>
struct HotT {
    R sh[3], sl[3], vh[3], vl[3], oa[3];
    R w0, pcol, pthr, nsig;
    int nday, steps, hop;
    int cell;                  // packed (ht << 16) | (td << 8) | fd
    int ci;                    // (ht * ftd + td) * ffd + fd, -1 = none
    R run_w;                   // weight-steps deposited in cell ci, not yet flushed
    R W;                       // current weight: exact W0 2^(-c n_day) at cell changes and
                               // events, times 2^(-c) per day-side step in between
    int hist_key, hist_cnt;    // speed bin of the histogram's run (-1 = none), its steps
    int inst;                  // -1 = empty slot
};
using Hot = HotT<float>;

// The general loop's: a step of it may count no speed, so its histogram's run keeps a cell of its own.
// As a member of HotT it changed ptxas' choices in the lean loops, which have no such run (0 -> 8 B of
// spill stores at 96 registers): 3e5 Moon-like particles 6.77 -> 6.82 ms, 1e6 Europa-like in FP64 24.9 ->
// 25.1 ms. So did a finish() that leaves out their empty flush_hist (44 against 24 B in the FP64 loop).
template <typename R>
struct GeneralHotT : HotT<R> {
    int hist_ci = -1;
};
template <int kMode, typename R>
using HotOf = std::conditional_t<Mode<kMode>::kAny, GeneralHotT<R>, HotT<R>>;

// Cell of the histogram's run.
template <int kMode, typename R>
__device__ __forceinline__ int &hist_cell(HotT<R> &h) {
    if constexpr (Mode<kMode>::kAny) return static_cast<GeneralHotT<R> &>(h).hist_ci;
    else return h.ci;
}

// Bounds of the current cell: r^2 in (r2lo, r2hi], z|z| in (r^2 zlo, r^2 zhi], longitude between
// the directions (s0, c0) and (s1, c1).
template <typename R>
struct BoundsT {
    R r2lo, r2hi, zlo, zhi, s0, c0, s1, c1;
};

// The boundary tables of an instance in the engine's precision: from device memory (the served
// queue) or from the block's shared memory (a solve of one instance, OneArgsT), where a cell
// change needs a 32-bit address and no descriptor load.
template <typename R> struct GlobalTab;
// Collision rate n * sigma of a cell from the background density.
__device__ __forceinline__ double background_rate(const FastInst &I, int ht, int ci) {
    if (I.t.n_bg && I.p.runner == DSMC_RUNNER_ADVANCED && ht < I.p.collide_ht_max && ci < I.t.n_bg_len)
        return __ldg(I.t.n_bg + ci) * I.p.cross_section;
    return 0.0;
}

template <> struct GlobalTab<float> {
    const FastInst &I;
    __device__ float rate(int ht, int ci) const { return static_cast<float>(background_rate(I, ht, ci)); }
    __device__ float rb2(int j) const { return __ldg(I.rb2 + j); }
    __device__ float sbs(int j) const { return __ldg(I.sbs + j); }
    __device__ float2 lon(int j) const { return __ldg(I.lonb + j); }
};
template <> struct GlobalTab<double> {
    const FastInst &I;
    __device__ double rate(int ht, int ci) const { return background_rate(I, ht, ci); }
    __device__ double rb2(int j) const { return __ldg(I.rb2d + j); }
    __device__ double sbs(int j) const { return __ldg(I.sbsd + j); }
    __device__ double2 lon(int j) const { return __ldg(I.lonbd + j); }
};

extern __shared__ double2 smem_tables[];

// Columns first, then rows, both with room for the engine's 255, then hd + 1 shells.
template <typename R>
struct SharedTab {
    using V2 = std::conditional_t<std::is_same<R, double>::value, double2, float2>;
    static constexpr int kRows = 256;
    const FastInst &I;
    __device__ static V2 *lonb() { return reinterpret_cast<V2 *>(smem_tables); }
    __device__ static R *sbsb() { return reinterpret_cast<R *>(lonb() + kRows); }
    __device__ static R *rb2b() { return sbsb() + kRows; }
    __device__ R rate(int, int ci) const {
        if constexpr (std::is_same<R, double>::value) return I.nsigd ? __ldg(I.nsigd + ci) : 0.0;
        else return I.nsig ? __ldg(I.nsig + ci) : 0.0f;
    }
    __device__ R rb2(int j) const { return rb2b()[j]; }
    __device__ R sbs(int j) const { return sbsb()[j]; }
    __device__ V2 lon(int j) const { return lonb()[j]; }
    // every thread of the block calls it, before the first use
    __device__ static void fill(const FastInst &I) {
        const GlobalTab<R> g{I};
        for (int j = threadIdx.x; j <= I.p.ffd; j += blockDim.x) lonb()[j] = g.lon(j);
        for (int j = threadIdx.x; j <= I.p.ftd; j += blockDim.x) sbsb()[j] = g.sbs(j);
        for (int j = threadIdx.x; j <= I.p.hd; j += blockDim.x) rb2b()[j] = g.rb2(j);
        __syncthreads();
    }
};

template <class A, typename R>
using TabOf = std::conditional_t<A::kOne, SharedTab<R>, GlobalTab<R>>;

template <typename R>
__device__ __forceinline__ void load_hot(const SlotsT<R> &s, long long i, long long S, HotT<R> &h) {
    h.inst = s.inst[i];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        h.sh[k] = s.sh[k * S + i];
        h.vh[k] = s.vh[k * S + i];
        h.oa[k] = s.oa[k * S + i];
        if constexpr (is_f64<R>()) {
            h.sl[k] = 0.0;
            h.vl[k] = 0.0;
        } else {
            h.sl[k] = s.sl[k * S + i];
            h.vl[k] = s.vl[k * S + i];
        }
    }
    h.w0 = s.w0[i];
    h.nday = s.nday[i];
    h.steps = s.steps[i];
    h.hop = s.hop[i];
    h.cell = s.cell[i];
    h.ci = s.run_cell[i];
    h.run_w = s.run_w[i];
    h.W = s.wcur[i];
    h.hist_key = s.hist_key[i];
    h.hist_cnt = s.hist_cnt[i];
    h.pcol = s.pcol[i];
    h.pthr = s.pthr[i];
    h.nsig = 0.0f;
}

template <typename R>
__device__ __forceinline__ void store_hot(const SlotsT<R> &s, long long i, long long S,
                                          const HotT<R> &h) {
    s.inst[i] = h.inst;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        s.sh[k * S + i] = h.sh[k];
        s.vh[k * S + i] = h.vh[k];
        s.oa[k * S + i] = h.oa[k];
        if constexpr (!is_f64<R>()) {
            s.sl[k * S + i] = h.sl[k];
            s.vl[k * S + i] = h.vl[k];
        }
    }
    s.w0[i] = h.w0;
    s.nday[i] = h.nday;
    s.steps[i] = h.steps;
    s.hop[i] = h.hop;
    s.cell[i] = h.cell;
    s.run_cell[i] = h.ci;
    s.run_w[i] = h.run_w;
    s.wcur[i] = h.W;
    s.hist_key[i] = h.hist_key;
    s.hist_cnt[i] = h.hist_cnt;
    s.pcol[i] = h.pcol;
    s.pthr[i] = h.pthr;
}

template <typename R>
__device__ __forceinline__ void set_pos(HotT<R> &h, const double s[3]) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        h.sh[k] = static_cast<R>(s[k]);
        h.sl[k] = static_cast<R>(s[k] - static_cast<double>(h.sh[k]));
    }
}

template <typename R>
__device__ __forceinline__ void set_vel(HotT<R> &h, const double v[3]) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        h.vh[k] = static_cast<R>(v[k]);
        h.vl[k] = static_cast<R>(v[k] - static_cast<double>(h.vh[k]));
    }
}

template <typename R>
__device__ __forceinline__ void get_pos(const HotT<R> &h, double s[3]) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if constexpr (is_f64<R>()) s[k] = h.sh[k];
        else s[k] = static_cast<double>(h.sh[k]) + static_cast<double>(h.sl[k]);
    }
}

template <typename R>
__device__ __forceinline__ void get_vel(const HotT<R> &h, double v[3]) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if constexpr (is_f64<R>()) v[k] = h.vh[k];
        else v[k] = static_cast<double>(h.vh[k]) + static_cast<double>(h.vl[k]);
    }
}

// Position component k in the engine's precision (hi + lo in FP32, the double in FP64).
template <typename R>
__device__ __forceinline__ R pos(const HotT<R> &h, int k) {
    if constexpr (is_f64<R>()) return h.sh[k];
    else return h.sh[k] + h.sl[k];
}

__device__ __forceinline__ int pack_cell(int ht, int td, int fd) { return (ht << 16) | (td << 8) | fd; }

__device__ __forceinline__ float fma_r(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_r(double a, double b, double c) { return fma(a, b, c); }

// Latitude row and longitude column of position (x, y, z) with r2 = |s|^2, moved from the
// current (td, fd) by boundary comparisons. Row td covers latitudes (b_td, b_td+1] and column fd
// longitudes (phi_fd, phi_fd+1], the upper-inclusive cells of grid_spherical_to_index
// (src/common/grid.c:28-39).
template <class T, typename R>
__device__ __forceinline__ void track_angles(const T &tab, R x, R y, R z, R r2, int &td, int &fd) {
    const FastInst &I = tab.I;
    const int ftd = I.p.ftd, ffd = I.p.ffd;
    const R zz = z * fabs(z);
    for (int it = 0; it < 64 && td + 1 < ftd && zz > r2 * tab.sbs(td + 1); it++) td++;
    for (int it = 0; it < 64 && td > 0 && zz <= r2 * tab.sbs(td); it++) td--;
    for (int it = 0; it < 2 * 256; it++) {
        const auto hi = tab.lon(fd + 1);
        if (x * hi.y - y * hi.x > R(0)) { fd = fd + 1 == ffd ? 0 : fd + 1; continue; }
        const auto lo = tab.lon(fd);
        if (x * lo.y - y * lo.x <= R(0) && !(fd == 0 && x >= R(0) && y > R(0))) {
            fd = fd == 0 ? ffd - 1 : fd - 1;
            continue;
        }
        break;
    }
}

template <class T, typename R>
__device__ __forceinline__ void track_shell(const T &tab, R r2, int &ht) {
    const int hd = tab.I.p.hd;
    for (int it = 0; it < 64 && ht + 1 < hd && r2 > tab.rb2(ht + 1); it++) ht++;
    for (int it = 0; it < 64 && ht > 0 && r2 <= tab.rb2(ht); it++) ht--;
}

// Cell of a position from scratch: an estimate from the angles, then the comparison fix-up.
template <class T, typename R>
__device__ __forceinline__ int cell_from_scratch(const T &tab, const R x, const R y, const R z) {
    const FastInst &I = tab.I;
    const R r2 = x * x + y * y + z * z;
    const float xf = static_cast<float>(x), yf = static_cast<float>(y), zf = static_cast<float>(z);
    const float r = sqrtf(static_cast<float>(r2));
    const float th = asinf(fminf(1.0f, fmaxf(-1.0f, zf / r)));
    float ph = atan2f(xf, yf);
    if (ph < 0.0f) ph += 2.0f * kPiF;
    int td = static_cast<int>((th + 0.5f * kPiF) / kPiF * I.p.ftd);
    int fd = static_cast<int>(ph / (2.0f * kPiF) * I.p.ffd);
    td = min(max(td, 0), I.p.ftd - 1);
    fd = min(max(fd, 0), I.p.ffd - 1);
    track_angles(tab, x, y, z, r2, td, fd);
    int ht;
    if (I.p.use_exp_grid) {
        // FP32 estimate; track_shell below settles the exact shell
        const float arg = static_cast<float>(I.p.alpha2 / I.p.unih) * (r - static_cast<float>(I.p.Radii)) + 1.0f;
        ht = arg <= 1.0f ? 0 : static_cast<int>(logf(arg) * static_cast<float>(1.0 / I.p.log1p_alpha2));
    } else {
        ht = static_cast<int>((static_cast<double>(r) - I.p.Radii) / I.p.unih);
    }
    ht = min(max(ht, 0), I.p.hd - 1);
    track_shell(tab, r2, ht);
    return pack_cell(ht, td, fd);
}

// Fixed-point deposit of a weight sum: W x 2^24 rounded once.
__device__ __forceinline__ unsigned long long fixed_of(float w) { return __float2ull_rn(w * 16777216.0f); }
__device__ __forceinline__ unsigned long long fixed_of(double w) { return __double2ull_rn(w * 16777216.0); }

// Flushes the weight-steps of the current cell as one 64-bit fixed-point atomic (W x 2^24
// summed over the steps spent in the cell, rounded once). The sum of a run is a function of the
// particle's own trajectory only, so the grid stays independent of thread order.
template <typename R>
__device__ __forceinline__ void flush_cell(const FastInst &I, HotT<R> &h) {
    if (h.ci >= 0 && h.run_w > R(0)) atomicAdd(&I.t.density[h.ci], fixed_of(h.run_w));
    h.run_w = R(0);
}

// Adds the histogram's run to its bin of cell ci, the run's: cell x bins may take more than 31 bits (255 x
// 255 x 34 cells of 1024 bins are 2.26e9 entries), so the index is formed here.
template <typename R>
__device__ __forceinline__ void flush_hist(const FastInst &I, HotT<R> &h, int ci) {
    if (h.hist_key >= 0 && h.hist_cnt)
        atomicAdd(&I.t.speed_hist[static_cast<long long>(ci) * I.p.n_speed_bins + h.hist_key],
                  static_cast<unsigned long long>(h.hist_cnt));
    h.hist_key = -1;
    h.hist_cnt = 0;
}

// Makes `cell` the current cell: flushes the previous cell's deposits, loads the eight bounds
// and the collision rate n * sigma of the new cell.
template <class T, typename R>
__device__ __forceinline__ void enter_cell(const T &tab, HotT<R> &h, BoundsT<R> &b, int cell) {
    const FastInst &I = tab.I;
    flush_cell(I, h);
    const int ht = cell >> 16, td = (cell >> 8) & 0xff, fd = cell & 0xff;
    h.cell = cell;
    h.ci = (ht * I.p.ftd + td) * I.p.ffd + fd;
    b.r2lo = tab.rb2(ht);
    b.r2hi = tab.rb2(ht + 1);
    b.zlo = tab.sbs(td);
    b.zhi = tab.sbs(td + 1);
    const auto lo = tab.lon(fd), hi = tab.lon(fd + 1);
    b.s0 = lo.x;
    b.c0 = lo.y;
    b.s1 = hi.x;
    b.c1 = hi.y;
    h.nsig = tab.rate(ht, h.ci);
}

template <typename R>
__device__ __forceinline__ R exp2_r(R x) {
    if constexpr (is_f64<R>()) return exp2(x);
    else return exp2f(x);
}

// FP32 engines keep the day constant in FP32, FP64 engines in FP64.
template <typename R>
__device__ __forceinline__ R c_day_of(const FastInst &I) {
    if constexpr (is_f64<R>()) return I.c_day_d;
    else return I.c_day;
}

// The particle left its cell: walk to the new cell one boundary at a time. Each move keeps the
// shared boundary from the registers and loads only the next one, so a typical crossing costs
// one table load. Same cells as track_shell / track_angles. in_r, in_t, in_f are the step's own
// inside tests per coordinate; only the coordinates that failed are walked (7 % faster on
// the 1e8-particle Ceres-like workload than walking all three, identical cells). Returns whether
// the cell changed.
template <bool kNoBg, class T, typename R>
__device__ __forceinline__ bool move_cell(const T &tab, HotT<R> &h, BoundsT<R> &b, R x, R y,
                                          R r2, R zz, bool in_r, bool in_t, bool in_f) {
    const FastInst &I = tab.I;
    int ht = h.cell >> 16, td = (h.cell >> 8) & 0xff, fd = h.cell & 0xff;
    // the three walks are independent (shells by r^2, rows by z|z| / r^2, columns by the
    // longitude tests), so a coordinate still inside its two bounds needs no walk. Each walk
    // goes one way only: after a move up the old upper bound is the new lower one, which the
    // particle is above, so the downward test cannot pass (and the other way round); the
    // walks test one bound per move (same cells as testing both).
    if (!in_r) {
        const int hd = I.p.hd;
        if (r2 > b.r2hi) {
            for (int it = 0; it < 64 && r2 > b.r2hi && ht + 1 < hd; it++) {
                ht++;
                b.r2lo = b.r2hi;
                b.r2hi = tab.rb2(ht + 1);
            }
        } else {
            for (int it = 0; it < 64 && r2 <= b.r2lo && ht > 0; it++) {
                ht--;
                b.r2hi = b.r2lo;
                b.r2lo = tab.rb2(ht);
            }
        }
    }
    if (!in_t) {
        const int ftd = I.p.ftd;
        if (zz > r2 * b.zhi) {
            for (int it = 0; it < 64 && zz > r2 * b.zhi && td + 1 < ftd; it++) {
                td++;
                b.zlo = b.zhi;
                b.zhi = tab.sbs(td + 1);
            }
        } else {
            for (int it = 0; it < 64 && zz <= r2 * b.zlo && td > 0; it++) {
                td--;
                b.zhi = b.zlo;
                b.zlo = tab.sbs(td);
            }
        }
    }
    if (!in_f) {
        const int ffd = I.p.ffd;
        if (x * b.c1 - y * b.s1 > R(0)) {
            for (int it = 0; it < 512 && x * b.c1 - y * b.s1 > R(0); it++) {
                fd = fd + 1 == ffd ? 0 : fd + 1;
                b.s0 = b.s1;
                b.c0 = b.c1;
                const auto q = tab.lon(fd + 1);
                b.s1 = q.x;
                b.c1 = q.y;
            }
        } else {
            for (int it = 0; it < 512 && x * b.c0 - y * b.s0 <= R(0) && !(fd == 0 && x >= R(0) && y > R(0));
                 it++) {
                fd = fd == 0 ? ffd - 1 : fd - 1;
                b.s1 = b.s0;
                b.c1 = b.c0;
                const auto q = tab.lon(fd);
                b.s0 = q.x;
                b.c0 = q.y;
            }
        }
    }
    const int cell = pack_cell(ht, td, fd);
    if (cell == h.cell) return false;
    // the run of a flying particle has a cell and no negative weight: flushed without the tests
    // of flush_cell (a run of zero adds zero)
    atomicAdd(&I.t.density[h.ci], fixed_of(h.run_w));
    h.run_w = R(0);
    h.cell = cell;
    h.ci = (ht * I.p.ftd + td) * I.p.ffd + fd;
    h.W = h.w0 * exp2_r<R>(-c_day_of<R>(I) * static_cast<R>(h.nday));   // re-anchor the running weight
    if (!kNoBg) h.nsig = tab.rate(ht, h.ci);
    return true;
}

__device__ __forceinline__ double cdf_eval(const double *coef, const double *box, int degree,
                                           double x) {
    const double t = (x - box[2]) / box[3];
    double r = 0.0;
    for (int i = 0; i <= degree; i++) r = r * t + coef[i];
    return r;
}

// Bisection of the fitted reverse-cumulative speed distribution (collision.c:43-101).
__device__ double cdf_sample(const double *coef, const double *box, double total, int degree,
                             double u) {
    const double at_max = cdf_eval(coef, box, degree, box[1]);
    const double ranking = u * (total - at_max) + at_max;
    double v0 = box[0], v1 = box[1];
    for (int iter = 0; iter < 100; iter++) {
        const double vm = (v0 + v1) * 0.5;
        const double fm = cdf_eval(coef, box, degree, vm) - ranking;
        const double f1 = cdf_eval(coef, box, degree, v1) - ranking;
        if (fm * f1 < 0) v0 = vm;
        else v1 = vm;
        if (fabs(v1 - v0) < 0.01) break;
    }
    return (v0 + v1) * 0.5;
}

__device__ __forceinline__ void unit_sphere_f(float zu, float pu, float o[3]) {
    const float z = 2.0f * zu - 1.0f;
    const float rr = sqrtf(fmaxf(0.0f, 1.0f - z * z));
    float sn, cs;
    sincosf(2.0f * kPiF * pu, &sn, &cs);
    o[0] = rr * cs;
    o[1] = rr * sn;
    o[2] = z;
}

// The FP64 path's unit vector: the plain FP64 kernel's map of two uniforms.
__device__ __forceinline__ void unit_sphere_d(double zu, double pu, double o[3]) {
    const double z = 2.0 * zu - 1.0;
    const double rr = sqrt(fmax(0.0, 1.0 - z * z));
    double sn, cs;
    sincos(2.0 * kPi * pu, &sn, &cs);
    o[0] = rr * cs;
    o[1] = rr * sn;
    o[2] = z;
}

struct StatAcc {
    unsigned steps = 0, escaped = 0, collisions = 0, bound = 0, finished = 0, drift = 0;
    int inst = -1;
};

// Adds the thread's statistics into its instance's counters: lanes of one instance are summed
// with one warp reduction and one atomic per counter. Every lane of the warp must call it.
template <typename A>
__device__ void flush_stats(const A &a, StatAcc &st) {
    const unsigned full = 0xffffffffu;
    const int key = st.inst;
    const unsigned group = __match_any_sync(full, key);
    const unsigned v[6] = {st.steps, st.escaped, st.collisions, st.bound, st.finished, st.drift};
    const int slot_of[6] = {kStatSteps, kStatEscaped, kStatCollisions, kStatBound, kStatFinished,
                            kStatDrift};
    const bool leader = (threadIdx.x & 31) == (__ffs(group) - 1);
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const unsigned sum = __reduce_add_sync(group, v[k]);
        if (leader && key >= 0 && sum)
            atomicAdd(&a.inst(key).t.stats[slot_of[k]], static_cast<unsigned long long>(sum));
    }
    st = StatAcc{};
}

// The previous instance's share of the counters, lane by lane (an instance switch inside a
// launch happens at most once per particle and is rare).
template <typename A>
__device__ void flush_stats_lane(const A &a, StatAcc &st) {
    if (st.inst >= 0) {
        unsigned long long *dst = a.inst(st.inst).t.stats;
        if (st.steps) atomicAdd(dst + kStatSteps, static_cast<unsigned long long>(st.steps));
        if (st.escaped) atomicAdd(dst + kStatEscaped, static_cast<unsigned long long>(st.escaped));
        if (st.collisions) atomicAdd(dst + kStatCollisions, static_cast<unsigned long long>(st.collisions));
        if (st.bound) atomicAdd(dst + kStatBound, static_cast<unsigned long long>(st.bound));
        if (st.drift) atomicAdd(dst + kStatDrift, static_cast<unsigned long long>(st.drift));
        if (st.finished) {
            atomicAdd(dst + kStatFinished, static_cast<unsigned long long>(st.finished));
            atomicAdd(&a.ctr->finished, static_cast<unsigned long long>(st.finished));
        }
    }
    st = StatAcc{};
}

template <typename R>
__device__ __forceinline__ R weight(const FastInst &I, const HotT<R> &h) {
    return h.w0 * exp2_r<R>(-c_day_of<R>(I) * static_cast<R>(h.nday));
}

// Row and column of the reference model's angles (grid_spherical_to_index, grid.c:28-39).
__device__ __forceinline__ void ref_index(float thi, float fi, int ftd, int ffd, int &td, int &fd) {
    td = static_cast<int>(ceilf((thi + 0.5f * kPiF) / kPiF * ftd)) - 1;
    fd = static_cast<int>(ceilf(fi / (2.0f * kPiF) * ffd)) - 1;
    td = min(max(td, 0), ftd - 1);
    fd = min(max(fd, 0), ffd - 1);
}

__device__ __forceinline__ void ref_index(double thi, double fi, int ftd, int ffd, int &td, int &fd) {
    td = static_cast<int>(ceil((thi + kPi / 2.0) / kPi * ftd)) - 1;
    fd = static_cast<int>(ceil(fi / (2.0 * kPi) * ffd)) - 1;
    td = min(max(td, 0), ftd - 1);
    fd = min(max(fd, 0), ffd - 1);
}

// Latitude and longitude of the current position, computed in FP64 (pos_to_angles,
// ballistic.c:29-33) and returned in the engine's precision.
template <typename R>
__device__ __forceinline__ void angles_of(const HotT<R> &h, R &thi, R &fi) {
    double s[3];
    get_pos(h, s);
    const double Ri = sqrt(s[0] * s[0] + s[1] * s[1] + s[2] * s[2]);
    thi = static_cast<R>(asin(s[2] / Ri));
    double f = atan2(s[0], s[1]);
    if (f < 0) f += 2.0 * kPi;
    fi = static_cast<R>(f);
}

// Orbital energy per unit mass |v|^2 / 2 - GM / |s| of the current state in FP64, for the
// per-hop energy-drift guard: 1 / |s| from the FP32 reciprocal square root and one Newton step in
// FP64 (relative error ~1e-14), so the event path takes no FP64 square root or division.
template <typename R>
__device__ __forceinline__ double orbital_energy(const FastInst &I, const HotT<R> &h) {
    double s[3], v[3];
    get_pos(h, s);
    get_vel(h, v);
    const double r2 = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
    double ir = rsqrtf(static_cast<float>(r2));
    ir = ir * (1.5 - 0.5 * r2 * ir * ir);
    return 0.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) - I.p.GM * ir;
}

// The hop's energy baseline: taken at every launch and after every collision.
template <class A, typename R>
__device__ __forceinline__ void drift_start(const A &a, long long i, const FastInst &I,
                                            const HotT<R> &h) {
    if (I.drift_abs > 0.0) a.s.e0[i] = static_cast<float>(orbital_energy(I, h));
}

// The hop ended (landing, escape radius, hop or life cap): counts it when the energy moved by
// more than the guard's bound since the baseline.
template <class A, typename R>
__device__ __forceinline__ void drift_check(const A &a, long long i, const FastInst &I,
                                            const HotT<R> &h, StatAcc &st) {
    if (I.drift_abs > 0.0 &&
        fabs(orbital_energy(I, h) - static_cast<double>(a.s.e0[i])) > I.drift_abs)
        st.drift++;
}

__device__ __forceinline__ void horizon_add(const FastInst &I, int td, int fd, float W) {
    atomicAdd(&I.t.horizon[td * I.p.ffd + fd], __float2ull_rn(W * 16777216.0f));
}

__device__ __forceinline__ void horizon_add(const FastInst &I, int td, int fd, double W) {
    atomicAdd(&I.t.horizon[td * I.p.ffd + fd], __double2ull_rn(W * DSMC_FIXED_SCALE));
}

// Old acceleration GM s / r^3 of a launch point (ballistic.c:176-181; the FP32 engine keeps it
// times -dt) and the hop's start. The energy baseline of the drift guard comes from e_launch when
// the launch already formed it.
template <class A, typename R>
__device__ __forceinline__ void start_hop_state(const A &a, long long i,
                                                const FastInst &I, HotT<R> &h,
                                                const double *e_launch) {
    if constexpr (is_f64<R>()) {
        const double sx = h.sh[0], sy = h.sh[1], sz = h.sh[2];
        const double ir = rsqrt(sx * sx + sy * sy + sz * sz);
        const double g = I.p.GM * (ir * ir * ir);
        h.oa[0] = g * sx;
        h.oa[1] = g * sy;
        h.oa[2] = g * sz;
    } else {
        const float sx = h.sh[0] + h.sl[0], sy = h.sh[1] + h.sl[1], sz = h.sh[2] + h.sl[2];
        const float ir = rsqrtf(fmaf(sx, sx, fmaf(sy, sy, sz * sz)));
        const float g = -static_cast<float>(I.p.GM * I.p.dt_step) * (ir * ir * ir);
        h.oa[0] = g * sx;
        h.oa[1] = g * sy;
        h.oa[2] = g * sz;
    }
    h.hop = 0;
    if (!e_launch) drift_start(a, i, I, h);
    else if (I.drift_abs > 0.0) a.s.e0[i] = static_cast<float>(*e_launch);
}

// Orbital energy of a launch from the |v|^2 and |s|^2 its bound test formed: 1 / |s| as in
// orbital_energy, so the baseline equals orbital_energy of the launched state.
__device__ __forceinline__ double launch_energy(const FastInst &I, double v2, double r2) {
    double ir = rsqrtf(static_cast<float>(r2));
    ir = ir * (1.5 - 0.5 * r2 * ir * ir);
    return 0.5 * v2 - I.p.GM * ir;
}

// Launch from the current surface position (ballistic.c:156-181; config: flux-weighted
// Maxwell-Boltzmann). Returns false when the reference's launch-speed escape test fires.
// kCfg: every instance of the launch is a config-model problem, so the reference-model branches
// of the event code are compiled out (shorter code on the path that high-gravity bodies take every
// few hundred steps). The FP32 engine maps the random words in FP32 with reciprocal square roots;
// the FP64 engine takes the plain FP64 kernel's maps.
template <int kMode, class A, typename R>
__device__ __forceinline__ bool launch(const A &a, long long i, const FastInst &I, HotT<R> &h,
                       StatAcc &st, R local_T, R thi, R fi) {
    const dsmc_params &p = I.p;
    Philox rng;
    rng.init(p.seed, p.instance, a.s.pid[i]);
    rng.event = a.s.evt[i];
    philox_next<Mode<kMode>::kRoll>(rng);
    a.s.evt[i] = rng.event;
    double s[3];
    get_pos(h, s);
    double vd[3];
    double e_launch = 0.0;
    bool have_e = false;
    if constexpr (is_f64<R>()) {
        if (Mode<kMode>::ref(p)) {
            // velocity_sample / velocity_sticking (velocity.c:49-73), ballistic.c:156-173
            const double KF = 2.0 * kPi * p.Radii * fabs(cos(thi)) / p.P;
            int idx = local_T >= 220.0 ? 20 : static_cast<int>(ceil(local_T / 10.0)) - 2;
            idx = idx < 0 ? 0 : (idx >= 23 ? 22 : idx);
            const double vr = I.t.vt_speeds[idx * 1000 + rng.w[0] % static_cast<uint32_t>(I.t.vt_count[idx])];
            double v_old[3];
            get_vel(h, v_old);
            const double vold2 = v_old[0] * v_old[0] + v_old[1] * v_old[1] + v_old[2] * v_old[2];
            const double vout = sqrt(p.alpha * vr * vr + (1.0 - p.alpha) * vold2);
            const double flyd = rng.raw(1) / kTwo32 * kPi + thi - kPi / 2.0;
            const double xi = rng.raw(2) / kTwo32 * kPi + fi - kPi / 2.0;
            vd[0] = cos(flyd) * sin(xi) * vout + KF * sin(fi + kPi / 2.0);
            vd[1] = cos(flyd) * cos(xi) * vout + KF * cos(fi + kPi / 2.0);
            vd[2] = sin(flyd) * vout;
            if (sqrt(vd[0] * vd[0] + vd[1] * vd[1] + vd[2] * vd[2]) >= p.ve) return false;
        } else {
            const double sigma = sqrt(p.kB_over_m * local_T);
            const double vn = sigma * sqrt(-2.0 * log(1.0 - rng.raw(0) / kTwo32));
            const double rho = sqrt(-2.0 * log(1.0 - rng.raw(1) / kTwo32));
            double sa, ca;
            sincos(2.0 * kPi * (rng.raw(2) / kTwo32), &sa, &ca);
            const double t1 = rho * ca, t2 = rho * sa;
            const double ir = rsqrt(s[0] * s[0] + s[1] * s[1] + s[2] * s[2]);
            const double n[3] = {s[0] * ir, s[1] * ir, s[2] * ir};
            double e[3] = {-n[1], n[0], 0.0};
            const double le2 = e[0] * e[0] + e[1] * e[1];
            if (le2 < 1e-24) { e[0] = 1.0; e[1] = 0.0; }
            else { const double il = rsqrt(le2); e[0] *= il; e[1] *= il; }
            const double nt[3] = {n[1] * e[2] - n[2] * e[1], n[2] * e[0] - n[0] * e[2], n[0] * e[1] - n[1] * e[0]};
            const double omega = p.P > 0.0 ? 2.0 * kPi / p.P : 0.0;
            const double rot[3] = {omega * s[1], -omega * s[0], 0.0};
#pragma unroll
            for (int k = 0; k < 3; k++) vd[k] = vn * n[k] + (sigma * t1) * e[k] + (sigma * t2) * nt[k] + rot[k];
            // FP64 escape/bound classification: E < 0 exactly when (v^2)^2 r^2 < (2 GM)^2
            const double v2 = vd[0] * vd[0] + vd[1] * vd[1] + vd[2] * vd[2];
            const double rr = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
            if (v2 * v2 * rr < 4.0 * p.GM * p.GM) st.bound++;
            e_launch = launch_energy(I, v2, rr);
            have_e = true;
        }
    } else {
        float v[3];
        if (Mode<kMode>::ref(p)) {
            const float KF = 2.0f * kPiF * static_cast<float>(p.Radii) * fabsf(cosf(thi)) / static_cast<float>(p.P);
            int idx = local_T >= 220.0f ? 20 : static_cast<int>(ceilf(local_T / 10.0f)) - 2;
            idx = idx < 0 ? 0 : (idx >= 23 ? 22 : idx);
            const float vr = static_cast<float>(I.t.vt_speeds[idx * 1000 + rng.w[0] % static_cast<uint32_t>(I.t.vt_count[idx])]);
            float vold2 = 0.0f;
#pragma unroll
            for (int k = 0; k < 3; k++) vold2 += h.vh[k] * h.vh[k];
            const float alpha = static_cast<float>(p.alpha);
            const float vout = sqrtf(alpha * vr * vr + (1.0f - alpha) * vold2);
            const float flyd = static_cast<float>(rng.w[1]) * (kPiF / 4294967296.0f) + thi - 0.5f * kPiF;
            const float xi = static_cast<float>(rng.w[2]) * (kPiF / 4294967296.0f) + fi - 0.5f * kPiF;
            float sf, cf, sx, cx, sr, cr;
            sincosf(flyd, &sf, &cf);
            sincosf(xi, &sx, &cx);
            sincosf(fi + 0.5f * kPiF, &sr, &cr);
            v[0] = cf * sx * vout + KF * sr;
            v[1] = cf * cx * vout + KF * cr;
            v[2] = sf * vout;
            if (sqrtf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) >= static_cast<float>(p.ve)) return false;
        } else {
            // the same maps of the random words as the FP64 path: log(1 - u) and angle 2 pi u
            const float sigma = sqrtf(static_cast<float>(p.kB_over_m) * local_T);
            const float vn = sigma * sqrtf(-2.0f * logf(1.0f - unit_open(rng.w[0])));
            const float rho = sqrtf(-2.0f * logf(1.0f - unit_open(rng.w[1])));
            float sa, ca;
            __sincosf(2.0f * kPiF * unit_open(rng.w[2]), &sa, &ca);   // argument in [0, 2 pi)
            const float t1 = rho * ca, t2 = rho * sa;
            // the event path stays short (no divisions, no FP64 square roots): unit normal and
            // east vector by reciprocal square roots
            const float px = h.sh[0] + h.sl[0], py = h.sh[1] + h.sl[1], pz = h.sh[2] + h.sl[2];
            const float ir = rsqrtf(fmaf(px, px, fmaf(py, py, pz * pz)));
            const float n[3] = {px * ir, py * ir, pz * ir};
            float e[3] = {-n[1], n[0], 0.0f};
            const float le2 = fmaf(e[0], e[0], e[1] * e[1]);
            if (le2 < 1e-12f) { e[0] = 1.0f; e[1] = 0.0f; }
            else { const float il = rsqrtf(le2); e[0] *= il; e[1] *= il; }
            const float nt[3] = {n[1] * e[2] - n[2] * e[1], n[2] * e[0] - n[0] * e[2], n[0] * e[1] - n[1] * e[0]};
            const float omega = p.P > 0.0 ? static_cast<float>(2.0 * kPi / p.P) : 0.0f;
            const float rot[3] = {omega * static_cast<float>(s[1]), -omega * static_cast<float>(s[0]), 0.0f};
#pragma unroll
            for (int k = 0; k < 3; k++) v[k] = vn * n[k] + (sigma * t1) * e[k] + (sigma * t2) * nt[k] + rot[k];
            // FP64 escape/bound classification of the launch: E = v^2/2 - GM/r < 0 exactly when
            // (v^2)^2 r^2 < (2 GM)^2, which needs no square root or division
            const double v2 = static_cast<double>(v[0]) * v[0] + static_cast<double>(v[1]) * v[1] +
                              static_cast<double>(v[2]) * v[2];
            const double rr = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
            if (v2 * v2 * rr < 4.0 * p.GM * p.GM) st.bound++;
            e_launch = launch_energy(I, v2, rr);
            have_e = true;
        }
        vd[0] = v[0];
        vd[1] = v[1];
        vd[2] = v[2];
    }
    set_vel(h, vd);
    start_hop_state(a, i, I, h, have_e ? &e_launch : nullptr);
    return true;
}

// Cell of a launch point from the latitude and longitude the particle had when it landed,
// starting in the lowest shell, moved by the comparison walks (no asin, atan2 or log).
template <class T, typename R>
__device__ __forceinline__ void enter_cell_near(const T &tab, HotT<R> &h, BoundsT<R> &b) {
    const R x = pos(h, 0), y = pos(h, 1), z = pos(h, 2);
    const R r2 = fma_r(x, x, fma_r(y, y, z * z));
    int ht = 0, td = (h.cell >> 8) & 0xff, fd = h.cell & 0xff;
    track_shell(tab, r2, ht);
    track_angles(tab, x, y, z, r2, td, fd);
    enter_cell(tab, h, b, pack_cell(ht, td, fd));
}

// Longitude of the centre of column fd (the reference's freeze scan, ballistic.c:140).
template <typename R>
__device__ __forceinline__ R column_centre(int fd, int ffd) {
    if constexpr (is_f64<R>()) return (fd + 0.5) / ffd * 2.0 * kPi;
    else return (fd + 0.5f) / ffd * 2.0f * kPiF;
}

// Turns the position by `cols` columns of longitude (the advanced runner's freeze scan,
// advanced.c:290-300).
template <typename R>
__device__ __forceinline__ void turn_to_column(HotT<R> &h, int cols, int ffd) {
    const double rot_fi = static_cast<double>(cols) / ffd * 2.0 * kPi;
    const double cs = cos(rot_fi), sn = sin(rot_fi);
    double s[3];
    get_pos(h, s);
    const double n0 = s[0] * cs - s[1] * sn, n1 = s[0] * sn + s[1] * cs;
    s[0] = n0;
    s[1] = n1;
    set_pos(h, s);
}

// Start of a hop (ballistic.c:124-181, advanced.c:271-333): weight and life checks, the
// reference freeze scan, the launch and the starting cell. Returns 0 when the particle flies,
// else its fate.
template <int kMode, class A, typename R>
__device__ __forceinline__ int hop_top(const A &a, long long i, const FastInst &I, HotT<R> &h,
                       BoundsT<R> &b, StatAcc &st, R thi, R fi, R local_T, bool first) {
    const dsmc_params &p = I.p;
    const R W = weight(I, h);
    if (W < static_cast<R>(p.w_min)) return DSMC_FATE_PHOTOLYSED;
    if (p.life_step_cap > 0 && h.steps >= p.life_step_cap) return DSMC_FATE_STEP_CAP;
    if (Mode<kMode>::ref(p)) {
        const int ftd = p.ftd, ffd = p.ffd;
        int td, fd;
        ref_index(thi, fi, ftd, ffd, td, fd);
        const double *T = I.t.T_map;
        local_T = static_cast<R>(T[td * ffd + fd]);
        if (local_T < static_cast<R>(p.freeze_T)) {
            bool found = false;
            float rest = a.s.rest[i];
            if (I.t.warm) {
                if (p.runner != DSMC_RUNNER_BALLISTIC) horizon_add(I, td, fd, W);
                const int wait = I.t.warm[td * ffd + fd];
                for (int k = wait ? wait : ffd; k > 0; k--) rest += static_cast<float>(p.dt_rot);
                if (wait) {
                    found = true;
                    if (p.runner == DSMC_RUNNER_BALLISTIC) {
                        fd = (fd + wait) % ffd;
                    } else {
                        turn_to_column(h, wait - fd, ffd);
                        fd = wait % ffd;
                    }
                    fi = column_centre<R>(fd, ffd);
                }
            } else if (p.runner == DSMC_RUNNER_BALLISTIC) {
                for (int add = 0; add < ffd; add++) {
                    rest += static_cast<float>(p.dt_rot);
                    const int check = (fd + add + 1) % ffd;
                    if (T[td * ffd + check] >= p.freeze_T) {
                        fd = check;
                        fi = column_centre<R>(fd, ffd);
                        found = true;
                        break;
                    }
                }
            } else {
                horizon_add(I, td, fd, W);
                for (int add = 1; add <= ffd; add++) {
                    rest += static_cast<float>(p.dt_rot);
                    if (T[td * ffd + (add % ffd)] >= p.freeze_T) {
                        turn_to_column(h, add - fd, ffd);
                        fd = add % ffd;
                        fi = column_centre<R>(fd, ffd);
                        found = true;
                        break;
                    }
                }
            }
            a.s.rest[i] = rest;
            if (!found) {
                horizon_add(I, td, fd, W);
                return DSMC_FATE_FROZEN;
            }
            local_T = static_cast<R>(T[td * ffd + fd]);
        }
    }
    if (!launch<kMode>(a, i, I, h, st, local_T, thi, fi)) return DSMC_FATE_ESCAPED;
    // the running weight restarts from its exact value at every launch (and at every cell
    // change): points of the particle's own trajectory, so results do not depend on where
    // kernel launches begin or end (the launch changes neither w0 nor the day count)
    h.W = W;
    const TabOf<A, R> tab{I};
    if (Mode<kMode>::kHist) flush_hist(I, h, h.ci);
    if (first)
        enter_cell(tab, h, b, cell_from_scratch(tab, pos(h, 0), pos(h, 1), pos(h, 2)));
    else
        enter_cell_near(tab, h, b);
    return 0;
}

// Latitude and longitude of the current position in FP32 (the reference model's relaunch
// angles, ballistic.c:245-247).
__device__ __forceinline__ void angles_of_f(const Hot &h, float &thi, float &fi) {
    const float x = h.sh[0] + h.sl[0], y = h.sh[1] + h.sl[1], z = h.sh[2] + h.sl[2];
    thi = asinf(fminf(1.0f, fmaxf(-1.0f, z * rsqrtf(fmaf(x, x, fmaf(y, y, z * z))))));
    fi = atan2f(x, y);
    if (fi < 0.0f) fi += 2.0f * kPiF;
}

// Face of the icosphere containing unit direction n, from the FP32 tables: the nearest of the 20
// base-face centroids, then one corner-cut test triple per subdivision level (the FP64 descent of
// locate_face on FP32 copies).
__device__ __forceinline__ int locate_face_f(const float4 *tab, int nlevel, const float n[3]) {
    int node = 0;
    float best = -2.0f;
#pragma unroll 4
    for (int f = 0; f < 20; f++) {
        const float4 c = __ldg(tab + f);
        const float d = c.x * n[0] + c.y * n[1] + c.z * n[2];
        if (d > best) { best = d; node = f; }
    }
    int offset = 0, width = 20;
    for (int level = 0; level < nlevel; level++) {
        const float4 *pl = tab + 20 + 3 * (offset + node);
        const float4 a = __ldg(pl), b = __ldg(pl + 1), c = __ldg(pl + 2);
        const int child = (a.x * n[0] + a.y * n[1] + a.z * n[2] > 0.0f) ? 0
                        : (b.x * n[0] + b.y * n[1] + b.z * n[2] > 0.0f) ? 1
                        : (c.x * n[0] + c.y * n[1] + c.z * n[2] > 0.0f) ? 2 : 3;
        node = node * 4 + child;
        offset += width;
        width *= 4;
    }
    return node;
}

// Landing (ballistic.c:239-264): polar deposit (reference) or night freeze-out / day-side
// re-emission point (config). Returns 0 to start a new hop, else the fate.
template <int kMode, class A, typename R>
__device__ __forceinline__ int land(const A &a, long long i, const FastInst &I, HotT<R> &h, R &thi,
                    R &fi, R &local_T) {
    const dsmc_params &p = I.p;
    int td, fd;
    if (Mode<kMode>::ref(p)) {
        if constexpr (is_f64<R>()) angles_of(h, thi, fi);
        else angles_of_f(h, thi, fi);
        ref_index(thi, fi, p.ftd, p.ffd, td, fd);
        if (td <= 1 || td >= p.ftd - 2) {
            horizon_add(I, td, fd, static_cast<R>(0.05) * weight(I, h));
            h.w0 *= static_cast<R>(0.95);
        }
        return 0;
    }
    if constexpr (is_f64<R>()) {
        // FP64 normal and face descent (the plain kernel's landing arithmetic)
        double s[3];
        get_pos(h, s);
        const double r2 = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
        const double Ri = sqrt(r2);
        const double nd[3] = {s[0] / Ri, s[1] / Ri, s[2] / Ri};
        if (nd[0] * p.sun[0] + nd[1] * p.sun[1] + nd[2] * p.sun[2] <= 0.0) {
            td = (h.cell >> 8) & 0xff;
            fd = h.cell & 0xff;
            track_angles(TabOf<A, R>{I}, s[0], s[1], s[2], r2, td, fd);
            horizon_add(I, td, fd, weight(I, h));
            return DSMC_FATE_FROZEN;
        }
        const double sn[3] = {nd[0] * p.Radii, nd[1] * p.Radii, nd[2] * p.Radii};
        set_pos(h, sn);
        const int face = locate_face(I.t, nd);
        a.s.face[i] = face;
        local_T = I.t.face_T[face];
        return 0;
    } else {
        // FP32 normal; the landing cell of a night-side freeze-out by comparison walks from the
        // last cell (the upper-inclusive cells of grid_spherical_to_index without asin or atan2)
        const float x = h.sh[0] + h.sl[0], y = h.sh[1] + h.sl[1], z = h.sh[2] + h.sl[2];
        const float r2 = fmaf(x, x, fmaf(y, y, z * z));
        const float ir = rsqrtf(r2);
        const float n[3] = {x * ir, y * ir, z * ir};
        if (fmaf(n[0], static_cast<float>(p.sun[0]), fmaf(n[1], static_cast<float>(p.sun[1]),
                                                          n[2] * static_cast<float>(p.sun[2]))) <= 0.0f) {
            td = (h.cell >> 8) & 0xff;
            fd = h.cell & 0xff;
            track_angles(TabOf<A, R>{I}, x, y, z, r2, td, fd);
            horizon_add(I, td, fd, weight(I, h));
            return DSMC_FATE_FROZEN;
        }
        // day side: re-emission from the surface point below the landing point
        const double nd[3] = {n[0], n[1], n[2]};
        const double s[3] = {nd[0] * p.Radii, nd[1] * p.Radii, nd[2] * p.Radii};
        set_pos(h, s);
        int face;
        if (I.face_f) {
            // hops are short next to the face size on high-gravity bodies: try the face of the
            // last launch point first (three sign tests), descend the tree only when the point
            // left it
            const int last = a.s.face[i];
            const int nnode = 20 * ((1 << (2 * I.t.nlevel)) - 1) / 3;
            const float4 *ed = I.face_f + 20 + 3 * nnode + 3 * last;
            bool inside = last >= 0;
            if (inside) {
                const float4 e0 = __ldg(ed), e1 = __ldg(ed + 1), e2 = __ldg(ed + 2);
                inside = (e0.x * n[0] + e0.y * n[1] + e0.z * n[2] >= 0.0f) &
                         (e1.x * n[0] + e1.y * n[1] + e1.z * n[2] >= 0.0f) &
                         (e2.x * n[0] + e2.y * n[1] + e2.z * n[2] >= 0.0f);
            }
            face = inside ? last : locate_face_f(I.face_f, I.t.nlevel, n);
            a.s.face[i] = face;
        } else {
            face = locate_face(I.t, nd);
        }
        local_T = static_cast<float>(I.t.face_T[face]);
        return 0;
    }
}

// End of a particle's life: per-particle rows (layout of ballistic.c:120,273-276 and
// advanced.c:262-267,439-444), counters, deposits flushed.
template <int kMode, class A, typename R>
__device__ __forceinline__ void finish(const A &a, long long i, const FastInst &I, HotT<R> &h,
                       StatAcc &st, int fate) {
    const dsmc_params &p = I.p;
    const DevTables &t = I.t;
    const bool ref = p.model == DSMC_MODEL_REFERENCE, adv = p.runner == DSMC_RUNNER_ADVANCED;
    const unsigned pid = a.s.pid[i];
    const int ncol = a.s.ncol[i];
    const long long slot = static_cast<long long>(pid) - t.out_base;
    if (slot >= 0 && slot < t.out_cap) {
        if (t.ttime && (fate != DSMC_FATE_ESCAPED || !ref)) {
            R thi, fi;
            angles_of(h, thi, fi);
            const float rest = a.s.rest[i];
            const double flight = static_cast<double>(h.steps) * p.dt_step;
            t.ttime[1 * t.out_cap + slot] = thi;
            t.ttime[2 * t.out_cap + slot] = flight + rest;
            t.ttime[3 * t.out_cap + slot] = weight(I, h);
            t.ttime[4 * t.out_cap + slot] = flight;
            if (adv || !ref) {
                t.ttime[7 * t.out_cap + slot] = rest;
                t.ttime[8 * t.out_cap + slot] = ncol;
            }
        }
        if (t.fate) t.fate[slot] = fate;
        if (t.steps) t.steps[slot] = h.steps;
    }
    st.finished++;
    st.collisions += ncol;
    if (fate == DSMC_FATE_ESCAPED) st.escaped++;
    flush_cell(I, h);
    flush_hist(I, h, hist_cell<kMode>(h));
    h.ci = -1;
    h.inst = -1;
}

// A collision against a partner drawn from the cell's fitted speed CDF (advanced.c:374-396).
template <int kMode, class A, typename R>
__device__ __forceinline__ void collide(const A &a, long long i, const FastInst &I, HotT<R> &h,
                        long long pidx) {
    const dsmc_params &p = I.p;
    const DevTables &t = I.t;
    Philox rng;
    rng.init(p.seed, p.instance, a.s.pid[i]);
    rng.event = a.s.evt[i];
    philox_next<Mode<kMode>::kRoll>(rng);
    const double *coef = t.cdf_coef + DSMC_CDF_STRIDE * pidx;
    const double *box = t.cdf_box + 4 * pidx;
    double v[3];
    get_vel(h, v);
    const double vv2 = cdf_sample(coef, box, t.cdf_total[pidx], t.cdf_degree, rng.raw(0) / kTwo32);
    double col_p = -1.0;
    if (p.scatter == DSMC_SCATTER_REFERENCE) {
        const double thi2 = kPi * rng.raw(1) / kTwo32 - kPi / 2.0;
        const double fi2 = 2.0 * kPi * rng.raw(2) / kTwo32;
        const double v2[3] = {vv2 * cos(thi2) * cos(fi2), vv2 * cos(thi2) * sin(fi2), vv2 * sin(thi2)};
        for (int k = 0; k < 3; k++) v[k] = (v[k] + v2[k]) + 0.5 * (v[k] - v2[k]);
        if (p.redraw_col_threshold) col_p = rng.raw(3) / kTwo32;
    } else {
        double d2[3], om[3];
        if constexpr (is_f64<R>()) {
            // the plain FP64 kernel's maps of the random words
            unit_sphere_d(rng.raw(1) / kTwo32, rng.raw(2) / kTwo32, d2);
            if (p.redraw_col_threshold) col_p = rng.raw(3) / kTwo32;
            philox_next<Mode<kMode>::kRoll>(rng);
            unit_sphere_d(rng.raw(0) / kTwo32, rng.raw(1) / kTwo32, om);
        } else {
            float d2f[3], omf[3];
            unit_sphere_f(unit_open(rng.w[1]), unit_open(rng.w[2]), d2f);
            if (p.redraw_col_threshold) col_p = rng.raw(3) / kTwo32;
            philox_next<Mode<kMode>::kRoll>(rng);
            unit_sphere_f(unit_open(rng.w[0]), unit_open(rng.w[1]), omf);
            for (int k = 0; k < 3; k++) { d2[k] = d2f[k]; om[k] = omf[k]; }
        }
        double g2 = 0.0, vcm[3];
        for (int k = 0; k < 3; k++) {
            const double v2k = vv2 * d2[k];
            g2 += (v[k] - v2k) * (v[k] - v2k);
            vcm[k] = 0.5 * (v[k] + v2k);
        }
        const double hg = 0.5 * sqrt(g2);
        for (int k = 0; k < 3; k++) v[k] = vcm[k] + hg * om[k];
    }
    a.s.evt[i] = rng.event;
    a.s.ncol[i] += 1;
    if (col_p >= 0.0) {
        if constexpr (is_f64<R>()) h.pthr = -log1p(-col_p);
        else h.pthr = -log1pf(-static_cast<float>(col_p));
    }
    set_vel(h, v);
    h.pcol = R(0);
    drift_start(a, i, I, h);
}

// Next work index of the device queue: one atomic per group of lanes asking together.
__device__ __forceinline__ unsigned long long grab_work(FastCounters *ctr) {
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    const unsigned rank = __popc(m & ((1u << lane) - 1u));
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(&ctr->next, static_cast<unsigned long long>(__popc(m)));
    base = __shfl_sync(m, base, leader);
    return base + rank;
}

template <typename A>
__device__ __forceinline__ int find_inst(const A &a, unsigned long long w) {
    if constexpr (A::kOne) return 0;
    int lo = 0, hi = static_cast<int>(a.ctr->ninst) - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (static_cast<unsigned long long>(a.inst(mid).work_base) <= w) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Fills an empty slot with the next particle of the queue, at its starting point; hop_top then
// launches it. Returns false when the queue is empty.
template <int kMode, class A, typename R>
__device__ __forceinline__ bool take_next(const A &a, long long i, HotT<R> &h, StatAcc &st, R &thi,
                                          R &fi, R &local_T) {
    local_T = R(0);
    const unsigned long long w = grab_work(a.ctr);
    if (w >= a.ctr->total) return false;
    const int ii = find_inst(a, w);
    const FastInst &I = a.inst(ii);
    const dsmc_params &p = I.p;
    if (ii != st.inst) {
        flush_stats_lane(a, st);
        st.inst = ii;
    }
    const unsigned pid = static_cast<unsigned>(I.pid_begin + static_cast<long long>(w - I.work_base));
    h.inst = ii;
    Philox rng;
    rng.init(p.seed, p.instance, pid);
    philox_next<Mode<kMode>::kRoll>(rng);
    h.w0 = R(1);
    h.nday = 0;
    h.steps = 0;
    h.hop = 0;
    h.pcol = R(0);
    h.ci = -1;
    h.run_w = R(0);
    h.hist_key = -1;
    h.hist_cnt = 0;
    const double zero[3] = {0.0, 0.0, 0.0};
    set_vel(h, zero);
    double col_p = 0.0;
    double s[3];
    if (Mode<kMode>::ref(p)) {
        const bool adv = p.runner == DSMC_RUNNER_ADVANCED;
        if (adv) col_p = rng.raw(0) / kTwo32;
        const int o = adv ? 1 : 0;
        const double th = rng.raw(o) / kTwo32 * kPi - kPi / 2.0;
        const double ph = rng.raw(o + 1) / kTwo32 * 2.0 * kPi;
        s[0] = p.Radii * cos(th) * sin(ph);
        s[1] = p.Radii * cos(th) * cos(ph);
        s[2] = p.Radii * sin(th);
        thi = static_cast<R>(th);
        fi = static_cast<R>(ph);
        int td, fd;
        ref_index(thi, fi, p.ftd, p.ffd, td, fd);
        local_T = static_cast<R>(I.t.T_map[td * p.ffd + fd]);
    } else {
        const int f = pick_face(I.t, rng.raw(0) / kTwo32);
        a.s.face[i] = f;
        double u1 = rng.raw(1) / kTwo32, u2 = rng.raw(2) / kTwo32;
        col_p = rng.raw(3) / kTwo32;
        if (u1 + u2 > 1.0) { u1 = 1.0 - u1; u2 = 1.0 - u2; }
        const double *fv = I.t.face_verts + 9 * f;
        double q[3];
        for (int k = 0; k < 3; k++) q[k] = fv[k] + u1 * (fv[3 + k] - fv[k]) + u2 * (fv[6 + k] - fv[k]);
        // |q|^-1 from the FP32 estimate and one Newton step in FP64 (relative error ~1e-14)
        const double q2 = q[0] * q[0] + q[1] * q[1] + q[2] * q[2];
        double iq = rsqrtf(static_cast<float>(q2));
        iq = iq * (1.5 - 0.5 * q2 * iq * iq);
        for (int k = 0; k < 3; k++) s[k] = q[k] * (p.Radii * iq);
        local_T = static_cast<R>(I.t.face_T[f]);
        thi = fi = R(0);   // the config model's launch does not use the angles
    }
    a.s.pid[i] = pid;
    a.s.evt[i] = rng.event;
    a.s.ncol[i] = 0;
    a.s.rest[i] = 0.0f;
    if (p.runner != DSMC_RUNNER_ADVANCED) {
        h.pthr = R(0);
    } else {
        if constexpr (is_f64<R>()) h.pthr = -log1p(-col_p);
        else h.pthr = -log1pf(-static_cast<float>(col_p));
    }
    set_pos(h, s);
    const long long slot = static_cast<long long>(pid) - I.t.out_base;
    if (I.t.ttime && slot >= 0 && slot < I.t.out_cap) {
        if (p.model != DSMC_MODEL_REFERENCE) angles_of(h, thi, fi);
        I.t.ttime[slot] = thi;
        if (p.runner == DSMC_RUNNER_ADVANCED || p.model != DSMC_MODEL_REFERENCE) {
            I.t.ttime[5 * I.t.out_cap + slot] = fi;
            I.t.ttime[6 * I.t.out_cap + slot] = local_T;
        }
    }
    return true;
}

// Fills an empty slot with the next particle and launches it; particles that end at their first
// launch are finished here and the next one is taken.
template <int kMode, class A, typename R>
__device__ __forceinline__ bool start_next(const A &a, long long i, HotT<R> &h, BoundsT<R> &b, StatAcc &st) {
    R thi, fi, local_T;
    while (take_next<kMode>(a, i, h, st, thi, fi, local_T)) {
        const FastInst &I = a.inst(h.inst);
        const int fate = hop_top<kMode>(a, i, I, h, b, st, thi, fi, local_T, true);
        if (fate == 0) return true;
        finish<kMode>(a, i, I, h, st, fate);
    }
    return false;
}

// Position of the particle being pushed, with |s|^2 and the acceleration there (FP32: the velocity
// change -a dt of a step; FP64: a).
template <typename R>
struct PosT { R x, y, z, r2, a[3]; };

__device__ __forceinline__ void gravity(PosT<float> &q, float GM) {
    const float ir = rsqrtf(q.r2);
    const float g = -GM * (ir * ir * ir);
    const F2 a = mul2(F2{g, g}, F2{q.x, q.y});
    q.a[0] = a.x;
    q.a[1] = a.y;
    q.a[2] = g * q.z;
}

__device__ __forceinline__ void gravity(PosT<double> &q, double GM) {
    const double ir = rsqrt(q.r2);
    const double g = GM * (ir * ir * ir);
    q.a[0] = g * q.x;
    q.a[1] = g * q.y;
    q.a[2] = g * q.z;
}

// The step's inside tests against the current cell's bounds. warp_kernel's unrolled steps keep only
// their conjunction and repeat the three in the slow path: kept for it, each test cost a step an
// instruction to hold (1e7 Ceres-like particles 281 against 278 ms).
template <typename R>
__device__ __forceinline__ bool in_shell(const PosT<R> &q, const BoundsT<R> &b) {
    return (q.r2 > b.r2lo) & (q.r2 <= b.r2hi);
}
template <typename R>
__device__ __forceinline__ bool in_row(const PosT<R> &q, const BoundsT<R> &b) {
    const R zz = q.z * fabs(q.z);
    return (zz > q.r2 * b.zlo) & (zz <= q.r2 * b.zhi);
}
template <typename R>
__device__ __forceinline__ bool in_column(const PosT<R> &q, const BoundsT<R> &b) {
    return (q.x * b.c0 - q.y * b.s0 > R(0)) & (q.x * b.c1 - q.y * b.s1 <= R(0));
}

template <typename R>
__device__ __forceinline__ void start_pos(const HotT<R> &h, PosT<R> &q) {
    q.x = pos(h, 0);
    q.y = pos(h, 1);
    q.z = pos(h, 2);
    q.r2 = fma_r(q.x, q.x, fma_r(q.y, q.y, q.z * q.z));
}

// One Verlet step of the reference's variant. FP32: (hi, lo) position and velocity sums, and the
// acceleration carried as the velocity change -a * dt (c1 = 1.5 dt, c2 = dt / 6; three multiplies
// fewer per step, and at a power-of-two dt the same roundings as a and dt kept apart); FP64: plain
// doubles with c1 = 1.5 dt^2, c2 = dt^2 / 6. q holds the current position on entry and the new one
// on exit; d the displacement.
// The FP32 update runs in packed pairs: x and y of a vector side by side, and for z the position
// and velocity sums side by side. The acceleration keeps its minus sign because packed operands
// take no negation. 1e7 Ceres-like particles: 2.23e11 -> 2.32e11 particle-steps/s, 3e6
// Moon-like: 1.28e11 -> 1.37e11, the 16-exosphere batch 1.32e11 -> 1.41e11; bit-identical.
__device__ __forceinline__ void verlet_step(Hot &h, PosT<float> &q, float dt, float c1, float c2,
                                            float d[3]) {
    const F2 a{q.a[0], q.a[1]}, dt2{dt, dt}, c12{c1, c1}, c22{c2, c2};
    const F2 dxy = fma2(F2{h.vh[0], h.vh[1]}, dt2,
                        fma2(F2{h.vl[0], h.vl[1]}, dt2, fma2(a, c12, mul2(F2{h.oa[0], h.oa[1]}, c22))));
    const float dz = fmaf(h.vh[2], dt, fmaf(h.vl[2], dt, fmaf(q.a[2], c1, h.oa[2] * c2)));
    accumulate2(h.sh[0], h.sh[1], h.sl[0], h.sl[1], dxy);
    accumulate2(h.vh[0], h.vh[1], h.vl[0], h.vl[1], a);
    accumulate2(h.sh[2], h.vh[2], h.sl[2], h.vl[2], F2{dz, q.a[2]});
    h.oa[0] = a.x;
    h.oa[1] = a.y;
    h.oa[2] = q.a[2];
    d[0] = dxy.x;
    d[1] = dxy.y;
    d[2] = dz;
    const F2 xy = add2(F2{h.sh[0], h.sh[1]}, F2{h.sl[0], h.sl[1]});
    q.x = xy.x;
    q.y = xy.y;
    q.z = h.sh[2] + h.sl[2];
    q.r2 = fmaf(q.x, q.x, fmaf(q.y, q.y, q.z * q.z));
}

__device__ __forceinline__ void verlet_step(HotT<double> &h, PosT<double> &q, double dt, double c1,
                                            double c2, double d[3]) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        d[k] = fma(h.vh[k], dt, -fma(q.a[k], c1, h.oa[k] * c2));
        h.sh[k] += d[k];
        h.vh[k] -= q.a[k] * dt;
        h.oa[k] = q.a[k];
    }
    q.x = h.sh[0];
    q.y = h.sh[1];
    q.z = h.sh[2];
    q.r2 = fma(q.x, q.x, fma(q.y, q.y, q.z * q.z));
}

// Event gathering (see fast_kernel): Verlet steps per chunk between the warp's votes.
constexpr int kChunk = 32;

// Adds the step to the speed histogram's run of one bin in one cell; `from` is the run's cell. The
// histogram loop (mode 4) counts every step, so the run's cell is the one the step started in; in the
// general loop a step may count nothing, so the cell is kept beside the run and the run is settled at
// the end of a launch (the slots have no room for it). 1e6 Ceres-like particles: 41.6 and 62.8 ms, the
// time of runs under a 32-bit index of cell and bin; with the run settled by the cell walk 42.4 and
// 63.7 ms, with a 64-bit index 43.3 and 63.3 ms.
template <typename R>
__device__ __forceinline__ void count_speed(const FastInst &I, const StepConst<R> &k, HotT<R> &h, int from) {
    const R sp = sqrt(fma_r(h.vh[0], h.vh[0], fma_r(h.vh[1], h.vh[1], h.vh[2] * h.vh[2])));
    const int bin = min(static_cast<int>(static_cast<float>(sp) * k.inv_bw), k.nbins - 1);
    if ((bin == h.hist_key) & (from == h.ci)) {
        h.hist_cnt++;
    } else {
        flush_hist(I, h, from);
        h.hist_key = bin;
        h.hist_cnt = 1;
    }
}

// The rest of a segment of a particle whose position is not a number (a launch draw of exactly 1
// in FP32, about once in 1e7 launches, gives it an infinite speed): every test of every step is
// false, so it stays in its cell, outside the day side, and deposits its weight until the segment
// ends. Stepping it instead sent it through the cell walk on every step, 0.37 us a step, which
// was the length of a whole solve of 3e5 Moon-like particles (10.7 ms with such a particle, 8.6 ms
// without). Returns the steps taken; the deposits are summed one by one, as the loop would.
template <typename R>
__device__ __forceinline__ int drift_nowhere(HotT<R> &h, int taken, int n) {
    h.run_w += h.W;   // the step that found it
    for (; taken < n; taken++) h.run_w += h.W;
    return taken;
}

// kMaxThreads x kMinBlocks: the register budget the allocation must respect (65536 registers
// per SM shared by kMinBlocks blocks of kMaxThreads). The launch shape picks the variant.
// kMode: see Mode. A: the queue (FastArgsT) or one instance (OneArgsT). R: float (FAST_FP32) or
// double (FAST_FP64).
// The step loop runs in segments: an inner loop pushes the particle until an event (landing,
// escape, cap) or the end of the launch's step budget, so the per-step path carries no instance
// or restart checks, and the lean loops settle their step counters once per segment. This
// structure measured 21 % faster than one flat loop over steps with the same arithmetic (and
// bit-identical results).
template <int kMaxThreads, int kMinBlocks, int kMode, int kUnroll, class A, typename R>
__global__ void __launch_bounds__(kMaxThreads, kMinBlocks) fast_kernel(const __grid_constant__ A a) {
    using M = Mode<kMode>;
    using Tab = TabOf<A, R>;
    constexpr bool kLean = !M::kAny;
    if constexpr (A::kOne) SharedTab<R>::fill(a.one);
    const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long long i = a.slot(t);
    HotOf<kMode, R> h;
    if (i >= 0) load_hot(a.s, i, a.nslots, h);
    else h.inst = -1;
    StatAcc st;
    st.inst = h.inst;
    BoundsT<R> b;
    bool alive = h.inst >= 0;
    if (alive) {
        // reload the cached bounds of the saved cell without flushing its pending deposits
        const int ci = h.ci;
        const R run_w = h.run_w;
        h.ci = -1;
        enter_cell(Tab{a.inst(h.inst)}, h, b, h.cell);
        h.ci = ci;
        h.run_w = run_w;
    } else if (i >= 0) {
        // a queue of fewer particles than slots starts on the lanes that fill_warps chose
        const long long warps = a.ctr->fill_warps;
        if (warps == 0 || ((t >> 5) < warps && (t & 31) * warps + (t >> 5) < static_cast<long long>(a.ctr->total)))
            alive = start_next<kMode>(a, i, h, b, st);
    }
    int cur = -1;
    StepConst<R> kreg;
    R dt = R(0), c1 = R(0), c2 = R(0);
    if constexpr (A::kOne) {
        dt = a.k.dt; c1 = a.k.c1; c2 = a.k.c2;
    }
    const FastInst *Ip = nullptr;
    int budget = a.K;

    while (alive && budget > 0) {
        if constexpr (!A::kOne) {
            if (h.inst != cur) {
                cur = h.inst;
                Ip = &a.inst(cur);
                kreg = step_consts<R>(*Ip);
                dt = kreg.dt; c1 = kreg.c1; c2 = kreg.c2;
            }
        }
        const StepConst<R> &k = [&]() -> const StepConst<R> & {
            if constexpr (A::kOne) return a.k;
            else return kreg;
        }();
        const FastInst &I = [&]() -> const FastInst & {
            if constexpr (A::kOne) return a.one;
            else return *Ip;
        }();
        // One segment: steps until an event or the end of the launch's budget. The lean loops
        // also stop at the life cap (config model) or the hop cap (reference model), so their
        // step counters are settled once per segment.
        PosT<R> q;
        start_pos(h, q);
        const int n = M::kCfg ? min(budget, k.life_cap - h.steps)
                    : M::kRef ? min(budget, k.hop_cap - h.hop) : budget;
        // the step of this segment that the skip-first rule leaves without a deposit
        const int skip = M::kRef && (k.flags & kFlagSkipFirst) && h.hop == 0 ? 1 : 0;
        int taken = 0;
        int event = 0;   // 1 landed (or hop cap), 2 escaped, 3 life cap
        // Lanes whose particle lands leave the step loop and run their event code while the warp
        // serialises it against the lanes still stepping. Where hops are short (high-gravity
        // bodies, a landing every ~200 steps) that leaves most lanes idle, so there the warp
        // steps in chunks of kChunk and, between chunks, lets the stopped lanes wait until they
        // have idled `limit` lane-chunks in all: then every waiting lane takes its event
        // together. Long hops (Ceres-like) keep the free-running loop. The limit is the largest
        // of the instances of the lanes that enter the segment together, so it is uniform.
        const unsigned peers = __activemask();
        int limit;
        if constexpr (A::kOne) limit = a.gather;
        else limit = static_cast<int>(__reduce_max_sync(peers, static_cast<unsigned>(I.gather)));
        const bool gather = limit > 0;
        const int npeer = __popc(peers);
        int idle = 0;
        for (;;) {
        const int lim = gather ? min(n, taken + kChunk) : n;
        if constexpr (kUnroll > 1) {
        static_assert(kMode == 1, "the sparse loop exists for the lean ballistic loop");
        gravity(q, k.GM);
        while (!event && taken < lim) {
            R d[3];
            bool in_r = true, in_t = true, in_f = true, left = false;
            auto settle = [&]() {   // a step's photolysis and deposit, once the cell is known
                if (fma_r(q.x, k.sx, fma_r(q.y, k.sy, q.z * k.sz)) > R(0)) {
                    h.nday++;
                    h.W *= k.fday;
                }
                h.run_w += h.W;
            };
            const bool whole = taken + kUnroll <= lim;
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                verlet_step(h, q, dt, c1, c2, d);
                gravity(q, k.GM);
                taken++;
                const R zz = q.z * fabs(q.z);
                in_r = (q.r2 > b.r2lo) & (q.r2 <= b.r2hi);
                in_t = (zz > q.r2 * b.zlo) & (zz <= q.r2 * b.zhi);
                in_f = (q.x * b.c0 - q.y * b.s0 > R(0)) & (q.x * b.c1 - q.y * b.s1 <= R(0));
                if (!(in_r & in_t & in_f)) {
                    left = true;
                    break;
                }
                settle();
                if (u == 0 && !whole) break;
            }
            if (left) {
                if (q.r2 <= k.rl2) {
                    event = 1;
                    break;
                }
                if (q.r2 >= k.re2) {
                    event = 2;
                    break;
                }
                if (!move_cell<true>(Tab{I}, h, b, q.x, q.y, q.r2, q.z * fabs(q.z), in_r, in_t, in_f) &&
                    q.r2 != q.r2) {
                    taken = drift_nowhere(h, taken, n);
                    break;
                }
                settle();
            }
        }
        } else {
        while (!event && taken < lim) {
            R d[3];
            gravity(q, k.GM);
            verlet_step(h, q, dt, c1, c2, d);
            taken++;
            const int ii = kLean ? 1 : h.hop;
            if (!kLean) {
                h.steps++;
                h.hop++;
            }
            const int from = h.ci;
            const R zz = q.z * fabs(q.z);
            const bool in_r = (q.r2 > b.r2lo) & (q.r2 <= b.r2hi);
            const bool in_t = (zz > q.r2 * b.zlo) & (zz <= q.r2 * b.zhi);
            const bool in_f = (q.x * b.c0 - q.y * b.s0 > R(0)) & (q.x * b.c1 - q.y * b.s1 <= R(0));
            if (!(in_r & in_t & in_f)) {
                if (q.r2 <= k.rl2) {
                    event = 1;
                    break;
                }
                if (q.r2 >= k.re2) {
                    event = 2;
                    break;
                }
                if (!move_cell<!M::kAny && !M::kCol>(Tab{I}, h, b, q.x, q.y, q.r2, zz, in_r, in_t, in_f) &&
                    kMode == 1 && q.r2 != q.r2) {
                    taken = drift_nowhere(h, taken, n);
                    break;
                }
            }
            const bool day = M::kRef || (M::kAny && (k.flags & kFlagRef))
                                 ? ((h.cell & 0xff) < k.half_ffd)
                                 : (fma_r(q.x, k.sx, fma_r(q.y, k.sy, q.z * k.sz)) > R(0));
            if (day) {
                h.nday++;
                h.W *= k.fday;
            }
            if (M::kCfg || (M::kRef && taken != skip) ||
                (M::kAny && !((k.flags & kFlagSkipFirst) && ii == 0))) {
                bool collided = false;
                if ((M::kAny ? (k.flags & kFlagCollide) != 0 : M::kCol) &&
                    (A::kOne ? h.nsig != R(0) : h.nsig > R(0))) {
                    const R rate = A::kOne ? fabs(h.nsig) : h.nsig;
                    h.pcol = fma_r(sqrt(fma_r(d[0], d[0], fma_r(d[1], d[1], d[2] * d[2]))), rate, h.pcol);
                    if (h.pcol > h.pthr && (!A::kOne || h.nsig > R(0))) {
                        const int ht = h.cell >> 16, td = (h.cell >> 8) & 0xff, fd = h.cell & 0xff;
                        const long long pidx = (static_cast<long long>(td) * I.p.ffd + fd) * I.p.hd + ht;
                        if (A::kOne || (ht < k.col_ht && __ldg(I.t.cdf_valid + pidx))) {
                            collide<kMode>(a, i, I, h, pidx);
                            collided = true;
                        }
                    }
                }
                if (!collided) {
                    h.run_w += h.W;
                    if (M::kHist || (M::kAny && (k.flags & kFlagHist))) {
                        count_speed(I, k, h, M::kHist ? from : hist_cell<kMode>(h));
                        if (M::kAny) hist_cell<kMode>(h) = h.ci;
                    }
                }
            }
            if (!kLean) {
                if (h.steps >= k.life_cap) event = 3;
                else if (h.hop >= k.hop_cap) event = 1;
            }
        }
        }
        if (!gather) break;
        const int stopped = __popc(__ballot_sync(peers, event != 0 || taken >= n));
        idle += stopped;
        if (stopped == npeer || idle >= limit) break;
        }
        budget -= taken;
        st.steps += taken;
        if (kLean) {
            h.steps += taken;
            if (M::kCfg && !event && h.steps >= k.life_cap) event = 3;
            if (M::kRef) {
                h.hop += taken;
                if (!event && h.hop >= k.hop_cap) event = 1;
            }
        }
        if (event) {
            drift_check(a, i, I, h, st);
            int fate = 0;
            if (event == 2) {
                fate = DSMC_FATE_ESCAPED;
            } else if (event == 3) {
                fate = DSMC_FATE_STEP_CAP;
            } else {
                R thi, fi, local_T = R(0);
                fate = land<kMode>(a, i, I, h, thi, fi, local_T);
                if (fate == 0) fate = hop_top<kMode>(a, i, I, h, b, st, thi, fi, local_T, false);
            }
            if (fate) {
                finish<kMode>(a, i, I, h, st, fate);
                alive = start_next<kMode>(a, i, h, b, st);
            }
        }
    }
    if (M::kAny && h.inst >= 0) flush_hist(a.inst(h.inst), h, hist_cell<kMode>(h));
    if (i >= 0) store_hot(a.s, i, a.nslots, h);
    // statistics of this launch, per instance; the finished count also drives the host loop
    const unsigned fin = st.finished;
    flush_stats(a, st);
    const unsigned wfin = __reduce_add_sync(0xffffffffu, fin);
    if ((threadIdx.x & 31) == 0 && wfin) atomicAdd(&a.ctr->finished, static_cast<unsigned long long>(wfin));
}

enum Event { kEvNone = 0, kEvLanded, kEvEscaped, kEvCap, kEvEmpty, kEvResume };

// The step loop of fast_kernel kept in step warp by warp: all lanes take up to kUnroll steps in a
// row without a branch back, the next step's reciprocal square root beside this step's cell tests;
// a lane that leaves its cell (or collides) stops there, and the lanes that did take the slow path
// together; events (landing, escape, cap, an empty slot) run at one place, for all lanes that have
// one, once the lanes that wait have idled `limit` iterations in all. Against fast_kernel, whose
// lanes take every cell change as it comes, a change costs its lane the rest of the iteration, but
// the change's code runs once per iteration and not once per step (a warp of long hops changes a
// cell on half of its steps), the branches per step halve, and the event code exists once.
// A launch runs a.K / kUnroll iterations, at least one, so a lane takes at most max(a.K, kUnroll) steps.
// Measured at kUnroll 8: 1e7 Ceres-like particles 278 ms against 291.5 ms, 3e5 of the reference
// model 72 against 103 ms; 4 and 12 steps in a row ran the former in 307 and 297 ms. Few particles,
// whose warps have nothing to hide a branch behind: 512 Ceres-like 1.60 ms at 12 steps in a row,
// 1.77 at 8, 3.4 in fast_kernel; 500 of the reference model with collisions 42.9 ms at 12, 46.7 at
// 8, 59.4 in fast_kernel. It loses where events are frequent for the steps they wait: 3e6 Moon-like
// particles 44.7 against 42.5 ms, with histograms 50 against 45 ms, collisions 62 against 49 ms.
template <int kMaxThreads, int kMinBlocks, int kMode, int kUnroll>
__global__ void __launch_bounds__(kMaxThreads, kMinBlocks) warp_kernel(const __grid_constant__ OneArgsT<float> a) {
    using A = OneArgsT<float>;
    using R = float;
    using M = Mode<kMode>;
    using Tab = TabOf<A, R>;
    constexpr unsigned kAll = 0xffffffffu;
    SharedTab<R>::fill(a.one);
    const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long long i = a.slot(t);
    HotT<R> h;
    if (i >= 0) load_hot(a.s, i, a.nslots, h);
    else h.inst = -1;
    StatAcc st;
    st.inst = h.inst;
    const FastInst &I = a.one;
    const StepConst<R> &k = a.k;
    BoundsT<R> b;
    bool flying = h.inst >= 0;
    int event = flying ? kEvResume : kEvNone;

    if (flying) {
        // reload the cached bounds of the saved cell without flushing its pending deposits
        const int ci = h.ci;
        const R run_w = h.run_w;
        h.ci = -1;
        enter_cell(Tab{I}, h, b, h.cell);
        h.ci = ci;
        h.run_w = run_w;
    } else if (i >= 0) {
        // a queue of fewer particles than slots starts on the lanes that fill_warps chose
        const long long warps = a.ctr->fill_warps;
        if (warps == 0 || ((t >> 5) < warps && (t & 31) * warps + (t >> 5) < static_cast<long long>(a.ctr->total)))
            event = kEvEmpty;
    }
    PosT<R> q;
    int n = 0, taken = 0, skip = 0, idle = 0;
    const int limit = a.gather * kChunk / kUnroll;   // lane-chunks of kChunk steps in lane-iterations

    const bool work = __any_sync(kAll, event != kEvNone);
    const int iters = a.K / kUnroll > 0 ? a.K / kUnroll : 1;
    for (int it = 0; work; it++) {
        const bool last = it >= iters;
        const unsigned ev = __ballot_sync(kAll, event != kEvNone);
        if (ev || last) {
            idle += __popc(ev);
            const unsigned fly = __ballot_sync(kAll, flying && !event);
            if (idle >= limit || !fly || last) {
                idle = 0;
                if (event) {
                    int fate = event == kEvResume ? 0 : -1;
                    R thi = R(0), fi = R(0), local_T = R(0);
                    if (event == kEvLanded || event == kEvEscaped || event == kEvCap) {
                        st.steps += taken;
                        h.steps += taken;
                        taken = 0;
                        drift_check(a, i, I, h, st);
                        fate = event == kEvEscaped ? DSMC_FATE_ESCAPED
                             : event == kEvCap ? DSMC_FATE_STEP_CAP : land<kMode>(a, i, I, h, thi, fi, local_T);
                    }
                    if (event != kEvResume) {
                        bool first = false;
                        for (;;) {
                            if (fate) {
                                if (fate > 0) finish<kMode>(a, i, I, h, st, fate);
                                flying = take_next<kMode>(a, i, h, st, thi, fi, local_T);
                                if (!flying) break;
                                first = true;
                            }
                            fate = hop_top<kMode>(a, i, I, h, b, st, thi, fi, local_T, first);
                            if (!fate) break;
                        }
                    }
                    event = 0;
                    if (flying) {
                        start_pos(h, q);
                        gravity(q, k.GM);
                        n = 0x7fffffff;
                        if (!M::kRef) n = min(n, k.life_cap - h.steps);
                        if (!M::kCfg) n = min(n, k.hop_cap - h.hop);
                        // the step that the skip-first rule leaves without a deposit
                        skip = !M::kCfg && (k.flags & kFlagSkipFirst) && h.hop == 0 ? 1 : 0;
                        taken = 0;
                    }
                }
                __syncwarp();
            }
            if (last || !__any_sync(kAll, flying)) break;
        }
        R d[3];
        bool left = false, struck = false;
        auto settle = [&]() {   // a step's photolysis and deposit, once the cell is known
            const bool day = M::kRef ? ((h.cell & 0xff) < k.half_ffd)
                                     : (fma_r(q.x, k.sx, fma_r(q.y, k.sy, q.z * k.sz)) > R(0));
            if (day) {
                h.nday++;
                h.W *= k.fday;
            }
            if (M::kRef && taken == skip) return;
            if (M::kCol && h.nsig != R(0)) {
                h.pcol = fma_r(sqrt(fma_r(d[0], d[0], fma_r(d[1], d[1], d[2] * d[2]))), fabs(h.nsig), h.pcol);
                struck = h.pcol > h.pthr && h.nsig > R(0);
                if (struck) return;
            }
            h.run_w += h.W;
        };
        if (flying && !event) {
            const bool whole = n - taken >= kUnroll;
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                verlet_step(h, q, k.dt, k.c1, k.c2, d);
                gravity(q, k.GM);
                taken++;
                if (!(in_shell(q, b) & in_row(q, b) & in_column(q, b))) {
                    left = true;
                    break;
                }
                settle();
                if (M::kCol && struck) break;
                if (u == 0 && !whole) break;
            }
        }
        __syncwarp();
        if (left) {
            if (q.r2 <= k.rl2) {
                event = kEvLanded;
            } else if (q.r2 >= k.re2) {
                event = kEvEscaped;
            } else if (!move_cell<!M::kCol>(Tab{I}, h, b, q.x, q.y, q.r2, q.z * fabs(q.z), in_shell(q, b),
                                            in_row(q, b), in_column(q, b)) &&
                       kMode == 1 && q.r2 != q.r2) {
                // to the end of its life, or of this launch: there it waits, as a lane that no
                // longer flies, with its steps settled
                const int rest = (iters - 1 - it) * kUnroll;
                taken = drift_nowhere(h, taken, n - taken > rest ? taken + rest : n);
                if (taken < n) {
                    st.steps += taken;
                    h.steps += taken;
                    taken = 0;
                    flying = false;
                }
            } else {
                settle();
            }
        }
        if (M::kCol && struck) {
            const int ht = h.cell >> 16, td = (h.cell >> 8) & 0xff, fd = h.cell & 0xff;
            collide<kMode>(a, i, I, h, (static_cast<long long>(td) * I.p.ffd + fd) * I.p.hd + ht);
        }
        if (flying && !event && taken >= n)
            event = !M::kRef && h.steps + taken >= k.life_cap ? kEvCap : kEvLanded;
    }
    if (flying) {
        st.steps += taken;
        h.steps += taken;
        if (!M::kCfg) h.hop += taken;
    }
    if (i >= 0) store_hot(a.s, i, a.nslots, h);
    // statistics of this launch, per instance; the finished count also drives the host loop
    const unsigned fin = st.finished;
    flush_stats(a, st);
    const unsigned wfin = __reduce_add_sync(kAll, fin);
    if ((threadIdx.x & 31) == 0 && wfin) atomicAdd(&a.ctr->finished, static_cast<unsigned long long>(wfin));
}

}  // namespace
}  // namespace dsmc
