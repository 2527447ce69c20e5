// kernel_plain.cu - the plain FP64 path: one thread per test particle for its whole life.
//
// This translation unit is compiled with -fmad=false so that every double operation rounds on
// its own, as the reference's x86-64 build does (SSE2, no FMA contraction). With fed initial
// states the push is then bit-identical to the reference's verlet_step
// (src/common/integrator.c:4-55). Transcendentals (sin, cos, asin, atan2, log, exp) come from
// CUDA's libm and may differ from glibc in the last place; everything else follows the reference
// runners' operation order (src/dsmc/ballistic.c:97-281, src/dsmc/advanced.c:236-451).
//
// Deposits are unsigned 64-bit fixed point (W * 2^24, rounded to nearest per step, the integers
// of one visit to a cell added together and flushed with one atomicAdd), so the grids are
// independent of thread order and bit-reproducible.
//
// A step's cost was the index formulas: asin, atan2, log and three divisions in FP64, 1.2e10
// particle-steps/s at any size. The cell's limits, moved inwards by more than the formulas'
// rounding, now settle most steps (struct Safe), and with the run of deposits and 128 registers
// the path runs 3.5e10 (2e6 Ceres-like particles 1197 -> 403 ms), results bit for bit the same.
#include "dsmc_device.cuh"
#include "dsmc_kernels.h"

namespace dsmc {
namespace {

__device__ __forceinline__ double len3(const double a[3]) {
    return sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
}

__device__ __forceinline__ void to_angles(const double s[3], double Ri, double &thi, double &fi) {
    thi = asin(s[2] / Ri);
    fi = atan2(s[0], s[1]);
    if (fi < 0) fi += 2.0 * kPi;
}

__device__ __forceinline__ void to_index(double thi, double fi, int ftd, int ffd, int &td,
                                         int &fd) {
    td = static_cast<int>(ceil((thi + kPi / 2.0) / kPi * ftd)) - 1;
    fd = static_cast<int>(ceil(fi / (2.0 * kPi) * ffd)) - 1;
    td = td < 0 ? 0 : (td >= ftd ? ftd - 1 : td);
    fd = fd < 0 ? 0 : (fd >= ffd ? ffd - 1 : fd);
}

__device__ __forceinline__ double cdf_eval(const double *coef, const double *box, int degree,
                                           double x) {
    double t = (x - box[2]) / box[3];
    double r = 0.0;
    for (int i = 0; i <= degree; i++) r = r * t + coef[i];
    return r;
}

// collision_sample_speed, src/common/collision.c:43-101: bisection of the fitted
// reverse-cumulative speed distribution.
__device__ double cdf_sample(const double *coef, const double *box, double total, int degree,
                             double u) {
    double vmax = box[1];
    double at_max = cdf_eval(coef, box, degree, vmax);
    double ranking = u * (total - at_max) + at_max;
    double v0 = box[0], v1 = vmax;
    for (int iter = 0; iter < 100; iter++) {
        double vm = (v0 + v1) * 0.5;
        double fm = cdf_eval(coef, box, degree, vm) - ranking;
        double f1 = cdf_eval(coef, box, degree, v1) - ranking;
        if (fm * f1 < 0) v0 = vm;
        else v1 = vm;
        if (fabs(v1 - v0) < 0.01) break;
    }
    return (v0 + v1) * 0.5;
}

__device__ __forceinline__ void unit_sphere(double zu, double pu, double o[3]) {
    double z = 2.0 * zu - 1.0;
    double r = sqrt(fmax(0.0, 1.0 - z * z));
    double ph = 2.0 * kPi * pu;
    o[0] = r * cos(ph);
    o[1] = r * sin(ph);
    o[2] = z;
}

// Turns the position by `cols` columns of longitude (advanced.c:290-300).
__device__ __forceinline__ void turn_to_column(double s[3], int cols, int ffd) {
    const double rot_fi = static_cast<double>(cols) / ffd * 2.0 * kPi;
    const double cs = cos(rot_fi), sn = sin(rot_fi);
    const double n0 = s[0] * cs - s[1] * sn, n1 = s[0] * sn + s[1] * cs;
    s[0] = n0;
    s[1] = n1;
}

// Limits of the current cell, each moved inwards by a margin far above the rounding of the index
// formulas (asin, atan2, log and the divisions: below 1e-14 relative). A position inside all of
// them has the cell's indices by the formulas too, so the step need not evaluate them; a position
// within a margin of an edge, or outside, goes through the formulas as before.
constexpr double kAngleMargin = 1e-12, kRadiusMargin = 1e-9;
struct Safe {
    double rlo = 1.0, rhi = 0.0;          // radius; empty until a cell is set
    double zlo, zhi;                      // z / r
    double s0, c0, s1, c1;                // (sine, cosine) of the two longitudes

    __device__ __forceinline__ void none() { rlo = 1.0; rhi = 0.0; }
    __device__ __forceinline__ void set(const dsmc_params &p, const double *edges, int ht, int td, int fd) {
        const double *zs = edges + p.hd + 1, *lon = zs + p.ftd + 1;
        const double extra = p.use_exp_grid ? 1e-12 * fabs(p.unih / p.alpha2) : 0.0;
        const double r0 = edges[ht], r1 = edges[ht + 1];
        rlo = ht > 0 ? r0 + (kRadiusMargin * fabs(r0) + extra) : 0.0;
        rhi = r1 - (kRadiusMargin * fabs(r1) + extra);
        zlo = td > 0 ? zs[td] + kAngleMargin : -2.0;
        zhi = td < p.ftd - 1 ? zs[td + 1] - kAngleMargin : 2.0;
        s0 = lon[2 * fd];
        c0 = lon[2 * fd + 1];
        s1 = lon[2 * fd + 2];
        c1 = lon[2 * fd + 3];
    }
    __device__ __forceinline__ bool holds(const double s[3], double r) const {
        const double m = kAngleMargin * (fabs(s[0]) + fabs(s[1]));
        return (r > rlo) & (r < rhi) & (s[2] > r * zlo) & (s[2] < r * zhi) &
               (s[0] * c0 - s[1] * s0 > m) & (s[1] * s1 - s[0] * c1 > m);
    }
};

struct Acc {
    unsigned long long steps = 0, escaped = 0, collisions = 0, bound = 0, finished = 0, drift = 0;
};

// Orbital energy per unit mass |v|^2 / 2 - GM / |s| of the per-hop energy-drift guard.
__device__ __forceinline__ double orbital_energy(const dsmc_params &p, const double s[3],
                                                 const double v[3]) {
    return 0.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) - p.GM / len3(s);
}

// Velocity-record replay modes (see launch_plain_record): kCount counts the deposited visits of
// each particle per (td, ht) bucket into the particle's own row; kRecord turns those rows into
// write cursors and stores the visits that fall below the per-bucket cap. Both modes leave the
// density and horizon grids untouched.
enum Mode { kSolve = 0, kCount = 1, kRecord = 2 };

template <int kMode>
__device__ void particle_life(const dsmc_params &p, const DevTables &t, long long pid,
                              Acc &acc, const RecordArgs &ra) {
    const int ftd = p.ftd, ffd = p.ffd, hd = p.hd;
    const bool ref = p.model == DSMC_MODEL_REFERENCE;
    const bool adv = p.runner == DSMC_RUNNER_ADVANCED;
    const double h = p.dt_step;

    Philox rng;
    rng.init(p.seed, p.instance, static_cast<uint32_t>(pid));

    int fate = DSMC_FATE_ALIVE, num_col = 0, td, fd;
    long long steps = 0;
    double real_col_p = 0.0, col_p = 0.0, time = 0.0, W = 1.0, flight_time = 0.0,
           rest_time = 0.0, thi, fi, local_T, s[3], v[3] = {0.0, 0.0, 0.0};
    // energy-drift guard: E at the hop's launch (or last collision) against E where it ends
    const double drift_abs = p.drift_tol * p.GM / p.Radii;
    double E_start = 0.0;

    rng.next();
    if (ref) {
        if (adv) col_p = rng.raw(0) / kTwo32;
        const int o = adv ? 1 : 0;
        thi = rng.raw(o) / kTwo32 * kPi - kPi / 2.0;
        fi = rng.raw(o + 1) / kTwo32 * 2.0 * kPi;
        s[0] = p.Radii * cos(thi) * sin(fi);
        s[1] = p.Radii * cos(thi) * cos(fi);
        s[2] = p.Radii * sin(thi);
        to_index(thi, fi, ftd, ffd, td, fd);
        local_T = t.T_map[td * ffd + fd];
    } else {
        const int f = pick_face(t, rng.raw(0) / kTwo32);
        double u1 = rng.raw(1) / kTwo32, u2 = rng.raw(2) / kTwo32;
        col_p = rng.raw(3) / kTwo32;
        if (u1 + u2 > 1.0) { u1 = 1.0 - u1; u2 = 1.0 - u2; }
        const double *a = t.face_verts + 9 * f;
        double q[3];
        for (int k = 0; k < 3; k++)
            q[k] = a[k] + u1 * (a[3 + k] - a[k]) + u2 * (a[6 + k] - a[k]);
        const double lq = len3(q);
        for (int k = 0; k < 3; k++) s[k] = q[k] * (p.Radii / lq);
        to_angles(s, len3(s), thi, fi);
        to_index(thi, fi, ftd, ffd, td, fd);
        local_T = t.face_T[f];
    }
    const long long slot = pid - t.out_base;
    const bool record = kMode == kSolve && t.ttime && slot >= 0 && slot < t.out_cap;
    if (record) {
        t.ttime[0 * t.out_cap + slot] = thi;
        if (adv || !ref) {
            t.ttime[5 * t.out_cap + slot] = fi;
            t.ttime[6 * t.out_cap + slot] = local_T;
        }
    }

    Safe safe;                             // limits of the cell (ht, td, fd) of the last step
    int ht = 0;
    unsigned long long run = 0;            // deposits of that cell not yet added to the grid
    auto flush = [&]() {
        if (kMode == kSolve && run) atomicAdd(&t.density[static_cast<long long>(ht) * ftd * ffd + td * ffd + fd], run);
        run = 0;
    };
    // velocity-record modes: visits of the particle in bucket (td, ht), kept here while it lasts
    int *row = kMode != kSolve ? ra.rows + (pid - ra.row_base) * static_cast<long long>(ftd * hd) : nullptr;
    int bucket = -1, visits = 0;
    int todo = kMode == kRecord ? ra.todo[pid - ra.row_base] : 0;
    if (kMode == kRecord && todo == 0) return;

    for (;;) {
        if (W < p.w_min) { fate = DSMC_FATE_PHOTOLYSED; break; }
        if (p.life_step_cap > 0 && steps >= p.life_step_cap) { fate = DSMC_FATE_STEP_CAP; break; }

        if (ref) {
            // Launch, ballistic.c:125-173 and advanced.c:272-326.
            const double KF = 2.0 * kPi * p.Radii * fabs(cos(thi)) / p.P;
            to_index(thi, fi, ftd, ffd, td, fd);
            local_T = t.T_map[td * ffd + fd];
            if (local_T < p.freeze_T) {
                if (adv && kMode == kSolve) atomicAdd(&t.horizon[td * ffd + fd], to_fixed(W));
                const int wait = t.warm[td * ffd + fd];
                const bool found = wait > 0;
                for (int k = found ? wait : ffd; k > 0; k--) {
                    time += p.dt_rot;
                    if (adv) rest_time += p.dt_rot;
                }
                if (found) {
                    if (adv) {
                        turn_to_column(s, wait - fd, ffd);
                        fd = wait % ffd;
                    } else {
                        fd = (fd + wait) % ffd;
                    }
                    fi = (fd + 0.5) / ffd * 2.0 * kPi;
                }
                if (!found) {
                    if (kMode == kSolve) atomicAdd(&t.horizon[td * ffd + fd], to_fixed(W));
                    fate = DSMC_FATE_FROZEN;
                    break;
                }
                local_T = t.T_map[td * ffd + fd];
            }
            rng.next();
            // velocity_sample (velocity.c:49-68) and velocity_sticking (velocity.c:70-73)
            int idx = local_T >= 220.0 ? 20 : static_cast<int>(ceil(local_T / 10.0)) - 2;
            idx = idx < 0 ? 0 : (idx >= 23 ? 22 : idx);
            const double vr = t.vt_speeds[idx * 1000 + rng.w[0] % static_cast<uint32_t>(t.vt_count[idx])];
            const double v_old_sq = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
            const double vout = sqrt(p.alpha * vr * vr + (1.0 - p.alpha) * v_old_sq);
            const double flyd = rng.raw(1) / kTwo32 * kPi + thi - kPi / 2.0;
            const double xi = rng.raw(2) / kTwo32 * kPi + fi - kPi / 2.0;
            double sf, cf, sx, cx, sr, cr;
            sincos(flyd, &sf, &cf);
            sincos(xi, &sx, &cx);
            sincos(fi + kPi / 2.0, &sr, &cr);
            v[0] = cf * sx * vout;
            v[1] = cf * cx * vout;
            v[2] = sf * vout;
            v[0] += KF * sr;
            v[1] += KF * cr;
            if (len3(v) >= p.ve) { fate = DSMC_FATE_ESCAPED; break; }
        } else {
            // Flux-weighted Maxwell-Boltzmann: Rayleigh normal, Gaussian tangential components.
            rng.next();
            const double sigma = sqrt(p.kB_over_m * local_T);
            const double vn = sigma * sqrt(-2.0 * log(1.0 - rng.raw(0) / kTwo32));
            const double rho = sqrt(-2.0 * log(1.0 - rng.raw(1) / kTwo32));
            const double ang = 2.0 * kPi * (rng.raw(2) / kTwo32);
            double sa, ca;
            sincos(ang, &sa, &ca);
            const double t1 = rho * ca, t2 = rho * sa;
            const double R = len3(s);
            const double n[3] = {s[0] / R, s[1] / R, s[2] / R};
            double e[3] = {-n[1], n[0], 0.0};
            const double le = sqrt(e[0] * e[0] + e[1] * e[1]);
            if (le < 1e-12) { e[0] = 1.0; e[1] = 0.0; }
            else { e[0] /= le; e[1] /= le; }
            const double nt[3] = {n[1] * e[2] - n[2] * e[1], n[2] * e[0] - n[0] * e[2],
                                  n[0] * e[1] - n[1] * e[0]};
            const double omega = p.P > 0.0 ? 2.0 * kPi / p.P : 0.0;
            const double rot[3] = {omega * s[1], -omega * s[0], 0.0};
            for (int k = 0; k < 3; k++)
                v[k] = vn * n[k] + (sigma * t1) * e[k] + (sigma * t2) * nt[k] + rot[k];
            const double E = 0.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) - p.GM / len3(s);
            if (E < 0.0) acc.bound++;
        }

        double Ri = len3(s);
        double oa[3];
        for (int k = 0; k < 3; k++) oa[k] = p.GM * s[k] / (Ri * Ri * Ri);
        E_start = orbital_energy(p, s, v);

        for (long long ii = 0; ii < p.hop_step_cap; ii++) {
            flight_time += h;
            time += h;
            steps++;
            // verlet_step, integrator.c:12-54
            const double R03 = Ri * Ri * Ri;   // Ri = |s|
            const double h2 = h * h;
            const double g = p.GM / R03;
            double ns[3];
            for (int k = 0; k < 3; k++)
                ns[k] = s[k] + v[k] * h - g * s[k] * (1.5 * h2) - oa[k] * (h2 / 6.0);
            const double dx = ns[0] - s[0], dy = ns[1] - s[1], dz = ns[2] - s[2];
            for (int k = 0; k < 3; k++) v[k] -= g * s[k] * h;
            for (int k = 0; k < 3; k++) oa[k] = g * s[k];
            const double Rn = len3(ns);
            if (Rn >= p.max_height && !(Rn <= p.Radii)) {
                // the angles are those of the last step inside, or of the launch
                if (ii > 0) to_angles(s, Ri, thi, fi);
                fate = DSMC_FATE_ESCAPED;
            }
            s[0] = ns[0]; s[1] = ns[1]; s[2] = ns[2];
            Ri = Rn;
            if (Ri <= p.Radii || fate != DSMC_FATE_ALIVE) break;

            if (!safe.holds(s, Ri)) {
                flush();
                double a, b;
                to_angles(s, Ri, a, b);
                to_index(a, b, ftd, ffd, td, fd);
                if (p.use_exp_grid) {
                    const double arg = p.alpha2 * (Ri - p.Radii) / p.unih + 1.0;
                    ht = arg <= 1.0 ? 0 : static_cast<int>(ceil(log(arg) / p.log1p_alpha2)) - 1;
                } else {
                    ht = static_cast<int>(ceil((Ri - p.Radii) / p.unih)) - 1;
                }
                if (ht < 0) ht = 0;
                if (ht < hd && t.edges) safe.set(p, t.edges, ht, td, fd);
                else safe.none();
            }
            const bool day = ref ? (fd < ffd / 2)
                                 : (s[0] * p.sun[0] + s[1] * p.sun[1] + s[2] * p.sun[2] > 0.0);
            if (day) W *= p.wdecay;

            const bool deposit = !(p.skip_first_deposit && ii == 0) && ht < hd;
            if (deposit) {
                bool collided = false;
                if (adv && t.n_bg && ht < p.collide_ht_max) {
                    const long long atm = static_cast<long long>(ht) * ftd * ffd + td * ffd + fd;
                    const double nloc = atm < t.n_bg_len ? t.n_bg[atm] : 0.0;
                    const double ds = sqrt(dx * dx + dy * dy + dz * dz);
                    real_col_p += ds * nloc * p.cross_section;
                    const long long pc = static_cast<long long>(td) * ffd * hd +
                                         static_cast<long long>(fd) * hd + ht;
                    if (col_p < 1.0 - exp(-real_col_p) && t.cdf_valid[pc]) {
                        real_col_p = 0.0;
                        num_col++;
                        const double *coef = t.cdf_coef + DSMC_CDF_STRIDE * pc;
                        const double *box = t.cdf_box + 4 * pc;
                        rng.next();
                        if (p.scatter == DSMC_SCATTER_REFERENCE) {
                            // advanced.c:381-395 and collision.c:35-40
                            const double vv2 = cdf_sample(coef, box, t.cdf_total[pc],
                                                          t.cdf_degree, rng.raw(0) / kTwo32);
                            const double thi2 = kPi * rng.raw(1) / kTwo32 - kPi / 2.0;
                            const double fi2 = 2.0 * kPi * rng.raw(2) / kTwo32;
                            const double v2[3] = {vv2 * cos(thi2) * cos(fi2),
                                                  vv2 * cos(thi2) * sin(fi2), vv2 * sin(thi2)};
                            for (int k = 0; k < 3; k++) {
                                const double del = v[k] - v2[k], vcm = v[k] + v2[k];
                                v[k] = vcm + 0.5 * del;
                            }
                            if (p.redraw_col_threshold) col_p = rng.raw(3) / kTwo32;
                        } else {
                            // isotropic elastic hard sphere, equal masses
                            const double vv2 = cdf_sample(coef, box, t.cdf_total[pc],
                                                          t.cdf_degree, rng.raw(0) / kTwo32);
                            double d2[3], om[3];
                            unit_sphere(rng.raw(1) / kTwo32, rng.raw(2) / kTwo32, d2);
                            if (p.redraw_col_threshold) col_p = rng.raw(3) / kTwo32;
                            rng.next();
                            unit_sphere(rng.raw(0) / kTwo32, rng.raw(1) / kTwo32, om);
                            double gv[3], vcm[3];
                            for (int k = 0; k < 3; k++) {
                                const double v2k = vv2 * d2[k];
                                gv[k] = v[k] - v2k;
                                vcm[k] = 0.5 * (v[k] + v2k);
                            }
                            const double gl = len3(gv);
                            for (int k = 0; k < 3; k++) v[k] = vcm[k] + 0.5 * gl * om[k];
                        }
                        collided = true;
                        E_start = orbital_energy(p, s, v);
                    }
                }
                if (kMode != kSolve) {
                    // count_nn is keyed by (td, ht) without fd, ballistic.c:216-229
                    const int b = td * hd + ht;
                    if (b != bucket) {
                        if (bucket >= 0) row[bucket] = visits;
                        bucket = b;
                        visits = row[b];
                    }
                    const int cur = visits++;
                    if (kMode == kRecord && cur < ra.cap) {
                        const long long slot = static_cast<long long>(b) * ra.cap + cur;
                        ra.rec_v[3 * slot] = v[0];
                        ra.rec_v[3 * slot + 1] = v[1];
                        ra.rec_v[3 * slot + 2] = v[2];
                        ra.rec_fd[slot] = fd;
                        ra.rec_key[slot] = (static_cast<unsigned long long>(pid) << 32) |
                                           static_cast<unsigned long long>(steps);
                        if (--todo == 0) return;   // its last record
                    }
                } else if (!collided) {
                    run += to_fixed(W);
                    if (t.speed_hist && p.n_speed_bins > 0) {
                        const long long cell = static_cast<long long>(ht) * ftd * ffd + td * ffd + fd;
                        int b = static_cast<int>(len3(v) / p.speed_bin_width);
                        if (b >= p.n_speed_bins) b = p.n_speed_bins - 1;
                        atomicAdd(&t.speed_hist[cell * p.n_speed_bins + b], 1ull);
                    }
                }
            }
            if (p.life_step_cap > 0 && steps >= p.life_step_cap) {
                to_angles(s, Ri, thi, fi);
                fate = DSMC_FATE_STEP_CAP;
                break;
            }
        }
        // the deposits of the hop's last cell; the landing code below moves (td, fd)
        flush();
        safe.none();
        // the hop ended (landing, escape radius, hop or life cap)
        if (p.drift_tol > 0.0 && fabs(orbital_energy(p, s, v) - E_start) > drift_abs) acc.drift++;
        if (fate != DSMC_FATE_ALIVE) break;

        // Landing, ballistic.c:239-264.
        Ri = len3(s);
        to_angles(s, Ri, thi, fi);
        to_index(thi, fi, ftd, ffd, td, fd);
        if (ref) {
            if (td <= 1 || td >= ftd - 2) {
                if (kMode == kSolve) atomicAdd(&t.horizon[td * ffd + fd], to_fixed(0.05 * W));
                W *= 0.95;
            }
        } else {
            const double nrm[3] = {s[0] / Ri, s[1] / Ri, s[2] / Ri};
            if (nrm[0] * p.sun[0] + nrm[1] * p.sun[1] + nrm[2] * p.sun[2] <= 0.0) {
                if (kMode == kSolve) atomicAdd(&t.horizon[td * ffd + fd], to_fixed(W));
                fate = DSMC_FATE_FROZEN;
                break;
            }
            for (int k = 0; k < 3; k++) s[k] = nrm[k] * p.Radii;
            local_T = t.face_T[locate_face(t, nrm)];
        }
    }

    if (kMode == kCount && bucket >= 0) row[bucket] = visits;
    acc.steps += steps;
    acc.collisions += num_col;
    acc.finished++;
    if (fate == DSMC_FATE_ESCAPED) acc.escaped++;
    if (kMode == kSolve && t.fate && slot >= 0 && slot < t.out_cap) t.fate[slot] = fate;
    if (kMode == kSolve && t.steps && slot >= 0 && slot < t.out_cap) t.steps[slot] = steps;
    if (record && (fate != DSMC_FATE_ESCAPED || !ref)) {
        t.ttime[1 * t.out_cap + slot] = thi;
        t.ttime[2 * t.out_cap + slot] = time;
        t.ttime[3 * t.out_cap + slot] = W;
        t.ttime[4 * t.out_cap + slot] = flight_time;
        if (adv || !ref) {
            t.ttime[7 * t.out_cap + slot] = rest_time;
            t.ttime[8 * t.out_cap + slot] = static_cast<double>(num_col);
        }
    }
}

// `lanes` threads of each warp take particles (see plain_shape). Four blocks of 128 per SM (128
// registers, 64 B of spill stores): 2e6 Ceres-like particles run 403 ms against 661 ms at the 250
// registers ptxas takes by itself and 390 ms at five blocks, 1e5 27.6, 37.7 and 28 ms.
template <int kMode>
__global__ void __launch_bounds__(128, 4) plain_fp64_kernel(const __grid_constant__ dsmc_params p,
                                                            const __grid_constant__ DevTables t,
                                                            long long pid_begin, long long n, int lanes,
                                                            const RecordArgs ra) {
    Acc acc;
    const int lane = threadIdx.x & 31;
    const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
    const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    for (long long i = warp * lanes + lane; lane < lanes && i < n; i += warps * lanes)
        particle_life<kMode>(p, t, pid_begin + i, acc, ra);
    if (kMode == kSolve) {
        warp_add_stat(&t.stats[kStatSteps], acc.steps);
        warp_add_stat(&t.stats[kStatEscaped], acc.escaped);
        warp_add_stat(&t.stats[kStatCollisions], acc.collisions);
        warp_add_stat(&t.stats[kStatBound], acc.bound);
        warp_add_stat(&t.stats[kStatFinished], acc.finished);
        warp_add_stat(&t.stats[kStatDrift], acc.drift);
    }
}

// Turns per-particle visit counts into write cursors: for each bucket, an exclusive scan over
// the chunk's particles in pid order, starting from the records the bucket already holds. Also
// counts each particle's records below the cap: the replay skips a particle without any and
// leaves one after its last, so it costs what the first particles of each bucket cost (a chunk of
// 5000 reference-model particles: 60 ms for the replay of whole lives, as the count pass).
// A cursor stays at the cap once it is there: the visits of a bucket may be more than an int holds (a
// chunk is up to 67 million particles, a life 13,000 steps in the mean), and a cursor that wrapped would
// be below the cap again.
__global__ void record_scan_kernel(int *rows, int nrows, int nb, int cap, int *todo, int *filled) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    int run = filled[b];
    for (int q = 0; q < nrows; q++) {
        const long long i = static_cast<long long>(q) * nb + b;
        const int own = min(rows[i], cap - run);   // its records below the cap
        rows[i] = run;
        if (own) atomicAdd(todo + q, own);
        run += own;
    }
    filled[b] = run;
}

// Blocks, and particles per warp, of a launch over n particles.
struct PlainShape { unsigned blocks; int lanes; };

PlainShape plain_shape(long long n, int num_sms) {
    const int block = 128;
    // few particles spread over the resident warps (16 per SM), so that a landing, the long part
    // of a life on the reference model, holds up few others: the velocity record of 5000
    // reference-model particles takes 55 ms against 65 ms at 4 warps per SM, 1e5 Ceres-like
    // particles fill the warps either way
    const long long warps = static_cast<long long>(num_sms) * 16;
    long long lanes = (n + warps - 1) / warps;
    lanes = lanes > 32 ? 32 : lanes;
    const long long per_block = block / 32 * lanes;
    const long long blocks = (n + per_block - 1) / per_block;
    // Enough blocks for every particle its own thread, capped at a few waves of resident blocks
    // (the grid-stride loop covers the rest).
    const long long cap = static_cast<long long>(num_sms) * 16 * 64;
    return {static_cast<unsigned>(blocks > cap ? cap : blocks), static_cast<int>(lanes)};
}

// Fed-state push: integrate each (s, v) with the reference's Verlet variant for up to nsteps
// steps, starting from oa = GM s / r^3 (ballistic.c:176-181), stopping at landing or escape.
__global__ void push_fp64_kernel(const dsmc_params p, long long n, int nsteps, double *pos,
                                 double *vel, int *status, int *taken) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
    double v[3] = {vel[3 * i], vel[3 * i + 1], vel[3 * i + 2]};
    const double h = p.dt_step;
    double Ri = len3(s);
    double oa[3];
    for (int k = 0; k < 3; k++) oa[k] = p.GM * s[k] / (Ri * Ri * Ri);
    int st = 0, k = 0;
    for (; k < nsteps && st == 0; k++) {
        const double R0 = len3(s);
        const double g = p.GM / (R0 * R0 * R0);
        const double h2 = h * h;
        double ns[3];
        for (int j = 0; j < 3; j++)
            ns[j] = s[j] + v[j] * h - g * s[j] * (1.5 * h2) - oa[j] * (h2 / 6.0);
        for (int j = 0; j < 3; j++) v[j] -= g * s[j] * h;
        for (int j = 0; j < 3; j++) oa[j] = g * s[j];
        s[0] = ns[0]; s[1] = ns[1]; s[2] = ns[2];
        Ri = len3(s);
        st = Ri <= p.Radii ? 1 : (Ri >= p.max_height ? 2 : 0);
    }
    for (int j = 0; j < 3; j++) { pos[3 * i + j] = s[j]; vel[3 * i + j] = v[j]; }
    status[i] = st;
    taken[i] = k;
}

}  // namespace

cudaError_t launch_push_fp64(const dsmc_params &p, long long n, int nsteps, double *pos,
                             double *vel, int *status, int *taken, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    push_fp64_kernel<<<static_cast<unsigned>((n + 127) / 128), 128, 0, stream>>>(p, n, nsteps, pos, vel,
                                                                                status, taken);
    return cudaGetLastError();
}

cudaError_t launch_plain_fp64(const dsmc_params &p, const DevTables &t, long long pid_begin,
                              long long n, int num_sms, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    const RecordArgs ra{};
    const PlainShape g = plain_shape(n, num_sms);
    plain_fp64_kernel<kSolve><<<g.blocks, 128, 0, stream>>>(p, t, pid_begin, n, g.lanes, ra);
    return cudaGetLastError();
}

cudaError_t launch_plain_record(const dsmc_params &p, const DevTables &t, long long pid_begin,
                                long long n, const RecordArgs &ra, int *filled, int num_sms,
                                cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    const PlainShape g = plain_shape(n, num_sms);
    plain_fp64_kernel<kCount><<<g.blocks, 128, 0, stream>>>(p, t, pid_begin, n, g.lanes, ra);
    const int nb = p.ftd * p.hd;
    const cudaError_t e = cudaMemsetAsync(ra.todo, 0, n * sizeof(int), stream);
    if (e != cudaSuccess) return e;
    record_scan_kernel<<<(nb + 127) / 128, 128, 0, stream>>>(ra.rows, static_cast<int>(n), nb, ra.cap, ra.todo,
                                                             filled);
    plain_fp64_kernel<kRecord><<<g.blocks, 128, 0, stream>>>(p, t, pid_begin, n, g.lanes, ra);
    return cudaGetLastError();
}

}  // namespace dsmc
