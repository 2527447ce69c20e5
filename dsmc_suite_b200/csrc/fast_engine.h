// fast_engine.h - resident-slot engine of the FAST paths (internal to the library).
//
// A fixed set of particle slots (one per resident thread) lives in HBM as structure-of-arrays.
// Each launch advances every slot by up to K Verlet steps; a slot whose particle ends takes the
// next particle from a device work queue that spans one or many problem instances. A solve of one
// instance launches kernels that carry its descriptor as a parameter; the served queue captures
// its launch loop once as a CUDA graph of G launches and replays it.
#pragma once

#include <vector>

#include "dsmc_device.cuh"

namespace dsmc {

// One problem instance as the fast kernel sees it.
struct FastInst {
    dsmc_params p;
    DevTables t;
    const float *rb2;        // [hd+1] squared shell boundaries, rb2[0] = R^2, rb2[hd] = r_top^2
    const float *sbs;        // [ftd+1] sin(b)|sin(b)| of latitude boundaries b_k
    const float2 *lonb;      // [ffd+1] (sin, cos) of longitude boundaries phi_k = 2 pi k / ffd
    // the same boundary tables in FP64 (FAST_FP64 solves; nullptr elsewhere)
    const double *rb2d, *sbsd;
    const double2 *lonbd;
    long long work_base;     // first work index of this instance in the queue
    long long n;             // particles
    long long pid_begin;     // particle id of the first particle
    float c_day;             // h / lifetime / ln 2 (W = W0 * 2^(-c_day * n_day))
    float r_land2, r_esc2;   // Radii^2, max_height^2
    double c_day_d;          // c_day in FP64
    int gather;              // lane-chunks a stopped lane may idle before its warp runs the events
                             // it gathered (0: no gathering), from the hop length (gather_chunks)
    double drift_abs;        // drift_tol * GM / Radii: the energy-drift guard's bound (0 = off)
    // collision rate n * sigma per cell in the engine's precision, negative where the cell has no
    // valid fit (the path integral grows there, no collision follows), 0 where nothing collides;
    // built for solves of one instance (nsig_kernel), nullptr in the served queue
    const float *nsig;
    const double *nsigd;
    const float4 *face_f;    // FP32 icosphere tables (config model), or nullptr: FP64 descent
};

// FP32 icosphere tables of an instance (floats; 0 when the problem has no icosphere) and their
// construction on the device from the problem's FP64 tables.
size_t face_floats_for(int nlevel);
size_t face_table_floats(const dsmc_params &p, const DevTables &t);
cudaError_t build_face_tables(const DevTables &t, float4 *out, cudaStream_t stream);

// Structure-of-arrays particle slots of an engine computing in R: float (the FAST_FP32 path:
// position and velocity as two-sum (hi, lo) pairs) or double (FAST_FP64: the lo arrays are
// carved but unused).
template <typename R>
struct SlotsT {
    int *inst;               // instance index, -1 = empty
    unsigned *pid;           // particle id within its instance
    unsigned *evt;           // Philox event counter
    R *sh, *sl, *vh, *vl, *oa;   // [3][S] each: position hi/lo, velocity hi/lo, old accel
                                 // (times -dt in the FP32 engine)
    R *w0;                   // weight factor outside photolysis
    int *nday;               // day-side steps (photolysis exponent)
    int *steps;              // steps in the particle's life
    int *hop;                // steps in the current hop
    int *cell;               // packed (ht << 16) | (td << 8) | fd
    int *run_cell;           // cell of the register deposit run, -1 = none
    R *run_w;                // weight-steps in run_cell not yet flushed (8-byte slot reserved)
    int *hist_key;           // speed bin of the histogram's run in run_cell, -1 = none
    int *hist_cnt;
    R *pcol, *pthr;          // accumulated collision probability and its threshold
    int *ncol;
    float *rest;             // freeze waiting time (reference model)
    R *wcur;                 // running weight (the hot loop's W between launches)
    int *face;               // icosphere face of the last launch point (config model), -1 = none
    float *e0;               // orbital energy at the hop's launch or last collision (drift guard)
};
using Slots = SlotsT<float>;

// Bytes of one slot in the structure-of-arrays block: run_w (an 8-byte slot), the 4-byte fields
// (inst pid evt nday steps hop cell run_cell hist_key hist_cnt ncol rest face e0) and the R fields
// (15 vector components, w0, pcol, pthr, wcur). carve_slots lays the arrays out over slot memory
// of fast_slot_bytes(nslots) bytes; nslots a multiple of 128 keeps every array 512-byte aligned.
template <typename R>
constexpr size_t slot_bytes_per_slot() { return 8 + 14 * 4 + 19 * sizeof(R); }
constexpr size_t kSlotBytesPerSlot = slot_bytes_per_slot<float>();
template <typename R>
SlotsT<R> carve_slots(void *mem, long long nslots);

// Device-side queue state. `total` and `ninst` live here rather than in the kernel arguments so
// that the host can append instances between launches of an already captured graph.
struct FastCounters {
    unsigned long long next;      // next work index
    unsigned long long finished;  // particles whose life ended
    unsigned long long total;     // work items in the queue (sum of the instances' particles)
    long long ninst;              // instances in the queue
    long long fill_warps;         // > 0: a queue of `total` particles, fewer than there are slots,
                                  // starts on this many warps (particle w + l * fill_warps on
                                  // lane l of warp w); 0: every slot takes from the queue
};

// The step loop's constants of one instance in the engine's precision.
template <typename R>
struct StepConst {
    R GM, dt, c1, c2;        // FP32: GM dt, dt, 1.5 dt, dt / 6; FP64: GM, dt, 1.5 dt^2, dt^2 / 6
    R rl2, re2;              // squared landing and escape radii
    R fday, sx, sy, sz;      // weight factor of a day-side step, direction to the sun
    float inv_bw;            // bins per m/s of the speed histogram
    int flags, half_ffd, life_cap, hop_cap, col_ht, nbins;
};
enum StepFlag { kFlagRef = 1, kFlagSkipFirst = 2, kFlagCollide = 4, kFlagHist = 8 };

template <typename R>
__host__ __device__ inline StepConst<R> step_consts(const FastInst &I) {
    const dsmc_params &p = I.p;
    StepConst<R> k;
    k.dt = static_cast<R>(p.dt_step);
    if constexpr (sizeof(R) == sizeof(double)) {
        k.GM = p.GM;
        k.c1 = 1.5 * p.dt_step * p.dt_step;
        k.c2 = p.dt_step * p.dt_step / 6.0;
        k.rl2 = p.Radii * p.Radii;
        k.re2 = p.max_height * p.max_height;
    } else {
        k.GM = static_cast<R>(p.GM * p.dt_step);
        k.c1 = static_cast<R>(1.5 * p.dt_step);
        k.c2 = static_cast<R>(p.dt_step / 6.0);
        k.rl2 = I.r_land2;
        k.re2 = I.r_esc2;
    }
    k.fday = static_cast<R>(p.wdecay);
    k.sx = static_cast<R>(p.sun[0]);
    k.sy = static_cast<R>(p.sun[1]);
    k.sz = static_cast<R>(p.sun[2]);
    k.half_ffd = p.ffd / 2;
    k.flags = (p.model == DSMC_MODEL_REFERENCE ? kFlagRef : 0) |
              (p.skip_first_deposit ? kFlagSkipFirst : 0) |
              (p.runner == DSMC_RUNNER_ADVANCED && I.t.n_bg ? kFlagCollide : 0) |
              (I.t.speed_hist && p.n_speed_bins > 0 ? kFlagHist : 0);
    const long long most = 0x7fffffffLL, life = p.life_step_cap, hop = p.hop_step_cap;
    k.life_cap = static_cast<int>(life <= 0 || life > most ? most : life);
    k.hop_cap = static_cast<int>(hop > most ? most : hop);
    k.col_ht = p.collide_ht_max;
    k.nbins = p.n_speed_bins;
    k.inv_bw = k.nbins > 0 ? static_cast<float>(1.0 / p.speed_bin_width) : 0.f;
    return k;
}

// Kernel arguments. The queue's size (total work items, instances) is read from the counters.
// FastArgsT: the served queue of many instances, whose descriptors lie in device memory.
template <typename R>
struct FastArgsT {
    static constexpr bool kOne = false;
    const FastInst *inst_;
    SlotsT<R> s;
    long long nslots;
    FastCounters *ctr;
    int K;
    __device__ const FastInst &inst(int k) const { return inst_[k]; }
    __device__ long long slot(long long i) const { return i; }
};

// OneArgsT: a solve of one instance, whose descriptor and step constants travel with the launch.
// They lie in the constant bank, where an arithmetic instruction reads its operand for free: the
// step loop keeps no constant in a register and an event reads its parameters without a load.
template <typename R>
struct OneArgsT {
    static constexpr bool kOne = true;
    FastInst one;
    StepConst<R> k;
    SlotsT<R> s;
    long long nslots;
    FastCounters *ctr;
    int K;
    int gather;               // lane-chunks of event gathering in this launch (see fast_kernel)
    const int *map;           // slot of each thread (-1: none), or nullptr: thread i has slot i
    __device__ const FastInst &inst(int) const { return one; }
    __device__ long long slot(long long i) const { return map ? map[i] : i; }
};

template <typename R> using OneKernel = void (*)(OneArgsT<R>);
using ServedKernel = void (*)(FastArgsT<float>);
// Lanes per SM up to which a launch runs the loops for few particles. 5e4 Moon-like particles (340
// per SM) take 3.5 ms in warp_kernel against 5.4 ms in the bulk loop, and the tail of 3e5 runs the
// solve in 6.6 against 8.4 ms (200 to 500 per SM are within 1 % on five solves). Below kTinyPerSm
// warp_kernel takes 12 steps in a row: 1e4 Ceres-like particles 2.03 ms, 2.23 at 8.
constexpr long long kSparsePerSm = 400, kTinyPerSm = 128, kAnyLanes = 1ll << 40;
// Steps in a row of the FP64 engine's loop for few particles, and of warp_kernel at most.
constexpr int kSparseUnroll = 8, kWarpUnroll = 12;
// The kernels of a solve of one instance for a register budget of blocks_per_sm blocks of 128
// threads (FP32: 4 or 5; FP64: 3, 4, or 5 in the lean loop) and a launch over lanes_per_sm live
// particles per SM. long_hops: the instance's events are not gathered.
OneKernel<float> one_kernel32(int blocks_per_sm, int mode, bool long_hops, long long lanes_per_sm);
OneKernel<double> one_kernel64(int blocks_per_sm, int mode, long long lanes_per_sm);
// The kernels of a queue of many instances (fast_served.cu lists the variants).
ServedKernel served_kernel(int variant, int mode);

// Dynamic shared memory of a OneArgsT kernel: 256 columns (pairs), 256 rows, hd + 1 shells.
inline size_t one_table_bytes(const dsmc_params &p, bool fp64) {
    return (3 * 256 + static_cast<size_t>(p.hd) + 1) * (fp64 ? sizeof(double) : sizeof(float));
}

// Pieces of the engine for callers that supply every buffer themselves (no allocation here):
// bytes of the slot arrays for nslots slots, of one instance descriptor and of the counters;
// fast_fill_instance builds one descriptor and its boundary tables in host memory (tab_host,
// tab_floats entries; d_tab is where the caller will copy them); fast_drain_external runs the
// launch loop without graphs on caller memory until the queue of `total` particles is empty, and
// gives up (cudaErrorLaunchTimeout) after stall_launches launches in a row in which no particle
// finished.
size_t fast_slot_bytes(long long nslots, bool fp64 = false);
size_t fast_inst_bytes();
size_t fast_counter_bytes();
// Expected steps of a typical hop: the ballistic flight time 2 v / g of a molecule launched at
// the thermal speed sqrt(k_B T / m) of a 235 K surface, over the time step.
double fast_hop_steps(const dsmc_params &p);
// Event gathering of an instance from its typical hop (see fast_kernel): 16 lane-chunks below
// 300 steps per hop, 4 below 600, none above.
int gather_chunks(const dsmc_params &p);
cudaError_t fast_fill_instance(const dsmc_params &p, const DevTables &t, long long pid_begin,
                               long long n, float *d_tab, size_t tab_floats, void *inst_host,
                               float *tab_host);
cudaError_t fast_drain_external(const void *d_inst, void *slot_mem, long long nslots, void *d_ctr,
                                long long total, int steps_per_launch, int block,
                                long long stall_launches, cudaStream_t stream,
                                long long *launches);

class FastEngine {
public:
    FastEngine() = default;
    ~FastEngine();
    FastEngine(const FastEngine &) = delete;
    FastEngine &operator=(const FastEngine &) = delete;

    // Solve particles [pid_begin, pid_begin + n) of one instance to the end of their lives, in
    // FP32 with two-sum compensation (fp64 false) or in FP64 (the FAST_FP64 path: the same
    // slots, queue, cell tracking and register deposits on double state and FP64 tables).
    cudaError_t run(const dsmc_params &p, const DevTables &t, bool fp64, long long pid_begin,
                    long long n, int num_sms, cudaStream_t stream);

    void set_shape(int blk, int per_sm, int k, int g) {
        block = blk;
        blocks_per_sm = per_sm;
        steps_per_launch = k;
        launches_per_graph = g;
    }
    long long slot_count() const { return nslots_; }

    // Launch shape (autotuned or set by the caller).
    int block = 128;          // threads per block
    int blocks_per_sm = 0;    // resident blocks per SM (0 = as many as fit)
    int steps_per_launch = 8192;
    int launches_per_graph = 8;
    long long launches = 0;   // launches issued by the last run

private:
    cudaError_t ensure_slots(int num_sms);
    cudaError_t upload_one(const dsmc_params &p, const DevTables &t, long long pid_begin, long long n,
                           cudaStream_t stream);
    cudaError_t launch_one(cudaStream_t stream, long long threads, const int *map, long long lanes_per_sm);
    void launch_served(cudaStream_t stream, int mode);
    cudaError_t drain(long long total, cudaStream_t stream);
    cudaError_t capture(cudaStream_t stream, int mode, cudaGraphExec_t *out);
    long long warps_for(long long live) const;
    bool long_hops() const { return inst_host_.gather == 0; }
    void free_graphs();

public:
    // Serving: an open queue that grows while it drains. serve_open resets the engine to an
    // empty queue with room for max_instances instances. serve_append adds one instance: its
    // boundary tables and descriptor are written on `upload` (which it synchronises), and the
    // larger queue is published on `compute` in stream order, so kernels already in flight are
    // not waited for; its statistics go to the engine's per-instance row `index`. serve_launch
    // enqueues one round (the captured graph, or one launch) without waiting. serve_release
    // frees an instance's boundary tables once all its particles have finished.
    cudaError_t serve_open(int num_sms, int max_instances, cudaStream_t stream);
    cudaError_t serve_append(const dsmc_params &p, const DevTables &t, long long n, int *index,
                             cudaStream_t upload, cudaStream_t compute);
    cudaError_t serve_launch(cudaStream_t stream, int mode);
    // Loop an instance may run in: 1 lean (config model, ballistic, no speed histogram, hop cap
    // not below the life cap), 2 lean with collisions (the same, collisional), 0 general only.
    // Every loop that can run an instance gives it identical results.
    static int loop_mode(const dsmc_params &p, const DevTables &t);
    void serve_release(int index, cudaStream_t stream);
    const FastCounters *serve_counters() const { return d_ctr_; }
    const unsigned long long *serve_stats_rows() const { return d_stats_; }
    int serve_instances() const { return ninst_; }
    int serve_capacity() const { return ninst_cap_; }
    // floats of an instance's table block: boundary tables, plus the FP32 icosphere tables of a
    // config-model problem with an icosphere of nlevel levels (nlevel < 0: none)
    static size_t serve_table_floats(const dsmc_params &p, int nlevel);
    void serve_set_pool(cudaMemPool_t pool) { pool_ = pool; }
    void serve_close(cudaStream_t stream);   // frees every instance's boundary tables
    size_t serve_fixed_bytes(int max_instances) const;

private:
    unsigned long long *d_stats_ = nullptr;   // [max_instances][kStatCount] (serving)
    int stats_cap_ = 0;
    cudaMemPool_t pool_ = nullptr;            // stream-ordered allocations (serving)
    std::vector<void *> inst_tabs_;           // boundary tables per instance (serving)
    unsigned long long serve_total_ = 0;
    void free_all();

    Slots slots_{};
    SlotsT<double> slots64_{};                // the same memory carved for FP64 state
    void *slot_mem_ = nullptr;
    bool fp64_ = false;                       // precision of run launches
    bool slot_fp64_ = false;                  // precision the slot memory is carved for
    long long nslots_ = 0;
    FastInst *d_inst_ = nullptr;
    int ninst_cap_ = 0;
    int ninst_ = 0;
    void *d_nsig_ = nullptr;                  // collision rates of a solve (FastInst::nsig)
    size_t nsig_cap_ = 0;
    float *d_tab_ = nullptr;
    size_t tab_cap_ = 0;
    std::vector<float> tab_host_;             // staging of d_tab_
    FastInst inst_host_{};                    // the instance of a solve
    FastCounters *d_ctr_ = nullptr;
    FastCounters *h_ctr_ = nullptr;           // [3] pinned: the last two launches', the start's
    cudaEvent_t round_[2] = {nullptr, nullptr};
    int *d_map_ = nullptr;                    // packed slots of a drain's last launches, in slot_mem_
    cudaGraphExec_t graph_mode_[3] = {nullptr, nullptr, nullptr};   // serving: loops 0, 1, 2
    int num_sms_ = 0;
    int variant_ = 4;
    int mode_ = 0;            // loop of a solve (see Mode in fast_kernel.cuh)
    bool one_ = false;        // a solve runs the kernels that take the instance with the launch
    size_t one_smem_ = 0;     // their shared memory (the boundary tables)
};

}  // namespace dsmc
