// fast_engine.cu - host side of the FAST paths: slots, boundary tables, the launch loop of a solve,
// and the served queue. The kernels are in fast_kernel.cuh.
#include "fast_engine.h"
#include "dsmc_kernels.h"

#include <algorithm>
#include <type_traits>
#include <cmath>
#include <cstring>
#include <vector>

namespace dsmc {

FastEngine::~FastEngine() { free_all(); }

void FastEngine::free_graphs() {
    for (cudaGraphExec_t &g : graph_mode_) {
        if (g) cudaGraphExecDestroy(g);
        g = nullptr;
    }
}

void FastEngine::free_all() {
    free_graphs();
    if (slot_mem_) cudaFree(slot_mem_);
    slot_mem_ = nullptr;
    if (d_inst_) cudaFree(d_inst_);
    d_inst_ = nullptr;
    if (d_tab_) cudaFree(d_tab_);
    d_tab_ = nullptr;
    if (d_nsig_) cudaFree(d_nsig_);
    d_nsig_ = nullptr;
    if (d_ctr_) cudaFree(d_ctr_);
    d_ctr_ = nullptr;
    if (h_ctr_) cudaFreeHost(h_ctr_);
    h_ctr_ = nullptr;
    d_map_ = nullptr;
    for (cudaEvent_t &e : round_) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
    if (d_stats_) cudaFree(d_stats_);
    d_stats_ = nullptr;
    stats_cap_ = 0;
    ninst_cap_ = 0;
    for (void *p : inst_tabs_)
        if (p) cudaFree(p);
    inst_tabs_.clear();
    nslots_ = 0;
}

namespace {

// FP64 variant for a launch shape: 5 blocks per SM (96 registers) in the lean loop, else 4 (128
// registers), 3 (168) when asked. More resident warps beat spill-free code, as in FP32: the lean
// loop runs 2e6 Ceres-like particles in 86.6 ms at 5 against 91.0 ms at 4 (1e6 Europa-like 25.7
// against 26.9 ms), and 1e7 at 4 in 63 ms against 73 ms at 3; the other loops spill over 450 B
// a thread at 5.
int pick_variant64(int blocks_per_sm, int mode) {
    if (mode == 1 && (blocks_per_sm == 0 || blocks_per_sm == 5)) return 5;
    return blocks_per_sm == 3 ? 3 : 4;
}

// Variant for a launch shape: blocks_per_sm names the register budget. The default (0) is the
// fastest measured on B200 for each loop (in the served queue's kernels), spills or not: the lean
// loop at 96 registers (20 warps per SM) beats 128 registers (16 warps) by 6 % and 80 (24 warps)
// by 3 %; the collision loop at 96 beats 128 by 1.5 % and 168 (no spills, 12 warps) by 15 %;
// the general loop at 128 beats 168 by 19 % and 96 by 18 %. Spill stores by ptxas, served queue and
// solve of one instance: lean 92 and 0 B, collision 336 and 92 B, general 372 and 40 B.
int pick_variant(int block, int blocks_per_sm, int mode) {
    if (block > 128) return blocks_per_sm >= 3 ? 1 : 0;
    if (blocks_per_sm == 2) return 3;
    if (blocks_per_sm == 3) return 2;
    if (blocks_per_sm == 4) return 4;
    if (blocks_per_sm == 5) return 5;
    return mode == 0 ? 4 : 5;
}

// Loop mode of one instance (see Mode in fast_kernel.cuh): 0 general, 1 and 2 the config model's
// lean loops without and with collisions, 3 and 5 the reference model's, 4 the config model with
// speed histograms.
int instance_mode(const dsmc_params &p, const DevTables &t) {
    const bool col = p.runner == DSMC_RUNNER_ADVANCED && t.n_bg;
    const bool hist = t.speed_hist && p.n_speed_bins > 0;
    if (p.model == DSMC_MODEL_REFERENCE) return hist || p.life_step_cap > 0 ? 0 : col ? 5 : 3;
    if (p.skip_first_deposit || p.life_step_cap <= 0 || p.hop_step_cap < p.life_step_cap || (hist && col))
        return 0;
    return hist ? 4 : col ? 2 : 1;
}

}  // namespace

namespace {

// FP32 copies of the icosphere's base-face centroids and corner-cut planes, as float4 (xyz, 0):
// [0, 20) centroids, then 3 planes per subdivision node, then per leaf face the normals of the 3
// planes through the origin and its edges, turned so that the face's cone is on their positive
// side (a point lies in face f iff its direction is on the positive side of all three). Built on
// the device from the problem's FP64 tables.
__global__ void face_tables_kernel(const double *cent, const double *planes, const double *verts,
                                   int nnode, int nface, float4 *out) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long long np = 20 + 3ll * nnode;
    if (i < 20) {
        out[i] = make_float4(static_cast<float>(cent[3 * i]), static_cast<float>(cent[3 * i + 1]),
                             static_cast<float>(cent[3 * i + 2]), 0.0f);
    } else if (i < np) {
        const double *q = planes + 3 * (i - 20);   // node (i-20)/3, plane (i-20)%3
        out[i] = make_float4(static_cast<float>(q[0]), static_cast<float>(q[1]), static_cast<float>(q[2]), 0.0f);
    } else if (i < np + 3ll * nface) {
        const long long f = (i - np) / 3;
        const int e = static_cast<int>((i - np) % 3);
        const double *v = verts + 9 * f;
        const double *p = v + 3 * e, *q = v + 3 * ((e + 1) % 3);
        double c[3] = {p[1] * q[2] - p[2] * q[1], p[2] * q[0] - p[0] * q[2], p[0] * q[1] - p[1] * q[0]};
        const double m[3] = {v[0] + v[3] + v[6], v[1] + v[4] + v[7], v[2] + v[5] + v[8]};
        if (c[0] * m[0] + c[1] * m[1] + c[2] * m[2] < 0.0)
            for (int k = 0; k < 3; k++) c[k] = -c[k];
        out[i] = make_float4(static_cast<float>(c[0]), static_cast<float>(c[1]), static_cast<float>(c[2]), 0.0f);
    }
}

}  // namespace

size_t face_floats_for(int nlevel) {
    const size_t nnode = static_cast<size_t>(20 * ((1 << (2 * nlevel)) - 1) / 3);
    const size_t nface = static_cast<size_t>(20) << (2 * nlevel);
    return 4 * (20 + 3 * nnode + 3 * nface);
}

size_t face_table_floats(const dsmc_params &p, const DevTables &t) {
    if (p.model != DSMC_MODEL_CONFIG || !t.base_centroid || !t.split_planes || !t.face_verts ||
        t.nlevel < 0)
        return 0;
    return face_floats_for(t.nlevel);
}

cudaError_t build_face_tables(const DevTables &t, float4 *out, cudaStream_t stream) {
    const int nnode = 20 * ((1 << (2 * t.nlevel)) - 1) / 3;
    const int nface = 20 << (2 * t.nlevel);
    const int n = 20 + 3 * nnode + 3 * nface;
    face_tables_kernel<<<(n + 127) / 128, 128, 0, stream>>>(t.base_centroid, t.split_planes,
                                                            t.face_verts, nnode, nface, out);
    return cudaGetLastError();
}

cudaError_t FastEngine::ensure_slots(int num_sms) {
    num_sms_ = num_sms;
    // one wave: as many blocks per SM as can be resident together
    int resident = 0;
    cudaError_t e0;
    if (fp64_) {
        if (block != 128) return cudaErrorInvalidValue;   // the FP64 engine runs 128-thread blocks
        variant_ = pick_variant64(blocks_per_sm, mode_);
        e0 = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, one_kernel64(variant_, mode_, kAnyLanes), block, one_smem_);
    } else {
        variant_ = pick_variant(block, blocks_per_sm, mode_);
        e0 = one_ ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, one_kernel32(variant_, mode_, long_hops(), kAnyLanes), block, one_smem_)
                  : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, served_kernel(variant_, mode_), block, 0);
    }
    if (e0 != cudaSuccess) return e0;
    if (resident < 1) return cudaErrorInvalidConfiguration;
    const int per_sm = (blocks_per_sm > resident || blocks_per_sm < 1) ? resident : blocks_per_sm;
    const long long want = static_cast<long long>(num_sms) * per_sm * block;
    // each part by itself, so that a call after one whose allocation failed goes on where that stopped
    cudaError_t e;
    if (!d_ctr_ && (e = cudaMalloc(&d_ctr_, sizeof(FastCounters))) != cudaSuccess) return e;
    if (!h_ctr_ && (e = cudaMallocHost(&h_ctr_, 3 * sizeof(FastCounters))) != cudaSuccess) return e;
    for (cudaEvent_t &r : round_)
        if (!r && (e = cudaEventCreateWithFlags(&r, cudaEventDisableTiming)) != cudaSuccess) return e;
    if (slot_mem_ && nslots_ == want && slot_fp64_ == fp64_) return cudaSuccess;
    free_graphs();
    if (slot_mem_) cudaFree(slot_mem_);
    slot_mem_ = nullptr;
    nslots_ = 0;
    const long long S = want;
    // behind the slots, the map of the drain's last launches (see drain): a counter, then one slot
    // per thread
    const size_t slot_bytes = (fast_slot_bytes(S, fp64_) + 255) & ~static_cast<size_t>(255);
    if ((e = cudaMalloc(&slot_mem_, slot_bytes + (S + 32) * sizeof(int))) != cudaSuccess) {
        slot_mem_ = nullptr;
        return e;
    }
    d_map_ = reinterpret_cast<int *>(static_cast<char *>(slot_mem_) + slot_bytes);
    slots_ = Slots{};
    slots64_ = SlotsT<double>{};
    if (fp64_) slots64_ = carve_slots<double>(slot_mem_, S);
    else slots_ = carve_slots<float>(slot_mem_, S);
    slot_fp64_ = fp64_;
    nslots_ = S;
    return cudaSuccess;
}

namespace {

// Idle limit (lane-chunks) of event gathering once the live slots are packed: a lane that waits
// then delays the end of the solve. 1e6 Europa-like particles in FP64 ran 25.7 ms at the full
// limit of 16, 25.1 ms at 2 and 25.4 ms at 0; 3e5 Moon-like 8.6, 8.25 and 8.4 ms.
constexpr int kTailGather = 2;

// Warps per SM that a few particles are spread over: one per scheduler. More warps of fewer lanes
// diverge less but take issue slots from one another; 1e4 Ceres-like particles ran 3.85 ms on 2
// warps per SM, 4.04 on 4, 4.49 on 8 and 5.84 on 20, 512 particles 3.1 to 3.3 ms on any (the
// first lanes of the slots, 4 full warps on each of a few SMs, took 4.4 and 3.7 ms).
constexpr int kSpreadWarpsPerSm = 4;

// The reference model launches into a half-space that the ground takes half of, so a particle lands
// every few steps and its events, which hold up the rest of its warp, are most of its life: 5000
// particles run 29.3 ms on 4 warps per SM, 24.6 on 8, 24.3 on 16 (FP64 44.9, 41.9, 40.7 ms).
constexpr int kSpreadWarpsPerSmRef = 16;

}  // namespace

// Warps that hold `live` particles: full ones, but at least one per scheduler; whole blocks, so
// that every thread of a launch has an entry in the map.
long long FastEngine::warps_for(long long live) const {
    const long long per_block = block / 32;
    const long long per_sm = inst_host_.p.model == DSMC_MODEL_REFERENCE ? kSpreadWarpsPerSmRef : kSpreadWarpsPerSm;
    long long w = std::max<long long>(per_sm * num_sms_, (live + 31) / 32);
    w = (w + per_block - 1) / per_block * per_block;
    return std::min(w, nslots_ / 32);
}

namespace {

// Offsets (in elements) of the boundary tables in one block: shells [hd+1] at 0, rows [ftd+1],
// columns [ffd+1] pairs.
struct BoundaryLayout { size_t sbs, lonb, count; };

template <typename R>
BoundaryLayout boundary_layout(const dsmc_params &p) {
    BoundaryLayout l;
    l.sbs = static_cast<size_t>(p.hd + 1);
    l.lonb = (l.sbs + (p.ftd + 1) + 1) & ~static_cast<size_t>(1);   // pairs start on a pair
    l.count = l.lonb + 2 * static_cast<size_t>(p.ffd + 1);
    return l;
}

template <typename R>
void fill_boundaries(const dsmc_params &p, const BoundaryLayout &l, R *tab) {
    R *rb2 = tab, *sbs = tab + l.sbs, *lon = tab + l.lonb;
    for (int j = 0; j <= p.hd; j++) {
        const double rj = p.use_exp_grid ? p.Radii + p.unih * (std::pow(1.0 + p.alpha2, j) - 1.0) / p.alpha2
                                         : p.Radii + j * p.unih;
        rb2[j] = static_cast<R>(rj * rj);
    }
    for (int j = 0; j <= p.ftd; j++) {
        const double sb = std::sin(static_cast<double>(j) / p.ftd * kPi - kPi / 2.0);
        sbs[j] = static_cast<R>(sb * std::fabs(sb));
    }
    sbs[0] = R(-1);
    sbs[p.ftd] = R(1);
    for (int j = 0; j <= p.ffd; j++) {
        const double ph = 2.0 * kPi * j / p.ffd;
        lon[2 * j] = static_cast<R>(std::sin(ph));
        lon[2 * j + 1] = static_cast<R>(std::cos(ph));
    }
    lon[0] = R(0); lon[1] = R(1);
    lon[2 * p.ffd] = R(0); lon[2 * p.ffd + 1] = R(1);
}

// The descriptor's scalars; the table pointers stay null.
void fill_inst(const dsmc_params &p, const DevTables &t, long long pid_begin, long long n, FastInst *I) {
    std::memset(I, 0, sizeof *I);
    I->p = p;
    I->t = t;
    I->n = n;
    I->pid_begin = pid_begin;
    I->c_day = static_cast<float>(p.dt_step / p.lifetime / std::log(2.0));
    I->c_day_d = p.dt_step / p.lifetime / std::log(2.0);
    I->gather = gather_chunks(p);
    I->drift_abs = p.drift_tol > 0.0 ? p.drift_tol * p.GM / p.Radii : 0.0;
    I->r_land2 = static_cast<float>(p.Radii * p.Radii);
    I->r_esc2 = static_cast<float>(p.max_height * p.max_height);
}

// Collision rates of a solve's cells (FastInst::nsig): what a cell change had to look up and
// convert, and whether the cell can collide at all, which was looked up on every step after the
// path integral had passed its threshold in a cell without a fit. The reference's phase 2, whose
// fits cover few cells, spent most of its steps there: 500 particles 73.6 -> 59.3 ms; 1e6 particles
// of the config-model phase 2 51.6 -> 49.4 ms.
template <typename R>
__global__ void nsig_kernel(const dsmc_params p, const DevTables t, R *out) {
    const long long ncell = static_cast<long long>(p.hd) * p.ftd * p.ffd;
    const long long c = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= ncell) return;
    const int fd = static_cast<int>(c % p.ffd), td = static_cast<int>(c / p.ffd % p.ftd),
              ht = static_cast<int>(c / p.ffd / p.ftd);
    R rate = R(0);
    if (ht < p.collide_ht_max && c < t.n_bg_len) rate = static_cast<R>(t.n_bg[c] * p.cross_section);
    if (!(rate > R(0))) rate = R(0);
    else if (!t.cdf_valid[(static_cast<long long>(td) * p.ffd + fd) * p.hd + ht]) rate = -rate;
    out[c] = rate;
}

// Packs the slots that still hold a particle over the first `warps` warps: the k-th found goes to
// lane k / warps of warp k % warps. map[0] counts (from -1, as the clear leaves it); map[32 + t]
// is the slot of thread t, -1 for none.
__global__ void pack_slots_kernel(const int *inst, long long nslots, int warps, int *map) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= nslots || inst[i] < 0) return;
    const int k = atomicAdd(map, 1) + 1;
    if (k < 32 * warps) map[32 + (k % warps) * 32 + k / warps] = static_cast<int>(i);
}

}  // namespace

// Boundary tables (FP32, and FP64 for an FP64 solve) and, for config-model problems, the FP32
// icosphere tables of the one instance of a solve. The descriptor itself travels with each launch.
cudaError_t FastEngine::upload_one(const dsmc_params &p, const DevTables &t, long long pid_begin,
                                   long long n, cudaStream_t stream) {
    const BoundaryLayout l = boundary_layout<float>(p);
    const size_t ff = face_table_floats(p, t);
    const size_t off64 = (l.count + 3) & ~static_cast<size_t>(3);                       // 16-byte starts
    const size_t off_face = (off64 + (fp64_ ? 2 * l.count : 0) + 3) & ~static_cast<size_t>(3);
    const size_t total = off_face + ff;
    cudaError_t e;
    if (total > tab_cap_) {
        if (d_tab_) cudaFree(d_tab_);
        d_tab_ = nullptr;
        tab_cap_ = 0;
        if ((e = cudaMalloc(&d_tab_, total * sizeof(float))) != cudaSuccess) return e;
        tab_cap_ = total;
    }
    tab_host_.assign(off_face, 0.0f);
    fill_boundaries(p, l, tab_host_.data());
    if (fp64_) fill_boundaries(p, l, reinterpret_cast<double *>(tab_host_.data() + off64));
    fill_inst(p, t, pid_begin, n, &inst_host_);
    inst_host_.rb2 = d_tab_;
    inst_host_.sbs = d_tab_ + l.sbs;
    inst_host_.lonb = reinterpret_cast<const float2 *>(d_tab_ + l.lonb);
    if (fp64_) {
        const double *d = reinterpret_cast<const double *>(d_tab_ + off64);
        inst_host_.rb2d = d;
        inst_host_.sbsd = d + l.sbs;
        inst_host_.lonbd = reinterpret_cast<const double2 *>(d + l.lonb);
    }
    if ((e = cudaMemcpyAsync(d_tab_, tab_host_.data(), off_face * sizeof(float), cudaMemcpyHostToDevice, stream)) != cudaSuccess)
        return e;
    if (ff) {
        float4 *face = reinterpret_cast<float4 *>(d_tab_ + off_face);
        inst_host_.face_f = face;
        if ((e = build_face_tables(t, face, stream)) != cudaSuccess) return e;
    }
    if (one_ && p.runner == DSMC_RUNNER_ADVANCED && t.n_bg) {
        const size_t ncell = static_cast<size_t>(p.hd) * p.ftd * p.ffd, need = ncell * (fp64_ ? 8 : 4);
        if (need > nsig_cap_) {
            if (d_nsig_) cudaFree(d_nsig_);
            d_nsig_ = nullptr;
            nsig_cap_ = 0;
            if ((e = cudaMalloc(&d_nsig_, need)) != cudaSuccess) return e;
            nsig_cap_ = need;
        }
        const unsigned blocks = static_cast<unsigned>((ncell + 255) / 256);
        if (fp64_) {
            nsig_kernel<<<blocks, 256, 0, stream>>>(p, t, static_cast<double *>(d_nsig_));
            inst_host_.nsigd = static_cast<const double *>(d_nsig_);
        } else {
            nsig_kernel<<<blocks, 256, 0, stream>>>(p, t, static_cast<float *>(d_nsig_));
            inst_host_.nsig = static_cast<const float *>(d_nsig_);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (!one_) {
        if (ninst_cap_ < 1) {
            if ((e = cudaMalloc(&d_inst_, sizeof(FastInst))) != cudaSuccess) return e;
            ninst_cap_ = 1;
        }
        e = cudaMemcpyAsync(d_inst_, &inst_host_, sizeof(FastInst), cudaMemcpyHostToDevice, stream);
    }
    return e;
}

// One launch of the solve's kernel over `threads` slots (map: see drain).
cudaError_t FastEngine::launch_one(cudaStream_t stream, long long threads, const int *map, long long lanes_per_sm) {
    const unsigned grid = static_cast<unsigned>(threads / block);   // whole blocks (see warps_for)
    auto fill = [&](auto &a, const auto &slots) {
        a.one = inst_host_;
        a.k = step_consts<std::decay_t<decltype(a.k.dt)>>(inst_host_);
        a.s = slots;
        a.nslots = nslots_;
        a.ctr = d_ctr_;
        a.K = steps_per_launch;
        a.map = map;
        a.gather = map ? std::min(inst_host_.gather, kTailGather) : inst_host_.gather;
    };
    if (slot_fp64_) {
        OneArgsT<double> a{};
        fill(a, slots64_);
        one_kernel64(variant_, mode_, lanes_per_sm)<<<grid, block, one_smem_, stream>>>(a);
    } else if (one_) {
        OneArgsT<float> a{};
        fill(a, slots_);
        one_kernel32(variant_, mode_, long_hops(), lanes_per_sm)<<<grid, block, one_smem_, stream>>>(a);
    } else {
        launch_served(stream, mode_ <= 2 ? mode_ : 0);
    }
    return cudaGetLastError();
}

// One launch of a served loop over every slot.
void FastEngine::launch_served(cudaStream_t stream, int mode) {
    FastArgsT<float> a{};
    a.inst_ = d_inst_;
    a.s = slots_;
    a.nslots = nslots_;
    a.ctr = d_ctr_;
    a.K = steps_per_launch;
    served_kernel(variant_, mode)<<<static_cast<unsigned>(nslots_ / block), block, 0, stream>>>(a);
}

// G launches of a served loop captured as one graph.
cudaError_t FastEngine::capture(cudaStream_t stream, int mode, cudaGraphExec_t *out) {
    cudaError_t e;
    cudaGraph_t g;
    *out = nullptr;
    if ((e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) return e;
    for (int k = 0; k < launches_per_graph; k++) launch_served(stream, mode);
    if ((e = cudaStreamEndCapture(stream, &g)) != cudaSuccess) return e;
    e = cudaGraphInstantiate(out, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) *out = nullptr;
    return e;
}

// Steps per slot after which a drain looks at its counters at the latest: the default launch. Shorter
// launches run in rounds of launches_per_graph, within these steps, so that a shape of short launches
// pays for a look, and in the tail for the packing, once a round: launches of 64 steps in rounds of 16
// run 512 Ceres-like particles in 4.8 ms and 2e6 in 106 ms, against 11.4 and 132 ms with a look after
// each (7.1 and 117 ms with the former kernels in a graph of 16); of 16 steps in rounds of 64, 14.2 and
// 211 ms against 53 and 328 (14.1 and 223).
constexpr int kStepsPerRound = 8192;

// Rounds of launches until every particle of the queue has finished.
//
// While the queue still holds several rounds' worth of particles the rounds run back to back,
// the host reading the counters of one while the next runs. Near the end of the queue the host
// waits for each: once the queue is empty the slots drain unevenly, and before each round the
// live ones are packed over as few warps as keep every scheduler busy (pack_slots_kernel), so
// that no warp is issued for a few lanes.
cudaError_t FastEngine::drain(long long total, cudaStream_t stream) {
    cudaError_t e;
    launches = 0;
    if (total <= 0) return cudaSuccess;
    FastCounters *start = h_ctr_ + 2;
    start->next = 0;
    start->finished = 0;
    start->total = static_cast<unsigned long long>(total);
    start->ninst = 1;
    start->fill_warps = total < nslots_ ? warps_for(total) : 0;
    if ((e = cudaMemcpyAsync(d_ctr_, start, sizeof(FastCounters), cudaMemcpyHostToDevice, stream)) != cudaSuccess)
        return e;
    int *inst = slot_fp64_ ? slots64_.inst : slots_.inst;
    if ((e = cudaMemsetAsync(inst, 0xff, nslots_ * sizeof(int), stream)) != cudaSuccess) return e;
    const long long whole = start->fill_warps ? start->fill_warps * 32 : nslots_;
    const int group = std::max(1, std::min(launches_per_graph, kStepsPerRound / steps_per_launch));
    const double round_steps = static_cast<double>(group) * steps_per_launch;
    const long long sure_steps = static_cast<long long>(group) * ((steps_per_launch + kWarpUnroll - 1) / kWarpUnroll);
    // Every launch advances each live particle by its steps (warp_kernel: by at least one of every
    // kWarpUnroll) or ends it, and every life is bounded by its step caps, so the queue drains. The
    // loop still gives up (launch-timeout status) if no particle finishes for 2^28 steps, which
    // would mean a logic error, not a long solve.
    long long issued = 0, seen = 0, live = total, quiet = 0;
    double rate = 0.0;                    // particles taken from the queue per step
    unsigned long long next = 0, finished = 0;
    for (;;) {
        const double left = rate > 0.0 ? (static_cast<double>(total) - static_cast<double>(next)) / rate : 0.0;
        const bool empty = next >= static_cast<unsigned long long>(total);
        long long threads = whole;
        const int *map = nullptr;
        if (one_ && empty && live < whole) {
            const long long w = warps_for(live);
            if ((e = cudaMemsetAsync(d_map_, 0xff, (32 + w * 32) * sizeof(int), stream)) != cudaSuccess) return e;
            pack_slots_kernel<<<static_cast<unsigned>((nslots_ + 255) / 256), 256, 0, stream>>>(
                inst, nslots_, static_cast<int>(w), d_map_);
            threads = w * 32;
            map = d_map_ + 32;
        }
        for (int k = 0; k < group; k++) {
            if ((e = launch_one(stream, threads, map, (live + num_sms_ - 1) / num_sms_)) != cudaSuccess)
                return e;
            launches++;
        }
        const int at = static_cast<int>(issued & 1);
        if ((e = cudaMemcpyAsync(h_ctr_ + at, d_ctr_, sizeof(FastCounters), cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
            (e = cudaEventRecord(round_[at], stream)) != cudaSuccess)
            return e;
        issued++;
        // one round ahead of the counters while the queue lasts for several more
        while (issued - seen > (left > 4.0 * round_steps ? 1 : 0)) {
            const int r = static_cast<int>(seen & 1);
            if ((e = cudaEventSynchronize(round_[r])) != cudaSuccess) return e;
            seen++;
            const FastCounters &c = h_ctr_[r];
            if (c.finished >= static_cast<unsigned long long>(total)) return cudaStreamSynchronize(stream);
            rate = static_cast<double>(c.next - next) / round_steps;
            quiet = c.finished == finished ? quiet + sure_steps : 0;
            next = c.next;
            finished = c.finished;
            live = total - static_cast<long long>(finished);
            if (quiet > (1ll << 28)) return cudaErrorLaunchTimeout;
        }
    }
}

cudaError_t FastEngine::run(const dsmc_params &p, const DevTables &t, bool fp64, long long pid_begin,
                            long long n, int num_sms, cudaStream_t stream) {
    launches = 0;
    if (p.ftd > 255 || p.ffd > 255 || p.hd > 32767) return cudaErrorInvalidValue;
    fp64_ = fp64;
    mode_ = instance_mode(p, t);
    if (fp64 && mode_ > 2) mode_ = 0;   // the FP64 engine has loops 0, 1 and 2
    // the kernels that take the instance with the launch exist for 128-thread blocks of the two
    // default register budgets (and FP64's two); other shapes run the served kernels
    inst_host_.gather = gather_chunks(p);
    one_ = fp64 || pick_variant(block, blocks_per_sm, mode_) >= 4;
    one_smem_ = one_ ? one_table_bytes(p, fp64) : 0;
    cudaError_t e = ensure_slots(num_sms);
    if (e != cudaSuccess || n <= 0) return e;   // of no particles: nothing issued that a later call would wait for
    e = upload_one(p, t, pid_begin, n, stream);
    if (e != cudaSuccess) return e;
    return drain(n, stream);
}

cudaError_t FastEngine::serve_open(int num_sms, int max_instances, cudaStream_t stream) {
    if (max_instances < 1) return cudaErrorInvalidValue;
    fp64_ = false;   // serving runs the FP32 engine
    one_ = false;
    mode_ = 0;   // the slots are sized for the general loop; every round picks its own loop
    cudaError_t e = ensure_slots(num_sms);
    if (e != cudaSuccess) return e;
    for (void *p : inst_tabs_)
        if (p) cudaFreeAsync(p, stream);
    inst_tabs_.assign(static_cast<size_t>(max_instances), nullptr);
    if (max_instances > ninst_cap_) {
        if (d_inst_) cudaFree(d_inst_);
        d_inst_ = nullptr;
        ninst_cap_ = 0;
        if ((e = cudaMalloc(&d_inst_, static_cast<size_t>(max_instances) * sizeof(FastInst))) != cudaSuccess) return e;
        ninst_cap_ = max_instances;
        free_graphs();
    }
    if (!d_stats_ || stats_cap_ < max_instances) {
        if (d_stats_) cudaFree(d_stats_);
        d_stats_ = nullptr;
        if ((e = cudaMalloc(&d_stats_, static_cast<size_t>(max_instances) * kStatCount * sizeof(unsigned long long))) != cudaSuccess)
            return e;
        stats_cap_ = max_instances;
    }
    if ((e = cudaMemsetAsync(d_stats_, 0, static_cast<size_t>(max_instances) * kStatCount * sizeof(unsigned long long), stream)) != cudaSuccess)
        return e;
    ninst_ = 0;
    serve_total_ = 0;
    launches = 0;
    if ((e = cudaMemsetAsync(d_ctr_, 0, sizeof(FastCounters), stream)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(slots_.inst, 0xff, nslots_ * sizeof(int), stream)) != cudaSuccess) return e;
    // the general loop, and the lean loops over the same slots, for rounds in which every queued
    // instance qualifies
    free_graphs();
    for (int m = 0; m <= 2 && launches_per_graph > 1; m++)
        if ((e = capture(stream, m, &graph_mode_[m])) != cudaSuccess) return e;
    return cudaStreamSynchronize(stream);
}

int FastEngine::loop_mode(const dsmc_params &p, const DevTables &t) {
    const int m = instance_mode(p, t);
    return m <= 2 ? m : 0;
}

namespace {

// Grows the served queue to `total` work items over `ninst` instances. Grabs made while the
// queue was empty pushed `next` past the old end without taking work (start_next returns on
// w >= total), so those indices are handed back first.
__global__ void publish_queue_kernel(FastCounters *c, unsigned long long old_total,
                                     unsigned long long total, long long ninst) {
    if (c->next > old_total) c->next = old_total;
    c->total = total;
    c->ninst = ninst;
}

}  // namespace

cudaError_t FastEngine::serve_append(const dsmc_params &p, const DevTables &t, long long n,
                                     int *index, cudaStream_t upload, cudaStream_t compute) {
    if (ninst_ >= ninst_cap_ || !d_stats_) return cudaErrorMemoryAllocation;
    if (p.ftd > 255 || p.ffd > 255 || p.hd > 32767 || n < 0 || n > (1ll << 32)) return cudaErrorInvalidValue;
    const size_t need = serve_table_floats(p, face_table_floats(p, t) ? t.nlevel : -1);
    const size_t base_need = static_cast<size_t>(p.hd + 1) + (p.ftd + 1) + 1 + 2 * static_cast<size_t>(p.ffd + 1);
    void *d_tab = nullptr;
    cudaError_t e = pool_ ? cudaMallocFromPoolAsync(&d_tab, need * sizeof(float), pool_, upload)
                          : cudaMallocAsync(&d_tab, need * sizeof(float), upload);
    if (e != cudaSuccess) return e;
    std::vector<float> tab(need, 0.0f);
    FastInst host;
    DevTables tt = t;
    tt.stats = d_stats_ + static_cast<size_t>(ninst_) * kStatCount;
    if ((e = fast_fill_instance(p, tt, 0, n, static_cast<float *>(d_tab), need, &host, tab.data())) != cudaSuccess) {
        cudaFreeAsync(d_tab, upload);
        return e;
    }
    host.work_base = static_cast<long long>(serve_total_);
    float4 *face = nullptr;
    if (face_table_floats(p, t)) {
        face = reinterpret_cast<float4 *>(static_cast<float *>(d_tab) + ((base_need + 3) & ~static_cast<size_t>(3)));
        host.face_f = face;
    }
    // The new descriptor lies beyond the instances the kernels in flight can see; it is written
    // on the upload stream while they run, and published on the compute stream after them.
    if ((e = cudaMemcpyAsync(d_tab, tab.data(), need * sizeof(float), cudaMemcpyHostToDevice, upload)) != cudaSuccess ||
        (e = cudaMemcpyAsync(d_inst_ + ninst_, &host, sizeof host, cudaMemcpyHostToDevice, upload)) != cudaSuccess ||
        (face && (e = build_face_tables(t, face, upload)) != cudaSuccess) ||
        (e = cudaStreamSynchronize(upload)) != cudaSuccess) {
        cudaFreeAsync(d_tab, upload);
        return e;
    }
    inst_tabs_[static_cast<size_t>(ninst_)] = d_tab;
    const unsigned long long old_total = serve_total_;
    serve_total_ += static_cast<unsigned long long>(n);
    publish_queue_kernel<<<1, 1, 0, compute>>>(d_ctr_, old_total, serve_total_, ninst_ + 1);
    if ((e = cudaGetLastError()) != cudaSuccess) {
        serve_total_ = old_total;
        return e;
    }
    *index = ninst_++;
    return cudaSuccess;
}

cudaError_t FastEngine::serve_launch(cudaStream_t stream, int mode) {
    if (launches_per_graph > 1) {
        const cudaError_t e = cudaGraphLaunch(graph_mode_[mode], stream);
        if (e == cudaSuccess) launches += launches_per_graph;
        return e;
    }
    launch_served(stream, mode);
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) launches += 1;
    return e;
}

void FastEngine::serve_release(int index, cudaStream_t stream) {
    if (index < 0 || index >= static_cast<int>(inst_tabs_.size())) return;
    if (inst_tabs_[static_cast<size_t>(index)]) cudaFreeAsync(inst_tabs_[static_cast<size_t>(index)], stream);
    inst_tabs_[static_cast<size_t>(index)] = nullptr;
}

void FastEngine::serve_close(cudaStream_t stream) {
    for (void *p : inst_tabs_)
        if (p) cudaFreeAsync(p, stream);
    inst_tabs_.clear();
}

size_t FastEngine::serve_table_floats(const dsmc_params &p, int nlevel) {
    // boundary tables, then (config model, icosphere of nlevel levels) the FP32 face tables
    const size_t base = static_cast<size_t>(p.hd + 1) + (p.ftd + 1) + 1 + 2 * static_cast<size_t>(p.ffd + 1);
    if (p.model != DSMC_MODEL_CONFIG || nlevel < 0) return base;
    return ((base + 3) & ~static_cast<size_t>(3)) + face_floats_for(nlevel);
}

size_t FastEngine::serve_fixed_bytes(int max_instances) const {
    return fast_slot_bytes(nslots_) + static_cast<size_t>(max_instances) * (sizeof(FastInst) + kStatCount * 8) +
           sizeof(FastCounters);
}

size_t fast_slot_bytes(long long nslots, bool fp64) {
    return static_cast<size_t>(nslots) * (fp64 ? slot_bytes_per_slot<double>() : slot_bytes_per_slot<float>()) + 256;
}

template <typename R>
SlotsT<R> carve_slots(void *mem, long long S) {
    char *b = static_cast<char *>(mem);
    auto take = [&](size_t each) { char *q = b; b += static_cast<size_t>(S) * each; return q; };
    constexpr size_t r = sizeof(R);
    SlotsT<R> s{};
    s.run_w = reinterpret_cast<R *>(take(8));
    s.inst = reinterpret_cast<int *>(take(4));
    s.pid = reinterpret_cast<unsigned *>(take(4));
    s.evt = reinterpret_cast<unsigned *>(take(4));
    s.sh = reinterpret_cast<R *>(take(3 * r));
    s.sl = reinterpret_cast<R *>(take(3 * r));
    s.vh = reinterpret_cast<R *>(take(3 * r));
    s.vl = reinterpret_cast<R *>(take(3 * r));
    s.oa = reinterpret_cast<R *>(take(3 * r));
    s.w0 = reinterpret_cast<R *>(take(r));
    s.nday = reinterpret_cast<int *>(take(4));
    s.steps = reinterpret_cast<int *>(take(4));
    s.hop = reinterpret_cast<int *>(take(4));
    s.cell = reinterpret_cast<int *>(take(4));
    s.run_cell = reinterpret_cast<int *>(take(4));
    s.hist_key = reinterpret_cast<int *>(take(4));
    s.hist_cnt = reinterpret_cast<int *>(take(4));
    s.pcol = reinterpret_cast<R *>(take(r));
    s.pthr = reinterpret_cast<R *>(take(r));
    s.ncol = reinterpret_cast<int *>(take(4));
    s.rest = reinterpret_cast<float *>(take(4));
    s.wcur = reinterpret_cast<R *>(take(r));
    s.face = reinterpret_cast<int *>(take(4));
    s.e0 = reinterpret_cast<float *>(take(4));
    return s;
}

template SlotsT<float> carve_slots<float>(void *, long long);
template SlotsT<double> carve_slots<double>(void *, long long);

size_t fast_inst_bytes() { return sizeof(FastInst); }

double fast_hop_steps(const dsmc_params &p) {
    const double g = p.GM / (p.Radii * p.Radii);
    const double v = std::sqrt(p.kB_over_m * 235.0);
    return g > 0.0 && p.dt_step > 0.0 ? 2.0 * v / (g * p.dt_step) : 1e30;
}

// Measured on B200 (particle-steps/s, gathering against the free-running loop): Moon-like
// (~200 steps per hop) 1.24e11 vs 8.2e10 at 16 lane-chunks, 1.17e11 at 4; Europa-like (~250)
// 1.31e11 vs 9.3e10; the reference model (dt 5 s, ~480) 6.8e10 at 4 vs 6.2e10 at 16; Ceres-like
// (~1160) and its collisional phase 2 are fastest free-running (gathering at 16 cost 5 %).
int gather_chunks(const dsmc_params &p) {
    const double hop = fast_hop_steps(p);
    return hop < 300.0 ? 16 : (hop < 600.0 ? 4 : 0);
}

size_t fast_counter_bytes() { return sizeof(FastCounters); }

cudaError_t fast_fill_instance(const dsmc_params &p, const DevTables &t, long long pid_begin,
                               long long n, float *d_tab, size_t tab_floats, void *inst_host,
                               float *tab_host) {
    const size_t need = static_cast<size_t>(p.hd + 1) + (p.ftd + 1) + 1 + 2 * (p.ffd + 1);
    if (need > tab_floats) return cudaErrorInvalidValue;
    const BoundaryLayout l = boundary_layout<float>(p);
    fill_boundaries(p, l, tab_host);
    FastInst &I = *static_cast<FastInst *>(inst_host);
    fill_inst(p, t, pid_begin, n, &I);
    I.rb2 = d_tab;
    I.sbs = d_tab + l.sbs;
    I.lonb = reinterpret_cast<const float2 *>(d_tab + l.lonb);
    return cudaSuccess;
}

cudaError_t fast_drain_external(const void *d_inst, void *slot_mem, long long nslots, void *d_ctr,
                                long long total, int steps_per_launch, int block,
                                long long stall_launches, cudaStream_t stream,
                                long long *launches) {
    *launches = 0;
    if (total <= 0) return cudaSuccess;
    if (nslots % block) return cudaErrorInvalidValue;
    const long long S = nslots;
    const Slots s = carve_slots<float>(slot_mem, S);
    cudaError_t e;
    FastCounters host{};
    host.total = static_cast<unsigned long long>(total);
    host.ninst = 1;
    if ((e = cudaMemcpyAsync(d_ctr, &host, sizeof host, cudaMemcpyHostToDevice, stream)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(s.inst, 0xff, S * sizeof(int), stream)) != cudaSuccess) return e;
    // the pageable source must stay valid until the copy has been made
    if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return e;
    FastArgsT<float> a{};
    a.inst_ = static_cast<const FastInst *>(d_inst);
    a.s = s;
    a.nslots = S;
    a.ctr = static_cast<FastCounters *>(d_ctr);
    a.K = steps_per_launch;
    const unsigned grid = static_cast<unsigned>(S / block);
    unsigned long long last = 0;
    long long stalled = 0;
    for (;;) {
        if (stalled > stall_launches) return cudaErrorLaunchTimeout;
        served_kernel(0, 0)<<<grid, block, 0, stream>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        *launches += 1;
        if ((e = cudaMemcpyAsync(&host, d_ctr, sizeof host, cudaMemcpyDeviceToHost, stream)) != cudaSuccess)
            return e;
        if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return e;
        if (host.finished >= static_cast<unsigned long long>(total)) return cudaSuccess;
        stalled = host.finished == last ? stalled + 1 : 0;
        last = host.finished;
    }
}

}  // namespace dsmc
