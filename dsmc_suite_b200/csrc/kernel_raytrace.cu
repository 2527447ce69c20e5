// kernel_raytrace.cu - Monte Carlo shadow flux of a body mesh on the GPU (the reference's
// src/raytracer/shadow_maker.c:198-238, which traces with Intel Embree on the CPU).
//
// For rotation phase t and face f: the sun direction s(t) = (cos(-za) sin(phi), cos(-za) cos(phi),
// sin(-za)) with phi = 2 pi (t + 1/2) / tt + pi; faces turned away (s . n < 0) get 0; otherwise
// Nmonte points of the face are drawn with rand_r from the seed t * nface + f + 42 (the
// reference's sequence), each lifted 1e-3 along the face normal and tested for any hit along s,
// and the face gets (1 - shadowed / Nmonte) (s . n).
//
// GPU design: one warp per (phase, face), its lanes the face's sample rays. The rays of a face start
// in one small box and share the direction, so the warp walks the BVH once for all of them: a slab
// test on the interval of origins (the per-ray test with each bound taken at its worst origin; the
// float operations are monotone, so a leaf that any ray of the face enters passes) lists the
// leaves they can enter, about 6 of a cratered sphere's. The rays then test the listed leaves
// together, each with the test of its own: which triangles a ray is tested against, and so every
// count, is that of a walk per ray. Such a walk took 2,820 instructions a ray at 5 of 32 lanes
// (11.8 ms for 20,480 faces x 24 phases x 50 samples on one thread per face). The lanes enter the
// face's random sequence at their own sample by jumping the linear congruential generator ahead.
// The BVH is built on the host (binned surface-area heuristic, at most 4 triangles per leaf,
// median splits below depth 40 so that every path fits the 64-entry traversal stack) and walked
// for any hit; triangles are stored as (v0, e1, e2) float4 triples for the Moller-Trumbore test.
// Compiled with -fmad=false so that the sample points and the flux factor follow the reference's
// FP64 operation order; the ray itself is FP32 like Embree's.
#include "dsmc_kernels.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <exception>
#include <thread>
#include <vector>

namespace dsmc {
namespace {

struct BvhNode {
    float lo[3];
    int first;      // inner node: index of the left child (right = first + 1); leaf: first triangle
    float hi[3];
    int count;      // 0 = inner node, else triangles in the leaf
};

constexpr int kLeaf = 4;
constexpr int kStack = 64;
constexpr int kMedianDepth = 40;

struct alignas(16) Box4 {   // bounds of three axes; the fourth lane makes the loops one vector wide
    float lo[4], hi[4];
    void clear() { for (int a = 0; a < 4; a++) { lo[a] = 1e38f; hi[a] = -1e38f; } }
    void add(const Box4 &b) {
        for (int a = 0; a < 4; a++) lo[a] = b.lo[a] < lo[a] ? b.lo[a] : lo[a];
        for (int a = 0; a < 4; a++) hi[a] = b.hi[a] > hi[a] ? b.hi[a] : hi[a];
    }
    void add_point(const float *p) {
        for (int a = 0; a < 4; a++) lo[a] = p[a] < lo[a] ? p[a] : lo[a];
        for (int a = 0; a < 4; a++) hi[a] = p[a] > hi[a] ? p[a] : hi[a];
    }
    float area() const {
        const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
        return dx < 0 ? 0.0f : 2.0f * (dx * dy + dy * dz + dz * dx);
    }
};
struct alignas(16) Tri {
    Box4 box;
    float cen[4];
    int id, bin;
};

// Same tree as one built triangle by triangle through an index list; the triangles themselves move,
// so every pass over a node reads memory in order, and the twelve bins are swept once from each
// side. Subtrees of the first levels go to threads of their own (disjoint ranges and nodes).
// 20,480 faces: 1.7 ms against 7.5 ms (and 3.4 ms on one thread).
struct Builder {
    std::vector<Tri> tri;
    std::vector<BvhNode> nodes;
    std::atomic<int> used{0};      // nodes handed out
    Builder(const std::vector<float> &V, const int *F, int n) : tri(n) {
        for (int k = 0; k < n; k++) {
            Tri &t = tri[k];
            t.id = k;
            t.box.clear();
            for (int a = 0; a < 3; a++) {
                for (int j = 0; j < 3; j++) {
                    const float x = V[3 * static_cast<size_t>(F[3 * k + j]) + a];
                    t.box.lo[a] = std::min(t.box.lo[a], x);
                    t.box.hi[a] = std::max(t.box.hi[a], x);
                }
                t.cen[a] = 0.5f * (t.box.lo[a] + t.box.hi[a]);
            }
            t.cen[3] = 0.0f;
        }
    }
    void build() {
        const int nface = static_cast<int>(tri.size());
        nodes.assign(2 * tri.size() + 1, BvhNode{});
        used = 1;
        split(0, 0, nface, 0);
        nodes.resize(static_cast<size_t>(used.load()));
    }
    void split(int node, int b, int e, int depth) {
        Box4 box, cb;   // of the triangles and of their centroids
        box.clear();
        cb.clear();
        for (int k = b; k < e; k++) {
            box.add(tri[k].box);
            cb.add_point(tri[k].cen);
        }
        for (int a = 0; a < 3; a++) { nodes[node].lo[a] = box.lo[a]; nodes[node].hi[a] = box.hi[a]; }
        if (e - b <= kLeaf) { nodes[node].first = b; nodes[node].count = e - b; return; }
        int axis = 0;
        for (int a = 1; a < 3; a++)
            if (cb.hi[a] - cb.lo[a] > cb.hi[axis] - cb.lo[axis]) axis = a;
        const float ext = cb.hi[axis] - cb.lo[axis], start = cb.lo[axis];
        if (!(ext > 0.0f)) { nodes[node].first = b; nodes[node].count = e - b; return; }   // coincident
        int mid = -1;
        if (depth < kMedianDepth) {
            constexpr int kBins = 12;
            int cnt[kBins] = {0};
            Box4 bb[kBins];
            for (auto &x : bb) x.clear();
            for (int k = b; k < e; k++) {
                const int i = std::min(std::max(static_cast<int>((tri[k].cen[axis] - start) / ext * kBins), 0), kBins - 1);
                tri[k].bin = i;
                cnt[i]++;
                bb[i].add(tri[k].box);
            }
            // triangles and areas on the two sides of every cut
            float al[kBins], ar[kBins];
            int nl[kBins], nr[kBins];
            Box4 side;
            side.clear();
            for (int s = 1, c = 0; s < kBins; s++) {
                side.add(bb[s - 1]);
                nl[s] = c += cnt[s - 1];
                al[s] = side.area();
            }
            side.clear();
            for (int s = kBins - 1, c = 0; s > 0; s--) {
                side.add(bb[s]);
                nr[s] = c += cnt[s];
                ar[s] = side.area();
            }
            float best = 1e38f;
            int best_i = -1;
            for (int s = 1; s < kBins; s++) {
                if (!nl[s] || !nr[s]) continue;
                const float cost = nl[s] * al[s] + nr[s] * ar[s];
                if (cost < best) { best = cost; best_i = s; }
            }
            if (best_i > 0) {
                Tri *p = std::partition(tri.data() + b, tri.data() + e, [&](const Tri &t) { return t.bin < best_i; });
                mid = static_cast<int>(p - tri.data());
            }
        }
        if (mid <= b || mid >= e) {   // median split along the axis
            mid = (b + e) / 2;
            std::nth_element(tri.data() + b, tri.data() + mid, tri.data() + e,
                             [&](const Tri &x, const Tri &y) { return x.cen[axis] < y.cen[axis]; });
        }
        const int left = used.fetch_add(2);
        nodes[node].first = left;
        nodes[node].count = 0;
        if (depth < 3 && e - b > 2000) {
            std::thread t;
            try {
                t = std::thread([&] { split(left, b, mid, depth + 1); });
            } catch (const std::exception &) {   // none to be had: this one builds both
                split(left, b, mid, depth + 1);
            }
            split(left + 1, mid, e, depth + 1);
            if (t.joinable()) t.join();
        } else {
            split(left, b, mid, depth + 1);
            split(left + 1, mid, e, depth + 1);
        }
    }
};

// glibc's rand_r: three steps of the ANSI C linear congruential generator, 11 + 10 + 10 bits.
__device__ __forceinline__ int rand_r_dev(unsigned int *seed) {
    unsigned int next = *seed;
    next = next * 1103515245u + 12345u;
    int result = static_cast<int>((next / 65536u) % 2048u);
    next = next * 1103515245u + 12345u;
    result = (result << 10) ^ static_cast<int>((next / 65536u) % 1024u);
    next = next * 1103515245u + 12345u;
    result = (result << 10) ^ static_cast<int>((next / 65536u) % 1024u);
    *seed = next;
    return result;
}

// State of rand_r's generator after `steps` steps from `seed` (x <- a x + c mod 2^32), by
// squaring the step.
__device__ __forceinline__ unsigned int lcg_jump(unsigned int seed, unsigned int steps) {
    unsigned int a = 1103515245u, c = 12345u, A = 1u, C = 0u;
    for (; steps; steps >>= 1) {
        if (steps & 1u) {
            A *= a;
            C = C * a + c;
        }
        c *= a + 1u;
        a *= a;
    }
    return A * seed + C;
}
constexpr unsigned int kStepsPerSample = 6;   // two rand_r calls of three steps

struct ShadowArgs {
    const BvhNode *nodes;
    const float4 *tris;     // [ntri][3]: v0, e1 = v1 - v0, e2 = v2 - v0 (BVH order)
    int nnodes;
    const int *facet;       // [nface][3], 0-based
    const double *spot;     // [npoint][3]
    const double *normal;   // [nface][3]
    int nface, tt, nmonte;
    double za;
    double *F;              // [nface][tt]
    int *overflow;          // traversal stack overflows (0 by construction of the tree)
};

__device__ bool slab(const BvhNode &n, const float o[3], const float inv[3], float tmax) {
    float t0 = 0.0f, t1 = tmax;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        float ta = (n.lo[a] - o[a]) * inv[a], tb = (n.hi[a] - o[a]) * inv[a];
        if (ta > tb) { const float x = ta; ta = tb; tb = x; }
        t0 = fmaxf(t0, ta);
        t1 = fminf(t1, tb);
    }
    return t0 <= t1;
}

// Moller-Trumbore with the ray parameter in [0, tmax] (Embree's tnear = 0, tfar = 1e30).
__device__ bool hit_triangle(const float4 *t, const float o[3], const float d[3], float tmax) {
    const float4 v0 = t[0], e1 = t[1], e2 = t[2];
    const float px = d[1] * e2.z - d[2] * e2.y, py = d[2] * e2.x - d[0] * e2.z, pz = d[0] * e2.y - d[1] * e2.x;
    const float det = e1.x * px + e1.y * py + e1.z * pz;
    if (det == 0.0f) return false;
    const float inv = 1.0f / det;
    const float sx = o[0] - v0.x, sy = o[1] - v0.y, sz = o[2] - v0.z;
    const float u = (sx * px + sy * py + sz * pz) * inv;
    if (u < 0.0f || u > 1.0f) return false;
    const float qx = sy * e1.z - sz * e1.y, qy = sz * e1.x - sx * e1.z, qz = sx * e1.y - sy * e1.x;
    const float v = (d[0] * qx + d[1] * qy + d[2] * qz) * inv;
    if (v < 0.0f || u + v > 1.0f) return false;
    const float tt = (e2.x * qx + e2.y * qy + e2.z * qz) * inv;
    return tt >= 0.0f && tt <= tmax;
}

__device__ bool occluded(const ShadowArgs &a, const float o[3], const float d[3]) {
    const float tmax = 1e30f;
    float inv[3];
#pragma unroll
    for (int k = 0; k < 3; k++) inv[k] = 1.0f / (d[k] != 0.0f ? d[k] : 1e-30f);
    int stack[kStack];
    int sp = 0, n = 0;
    for (int it = 0; it < 2 * a.nnodes + 2; it++) {
        const BvhNode nd = a.nodes[n];
        bool descend = false;
        if (slab(nd, o, inv, tmax)) {
            if (nd.count > 0) {
                for (int k = nd.first; k < nd.first + nd.count; k++)
                    if (hit_triangle(a.tris + 3 * k, o, d, tmax)) return true;
            } else if (sp < kStack) {
                stack[sp++] = nd.first + 1;
                n = nd.first;
                descend = true;
            } else {
                atomicAdd(a.overflow, 1);
            }
        }
        if (!descend) {
            if (sp == 0) return false;
            n = stack[--sp];
        }
    }
    return false;
}

// Whether any ray along d from an origin in [olo, ohi] passes slab(): the bounds of slab's interval,
// each taken at the origin that stretches it most.
__device__ bool slab_any(const BvhNode &n, const float olo[3], const float ohi[3], const float inv[3], float tmax) {
    float t0 = 0.0f, t1 = tmax;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const bool up = inv[a] >= 0.0f;
        t0 = fmaxf(t0, up ? (n.lo[a] - ohi[a]) * inv[a] : (n.hi[a] - olo[a]) * inv[a]);
        t1 = fminf(t1, up ? (n.hi[a] - olo[a]) * inv[a] : (n.lo[a] - ohi[a]) * inv[a]);
    }
    return t0 <= t1;
}

constexpr int kWarps = 8;          // warps per block
constexpr int kFacesPerWarp = 8;   // consecutive faces a warp works off
constexpr int kLeaves = 192;       // listed leaves per warp; a face with more walks ray by ray

__global__ void __launch_bounds__(32 * kWarps) shadow_kernel(const ShadowArgs a) {
    __shared__ double sun_of_phase[3];
    __shared__ int leaf_list[kWarps][kLeaves];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr unsigned kAll = 0xffffffffu;
    constexpr double kPi = 3.14159265358979323846;
    const long long groups = (a.nface + kWarps * kFacesPerWarp - 1) / (kWarps * kFacesPerWarp);
    for (long long g = blockIdx.x; g < groups * a.tt; g += gridDim.x) {
    const int t = static_cast<int>(g / groups);
    __syncthreads();
    if (threadIdx.x == 0) {
        const double fi = ((t + 0.5) / a.tt) * 2.0 * kPi + kPi;
        sun_of_phase[0] = cos(-a.za) * sin(fi);
        sun_of_phase[1] = cos(-a.za) * cos(fi);
        sun_of_phase[2] = sin(-a.za);
    }
    __syncthreads();
    const double sun[3] = {sun_of_phase[0], sun_of_phase[1], sun_of_phase[2]};
    const float d[3] = {static_cast<float>(sun[0]), static_cast<float>(sun[1]), static_cast<float>(sun[2])};
    const float tmax = 1e30f;
    float inv[3];
#pragma unroll
    for (int k = 0; k < 3; k++) inv[k] = 1.0f / (d[k] != 0.0f ? d[k] : 1e-30f);
    const double eps = static_cast<double>(1e-3f);   // the reference's float offset, promoted
    int *list = leaf_list[warp];
    const long long first = ((g % groups) * kWarps + warp) * kFacesPerWarp;
    for (int j = 0; j < kFacesPerWarp && first + j < a.nface; j++) {
        const int nf = static_cast<int>(first + j);
        const double *fn = a.normal + 3 * nf;
        const double c6 = sun[0] * fn[0] + sun[1] * fn[1] + sun[2] * fn[2];
        double *out = a.F + static_cast<long long>(nf) * a.tt + t;
        if (c6 < 0) {
            if (lane == 0) *out = 0.0;
            continue;
        }
        const double *A = a.spot + 3 * a.facet[3 * nf], *B = a.spot + 3 * a.facet[3 * nf + 1],
                     *C = a.spot + 3 * a.facet[3 * nf + 2];
        // box of the sample origins: a point of the face, lifted, rounded to float; the margin
        // covers the rounding of the barycentric sum
        float olo[3], ohi[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double lo = fmin(A[k], fmin(B[k], C[k])), hi = fmax(A[k], fmax(B[k], C[k]));
            const double up = eps * fn[k], m = 1e-12 * (fmax(fabs(lo), fabs(hi)) + fabs(up));
            olo[k] = __double2float_rd(lo + up - m);
            ohi[k] = __double2float_ru(hi + up + m);
        }
        // the leaves that a ray of this face can enter (every lane walks the same nodes)
        int stack[kStack];
        int sp = 0, n = 0, found = 0;
        for (int it = 0; it < 2 * a.nnodes + 2; it++) {
            const BvhNode nd = a.nodes[n];
            bool descend = false;
            if (slab_any(nd, olo, ohi, inv, tmax)) {
                if (nd.count > 0) {
                    if (found < kLeaves && lane == 0) list[found] = n;
                    found++;
                } else if (sp < kStack) {
                    stack[sp++] = nd.first + 1;
                    n = nd.first;
                    descend = true;
                } else if (lane == 0) {
                    atomicAdd(a.overflow, 1);
                }
            }
            if (!descend) {
                if (sp == 0) break;
                n = stack[--sp];
            }
        }
        __syncwarp();
        int shadowed = 0;
        for (unsigned int base = 0; base < static_cast<unsigned int>(a.nmonte); base += 32) {
            const unsigned int mc = base + lane;
            const bool mine = mc < static_cast<unsigned int>(a.nmonte);
            unsigned int seed = lcg_jump(static_cast<unsigned int>(t * a.nface + nf + 42),
                                         kStepsPerSample * mc);
            const double r1 = sqrt(static_cast<double>(rand_r_dev(&seed)) / 2147483647.0);
            const double r2 = static_cast<double>(rand_r_dev(&seed)) / 2147483647.0;
            const double wa = 1.0 - r1, wb = r1 * (1.0 - r2), wc = r1 * r2;
            float o[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double p = A[k] * wa + B[k] * wb + C[k] * wc;
                o[k] = static_cast<float>(p + eps * fn[k]);
            }
            bool hit = false;
            if (found <= kLeaves) {
                for (int l = 0; l < found && __any_sync(kAll, mine && !hit); l++) {
                    const BvhNode nd = a.nodes[list[l]];
                    if (mine && !hit && slab(nd, o, inv, tmax))
                        for (int k = nd.first; k < nd.first + nd.count && !hit; k++)
                            hit = hit_triangle(a.tris + 3 * k, o, d, tmax);
                    __syncwarp();
                }
            } else if (mine) {
                hit = occluded(a, o, d);
            }
            shadowed += __popc(__ballot_sync(kAll, mine && hit));
        }
        if (lane == 0) *out = (1.0 - static_cast<double>(shadowed) / a.nmonte) * c6;
        __syncwarp();
    }
    }
}

}  // namespace

cudaError_t shadow_flux(int npoint, const double *spot, int nface, const int *facet,
                        const double *normal, double za, int tt, int nmonte, double *F_host,
                        const std::function<void *(size_t)> &scratch, cudaStream_t stream,
                        long long *overflows, double *kernel_ms) {
    std::vector<float> V(3 * static_cast<size_t>(npoint));
    for (size_t k = 0; k < V.size(); k++) V[k] = static_cast<float>(spot[k]);
    Builder bld(V, facet, nface);
    bld.build();
    std::vector<float4> tris(3 * static_cast<size_t>(nface));
    for (int k = 0; k < nface; k++) {
        const int f = bld.tri[k].id;
        const float *v0 = &V[3 * static_cast<size_t>(facet[3 * f])], *v1 = &V[3 * static_cast<size_t>(facet[3 * f + 1])],
                    *v2 = &V[3 * static_cast<size_t>(facet[3 * f + 2])];
        tris[3 * k + 0] = make_float4(v0[0], v0[1], v0[2], 0.0f);
        tris[3 * k + 1] = make_float4(v1[0] - v0[0], v1[1] - v0[1], v1[2] - v0[2], 0.0f);
        tris[3 * k + 2] = make_float4(v2[0] - v0[0], v2[1] - v0[1], v2[2] - v0[2], 0.0f);
    }
    const size_t nn = bld.nodes.size(), nfc = static_cast<size_t>(nface), np = static_cast<size_t>(npoint);
    const size_t nF = nfc * static_cast<size_t>(tt);
    // one block from the caller: nodes, triangles, faces, vertices, normals, F, overflow count
    const size_t sizes[7] = {nn * sizeof(BvhNode), tris.size() * sizeof(float4), nfc * 3 * sizeof(int),
                             np * 3 * sizeof(double), nfc * 3 * sizeof(double), nF * sizeof(double), sizeof(int)};
    struct { void *p[7]; } b;
    size_t at[7], total = 0;
    for (int k = 0; k < 7; k++) {
        at[k] = total;
        total += (sizes[k] + 255) & ~size_t(255);
    }
    void *block = scratch(total);
    if (!block) return cudaErrorMemoryAllocation;
    for (int k = 0; k < 7; k++) b.p[k] = static_cast<char *>(block) + at[k];
    cudaError_t e;
    if ((e = cudaMemcpyAsync(b.p[0], bld.nodes.data(), nn * sizeof(BvhNode), cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(b.p[1], tris.data(), tris.size() * sizeof(float4), cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(b.p[2], facet, nfc * 3 * sizeof(int), cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(b.p[3], spot, np * 3 * sizeof(double), cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(b.p[4], normal, nfc * 3 * sizeof(double), cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
        (e = cudaMemsetAsync(b.p[6], 0, sizeof(int), stream)) != cudaSuccess)
        return e;
    ShadowArgs a{};
    a.nodes = static_cast<const BvhNode *>(b.p[0]);
    a.tris = static_cast<const float4 *>(b.p[1]);
    a.nnodes = static_cast<int>(nn);
    a.facet = static_cast<const int *>(b.p[2]);
    a.spot = static_cast<const double *>(b.p[3]);
    a.normal = static_cast<const double *>(b.p[4]);
    a.nface = nface;
    a.tt = tt;
    a.nmonte = nmonte;
    a.za = za;
    a.F = static_cast<double *>(b.p[5]);
    a.overflow = static_cast<int *>(b.p[6]);
    const int faces = kWarps * kFacesPerWarp;
    struct Events {
        cudaEvent_t e[2] = {nullptr, nullptr};
        ~Events() { for (cudaEvent_t x : e) if (x) cudaEventDestroy(x); }
    } ev;
    if ((e = cudaEventCreate(&ev.e[0])) != cudaSuccess || (e = cudaEventCreate(&ev.e[1])) != cudaSuccess ||
        (e = cudaEventRecord(ev.e[0], stream)) != cudaSuccess)
        return e;
    const long long blocks = std::min((nface + faces - 1ll) / faces * tt, 1ll << 30);
    shadow_kernel<<<static_cast<unsigned>(blocks), 32 * kWarps, 0, stream>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = cudaEventRecord(ev.e[1], stream)) != cudaSuccess) return e;
    int ovf = 0;
    if ((e = cudaMemcpyAsync(F_host, b.p[5], nF * sizeof(double), cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(&ovf, b.p[6], sizeof(int), cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(stream)) != cudaSuccess)
        return e;
    if (overflows) *overflows = ovf;
    float ms = 0.f;
    if (kernel_ms && cudaEventElapsedTime(&ms, ev.e[0], ev.e[1]) == cudaSuccess) *kernel_ms = ms;
    return cudaSuccess;
}

}  // namespace dsmc
