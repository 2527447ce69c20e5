// A CUDA runtime without a GPU, for tests of the library's host code: the objects of the library are
// linked with it in place of libcudart. Device memory is host memory (zeroed, within a limit that a
// test sets), copies and clears are made at once, and no kernel runs; a launch of a solve's step loop
// only counts, and the queue's counters read as finished after fake_finish_after of them. Streams
// keep which of their kernels the host, or another stream, has waited for: work issued on one stream
// while a kernel of another may still run counts as a race.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

struct CUstream_st { long long issued = 0; };
struct CUevent_st { CUstream_st *stream = nullptr; long long at = 0; };

namespace {
std::recursive_mutex mu;
std::map<char *, size_t> blocks;
size_t held = 0, limit = size_t(64) << 30;
long long allocs = 0, fail_at = -1, launches = 0, loops = 0, reads = 0, finish_after = 1, races = 0, device_syncs = 0,
          lowered = 0;
bool capturing = false;   // some stream of the process is being captured, by another thread
std::map<CUstream_st *, long long> waited;   // of every stream's kernels, those known to have ended
std::map<const void *, std::string> kernels;
std::map<const void *, int> smem_limit;
struct Config { dim3 g, b; size_t smem; cudaStream_t s; };
thread_local Config pushed;

using Lock = std::lock_guard<std::recursive_mutex>;

void ended(CUstream_st *s, long long at) {
    if (waited[s] < at) waited[s] = at;
}
void all_ended() {
    for (auto &w : waited) w.second = w.first->issued;
}
void touch(CUstream_st *s) {   // new work on s: kernels of other streams may still run
    for (auto &w : waited)
        if (w.first != s && w.first->issued > w.second) races++;
}
cudaError_t give(void **p, size_t n) {
    Lock l(mu);
    if (allocs++ == fail_at || held + n > limit) return cudaErrorMemoryAllocation;
    char *q = static_cast<char *>(std::calloc(n ? n : 1, 1));
    if (!q) return cudaErrorMemoryAllocation;
    blocks[q] = n;
    held += n;
    *p = q;
    return cudaSuccess;
}
cudaError_t take(void *p) {
    Lock l(mu);
    if (!p) return cudaSuccess;
    auto b = blocks.find(static_cast<char *>(p));
    if (b == blocks.end()) return cudaErrorInvalidValue;
    held -= b->second;
    blocks.erase(b);
    std::free(p);
    return cudaSuccess;
}
bool on_device(const void *p, size_t n) {
    auto b = blocks.upper_bound(static_cast<char *>(const_cast<void *>(p)));
    if (b == blocks.begin()) return false;
    --b;
    return static_cast<const char *>(p) + n <= b->first + b->second;
}
}  // namespace

extern "C" {

// what a test sets and reads
void fake_reset() {
    Lock l(mu);
    limit = size_t(64) << 30;
    allocs = launches = loops = reads = races = device_syncs = lowered = 0;
    fail_at = -1;
    finish_after = 1;
    capturing = false;
    smem_limit.clear();
    all_ended();
}
void fake_limit(size_t bytes) { limit = bytes; }
void fake_fail_at(long long k) { allocs = 0; fail_at = k; }
void fake_finish_after(long long k) { loops = 0; finish_after = k; }
void fake_capturing(int on) { capturing = on != 0; }
size_t fake_held() { return held; }
long long fake_allocs() { return allocs; }
long long fake_loops() { return loops; }
long long fake_reads() { return reads; }
long long fake_races() { return races; }
long long fake_device_syncs() { return device_syncs; }
long long fake_lowered() { return lowered; }
void *fake_stream() { cudaStream_t s; cudaStreamCreateWithFlags(&s, 0); return s; }

cudaError_t cudaMalloc(void **p, size_t n) { return give(p, n); }
cudaError_t cudaFree(void *p) { Lock l(mu); all_ended(); return take(p); }   // waits for the device
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return give(p, n); }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { return give(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return take(p); }
cudaError_t cudaMallocHost(void **p, size_t n) { return (*p = std::calloc(n, 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *, const cudaMemPoolProps *) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaErrorNotSupported; }

cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) {
    Lock l(mu);
    if (!on_device(p, n)) return cudaErrorInvalidValue;
    touch(s);
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *q, size_t n, cudaMemcpyKind kind, cudaStream_t s) {
    Lock l(mu);
    const bool to = kind == cudaMemcpyHostToDevice || kind == cudaMemcpyDeviceToDevice;
    if (to ? !on_device(d, n) : !on_device(q, n)) return cudaErrorInvalidValue;
    touch(s);
    std::memcpy(d, q, n);
    if (kind == cudaMemcpyDeviceToHost && n == 5 * 8) {   // the queue: next, finished, total, ...
        unsigned long long *c = static_cast<unsigned long long *>(d);
        reads++;
        c[0] = c[2];
        c[1] = loops >= finish_after ? c[2] : 0;
    }
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorNotSupported; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { Lock l(mu); *s = new CUstream_st; waited[*s] = 0; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { Lock l(mu); waited.erase(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { Lock l(mu); ended(s, s->issued); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {
    Lock l(mu);
    device_syncs++;
    if (capturing) return cudaErrorStreamCaptureUnsupported;
    all_ended();
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t e, unsigned) { Lock l(mu); if (e->stream) ended(e->stream, e->at); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = new CUevent_st; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { Lock l(mu); e->stream = s; e->at = s->issued; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { Lock l(mu); if (e->stream && waited.count(e->stream)) ended(e->stream, e->at); return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) {
    Lock l(mu);
    return !e->stream || !waited.count(e->stream) || waited[e->stream] >= e->at ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error"; }

cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { *n = 5; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
    Lock l(mu);
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
    if (smem_limit.count(f) && v < smem_limit[f]) lowered++;
    smem_limit[f] = v;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t smem, cudaStream_t s) {
    Lock l(mu);
    if (smem > 49152 && smem > static_cast<size_t>(smem_limit[f])) return cudaErrorInvalidValue;
    touch(s);
    s->issued++;
    launches++;
    const std::string &name = kernels[f];
    if (name.find("fast_kernel") != std::string::npos || name.find("warp_kernel") != std::string::npos) loops++;
    return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) { pushed = {g, b, smem, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
    *g = pushed.g;
    *b = pushed.b;
    *smem = pushed.smem;
    *static_cast<cudaStream_t *>(s) = pushed.s;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *) {
    Lock l(mu);
    kernels[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

}  // extern "C"
