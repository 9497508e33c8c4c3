// A CUDA runtime of host memory under the library's own host code: the entry
// points that hk_host.cpp, hk_engine.cpp and hk_server.cpp call, and in place of
// the kernels' launchers a log of what would have been launched.  It lets the
// host's decisions (form, pool, launches, streams, devices, captures, memory)
// be tested without a GPU.  Not a simulation: nothing is rendered.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

#include "hk_kernels.h"
#include "hk_lbvh.h"
#include "hk_wavefront.h"

namespace {
struct Stream { int device, priority; };
struct Event { int device; };
struct Exec { bool loop; hk::WfState W; };
struct Fake {
    std::recursive_mutex mu;
    int device = 0;
    size_t limit = SIZE_MAX, live = 0;
    std::map<void *, size_t> blocks;
    bool other_capture = false, broken = false;   // a capture of another thread in the default (global) mode
    int capturing_user = 0;                       // what cudaStreamIsCapturing says of the caller's streams
    bool in_capture = false;                      // the library's own
    hk::WfState W{};                              // of the last captured iteration
    uint64_t passes_left = 0;                     // passes that the render begun last needs in the worst case
    int fail_instantiate = 0, pinned = 0;
    std::string log;
} g;
thread_local cudaStreamCaptureMode t_mode = cudaStreamCaptureModeGlobal;
thread_local cudaError_t t_last = cudaSuccess;

void note(const std::string &s) {
    std::lock_guard<std::recursive_mutex> lk(g.mu);
    g.log += s + "\n";
}
int device_of(cudaStream_t s) { return s ? ((Stream *)s)->device : g.device; }
cudaError_t fail(cudaError_t e) { return t_last = e; }
// calls that a capture in global mode forbids to every thread that has not relaxed its own mode
bool unsafe() {
    if (!g.other_capture || t_mode == cudaStreamCaptureModeRelaxed) return false;
    g.broken = true;
    return true;
}
void finish(const hk::WfState &W) {
    W.ctr->next_work = W.ctr->total_work;
    W.ctr->active = 0;
    for (unsigned k = 0; k < W.ctr->seg_count; ++k) {   // the plan's jobs
        const hk::WfJob &J = W.jobs[W.segs[k].job];
        *J.finished = J.work_count;
    }
}
}  // namespace

#define LOCK std::lock_guard<std::recursive_mutex> lk(g.mu)
extern "C" {
// ---- what the tests set and read
const char *fake_log() { return g.log.c_str(); }
void fake_clear() { LOCK; g.log.clear(); }
void fake_limit(size_t n) { g.limit = n; }
size_t fake_live() { return g.live; }
void fake_device(int d) { g.device = d; }
void fake_other_capture(int on) { g.other_capture = on != 0; g.broken = false; }
int fake_capture_broken() { return g.broken; }
void fake_user_capturing(int on) { g.capturing_user = on; }
void fake_fail_instantiate(int on) { g.fail_instantiate = on; }
int fake_pinned() { return g.pinned; }
uint64_t fake_passes_left() { return g.passes_left; }
void *fake_stream(int device, int priority) { return new Stream{device, priority}; }

// ---- the runtime
cudaError_t cudaGetLastError() { cudaError_t e = t_last; t_last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int *d) { *d = g.device; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return unsafe() ? fail(cudaErrorStreamCaptureUnsupported) : cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *least, int *greatest) { *least = 0; *greatest = -5; return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m) { std::swap(*m, t_mode); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)180 << 30; return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) {
    LOCK;
    if (unsafe()) return fail(cudaErrorStreamCaptureUnsupported);
    if (g.live + n > g.limit) { note("malloc-failed"); return fail(cudaErrorMemoryAllocation); }
    *p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    g.blocks[*p] = n;
    g.live += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    LOCK;
    if (unsafe()) return fail(cudaErrorStreamCaptureUnsupported);
    auto it = g.blocks.find(p);
    if (it == g.blocks.end()) return fail(cudaErrorInvalidValue);
    munmap(p, it->second);
    g.live -= it->second;
    g.blocks.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMallocHost(void **p, size_t n) {
    if (unsafe()) return fail(cudaErrorStreamCaptureUnsupported);
    *p = calloc(1, n);
    ++g.pinned;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t) new Stream{g.device, 0}; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int p) { *s = (cudaStream_t) new Stream{g.device, p}; return cudaSuccess; }
cudaError_t cudaStreamGetPriority(cudaStream_t s, int *p) { *p = s ? ((Stream *)s)->priority : 0; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete (Stream *)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return unsafe() ? fail(cudaErrorStreamCaptureUnsupported) : cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
    *st = g.capturing_user ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t) new Event{g.device}; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (Event *)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    return ((Event *)e)->device == device_of(s) ? cudaSuccess : fail(cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { g.in_capture = true; return cudaSuccess; }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *, size_t,
                                          cudaStreamCaptureMode) {
    g.in_capture = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *gr) {
    g.in_capture = false;
    *gr = (cudaGraph_t)&g;
    return cudaSuccess;
}
cudaError_t cudaGraphCreate(cudaGraph_t *gr, unsigned) { *gr = (cudaGraph_t)&g; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned, unsigned) { *h = 1; return cudaSuccess; }
cudaError_t cudaGraphAddNode(cudaGraphNode_t *, cudaGraph_t, const cudaGraphNode_t *, size_t, cudaGraphNodeParams *np) {
    static cudaGraph_t body[1];
    np->conditional.phGraph_out = body;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    if (g.fail_instantiate) return fail(cudaErrorMemoryAllocation);
    *e = (cudaGraphExec_t) new Exec{g.W.cond != 0, g.W};
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete (Exec *)e; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
    LOCK;
    const Exec &e = *(Exec *)x;
    note((e.loop ? "loop priority " : "pair priority ") + std::to_string(((Stream *)s)->priority) + " device " +
         std::to_string(((Stream *)s)->device) + " capacity " + std::to_string(e.W.capacity));
    g.passes_left -= std::min<uint64_t>(g.passes_left, e.loop ? hk::kWfMaxLoops : 1);
    if (g.passes_left == 0) finish(e.W);
    return cudaSuccess;
}
}  // extern "C"

// ---- the kernels' launchers
namespace hk {
cudaError_t static_render_scratch(void **out) {
    static std::vector<unsigned long long> s(kStaticScratchWords);
    *out = s.data();
    return cudaSuccess;
}
cudaError_t launch_render(const DevScene &, const RenderLaunch &P, int grid, cudaStream_t) {
    note("mega grid " + std::to_string(grid) + " lanes " + std::to_string(P.lanes));
    return cudaSuccess;
}
cudaError_t launch_resolve(const float *, float *, int, int, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_trace(const DevScene &, uint64_t, const float *, int32_t *, float *, float *, float *, int, unsigned long long *,
                         cudaStream_t) { return cudaSuccess; }
cudaError_t launch_bsdf_batch(const DevScene &, int, int, uint64_t, const float *, const float *, const float *, const float *,
                              const float *, const float *, float *, float *, float *, int32_t *, float *, float *, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launch_texture_eval(const DevScene &, const DevTexture *, int, uint64_t, const float *, const float *, float *,
                                cudaStream_t) { return cudaSuccess; }
cudaError_t launch_emitter_sample(const DevScene &, int, uint64_t, const float *, float *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_camera_rays(const DevScene &, uint64_t, const float *, float *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_env_eval(const DevScene &, uint64_t, const float *, float *, float *, cudaStream_t) { return cudaSuccess; }
int render_occupancy(int, bool) { return kRenderBlocks; }
void build_bvh8_gpu(const float *, uint32_t, cudaStream_t, GpuBvh8 &) { throw HkError{HK_ERR_CUDA, "no device"}; }
void gather_tri_records(const float *, const int32_t *, const uint32_t *, uint32_t, float *, cudaStream_t) {}

cudaError_t wf_launch_init(const WfState &W, int slots, const WfJob &J, cudaStream_t) {
    W.ctr->active = 0;
    if (J.work_count > 0) {
        W.ctr->next_work = 0;
        W.ctr->total_work = J.work_count;
        // every slot's paths one after another, each to its depth, two vertices a pass
        g.passes_left = ((J.work_count + slots - 1) / slots * (uint64_t)J.depth + J.depth) / 2 + 1;
        note("begin slots " + std::to_string(slots) + " sample " + std::to_string((int64_t)J.sample_offset) + " image " +
             std::to_string((int64_t)J.image_index));
    }
    return cudaSuccess;
}
cudaError_t wf_launch_iteration(const DevScene &, const WfState &W, const WfLaunchConfig &, int, cudaStream_t) {
    if (g.in_capture) g.W = W;
    else { note("plain"); finish(W); }
    return cudaSuccess;
}
cudaError_t wf_launch_phase(const DevScene &, const WfState &W, const WfLaunchConfig &, int, int, cudaStream_t) {
    finish(W);
    return cudaSuccess;
}
cudaError_t wf_launch_counters_add(const WfState &, unsigned long long *, bool, cudaStream_t) { return cudaSuccess; }
int wf_occupancy(int, int, int, bool) { return 4; }
int wf_shade_occupancy(int, int, bool) { return 3; }
}  // namespace hk
