// Host driver of one wavefront engine (see hk_engine.h).
#include "hk_engine.h"

#include <algorithm>
#include <cstddef>
#include <cstring>

namespace hk {

namespace {
// bytes of an allocation's part
constexpr size_t part(size_t n) { return (n + 255) & ~(size_t)255; }
// the part of n bytes at p, which moves past it
char *take(char *&p, size_t n) {
    char *r = p;
    p += part(n);
    return r;
}
// queue arrays of one slot id per slot: 2 extend, 2 idle, the scene's shade queues, 1 finished
int queue_arrays(uint64_t shade_queues) { return 5 + __builtin_popcountll(shade_queues); }
}  // namespace

size_t WfEngine::bytes_for(int capacity, int nemitters, uint64_t shade_queues) {
    const size_t N = (size_t)capacity;
    const size_t shadow = N * (size_t)std::max(1, nemitters);
    return part(N * kSlotBytes) + part(N * sizeof(int) * queue_arrays(shade_queues)) + part(shadow * 16 * 3) +
           part(sizeof(WfCounters)) + part(sizeof(WfJob) * kWfMaxJobs) + part(sizeof(unsigned long long) * kWfMaxJobs) +
           part(sizeof(WfSeg) * kWfMaxSegs);
}

WfEngine::WfEngine(const DevScene &S, int sm_count, const WfEngineConfig &cfg) : S_(S), cfg_(cfg) {
    if (cfg_.capacity < 1024 || cfg_.capacity > (1 << 26))
        throw HkError{HK_ERR_INVALID, "wavefront capacity must be in [1024, 2^26]"};
    if (!valid_threads(cfg_)) throw HkError{HK_ERR_INVALID, "wavefront block sizes must be multiples of 32 up to 256"};
    if (!fits(cfg_.capacity, S.nemitters))
        throw HkError{HK_ERR_INVALID, "wavefront capacity x emitters must be below 2^31"};
    HK_CUDA(cudaGetDevice(&device_));
    const size_t N = (size_t)cfg_.capacity;
    W_.capacity = cfg_.capacity;
    W_.max_shadow = cfg_.capacity * std::max(1, S.nemitters);
    bytes_ = bytes_for(cfg_.capacity, S.nemitters, S.shade_queues);
    // one device allocation, carved up (256-byte aligned parts)
    mem_.alloc(bytes_);
    char *at = mem_.as<char>();
    char *rec = take(at, N * kSlotBytes);   // slot records
    int *q = (int *)take(at, N * sizeof(int) * queue_arrays(S.shade_queues));
    float4 *sh = (float4 *)take(at, (size_t)W_.max_shadow * 16 * 3);
    W_.ctr = (WfCounters *)take(at, sizeof(WfCounters));
    jobs_ = (WfJob *)take(at, sizeof(WfJob) * kWfMaxJobs);
    finished_ = (unsigned long long *)take(at, sizeof(unsigned long long) * kWfMaxJobs);
    segs_ = (WfSeg *)take(at, sizeof(WfSeg) * kWfMaxSegs);
    W_.jobs = jobs_;
    W_.segs = segs_;
    W_.ray_o.p = (float4 *)(rec + 0);
    W_.ray_d.p = (float4 *)(rec + 16);
    W_.beta.p = (float4 *)(rec + 32);
    W_.pix.p = (float4 *)(rec + 48);
    W_.rng.p = (uint4 *)(rec + 64);
    W_.hit.p = (float4 *)(rec + 80);
    W_.lacc.p = (float4 *)(rec + 96);
    W_.prev_pdf.p = (float *)(rec + 112);
    W_.eq[0] = q; W_.eq[1] = q + N;
    W_.idle[0] = q + 2 * N; W_.idle[1] = q + 3 * N;
    W_.fq = q + 4 * N;
    q += 5 * N;
    for (int t = 0; t < kWfTypes; ++t)
        if (S.shade_queues >> t & 1u) { W_.sq[t] = q; q += N; }
    W_.sh_o = sh; W_.sh_d = sh + W_.max_shadow; W_.sh_c = sh + 2 * (size_t)W_.max_shadow;
    int least = 0, greatest = 0;
    HK_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    HK_CUDA(cudaStreamCreateWithPriority(&streams_[0], cudaStreamNonBlocking, least));
    HK_CUDA(cudaStreamCreateWithPriority(&streams_[1], cudaStreamNonBlocking, greatest));
    stream_ = streams_[0];
    HK_CUDA(cudaEventCreateWithFlags(&ev_switch_, cudaEventDisableTiming));
    HK_CUDA(cudaEventCreateWithFlags(&ev_done_, cudaEventDisableTiming));
    HK_CUDA(cudaEventCreateWithFlags(&ev_plan_, cudaEventDisableTiming));
    // launch configuration: persistent grids of one wave of resident blocks
    L_.threads_extend = cfg_.threads_extend;
    L_.threads_shade = cfg_.threads_shade;
    L_.threads_shadow = cfg_.threads_extend;
    L_.threads_regen = 256;
    L_.lean_extend = cfg_.reg_lean & 1;
    L_.lean_shadow = (cfg_.reg_lean >> 1) & 1;
    L_.lean_shade = (cfg_.reg_lean >> 2) & 1;
    auto grid = [&](int which, int threads) {
        const bool lean = which == 0 ? L_.lean_extend : (which == 2 ? L_.lean_shadow : false);
        return std::max(1, sm_count * std::max(1, wf_occupancy(which, threads, S.accel, lean)));
    };
    L_.blocks_extend = grid(0, L_.threads_extend);
    L_.shade_queues = S.shade_queues;
    int nshade = 0;
    for (int q = 0; q < kWfTypes; ++q) {
        if (!(S.shade_queues >> q & 1u)) continue;
        L_.blocks_shade[q] = std::max(1, sm_count * std::max(1, wf_shade_occupancy(q, L_.threads_shade, L_.lean_shade)));
        ++nshade;
    }
    L_.blocks_shadow = grid(2, L_.threads_shadow);
    L_.blocks_regen = grid(3, L_.threads_regen);
    if (!cfg_.serve) {
        L_.nfork = std::min(kWfForks, nshade - 1);
        if (L_.nfork > 0) HK_CUDA(cudaEventCreateWithFlags(&L_.ev_fork, cudaEventDisableTiming));
        for (int f = 0; f < L_.nfork; ++f) {
            HK_CUDA(cudaStreamCreateWithFlags(&L_.fork[f], cudaStreamNonBlocking));
            HK_CUDA(cudaEventCreateWithFlags(&L_.ev_join[f], cudaEventDisableTiming));
        }
    }
    W_.recycle = cfg_.serve ? 1 : 0;
    // idle lanes before a refill, 8-wide tree: a refill costs the warp about 140
    // instructions and a partly filled test batch, an idle lane a 32nd of the
    // rest (64-sphere scene, ms of 33.5M paths at 4 / 8 / 12 lanes: closest hit
    // 24.5 / 21.8 / 21.0, shadow 33.7 / 33.0 / 33.5)
    const bool w8 = S.accel == kAccelBvh8;
    L_.fetch_steps = cfg_.fetch_steps > 0 ? cfg_.fetch_steps : 8;
    L_.fetch_min_idle = cfg_.fetch_min_idle > 0 ? std::min(32, cfg_.fetch_min_idle) : (w8 ? 12 : 1);
    L_.fetch_steps_shadow = cfg_.fetch_steps_shadow > 0 ? cfg_.fetch_steps_shadow : L_.fetch_steps;
    const int shadow_idle = cfg_.fetch_min_idle_shadow > 0 ? cfg_.fetch_min_idle_shadow : cfg_.fetch_min_idle;
    L_.fetch_min_idle_shadow = shadow_idle > 0 ? std::min(32, shadow_idle) : (w8 ? 8 : 1);
    HK_CUDA(cudaGetLastError());
    if (cfg_.serve) reset();
    else HK_CUDA(wf_launch_init(W_, W_.capacity, WfJob{}, stream_));   // begin or reset starts a render
}

// The host mirrors, in one pinned allocation made when a plan or a status first
// needs them: it takes 2 ms, twice the rest of an engine, and a render that
// starts with begin needs neither.
void WfEngine::pin_host() {
    if (host_.p) return;
    const size_t bytes = 2 * part(sizeof(WfCounters)) + part(sizeof(unsigned long long) * kWfMaxJobs) +
                         part(sizeof(WfJob) * kWfMaxJobs) + part(sizeof(WfSeg) * kWfMaxSegs);
    host_.alloc(bytes);
    std::memset(host_.p, 0, bytes);
    char *at = host_.p;
    h_ctr_ = (WfCounters *)take(at, sizeof(WfCounters));
    h_head_ = (WfCounters *)take(at, sizeof(WfCounters));
    h_fin_ = (unsigned long long *)take(at, sizeof(unsigned long long) * kWfMaxJobs);
    h_jobs_ = (WfJob *)take(at, sizeof(WfJob) * kWfMaxJobs);
    h_segs_ = (WfSeg *)take(at, sizeof(WfSeg) * kWfMaxSegs);
}

WfEngine::~WfEngine() {
    for (cudaStream_t s : streams_)
        if (s) cudaStreamSynchronize(s);
    if (exec_) cudaGraphExecDestroy(exec_);
    if (graph_) cudaGraphDestroy(graph_);
    if (loop_exec_) cudaGraphExecDestroy(loop_exec_);
    if (loop_graph_) cudaGraphDestroy(loop_graph_);
    for (cudaEvent_t e : {L_.ev_fork, L_.ev_join[0], L_.ev_join[1], L_.ev_join[2]})
        if (e) cudaEventDestroy(e);
    for (cudaStream_t s : L_.fork)
        if (s) cudaStreamDestroy(s);
    for (cudaEvent_t e : {ev_done_, ev_plan_, ev_switch_, pe_[0], pe_[1]})
        if (e) cudaEventDestroy(e);
    for (cudaStream_t s : streams_)
        if (s) cudaStreamDestroy(s);
}

void WfEngine::set_priority(bool high) {
    cudaStream_t target = streams_[high ? 1 : 0];
    if (target == stream_) return;
    HK_CUDA(cudaEventRecord(ev_switch_, stream_));
    HK_CUDA(cudaStreamWaitEvent(target, ev_switch_, 0));
    stream_ = target;
}

void WfEngine::reset(int slots) {
    set_plan({}, 0);
    HK_CUDA(wf_launch_init(W_, slots > 0 ? std::min(slots, W_.capacity) : W_.capacity, WfJob{}, stream_));
}

void WfEngine::begin(WfJob J, int slots) {
    J.finished = finished_;
    job_count_ = std::max(job_count_, 1);
    HK_CUDA(wf_launch_init(W_, std::min(slots, W_.capacity), J, stream_));
}

void WfEngine::set_job(int slot, WfJob J) {
    if (slot < 0 || slot >= kWfMaxJobs) throw HkError{HK_ERR_INVALID, "job slot out of range"};
    // Each slot has its own staging entry; a slot is rewritten only after its
    // previous job ended, long after that job's copy ran.
    pin_host();
    J.finished = finished_ + slot;
    job_count_ = std::max(job_count_, slot + 1);
    h_jobs_[slot] = J;
    HK_CUDA(cudaMemcpyAsync(jobs_ + slot, h_jobs_ + slot, sizeof(WfJob), cudaMemcpyHostToDevice, stream_));
    HK_CUDA(cudaMemsetAsync(finished_ + slot, 0, sizeof(unsigned long long), stream_));
}

void WfEngine::set_plan(const std::vector<WfSeg> &segs, uint64_t total) {
    if (segs.size() > (size_t)kWfMaxSegs) throw HkError{HK_ERR_INVALID, "dispatch plan has too many pieces"};
    pin_host();
    HK_CUDA(cudaEventSynchronize(ev_plan_));   // the staging copies of the previous plan have run
    if (!segs.empty()) {
        std::memcpy(h_segs_, segs.data(), sizeof(WfSeg) * segs.size());
        HK_CUDA(cudaMemcpyAsync(segs_, h_segs_, sizeof(WfSeg) * segs.size(), cudaMemcpyHostToDevice, stream_));
    }
    WfCounters &h = *h_head_;
    h.next_work = 0;
    h.total_work = total;
    h.seg_count = (unsigned)segs.size();
    h.job_count = (unsigned)job_count_;
    // the dispatch head: next_work, total_work, seg_count, job_count (first 24 bytes)
    HK_CUDA(cudaMemcpyAsync(W_.ctr, &h, offsetof(WfCounters, eq_count), cudaMemcpyHostToDevice, stream_));
    HK_CUDA(cudaEventRecord(ev_plan_, stream_));
}

void WfEngine::capture() {
    HK_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
    cudaError_t e0 = wf_launch_iteration(S_, W_, L_, 0, stream_);
    cudaError_t e1 = wf_launch_iteration(S_, W_, L_, 1, stream_);
    cudaError_t ec = cudaStreamEndCapture(stream_, &graph_);
    if (e0 != cudaSuccess || e1 != cudaSuccess || ec != cudaSuccess) {
        if (graph_) cudaGraphDestroy(graph_);
        graph_ = nullptr;
        throw HkError{HK_ERR_CUDA, "wavefront graph capture failed"};
    }
    HK_CUDA(cudaGraphInstantiate(&exec_, graph_, 0));
}

void WfEngine::capture_loop() {
    HK_CUDA(cudaGraphCreate(&loop_graph_, 0));
    cudaGraphConditionalHandle handle;
    HK_CUDA(cudaGraphConditionalHandleCreate(&handle, loop_graph_, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = handle;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t node;
    HK_CUDA(cudaGraphAddNode(&node, loop_graph_, nullptr, 0, &np));
    cudaGraph_t body = np.conditional.phGraph_out[0];
    WfState W = W_;
    W.cond = handle;
    HK_CUDA(cudaStreamBeginCaptureToGraph(stream_, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    const cudaError_t e0 = wf_launch_iteration(S_, W, L_, 0, stream_);
    const cudaError_t e1 = wf_launch_iteration(S_, W, L_, 1, stream_);
    const cudaError_t ec = cudaStreamEndCapture(stream_, &body);
    if (e0 != cudaSuccess || e1 != cudaSuccess || ec != cudaSuccess)
        throw HkError{HK_ERR_CUDA, "wavefront graph capture failed"};
    HK_CUDA(cudaGraphInstantiate(&loop_exec_, loop_graph_, 0));
}

void WfEngine::prepare_loop() {
    if (loop_exec_) return;
    if (loop_graph_) cudaGraphDestroy(loop_graph_);   // an earlier attempt failed half way
    loop_graph_ = nullptr;
    capture_loop();
}

void WfEngine::run_to_end() {
    prepare_loop();
    HK_CUDA(cudaGraphLaunch(loop_exec_, stream_));
}

void WfEngine::run(int iterations, bool use_graph, float *kernel_ms, int32_t *kernel_launches) {
    iterations += iterations & 1;   // the queues ping-pong: whole pairs only
    if (kernel_ms) {
        if (!pe_[0]) {
            HK_CUDA(cudaEventCreate(&pe_[0]));
            HK_CUDA(cudaEventCreate(&pe_[1]));
        }
        const int phase_launches[4] = {1, 1, __builtin_popcountll(L_.shade_queues), 1};
        for (int k = 0; k < iterations; ++k)
            for (int ph = 0; ph < 4; ++ph) {
                HK_CUDA(cudaEventRecord(pe_[0], stream_));
                HK_CUDA(wf_launch_phase(S_, W_, L_, k & 1, ph, stream_));
                HK_CUDA(cudaEventRecord(pe_[1], stream_));
                HK_CUDA(cudaEventSynchronize(pe_[1]));
                float ms = 0;
                HK_CUDA(cudaEventElapsedTime(&ms, pe_[0], pe_[1]));
                kernel_ms[ph] += ms;
                if (kernel_launches) kernel_launches[ph] += phase_launches[ph];
            }
        return;
    }
    if (!use_graph) {
        for (int k = 0; k < iterations; ++k) HK_CUDA(wf_launch_iteration(S_, W_, L_, k & 1, stream_));
        return;
    }
    if (!exec_) capture();
    for (int k = 0; k < iterations; k += 2) HK_CUDA(cudaGraphLaunch(exec_, stream_));
}

void WfEngine::fetch_status() {
    pin_host();
    HK_CUDA(cudaMemcpyAsync(h_ctr_, W_.ctr, offsetof(WfCounters, log_n), cudaMemcpyDeviceToHost, stream_));
    HK_CUDA(cudaMemcpyAsync(h_fin_, finished_, sizeof(unsigned long long) * kWfMaxJobs, cudaMemcpyDeviceToHost,
                            stream_));
    HK_CUDA(cudaEventRecord(ev_done_, stream_));
}

void WfEngine::add_counters(unsigned long long *out_dev, bool sum) {
    HK_CUDA(wf_launch_counters_add(W_, out_dev, sum, stream_));
}

int WfEngine::launch_log(int which, uint32_t *rays, int max) {
    unsigned n = 0;
    HK_CUDA(cudaMemcpyAsync(&n, &W_.ctr->log_n[which], sizeof n, cudaMemcpyDeviceToHost, stream_));
    HK_CUDA(cudaStreamSynchronize(stream_));
    const int k = (int)std::min<unsigned>(n, (unsigned)std::min(max, kWfLaunchLog));
    if (k > 0) {
        HK_CUDA(cudaMemcpyAsync(rays, &W_.ctr->log_rays[which][0], sizeof(uint32_t) * k, cudaMemcpyDeviceToHost,
                                stream_));
        HK_CUDA(cudaStreamSynchronize(stream_));
    }
    return (int)n;
}

}  // namespace hk
