// Host driver of one wavefront engine: the path-slot pool of one scene in HBM,
// its job table and dispatch plan, its own stream and the CUDA graph of its
// iterations.  hk_render_batch runs one engine per scene over a fixed batch;
// the serving loop keeps one engine per resident scene and adds jobs to it
// while it runs.
#pragma once
#include <algorithm>
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "hk_device.h"
#include "hk_hostutil.h"
#include "hk_wavefront.h"

namespace hk {

struct WfEngineConfig {
    int capacity = 1 << 21;   // path slots
    int threads_extend = 128;
    int threads_shade = 128;
    int fetch_steps = 0;      // binary tree: node visits between traversal refills (0: 8)
    int fetch_min_idle = 0;   // idle lanes before a warp refills while others traverse (0: per-kernel default)
    int fetch_steps_shadow = 0;      // the same for the shadow rays (0: the closest-hit value where one is given)
    int fetch_min_idle_shadow = 0;
    bool fit_capacity = false;   // capacity was chosen from the work, not by the caller
    bool serve = false;   // plans follow one another; one stream (run), no device-side loop
    int reg_lean = 0;   // bit 0: extend, bit 1: shadow, bit 2: untextured shade kernels with the smaller register budget
};

class WfEngine {
public:
    // S must stay valid (its device buffers alive) for the engine's lifetime.
    WfEngine(const DevScene &S, int sm_count, const WfEngineConfig &cfg);
    ~WfEngine();
    WfEngine(const WfEngine &) = delete;
    WfEngine &operator=(const WfEngine &) = delete;

    // Device bytes an engine of this capacity holds for a scene with nemitters emitters and these shade queues.
    // Shadow records are numbered in 32 bits: one for every slot and emitter.
    static bool fits(int capacity, int nemitters) { return (int64_t)capacity * std::max(1, nemitters) < (1ll << 31); }
    static bool valid_threads(const WfEngineConfig &c) {
        for (int t : {c.threads_extend, c.threads_shade})
            if (t % 32 != 0 || t <= 0 || t > 256) return false;
        return true;
    }
    static size_t bytes_for(int capacity, int nemitters, uint64_t shade_queues);
    size_t device_bytes() const { return bytes_; }
    const WfEngineConfig &config() const { return cfg_; }
    int device() const { return device_; }   // the device that was current when the engine was made: its memory, streams and events
    // The stream the engine's work goes to next (one of two of different priority).
    cudaStream_t stream() const { return stream_; }
    // Move later work to the high- or low-priority stream, ordered after all
    // earlier work: pending kernels of a high-priority engine are scheduled
    // before those of low-priority engines sharing the GPU.
    void set_priority(bool high);

    // Empty pool (the first `slots` slots idle, 0: all), zero statistics, empty plan.  Async on stream().
    void reset(int slots = 0);
    // The start of a render of one job: reset(slots), the job in entry 0 and its
    // plan, in one launch without staging copies.  Async, and never waits.
    void begin(WfJob J, int slots);
    // Job-table entry `slot`: its finished counter is zeroed and J.finished set.  Async;
    // the slot must not be in use by paths in flight.
    void set_job(int slot, WfJob J);
    // Dispatch plan: pieces sorted by plan_begin, `total` items.  Async.
    void set_plan(const std::vector<WfSeg> &segs, uint64_t total);
    // `iterations` (even) wavefront iterations, from the graph or as plain launches.
    // With kernel_ms (host float[4]) each phase is timed with events and added.
    void run(int iterations, bool use_graph, float *kernel_ms = nullptr, int32_t *kernel_launches = nullptr);
    // Iterations until the plan is dealt and no path is in flight, or at least
    // kWfMaxLoops pairs of them: one graph launch whose while node regen
    // steers, so the host neither polls nor overshoots.  Async.
    void run_to_end();
    // Make run_to_end's graph now (its first use does otherwise).
    void prepare_loop();
    // Copy the counters and the job table's finished counters to the host mirrors
    // and record done_event(); read them after the event completed.
    void fetch_status();
    cudaEvent_t done_event() const { return ev_done_; }
    const WfCounters &status() const { return *h_ctr_; }
    const unsigned long long *finished() const { return h_fin_; }
    // Add the statistics to a caller's 7-slot device array (sum: 5 slots, the
    // traversal totals over both ray kinds).  Async.
    void add_counters(unsigned long long *out_dev, bool sum = false);
    // Rays of each extend (which 0) / shadow (which 1) launch since the last
    // reset, in launch order: up to max of them into rays (host); returns the
    // number of launches.  Synchronises the engine's stream.
    int launch_log(int which, uint32_t *rays, int max);
    const WfState &state() const { return W_; }

private:
    void capture();
    void pin_host();
    void capture_loop();
    DevScene S_;
    WfEngineConfig cfg_;
    WfLaunchConfig L_{};
    WfState W_{};
    size_t bytes_ = 0;
    int device_ = 0;
    int job_count_ = 0;   // highest job slot ever set + 1
    DevBuf mem_;             // slot records, queues, shadow queue, counters, job table, plan
    PinnedBuf<char> host_;   // the host mirrors below, on first use
    WfCounters *h_ctr_ = nullptr, *h_head_ = nullptr;
    unsigned long long *h_fin_ = nullptr;
    WfJob *h_jobs_ = nullptr;
    WfSeg *h_segs_ = nullptr;
    WfJob *jobs_ = nullptr;   // device
    WfSeg *segs_ = nullptr;
    unsigned long long *finished_ = nullptr;
    cudaStream_t stream_ = nullptr;             // current: streams_[0] or streams_[1]
    cudaStream_t streams_[2] = {nullptr, nullptr};   // low, high priority
    cudaEvent_t ev_switch_ = nullptr;
    cudaEvent_t ev_done_ = nullptr, ev_plan_ = nullptr, pe_[2] = {nullptr, nullptr};
    cudaGraph_t graph_ = nullptr;
    cudaGraphExec_t exec_ = nullptr;
    cudaGraph_t loop_graph_ = nullptr;   // one while node over a pair of iterations
    cudaGraphExec_t loop_exec_ = nullptr;
};

}  // namespace hk
