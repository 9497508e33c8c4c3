// Wavefront pathMIS on sm_100a: the integrator of
// src/integrator/PathMISIntegrator.cpp:16-157 split at its ray casts so that
// every kernel runs one kind of work over a compacted queue.
//
//   regen   finished paths are splatted (ImageBlock::Put, src/core/Block.cpp:95)
//           into their job's film with 128-bit vector reductions; slots claim
//           new (job, tile, sample, pixel) work and start camera rays
//   extend  closest hit of every queued ray; the hit's material type picks
//           the shade queue
//   shade<T> one kernel per top-level BSDF type (and one for misses): emitter
//           hit with its MIS weight, next-event estimation over every emitter
//           (shadow rays queued with their contribution), BSDF sampling,
//           Russian roulette
//   shadow  any-hit of every queued shadow ray; unoccluded contributions are
//           added to their path's radiance
//
// This file holds regen and the launches of an iteration; the queue helpers and the
// shade kernels are in hk_wf_kernels.cuh, the extend and shadow kernels in
// hk_wf_trace.cuh.
//
// The estimator is the reference's: the next-event MIS weight of an
// unoccluded emitter is its own pl / (pl + pb) (the reference updates its
// carried weight exactly when the shadow ray is unoccluded, and uses it right
// away); the emitter-hit weight is computed from the pdf that the previous
// vertex's BSDF had for the direction it sampled, taken there and kept in the
// path's record, and forced to 1 after an EDiscrete sample; Russian roulette runs
// before the continuation ray is traced (the reference traces first and
// discards the hit of a terminated path, which changes nothing).
#include "hk_wf_kernels.cuh"

#include <algorithm>

namespace hk {

// The traversal and shade kernels are instantiated in hk_wf_trace_*.cu and
// hk_wf_shade_*.cu; this file only calls their launchers.
template <int kAccel>
cudaError_t wf_launch_extend_t(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template <int kAccel>
cudaError_t wf_launch_shadow_t(const DevScene &, const WfState &, const WfLaunchConfig &, cudaStream_t);
template <int kAccel>
int wf_trace_occupancy_t(int, int, bool);
#define HK_WF_SHADE_EXTERN(K)                                                                                           \
    extern template cudaError_t wf_launch_shade_t<K>(const DevScene &, const WfState &, const WfLaunchConfig &, int, \
                                                     cudaStream_t);                                                 \
    extern template int wf_shade_occupancy_t<K>(int, bool)
HK_WF_SHADE_EXTERN(0);
HK_WF_SHADE_EXTERN(1);
HK_WF_SHADE_EXTERN(2);
HK_WF_SHADE_EXTERN(3);
HK_WF_SHADE_EXTERN(4);
HK_WF_SHADE_EXTERN(5);
HK_WF_SHADE_EXTERN(6);
HK_WF_SHADE_EXTERN(7);
HK_WF_SHADE_EXTERN(8);
HK_WF_SHADE_EXTERN(9);
HK_WF_SHADE_EXTERN(11);
HK_WF_SHADE_EXTERN(12);
HK_WF_SHADE_EXTERN(13);
HK_WF_SHADE_EXTERN(14);
HK_WF_SHADE_EXTERN(15);
HK_WF_SHADE_EXTERN(16);
HK_WF_SHADE_EXTERN(17);
HK_WF_SHADE_EXTERN(18);
HK_WF_SHADE_EXTERN(19);
HK_WF_SHADE_EXTERN(20);
HK_WF_SHADE_EXTERN(21);
HK_WF_SHADE_EXTERN(23);
HK_WF_SHADE_EXTERN(24);
HK_WF_SHADE_EXTERN(25);
HK_WF_SHADE_EXTERN(26);
HK_WF_SHADE_EXTERN(27);
HK_WF_SHADE_EXTERN(28);
HK_WF_SHADE_EXTERN(29);
HK_WF_SHADE_EXTERN(30);
HK_WF_SHADE_EXTERN(31);
HK_WF_SHADE_EXTERN(32);
HK_WF_SHADE_EXTERN(33);
HK_WF_SHADE_EXTERN(35);
HK_WF_SHADE_EXTERN(36);
HK_WF_SHADE_EXTERN(37);
#undef HK_WF_SHADE_EXTERN
static_assert(kWfTypes == 38, "one shade kernel per queue");
// TwoSided BSDFs (10, 22, 34) have no kernel of their own: wf_queue_of sends them to the generic queue.
constexpr bool has_shade_kernel(int q) { return q == 0 || q == kWfGenericQueue || (q - 1) % kWfLeafTypes != kTwoSided; }

// ------------------------------------------------------------ regen
// Splat and retire the finished paths, then give finished and idle slots new
// work from the dispatch plan; slots that find none wait in the next idle
// list.  Queues read here: fq, idle[cur]; written: eq[cur], idle[cur ^ 1].
// Slot i of the n slots that want work (finished paths first, then idle
// slots) takes plan item next_work + i: the items are dealt without an
// atomic, and the last block to finish advances next_work by n.  An item
// whose pixel lies outside its image (the partial tiles at the right and
// bottom edges) counts as work done and leaves its slot idle until the next
// iteration.  Where no plan follows this one (W.recycle == 0), idle slots
// beyond the plan's end are dropped, so that a draining pool touches only the
// paths still in flight (a quarter of a 2^22-path image's iterations drain).
// Appends to the extend and idle lists, the per-job finished counts and the
// change of the in-flight count are gathered per block in shared memory and
// added once per block and round: a global atomic per warp on a handful of
// addresses serialises at the L2.
__global__ void __launch_bounds__(256) wf_regen_kernel(DevScene S, WfState W, int cur) {
    __shared__ unsigned s_finished[kWfMaxJobs];
    __shared__ int s_active;
    __shared__ unsigned s_warp[2][8];   // per-warp counts, then offsets, of the extend / idle appends
    __shared__ unsigned s_base[2];
    const int njobs = (int)W.ctr->job_count;
    const int nf = (int)W.ctr->fq_count;
    const uint64_t total = W.ctr->total_work;
    const uint64_t first = W.ctr->next_work;
    int n = nf + (int)W.ctr->idle_count[cur];
    const bool drained = !W.recycle && first + (uint64_t)n >= total;   // this pass deals the plan's last item
    if (drained) n = max(nf, (int)min((uint64_t)n, total - min(first, total)));
    const int nseg = (int)W.ctr->seg_count;
    const bool some = (int)(blockIdx.x * blockDim.x) < n;   // block-uniform: slots for this block
    if (some)
        for (int k = threadIdx.x; k < njobs; k += blockDim.x) s_finished[k] = 0u;
    if (threadIdx.x == 0) s_active = 0;
    __syncthreads();
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    unsigned long long dropped = 0;
    int active_delta = 0;
    for (int i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {   // block-uniform rounds
        const int i = i0 + (int)threadIdx.x;
        int slot = -1;
        bool started = false;
        if (i < n) {
            if (i < nf) {
                slot = W.fq[i];
                float4 p = W.pix[slot];
                float4 L = W.lacc[slot];
                const int pj = __float_as_int(p.z);
                const WfJob &J = W.jobs[pj];
                V3 val = v3(L.x, L.y, L.z);
                if (is_valid(val)) splat_film(S, J.film, (int)J.width, (int)J.height, p.x, p.y, val);
                else ++dropped;
                atomicAdd(&s_finished[pj], 1u);
                --active_delta;
            } else {
                slot = W.idle[cur][i - nf];
            }
            const uint64_t w = first + (uint64_t)i;
            if (w < total) {
                const WfSeg &G = W.segs[find_seg(W, w, nseg)];
                const int j = G.job;
                const WfJob &J = W.jobs[j];
                const uint64_t l = G.job_begin + (w - G.plan_begin);
                const uint32_t p = (uint32_t)(l % kWfTilePixels);
                const uint64_t ts = l / kWfTilePixels;
                uint32_t s, t;
                if (J.sample_major) {
                    const uint64_t ntiles = J.work_count / ((uint64_t)J.spp * kWfTilePixels);
                    t = (uint32_t)(ts % ntiles);
                    s = (uint32_t)(ts / ntiles);
                } else {
                    s = (uint32_t)(ts % J.spp);
                    t = (uint32_t)(ts / J.spp);
                }
                const uint32_t x = (t % J.tiles_x) * kWfTileSide + p % kWfTileSide;
                const uint32_t y = (t / J.tiles_x) * kWfTileSide + p / kWfTileSide;
                if (x >= J.width || y >= J.height) {
                    atomicAdd(&s_finished[j], 1u);   // counted as work done: no path
                } else {
                    Pcg32 rng;
                    rng.seed(mix_seed(J.seed, (uint64_t)J.sample_offset + s),
                             (uint64_t)y * J.width + x + (uint64_t)J.image_index * J.width * J.height);
                    float px = (float)x + rng.nextf(), py = (float)y + rng.nextf();
                    Ray r = camera_ray_job(S, J, px, py);
                    W.ray_o[slot] = f4(r.o, r.tmin);
                    W.ray_d[slot] = f4(r.d, r.tmax);
                    W.beta[slot] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
                    W.lacc[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    W.pix[slot] = make_float4(px, py, __int_as_float(j), __int_as_float(0));
                    W.rng[slot] = make_uint4((uint32_t)rng.state, (uint32_t)(rng.state >> 32), (uint32_t)rng.inc,
                                             (uint32_t)(rng.inc >> 32));
                    ++active_delta;
                    started = true;
                }
            }
        }
        // block-aggregated appends: one atomic per list per block and round
        const bool to_idle = i < n && !started && !drained;
        const unsigned be = __ballot_sync(0xffffffffu, started), bi = __ballot_sync(0xffffffffu, to_idle);
        if (lane == 0) {
            s_warp[0][warp] = __popc(be);
            s_warp[1][warp] = __popc(bi);
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            unsigned sum = 0;
            for (unsigned k = 0; k < nwarps; ++k) {
                const unsigned c = s_warp[threadIdx.x][k];
                s_warp[threadIdx.x][k] = sum;
                sum += c;
            }
            unsigned *ctr = threadIdx.x == 0 ? &W.ctr->eq_count[cur] : &W.ctr->idle_count[cur ^ 1];
            s_base[threadIdx.x] = sum ? atomicAdd(ctr, sum) : 0u;
        }
        __syncthreads();
        const unsigned below = (1u << lane) - 1u;
        if (started) W.eq[cur][s_base[0] + s_warp[0][warp] + __popc(be & below)] = slot;
        if (to_idle) W.idle[cur ^ 1][s_base[1] + s_warp[1][warp] + __popc(bi & below)] = slot;
        __syncthreads();   // s_warp and s_base are rewritten by the next round
    }
    if (dropped) atomicAdd(&W.ctr->dropped, dropped);
    // one atomic per warp into the block, one per block and job into HBM
    for (int o = 16; o > 0; o >>= 1) active_delta += __shfl_down_sync(0xffffffffu, active_delta, o);
    if (lane == 0 && active_delta) atomicAdd(&s_active, active_delta);
    __syncthreads();
    for (int k = threadIdx.x; some && k < njobs; k += blockDim.x)
        if (s_finished[k]) atomicAdd(W.jobs[k].finished, (unsigned long long)s_finished[k]);
    // the last block through resets the counters of the queues consumed here
    // and of those that the next phases fill, and decides whether the
    // device-side loop goes on
    if (threadIdx.x == 0) {
        WfCounters *c = W.ctr;
        if (s_active) atomicAdd(&c->active, (unsigned)s_active);
        __threadfence();
        if (atomicAdd(&c->regen_done, 1u) == gridDim.x - 1u) {
            __threadfence();
            const unsigned long long dealt = first + (uint64_t)n;
            const unsigned long long next = dealt < total ? dealt : total;
            c->regen_done = 0u;
            c->next_work = next;
            c->fq_count = 0u;
            c->idle_count[cur] = 0u;
            c->eq_count[cur ^ 1] = 0u;
            c->shadow_count = 0u;
            for (unsigned k = 0; k < kWfFetchParts; ++k) c->ext_fetch[k * kWfFetchStride] = c->sh_fetch[k * kWfFetchStride] = 0u;
            for (int t = 0; t < kWfTypes; ++t) c->sq_count[t] = 0u;
            if (W.cond && cur == 1) {
                const bool more = (atomicAdd(&c->active, 0u) != 0u || next < total) && ++c->loops < kWfMaxLoops;
                if (!more) c->loops = 0u;
                cudaGraphSetConditional(W.cond, more ? 1u : 0u);
            }
        }
    }
}

// Empty pool: the first `slots` slots in idle list 0, all queues and statistics
// zero.  With a job (work_count > 0) also the table of that one job and its plan:
// the whole start of a render in one launch, its input passed by value, so a
// caller can queue renders without the host waiting for a staging buffer.
__global__ void wf_init_kernel(WfState W, int slots, WfJob J) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += gridDim.x * blockDim.x) W.idle[0][i] = i;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        WfCounters *c = W.ctr;
        c->eq_count[0] = c->eq_count[1] = 0;
        c->idle_count[0] = (unsigned)slots;
        c->idle_count[1] = 0;
        for (int t = 0; t < kWfTypes; ++t) c->sq_count[t] = 0;
        c->fq_count = c->shadow_count = c->active = 0;
        for (unsigned k = 0; k < kWfFetchParts; ++k) c->ext_fetch[k * kWfFetchStride] = c->sh_fetch[k * kWfFetchStride] = 0;
        c->regen_done = c->loops = 0;
        c->rays = c->shadow_rays = c->dropped = 0;
        c->node_visits = c->tri_tests = c->node_visits_shadow = c->tri_tests_shadow = 0;
        c->log_n[0] = c->log_n[1] = 0;
        if (J.work_count > 0) {
            c->next_work = 0;
            c->total_work = J.work_count;
            c->seg_count = 1;
            c->job_count = 1;
            const_cast<WfJob *>(W.jobs)[0] = J;
            const_cast<WfSeg *>(W.segs)[0] = WfSeg{0, 0, 0, 0};
            *J.finished = 0;
        }
    }
}

// Add the engine's statistics to a caller's 7-slot u64 array, or to a 5-slot one
// with the traversal totals of both ray kinds (sum).  Other renders may add to
// the array meanwhile.
__global__ void wf_counters_add_kernel(const WfCounters *c, unsigned long long *out, bool sum) {
    if (threadIdx.x != 0) return;
    atomicAdd(out + 0, c->rays);
    atomicAdd(out + 1, c->shadow_rays);
    atomicAdd(out + 2, c->dropped);
    atomicAdd(out + 3, c->node_visits + (sum ? c->node_visits_shadow : 0));
    atomicAdd(out + 4, c->tri_tests + (sum ? c->tri_tests_shadow : 0));
    if (sum) return;
    atomicAdd(out + 5, c->node_visits_shadow);
    atomicAdd(out + 6, c->tri_tests_shadow);
}

// ------------------------------------------------------------ launchers
static cudaError_t launch_extend(const DevScene &S, const WfState &W, const WfLaunchConfig &C, int cur, cudaStream_t st) {
    return S.accel == kAccelBvh8 ? wf_launch_extend_t<kAccelBvh8>(S, W, C, cur, st) : wf_launch_extend_t<kAccelBvh2>(S, W, C, cur, st);
}
static cudaError_t launch_shadow(const DevScene &S, const WfState &W, const WfLaunchConfig &C, cudaStream_t st) {
    return S.accel == kAccelBvh8 ? wf_launch_shadow_t<kAccelBvh8>(S, W, C, st) : wf_launch_shadow_t<kAccelBvh2>(S, W, C, st);
}
// The shade kernels of the queues that the scene can reach.  They are dealt to
// the launch stream and its forks: each runs one wave or less in the later
// iterations, so side by side they fill the SMs that one alone leaves idle.
template <int kType>
struct ShadeLaunch {
    static void run(const DevScene &S, const WfState &W, const WfLaunchConfig &C, int nxt, cudaStream_t st, int &k) {
        if constexpr (has_shade_kernel(kType)) {
            if (C.shade_queues >> kType & 1u) {
                const int lane = k++ % (C.nfork + 1);
                wf_launch_shade_t<kType>(S, W, C, nxt, lane == 0 ? st : C.fork[lane - 1]);
            }
        }
        if constexpr (kType + 1 < kWfTypes) ShadeLaunch<kType + 1>::run(S, W, C, nxt, st, k);
    }
};
static cudaError_t launch_shade_all(const DevScene &S, const WfState &W, const WfLaunchConfig &C, int nxt, cudaStream_t st) {
    if (C.nfork > 0) {
        cudaEventRecord(C.ev_fork, st);
        for (int f = 0; f < C.nfork; ++f) cudaStreamWaitEvent(C.fork[f], C.ev_fork, 0);
    }
    int k = 0;
    ShadeLaunch<0>::run(S, W, C, nxt, st, k);
    for (int f = 0; f < C.nfork; ++f) {
        cudaEventRecord(C.ev_join[f], C.fork[f]);
        cudaStreamWaitEvent(st, C.ev_join[f], 0);
    }
    return cudaGetLastError();
}

cudaError_t wf_launch_counters_add(const WfState &W, unsigned long long *out, bool sum, cudaStream_t st) {
    wf_counters_add_kernel<<<1, 32, 0, st>>>(W.ctr, out, sum);
    return cudaGetLastError();
}

cudaError_t wf_launch_init(const WfState &W, int slots, const WfJob &J, cudaStream_t st) {
    wf_init_kernel<<<std::max(1, std::min((slots + 255) / 256, 4096)), 256, 0, st>>>(W, slots, J);
    return cudaGetLastError();
}

cudaError_t wf_launch_iteration(const DevScene &S, const WfState &W, const WfLaunchConfig &C, int cur, cudaStream_t st) {
    const int nxt = cur ^ 1;
    wf_regen_kernel<<<C.blocks_regen, C.threads_regen, 0, st>>>(S, W, cur);
    launch_extend(S, W, C, cur, st);
    launch_shade_all(S, W, C, nxt, st);
    launch_shadow(S, W, C, st);
    return cudaGetLastError();
}

cudaError_t wf_launch_phase(const DevScene &S, const WfState &W, const WfLaunchConfig &C, int cur, int phase,
                            cudaStream_t st) {
    const int nxt = cur ^ 1;
    switch (phase) {
    case 0:
        wf_regen_kernel<<<C.blocks_regen, C.threads_regen, 0, st>>>(S, W, cur);
            break;
    case 1: launch_extend(S, W, C, cur, st); break;
    case 2: launch_shade_all(S, W, C, nxt, st); break;
    default: launch_shadow(S, W, C, st); break;
    }
    return cudaGetLastError();
}

int wf_occupancy(int which, int threads, int accel, bool lean) {
    if (which == 3) {
        int n = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wf_regen_kernel, threads, 0);
        return n;
    }
    return accel == kAccelBvh8 ? wf_trace_occupancy_t<kAccelBvh8>(which, threads, lean)
                               : wf_trace_occupancy_t<kAccelBvh2>(which, threads, lean);
}
template <int kType>
static int shade_occupancy(int queue, int threads, bool lean) {
    if constexpr (has_shade_kernel(kType)) {
        if (queue == kType) return wf_shade_occupancy_t<kType>(threads, lean);
    }
    if constexpr (kType + 1 < kWfTypes) return shade_occupancy<kType + 1>(queue, threads, lean);
    return 0;
}
int wf_shade_occupancy(int queue, int threads, bool lean) { return shade_occupancy<0>(queue, threads, lean); }

}  // namespace hk
