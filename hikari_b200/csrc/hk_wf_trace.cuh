// Traversal kernels of the wavefront (extend: closest hit, shadow: any hit).
// Included by hk_wf_trace_*.cu alone, so a change here recompiles no shade
// kernel and no megakernel.
#pragma once
#include "hk_traverse8.cuh"
#include "hk_wf_kernels.cuh"

namespace hk {

// Two register budgets: kBlocks = 4 resident blocks of 256 threads (64
// registers) and, where hk_wavefront_config.reg_lean asks, kLeanBlocks = 5 (48
// registers, some spilling).  Left to itself the compiler takes 76-80
// registers, and the fewer resident warps cost 7% (64-sphere scene, shadow 0.265
// instead of 0.248 ns per ray); 56 with spilling costs 3%.
constexpr int kBlocks = 4;
constexpr int kLeanBlocks = 5;

// ------------------------------------------------------------ kernels
// Traces the n rays of a queue in the tree kAccel.
template <int kAccel, bool kAnyHit, class Load, class Store>
__device__ __forceinline__ void trace_rays(const DevScene &S, unsigned *fetch, unsigned n, int steps, int min_idle,
                                           Load load, Store store, TravStats &ts) {
    if constexpr (kAccel == kAccelBvh8) {
        // Every warp starts with an equal share of the queue, at most kClaim8
        // rays, so that a short queue (a small image, the last bounces of a large
        // one) is spread over all warps and costs no atomic: with chunks of 128
        // claimed from the start, 4096 rays of a Cornell box went to 32 warps and
        // took 58 us; so they take 12.  The rest is claimed 32 rays at a time: a
        // claim of 128 near the end kept a warp for a quarter of a launch of 2^21
        // rays while others idled (64-sphere scene, 0.304 ns per closest-hit ray,
        // 0.265 with 32).  One counter would bound cheap rays (Cornell box,
        // shadow 0.132 -> 0.190 ns), so the rest is cut into kWfFetchParts parts
        // with a counter and a cache line each; a warp moves on to the next part
        // when one is used up.
        const unsigned warps = gridDim.x * (blockDim.x / 32u), warp = blockIdx.x * (blockDim.x / 32u) + threadIdx.x / 32u;
        const unsigned own = min(kClaim8, (n + warps - 1u) / warps);
        const unsigned first = min(n, warp * own), last = min(n, first + own);
        auto claim = [&](unsigned &part) {
            const unsigned dealt = gridDim.x * (blockDim.x / 32u) * kClaim8;
            if (n <= dealt) return n;
            // entries of a part: a multiple of kClaim8
            const unsigned len = ((n - dealt + kWfFetchParts * kClaim8 - 1u) / (kWfFetchParts * kClaim8)) * kClaim8;
            for (unsigned k = 0; k < kWfFetchParts; ++k) {
                const unsigned at = atomicAdd(fetch + part * kWfFetchStride, kClaim8);
                if (at < len && dealt + part * len + at < n) return dealt + part * len + at;
                part = part + 1u == kWfFetchParts ? 0u : part + 1u;
            }
            return n;
        };
        trace_queue8<kAnyHit, kAnyHit ? kRangeUnit : kRangeWave>(S, first, last, n, warp % kWfFetchParts, min_idle, claim, load,
                                                                 store, ts);
    } else {
        Bvh2Walker wk;
        int stack_mem[kStackSize];
        wk.stack = stack_mem;
        trace_queue<kAnyHit>(S, wk, fetch, n, steps, min_idle, load,
                             [&](int i, const Bvh2Walker &w) { store(i, w.found, w.hit); }, ts);
    }
}
// Adds a warp's traversal statistics to the two counters (8-wide tree: every
// lane has the warp's; binary: its own).
template <int kAccel>
__device__ __forceinline__ void add_stats(const TravStats &ts, unsigned long long *visits, unsigned long long *tests) {
    unsigned long long nv = ts.nodes, nt = ts.tris;
    if constexpr (kAccel != kAccelBvh8)
        for (int o = 16; o > 0; o >>= 1) {
            nv += __shfl_down_sync(0xffffffffu, nv, o);
            nt += __shfl_down_sync(0xffffffffu, nt, o);
        }
    if (lane_id() == 0 && (nv || nt)) {
        atomicAdd(visits, nv);
        atomicAdd(tests, nt);
    }
}
// Counts the rays of a launch (which: 0 extend, 1 shadow); launches are stream-ordered.
__device__ __forceinline__ void log_launch(WfCounters *c, int which, unsigned n) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    atomicAdd(which ? &c->shadow_rays : &c->rays, (unsigned long long)n);
    const unsigned k = c->log_n[which];
    if (k < (unsigned)kWfLaunchLog) c->log_rays[which][k] = n;
    c->log_n[which] = k + 1;
}

template <int kAccel, int kMinBlocks>
__global__ void __launch_bounds__(256, kMinBlocks) wf_extend_kernel(DevScene S, WfState W, int cur, int steps, int min_idle) {
    const unsigned n = W.ctr->eq_count[cur];
    TravStats ts;
    int slot = -1;
    auto load = [&](int i) {
        slot = W.eq[cur][i];
        const float4 o = W.ray_o[slot], d = W.ray_d[slot];
        Ray r;
        r.o = xyz(o);
        r.d = xyz(d);
        r.tmin = o.w;
        r.tmax = d.w;
        return r;
    };
    auto store = [&](int, bool found, Hit h) {
        int type = 0;
        if (found) {
            const float4 *tp = S.tris + 3 * (size_t)h.tri;
            const float4 p1 = ldg4(tp + 1);
            if constexpr (kAccel == kAccelBvh8) {
                // t and the barycentrics with the reference's arithmetic (the binary walker has done it)
                const float4 o = W.ray_o[slot], d = W.ray_d[slot];
                refine_mt(xyz(o), xyz(d), xyz(ldg4(tp)), xyz(p1), xyz(ldg4(tp + 2)), o.w, d.w, h.t, h.u, h.v);
            }
            type = S.meshes[__float_as_int(p1.w)].shade_queue;
        }
        W.hit[slot] = make_float4(h.t, h.u, h.v, __int_as_float(found ? h.tri : -1));
        W.sq[type][warp_append_keyed(W.ctr->sq_count, type)] = slot;
    };
    trace_rays<kAccel, false>(S, W.ctr->ext_fetch, n, steps, min_idle, load, store, ts);
    add_stats<kAccel>(ts, &W.ctr->node_visits, &W.ctr->tri_tests);
    log_launch(W.ctr, 0, n);
}

template <int kAccel, int kMinBlocks>
__global__ void __launch_bounds__(256, kMinBlocks) wf_shadow_kernel(DevScene S, WfState W, int steps, int min_idle) {
    const unsigned n = min(W.ctr->shadow_count, (unsigned)W.max_shadow);
    TravStats ts;
    auto load = [&](int i) {
        const float4 o = W.sh_o[i], d = W.sh_d[i];
        Ray r;
        r.o = xyz(o);
        r.d = xyz(d);
        r.tmin = kRayEps;
        r.tmax = 1.0f - kRayEps;
        return r;
    };
    auto store = [&](int i, bool found, const Hit &) {
        if (!found) {
            const float4 c = W.sh_c[i];
            const int slot = __float_as_int(W.sh_o[i].w);
            red_add_v4(W.lacc + slot, c.x, c.y, c.z, 0.0f);
        }
    };
    trace_rays<kAccel, true>(S, W.ctr->sh_fetch, n, steps, min_idle, load, store, ts);
    add_stats<kAccel>(ts, &W.ctr->node_visits_shadow, &W.ctr->tri_tests_shadow);
    log_launch(W.ctr, 1, n);
}

// ------------------------------------------------------------ launchers
// dynamic shared memory of a launch (which: 0 extend, 2 shadow)
inline size_t wf_trace_smem(int which, int accel, int threads) {
    return accel == kAccelBvh8 ? trace8_smem(which == 2, threads) : 0;
}
template <int kAccel>
cudaError_t wf_launch_extend_t(const DevScene &S, const WfState &W, const WfLaunchConfig &C, int cur, cudaStream_t st) {
    const size_t smem = wf_trace_smem(0, kAccel, C.threads_extend);
    const int a = C.fetch_steps, b = C.fetch_min_idle;
    if (C.lean_extend) wf_extend_kernel<kAccel, kLeanBlocks><<<C.blocks_extend, C.threads_extend, smem, st>>>(S, W, cur, a, b);
    else wf_extend_kernel<kAccel, kBlocks><<<C.blocks_extend, C.threads_extend, smem, st>>>(S, W, cur, a, b);
    return cudaGetLastError();
}
template <int kAccel>
cudaError_t wf_launch_shadow_t(const DevScene &S, const WfState &W, const WfLaunchConfig &C, cudaStream_t st) {
    const size_t smem = wf_trace_smem(2, kAccel, C.threads_shadow);
    const int a = C.fetch_steps_shadow, b = C.fetch_min_idle_shadow;
    if (C.lean_shadow) wf_shadow_kernel<kAccel, kLeanBlocks><<<C.blocks_shadow, C.threads_shadow, smem, st>>>(S, W, a, b);
    else wf_shadow_kernel<kAccel, kBlocks><<<C.blocks_shadow, C.threads_shadow, smem, st>>>(S, W, a, b);
    return cudaGetLastError();
}
// which: 0 extend, 2 shadow; lean: the kLeanBlocks register budget
template <int kAccel>
int wf_trace_occupancy_t(int which, int threads, bool lean) {
    int n = 0;
    const size_t smem = wf_trace_smem(which, kAccel, threads);
    if (which == 0) {
        if (lean) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wf_extend_kernel<kAccel, kLeanBlocks>, threads, smem);
        else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wf_extend_kernel<kAccel, kBlocks>, threads, smem);
    } else {
        if (lean) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wf_shadow_kernel<kAccel, kLeanBlocks>, threads, smem);
        else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wf_shadow_kernel<kAccel, kBlocks>, threads, smem);
    }
    return n;
}

}  // namespace hk
