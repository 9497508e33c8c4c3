// Traversal of the 8-wide tree by warps that share their triangle tests, for
// kernels that trace a queue of rays: the wavefront's extend and shadow kernels
// and the ray queries.
//
// The 8-wide tree is walked by warps whose lanes hold one ray each and share
// one queue of triangle tests (trace_queue8): a step visits one node per lane,
// the triangles that the visits hit are appended to a 128-entry ring in shared
// memory as (triangle, owner lane), and a batch of 32 is tested, one triangle
// per lane, whenever 32 are pending.  The kernels are bound by instruction
// issue (76-80% of the slots) with the ALU pipe beside it (60-63%: the node
// test's byte permutes, min / max and compares run there at half rate), not by
// DRAM (under 15%), so what counts is warp instructions per ray.  A lane that tests its own
// triangles keeps the warp for as many rounds as the largest leaf group with
// the other lanes idle (13 active lanes per instruction); testing each step's
// triangles at once, shared out over the lanes, fills half of a round (14
// triangles on average) and pays for numbering triangles and finding owners in
// every round.  1024^2 x 32 spp, ns per ray when the ring was brought in, before
// the steps whose figures stand below (now 0.222 and 0.244 ns on the 64-sphere
// scene, 128 spp), own / shared out at once / ring:
// 64-sphere scene (1.3M triangles) shadow 0.319 / 0.280 / 0.245, closest hit
// 0.466 / 0.413 / 0.266; glass sphere (0.33M) shadow 0.485 / 0.391 / 0.324,
// closest hit 0.549 / 0.473 / 0.307; Cornell box (36 triangles, two visits a
// ray) shadow 0.124 / 0.129 / 0.120, closest hit 0.161 / 0.174 / 0.134.
#pragma once
#include "hk_traverse.cuh"

namespace hk {

constexpr unsigned kClaim8 = 32;       // rays that a warp claims at once
// Pending triangle tests per warp (a power of two, at least 2 x 32).  A step of
// a small scene queues a hundred (Cornell box: 3 per ray and visit), which a
// ring of 64 takes in passes; 256 take L1 from the nodes of large ones (whole
// render with 64 / 128 / 256, ms: Cornell box 29.3 / 28.2 / 28.0, 64-sphere scene
// 66.3 / 66.1 / 66.2, glass sphere 52.3 / 52.1 / 52.2).
constexpr unsigned kTriRing = 128;
constexpr unsigned kTriOwnerShift = kLeafCountShift;   // scenes hold fewer than 2^27 triangles: the owner lane sits above
constexpr uint32_t kTriMask = (1u << kTriOwnerShift) - 1u;

// Range of a queue's rays: any; [kRayEps, 1 - kRayEps], a segment between two
// points (the wavefront's shadow rays); from at least 0 on (its closest-hit
// rays).  Where a range starts at 0 the planes are formed with saturating FMAs,
// which clamp the near ones for nothing, instead of a max per child on the ALU
// pipe that bounds the walk; a segment's far planes are clamped the same way,
// and a strict comparison rejects boxes behind it or beyond it (both planes
// saturate to the same end; a box of zero thickness keeps the slack apart).
// Closest-hit distances are scaled by 2^-60, exactly, to stay below 1: the
// build's largest nodes are 2^46 across, and the least plane steps of scenes
// from 2^-46 on stay normal floats.  Shadow rays 0.244 -> 0.238 ns, closest-hit
// rays 0.266 -> 0.265 ns (64-sphere scene).
constexpr int kRangeAny = 0, kRangeUnit = 1, kRangeWave = 2;
constexpr float kNodeScale = 8.673617379884035e-19f;   // 2^-60

__device__ __forceinline__ float fma_sat(float a, float b, float c) {
    float r;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// A ray's constants of the node test.
struct NodeRay {
    V3 o;
    V3 i;                // 1 / d
    float tmin, tmax;    // tmax with the same slack
    uint32_t oct;        // slot_order of the ray | its octant << 5
};

template <bool kAnyHit, int kForm>
__device__ __forceinline__ void node_ray_begin(NodeRay &q, const Ray &ray) {
    q.o = ray.o;
    // |1/d| <= 1e20 keeps 2^23 steps of up to 2^38 (the largest step the build emits) finite
    const float tiny = 1e-20f, slack = 1.00000024f;
    const V3 d = ray.d;
    const V3 dd = v3(fabsf(d.x) < tiny ? copysignf(tiny, d.x) : d.x, fabsf(d.y) < tiny ? copysignf(tiny, d.y) : d.y,
                     fabsf(d.z) < tiny ? copysignf(tiny, d.z) : d.z);
    const V3 i = v3(1.0f / dd.x, 1.0f / dd.y, 1.0f / dd.z);
    q.i = i;
    const uint32_t oct = (i.x < 0.0f ? 1u : 0u) | (i.y < 0.0f ? 2u : 0u) | (i.z < 0.0f ? 4u : 0u);
    q.oct = slot_order(kAnyHit ? 7u ^ oct : oct) | oct << 5;
    q.tmin = ray.tmin;
    q.tmax = ray.tmax * slack + 1e-30f;
    if (kForm == kRangeWave) {
        q.i = q.i * kNodeScale;
        q.tmax = q.tmax * kNodeScale;
    }
}

// Children are visited from the highest nibble slot ^ ko down: near first for closest hits.  Any-hit
// rays go far first: they start on a surface whose own neighbourhood fills the
// near boxes without occluding, and what occludes them does so as well met last
// (visits and ns per shadow ray, near / far first: 64-sphere scene 9.95 / 9.54,
// 0.232 / 0.227; glass sphere 9.65 / 7.28, 0.309 / 0.261).
// Intersect the 8 children of a node (hk_bvh.h): its node group and triangle
// group (first triangle, hit triangle bits), and its slot word.  A hit child is
// one predicated or; with a meta byte per slot, shifted to its place for each
// child, and one queue entry per turn of the loop instead of one leaf, closest-
// hit rays took 0.272 ns instead of 0.258 and shadow rays 0.232 instead of 0.221
// (64-sphere scene; glass sphere 0.311 / 0.297 and 0.288 / 0.275, Cornell box
// 0.136 / 0.128 and 0.128 / 0.123).
template <int kForm>
__device__ __forceinline__ void visit8(const DevScene &S, uint32_t child, const NodeRay &q, uint2 &ng, uint2 &tg,
                                       uint32_t &slots) {
    const uint4 *np = S.wnodes + 5 * (size_t)child;
    const uint4 n0 = ldg4u(np), n1 = ldg4u(np + 1), n2 = ldg4u(np + 2), n3 = ldg4u(np + 3), n4 = ldg4u(np + 4);
    const uint32_t oct = q.oct >> 5;
    // plane step and offset per axis of the near (x) and far (y) planes; offsets
    // are shifted by -2^23 steps (qbyte_biased).  The far planes' constants are
    // scaled by 1 + 2^-22 (two ulps): the slack that keeps boxes of zero
    // thickness costs nothing per child.
    const float sx = __uint_as_float((n0.w << 23) & 0x7f800000u), sy = __uint_as_float((n0.w << 15) & 0x7f800000u),
                sz = __uint_as_float((n0.w << 7) & 0x7f800000u);
    const float px = __uint_as_float(n0.x) - q.o.x, py = __uint_as_float(n0.y) - q.o.y, pz = __uint_as_float(n0.z) - q.o.z;
    const float slack = 1.00000024f;
    const V3 f = q.i * slack;
    // a segment's distances count from its least one, where its planes saturate
    auto off = [&](float p, float i) { return kForm == kRangeUnit ? __fmaf_rn(p, i, -kRayEps) : p * i; };
    const float2 ax = make_float2(sx * q.i.x, sx * f.x), ay = make_float2(sy * q.i.y, sy * f.y),
                 az = make_float2(sz * q.i.z, sz * f.z);
    const float2 bx = make_float2(__fmaf_rn(-8388608.0f, ax.x, off(px, q.i.x)), __fmaf_rn(-8388608.0f, ax.y, off(px, f.x)));
    const float2 by = make_float2(__fmaf_rn(-8388608.0f, ay.x, off(py, q.i.y)), __fmaf_rn(-8388608.0f, ay.y, off(py, f.y)));
    const float2 bz = make_float2(__fmaf_rn(-8388608.0f, az.x, off(pz, q.i.z)), __fmaf_rn(-8388608.0f, az.y, off(pz, f.z)));
    // near / far planes per axis (lo planes first for a positive direction)
    const uint32_t nx0 = oct & 1u ? n3.z : n2.x, nx1 = oct & 1u ? n3.w : n2.y;
    const uint32_t fx0 = oct & 1u ? n2.x : n3.z, fx1 = oct & 1u ? n2.y : n3.w;
    const uint32_t ny0 = oct & 2u ? n4.x : n2.z, ny1 = oct & 2u ? n4.y : n2.w;
    const uint32_t fy0 = oct & 2u ? n2.z : n4.x, fy1 = oct & 2u ? n2.w : n4.y;
    const uint32_t nz0 = oct & 4u ? n4.z : n3.x, nz1 = oct & 4u ? n4.w : n3.y;
    const uint32_t fz0 = oct & 4u ? n3.x : n4.z, fz1 = oct & 4u ? n3.y : n4.w;
    uint32_t hits = 0;
    constexpr bool kUnit = kForm == kRangeUnit;
    const float t0 = kUnit ? kRayEps : q.tmin, t1 = kUnit ? (1.0f - kRayEps) * 1.00000024f : q.tmax;
    auto test_child = [&](auto kk, uint32_t xn, uint32_t xf, uint32_t yn, uint32_t yf, uint32_t zn, uint32_t zf) {
        constexpr int c = decltype(kk)::value, k = c & 3;
        if constexpr (kForm != kRangeAny) {
            const float2 tx = make_float2(fma_sat(qbyte_biased<k>(xn), ax.x, bx.x), fma_sat(qbyte_biased<k>(xf), ax.y, bx.y));
            const float2 ty = make_float2(fma_sat(qbyte_biased<k>(yn), ay.x, by.x), fma_sat(qbyte_biased<k>(yf), ay.y, by.y));
            const float2 tz = make_float2(fma_sat(qbyte_biased<k>(zn), az.x, bz.x), fma_sat(qbyte_biased<k>(zf), az.y, bz.y));
            const float tn = fmax3f(tx.x, ty.x, tz.x);
            const float tf3 = fmin3f(tx.y, ty.y, tz.y);
            const float tf = kUnit ? tf3 : fminf(tf3, t1);
            if (tn < tf) hits |= 0xfu << (4 * c);
            return;
        }
        const float2 tx = make_float2(__fmaf_rn(qbyte_biased<k>(xn), ax.x, bx.x), __fmaf_rn(qbyte_biased<k>(xf), ax.y, bx.y));
        const float2 ty = make_float2(__fmaf_rn(qbyte_biased<k>(yn), ay.x, by.x), __fmaf_rn(qbyte_biased<k>(yf), ay.y, by.y));
        const float2 tz = make_float2(__fmaf_rn(qbyte_biased<k>(zn), az.x, bz.x), __fmaf_rn(qbyte_biased<k>(zf), az.y, bz.y));
        const float tn = fmax3f(tx.x, ty.x, fmaxf(tz.x, t0));
        const float tf = fmin3f(tx.y, ty.y, fminf(tz.y, t1));
        if (tn <= tf) hits |= 0xfu << (4 * c);
    };
    test_child(std::integral_constant<int, 0>{}, nx0, fx0, ny0, fy0, nz0, fz0);
    test_child(std::integral_constant<int, 1>{}, nx0, fx0, ny0, fy0, nz0, fz0);
    test_child(std::integral_constant<int, 2>{}, nx0, fx0, ny0, fy0, nz0, fz0);
    test_child(std::integral_constant<int, 3>{}, nx0, fx0, ny0, fy0, nz0, fz0);
    test_child(std::integral_constant<int, 4>{}, nx1, fx1, ny1, fy1, nz1, fz1);
    test_child(std::integral_constant<int, 5>{}, nx1, fx1, ny1, fy1, nz1, fz1);
    test_child(std::integral_constant<int, 6>{}, nx1, fx1, ny1, fy1, nz1, fz1);
    test_child(std::integral_constant<int, 7>{}, nx1, fx1, ny1, fy1, nz1, fz1);
    slots = n1.z;
    ng = node_group(n1.x, slots, hits & slots, q.oct);
    tg = make_uint2(n1.y, hits & slots & kSlotTris);
}

// Shared memory of one warp of the 8-wide traversal kernels: the lanes' rays as
// the triangle test reads them (two float4 each), the short stacks (kShStack
// entries of 32 lanes), the ring; for closest-hit rays also the lanes' hits so
// far (t, u, v, triangle) and their tmax.  One base address per warp and
// constant offsets from it keep the addresses out of the registers.
template <bool kAnyHit>
struct WarpSmem {
    float4 rays[64];
    float4 hits[kAnyHit ? 1 : 32];
    uint2 stack[kShStack * 32];
    uint32_t ring[kTriRing];
    uint32_t tmaxs[kAnyHit ? 4 : 32];
};
constexpr size_t trace8_smem(bool any_hit, int threads) {
    return (size_t)(threads / 32) * (any_hit ? sizeof(WarpSmem<true>) : sizeof(WarpSmem<false>));
}

// Floats as unsigned integers in the floats' order, and back.
__device__ __forceinline__ uint32_t ordered_bits(float t) {
    const uint32_t b = __float_as_uint(t + 0.0f);   // -0 becomes +0
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_ordered(uint32_t b) {
    return __uint_as_float((b & 0x80000000u) ? (b & 0x7fffffffu) : ~b);
}

// Traverses n rays of a queue: lanes are refilled as in trace_queue
// (hk_traverse.cuh), node visits and triangle tests as described at the top.
// The warp starts with entries first to last - 1; claim(part), called by one
// lane, takes the next kClaim8 ones and returns the first of them (n or more:
// none are left); part is the warp's, kept from claim to claim.
// load(i) returns ray i; store(i, found, hit) consumes the result.  st counts
// the warp's visits and tests (the same in every lane).  kUnit: every ray's
// range is [kRayEps, 1 - kRayEps], a segment between two points.  A lane
// whose walk has ended, or whose any-hit ray is found occluded, waits until
// min_idle lanes are without a walk; the ring is then tested to its end, so no
// entry outlives its ray, the rays are stored and the lanes refilled.
//
// Closest-hit rays keep the hit that the serial loop keeps: tests run in the
// order a ray met its triangles (ring order, and lane order within a batch),
// a hit needs t <= tmax as of the batch's start, the least t of the batch
// wins, and of equal ones the latest.  That tmax shrinks a batch late only
// adds visits and tests, never a hit.
template <bool kAnyHit, int kForm, class Claim, class Load, class Store>
__device__ __forceinline__ void trace_queue8(const DevScene &S, unsigned first, unsigned last, unsigned n,
                                             unsigned part, int min_idle, Claim claim, Load load, Store store, TravStats &st) {
    constexpr bool kUnit = kForm == kRangeUnit;
    extern __shared__ float4 trace_smem[];
    const unsigned lane = threadIdx.x & 31u;
    WarpSmem<kAnyHit> &sm = reinterpret_cast<WarpSmem<kAnyHit> *>(trace_smem)[threadIdx.x >> 5];
    uint2 spill[kStackSize - kShStack];   // entries of the stack past the short one
    int sp = 0;

    NodeRay nr;
    uint2 ng = make_uint2(0u, 0u);
    int item = -1;
    bool live = false, found = false, exhausted = false;
    unsigned head = 0, pend = 0;              // warp-uniform: the ring's first entry and number of entries
    unsigned chunk_next = first, chunk_end = last;   // warp-uniform: unhanded entries of the warp's chunk

    // Test the ring's first cnt (at most 32) entries, one per lane.
    auto test_batch = [&](unsigned cnt) {
        __syncwarp();   // the entries and the rays are visible
        const bool act = lane < cnt;
        const uint32_t e = act ? sm.ring[(head + lane) & (kTriRing - 1u)] : 0u;
        const uint32_t own = e >> kTriOwnerShift, tri = e & kTriMask;
        head += cnt;
        pend -= cnt;
        if constexpr (kAnyHit) {
            bool hit = false;
            if (act) {
                const float4 *tp = S.tris + 3 * (size_t)tri;
                const float4 p0 = ldg4(tp), p1 = ldg4(tp + 1), p2 = ldg4(tp + 2);
                const float4 ro = sm.rays[2 * own], rd = sm.rays[2 * own + 1];
                hit = occludes_mt(xyz(ro), xyz(rd), xyz(p0), xyz(p1), xyz(p2), kUnit ? kRayEps : ro.w,
                                  kUnit ? 1.0f - kRayEps : rd.w);
            }
            const uint32_t occluded = __reduce_or_sync(0xffffffffu, hit ? 1u << own : 0u);
            if (occluded >> lane & 1u) {
                found = true;
                live = false;
            }
        } else {
            bool hit = false;
            float tt = 0.0f, uu = 0.0f, vv = 0.0f;
            if (act) {
                const float4 *tp = S.tris + 3 * (size_t)tri;
                const float4 p0 = ldg4(tp), p1 = ldg4(tp + 1), p2 = ldg4(tp + 2);
                const float4 ro = sm.rays[2 * own], rw = sm.rays[2 * own + 1];
                const uint32_t kp = __float_as_uint(rw.w);
                WatertightRay w;
                w.kx = (int)(kp & 3u);
                w.ky = (int)((kp >> 2) & 3u);
                w.kz = (int)((kp >> 4) & 3u);
                w.sx = rw.x;
                w.sy = rw.y;
                w.sz = rw.z;
                hit = intersect_watertight(w, xyz(ro), xyz(p0), xyz(p1), xyz(p2), ro.w, from_ordered(sm.tmaxs[own]), tt, uu,
                                           vv);
            }
            if (__any_sync(0xffffffffu, hit)) {   // also: every lane has read tmaxs
                const uint32_t key = ordered_bits(tt);
                if (hit) atomicMin(&sm.tmaxs[own], key);
                __syncwarp();
                const bool least = hit && sm.tmaxs[own] == key;
                if (least) sm.hits[own] = make_float4(tt, uu, vv, __uint_as_float(tri));
                __syncwarp();
                // equal least t of one ray in this batch: the latest stays
                const bool lost = least && __float_as_uint(sm.hits[own].w) != tri;
                if (__any_sync(0xffffffffu, lost)) {
                    for (unsigned l = 0; l < 32; ++l) {
                        if (lane == l && least) sm.hits[own] = make_float4(tt, uu, vv, __uint_as_float(tri));
                        __syncwarp();
                    }
                }
                nr.tmax = from_ordered(sm.tmaxs[lane]) * 1.00000024f + 1e-30f;
                if (kForm == kRangeWave) nr.tmax = nr.tmax * kNodeScale;
            }
        }
        __syncwarp();   // reads of the ring precede its next entries
    };

    for (;;) {
        // rays for idle lanes
        const unsigned want = __ballot_sync(0xffffffffu, item < 0 && !exhausted);
        const unsigned busy = __ballot_sync(0xffffffffu, item >= 0);
        if (want && (busy == 0u || __popc(want) >= min_idle)) {
            const unsigned k = __popc(want), rank = __popc(want & ((1u << lane) - 1u));
            const unsigned avail = chunk_end - chunk_next;
            unsigned idx = chunk_next + rank;
            if (k > avail) {   // warp-uniform: claim the next chunk for the lanes past the old one
                unsigned base = 0;
                if ((int)lane == __ffs(want) - 1) base = claim(part);
                base = __shfl_sync(0xffffffffu, base, __ffs(want) - 1);
                part = __shfl_sync(0xffffffffu, part, __ffs(want) - 1);
                if (rank >= avail) idx = base + (rank - avail);
                chunk_next = base + (k - avail);
                chunk_end = base + kClaim8;
            } else {
                chunk_next += k;
            }
            if (want >> lane & 1u) {
                if (idx < n) {
                    item = (int)idx;
                    const Ray r = load(item);
                    node_ray_begin<kAnyHit, kForm>(nr, r);
                    ng = root_group(S.nwnodes != 0, nr.oct);
                    sp = 0;
                    found = false;
                    live = S.nwnodes != 0;
                    sm.rays[2 * lane] = make_float4(r.o.x, r.o.y, r.o.z, r.tmin);
                    if constexpr (kAnyHit) {
                        sm.rays[2 * lane + 1] = make_float4(r.d.x, r.d.y, r.d.z, r.tmax);
                    } else {
                        const WatertightRay w = watertight_setup(r.d);
                        sm.rays[2 * lane + 1] = make_float4(
                            w.sx, w.sy, w.sz, __uint_as_float((uint32_t)w.kx | ((uint32_t)w.ky << 2) | ((uint32_t)w.kz << 4)));
                        sm.hits[lane].w = __int_as_float(-1);
                        sm.tmaxs[lane] = ordered_bits(r.tmax);
                    }
                } else {
                    exhausted = true;
                }
            }
        }
        if (!__any_sync(0xffffffffu, item >= 0)) break;
        const unsigned may = __ballot_sync(0xffffffffu, item >= 0 || !exhausted);
        unsigned walking = __ballot_sync(0xffffffffu, live);
        __syncwarp();
        for (;;) {
            uint2 tg = make_uint2(0u, 0u);
            uint32_t slots = 0;
            if (live) {   // one node per ray
                const uint32_t child = next_child(ng, nr.oct);
                if (ng.y & kSlotNode) {   // the tree's depth bound keeps sp below kStackSize
                    if (sp < kShStack) sm.stack[32 * sp + lane] = ng;
                    else if (sp < kStackSize) spill[sp - kShStack] = ng;
                    ++sp;
                }
                visit8<kForm>(S, child, nr, ng, tg, slots);
                if (!(ng.y & kSlotNode)) {
                    if (sp == 0) {
                        live = false;
                    } else {
                        --sp;
                        ng = sp < kShStack ? sm.stack[32 * sp + lane] : spill[sp - kShStack];
                    }
                }
            }
            const uint32_t cnt = __popc(tg.y);
            if (__any_sync(0xffffffffu, cnt != 0u)) {
                uint32_t incl = cnt;   // inclusive prefix of the counts in lane order
// shfl's own in-range predicate guards the addition
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                    asm volatile("{\n\t.reg .pred p;\n\t.reg .u32 v;\n\t"
                                 "shfl.sync.up.b32 v|p, %0, %1, 0, 0xffffffff;\n\t@p add.u32 %0, %0, v;\n\t}"
                                 : "+r"(incl) : "r"(o));
                const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
                st.tris += total;
                if (total <= kTriRing - pend) {
                    // leaf by leaf, from the highest slot down and the last position back: ring order is
                    // bit order (a hit leaf has all its triangles' bits set, so bit b & 3 counts them)
                    uint32_t at = head + pend + incl;
                    const uint32_t base = tg.x | (lane << kTriOwnerShift);
                    while (tg.y != 0u) {
                        const uint32_t b = 31u - __clz(tg.y), below = (1u << (b & 28u)) - 1u, leaf = b & 3u;
                        tg.y &= below;
                        at -= leaf;
                        const uint32_t e = base + __popc(slots & kSlotTris & below);
                        sm.ring[at & (kTriRing - 1u)] = e;
                        if (leaf > 1u) sm.ring[(at + 1u) & (kTriRing - 1u)] = e + 1u;
                        if (leaf > 2u) sm.ring[(at + 2u) & (kTriRing - 1u)] = e + 2u;
                    }
                    pend += total;
                    while (pend >= 32u) test_batch(32u);
                } else {   // more triangles than the ring has room for: in passes
                    uint32_t pos = incl - cnt, dealt = 0;
                    while (dealt < total) {
                        const uint32_t room = kTriRing - pend;
                        while (tg.y != 0u && pos < dealt + room) {
                            const uint32_t b = __ffs(tg.y) - 1;
                            tg.y &= tg.y - 1u;
                            sm.ring[(head + pend + (pos - dealt)) & (kTriRing - 1u)] = (tg.x + tri_offset(slots, b)) | (lane << kTriOwnerShift);
                            ++pos;
                        }
                        const uint32_t moved = min(total - dealt, room);
                        pend += moved;
                        dealt += moved;
                        while (pend >= 32u) test_batch(32u);
                    }
                }
            }
            // once min_idle of the lanes that could hold a ray walk none, end their rays and refill
            st.nodes += __popc(walking);
            walking = __ballot_sync(0xffffffffu, live);
            if (walking == 0u || __popc(may & ~walking) >= min_idle) break;
        }
        if (__any_sync(0xffffffffu, item >= 0 && !live)) {
            if (pend) test_batch(pend);   // fewer than 32 are left here
            if (item >= 0 && !live) {
                Hit h;
                h.t = h.u = h.v = 0.0f;
                h.tri = -1;
                if constexpr (!kAnyHit) {
                    const float4 r = sm.hits[lane];
                    h.t = r.x; h.u = r.y; h.v = r.z;
                    h.tri = __float_as_int(r.w);
                    found = h.tri >= 0;
                }
                store(item, found, h);
                item = -1;
            }
        }
        __syncwarp();   // every read of a lane's records precedes their replacement
    }
}

}  // namespace hk
