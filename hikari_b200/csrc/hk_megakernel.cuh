// The plain megakernel (the drop-in): PathMISIntegrator::Li per lane, persistent
// warps whose lanes take a new path as soon as theirs ends, samples splatted
// into the film with vector reductions.  Each instantiation (tree kind x
// texture lookups) is compiled in its own translation unit (hk_render_*.cu).
#pragma once
#include "hk_kernels.h"
#include "hk_shading.cuh"

namespace hk {

// ------------------------------------------------------------ integrator
struct PathCounters {
    uint32_t rays, shadow;
    TravStats trav;
};

// One path of a lane.  The BSDF record of a vertex stays here for the next one: where
// that hits an area light, its MIS weight asks for the previous BSDF's pdf
// of the sampled direction.  Taken at every vertex instead, the call cost 5 to 10% (Cornell
// box 423 -> 403 us at 2^14 paths, smooth materials 1076 -> 986).
struct Path {
    Pcg32 rng;
    Ray ray;          // the next ray to trace
    V3 L, beta;
    float px, py;     // film position
    float w_mats;     // MIS weight of an emitter hit, carried across vertices
    int depth;
    bool force_mats;  // the previous BSDF sample was EDiscrete
    int bsdf;         // the last shaded vertex's BSDF, its record and (a bumpMap or normalMap) its frames
    BRec rec;
};

// One vertex of PathMISIntegrator::Li (src/integrator/PathMISIntegrator.cpp:16-157):
// trace the path's ray, add the emission or the environment of what it meets,
// estimate direct light, sample the BSDF and leave the continuation ray in P.
// Returns false where the path has ended.  Every reference quirk is kept:
// Russian roulette p = 0.95 from depth rr_start (reference: every bounce), NEE
// over all emitters, MIS weight carried across bounces, unweighted environment
// on BSDF-sampled misses, the EDiscrete override and Eigen's |c| <= 1e-5 zero
// test on throughput and NEE values.  kTex: the scene has textured materials
// (texture lookups compiled in); the first hit's lookups filter with the
// camera ray's differentials, later hits have none (src/core/Intersection.cpp:35).
// bf: the frames of the last vertex whose BSDF is a bumpMap or normalMap (kTex only).
template <int kAccel, bool kTex>
__device__ __forceinline__ bool path_vertex(const DevScene &S, Path &P, BumpFrames &bf, int depth_max, int rr_start,
                                            PathCounters &pc) {
    Hit h;
    pc.rays++;
    if (!trace<kAccel, false>(S, P.ray, h, pc.trav)) {
        if (S.env_index >= 0 && (P.depth > 0 || !S.force_background)) P.L = P.L + P.beta * env_eval(S, P.ray.d);
        else if (P.depth == 0) P.L = ld3(S.background);
        return false;
    }
    Isect it;
    post_intersect(S, h, it);
    const DevMesh &m = S.meshes[it.mesh];
    const int bsdf = m.bsdf;
    if (m.emitter >= 0) {
        const DevAreaLight &AL = S.area_lights[__ldg(S.emitter_area + m.emitter)];
        ERec er;
        er.ref = P.ray.o; er.p = it.p; er.n = it.sh.n;
        V3 wi = er.p - er.ref; er.dist = norm(wi); er.wi = wi / er.dist;
        if (P.depth > 0) {
            if (P.force_mats) {
                P.w_mats = 1.0f;
            } else {
                const float plm = area_pdf(AL, er);
                float pbm;
                if constexpr (kTex) pbm = bsdf_pdf_b(S.bsdfs, P.bsdf, P.rec, bf);
                else pbm = bsdf_pdf_n(S.bsdfs, P.bsdf, P.rec);
                if (pbm + plm != 0.0f) P.w_mats = pbm / (pbm + plm);
            }
        }
        P.L = P.L + (P.beta * P.w_mats) * area_eval(AL, er);
    }
    float4 duv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float3 geo = make_float3(INFINITY, 0.0f, 0.0f);
    P.bsdf = bsdf;
    BRec &br = P.rec;
    if constexpr (kTex) {
        if (P.depth == 0 && S.ray_diff) {
            V3 rx, ry;
            camera_diff(S, S.cam, S.width, S.height, S.cam_aspect, P.px, P.py, rx, ry);
            duv = screen_partials(S, h, it, P.ray.o, rx, ry);
        }
        if (is_bump(S.bsdfs[bsdf])) bf = perturbed_frames(S, h, it, S.bsdfs[bsdf]);
        if (S.bsdfs[bsdf].geo_tex) geo = tex_geometry(S, h, it);
    }
    br.wi = to_local(it.sh, P.ray.d * -1.0f);
    br.eta = 0.0f;
    br.tu = it.u; br.tv = it.v; br.tex = kTex; br.duv = duv; br.geo = geo;
    for (int e = 0; e < S.nemitters; ++e) {
        ERec er;
        er.ref = it.p;
        er.dist = 0.0f;
        er.pdf = 0.0f;
        float u1 = P.rng.nextf();
        float ux = P.rng.nextf(), uy = P.rng.nextf();
        V3 ld = emitter_sample(S, e, er, ux, uy, u1);
        if (is_zero(ld)) continue;
        // the BSDF term first, the shadow ray only for a non-zero contribution
        // (an occluded ray adds nothing either way)
        br.wo = to_local(it.sh, er.wi);
        br.measure = kMeasureSolidAngle;
        const float pl = er.pdf;
        float pb;
        V3 f;
        if constexpr (kTex) {
            pb = bsdf_pdf_b(S.bsdfs, bsdf, br, bf);
            f = bsdf_eval_b(S.bsdfs, bsdf, br, bf);
        } else {
            pb = bsdf_pdf_n(S.bsdfs, bsdf, br);
            f = bsdf_eval_n(S.bsdfs, bsdf, br);
        }
        const float w = (pl + pb != 0.0f) ? pl / (pl + pb) : 1.0f;
        const float c = fabsf(br.wo.z);
        const V3 contrib = v3((((P.beta.x * f.x) * c) * ld.x) * w, (((P.beta.y * f.y) * c) * ld.y) * w,
                              (((P.beta.z * f.z) * c) * ld.z) * w);
        if (all_zero(contrib)) continue;
        Ray sr;
        sr.o = it.p; sr.d = er.p - it.p; sr.tmin = kRayEps; sr.tmax = 1.0f - kRayEps;
        Hit sh;
        pc.shadow++;
        if (!trace<kAccel, true>(S, sr, sh, pc.trav)) P.L = P.L + contrib;
    }
    br.wo = v3(0, 0, 0);
    br.measure = kMeasureUnknown;
    float sx = P.rng.nextf(), sy = P.rng.nextf();
    float u1 = needs_u1(S.bsdfs, bsdf) ? P.rng.nextf() : 0.0f;
    V3 F;
    if constexpr (kTex) F = bsdf_sample_b(S.bsdfs, bsdf, br, sx, sy, u1, bf);
    else F = bsdf_sample_n(S.bsdfs, bsdf, br, sx, sy, u1);
    P.beta = P.beta * F;
    if (is_zero(P.beta)) return false;
    P.force_mats = br.measure == kMeasureDiscrete;
    if (P.force_mats) P.w_mats = 1.0f;
    // Russian roulette (PathMISIntegrator.cpp:142-151) and the depth bound
    // before the continuation ray is traced: the reference traces first and
    // ends the path afterwards, discarding the hit; the trace draws no random
    // numbers, so the stream is consumed in the same order
    if (P.depth >= rr_start) {
        if (P.rng.nextf() < 0.95f) P.beta = P.beta * (1.0f / 0.95f);
        else return false;
    }
    ++P.depth;
    if (P.depth >= depth_max) return false;   // the next hit would not be shaded
    br.eta = 0.0f;
    P.ray.o = it.p;
    P.ray.d = to_world(it.sh, br.wo);
    P.ray.tmin = kRayEps;
    P.ray.tmax = __int_as_float(0x7f800000);
    return true;
}

// ------------------------------------------------------------ megakernel
// Paths are numbered sample by sample over the image, 16 x 16 tile by tile
// within a sample, and dealt to warps P.lanes at a time; a lane whose path has
// ended takes the next one at its warp's next vertex.  With a lane per pixel that
// ran its samples one after another, a warp waited at each sample for its
// longest path (roulette at p = 0.95: the longest of 32 has four times the
// mean's vertices), and a block for its slowest tile item.
//
// kRounds: the paths of a block start together.  A warp takes 32 new paths when its last
// one has ended, after a barrier of its block.  Where all paths are short there is
// little to wait for, and what a lane gains by going on alone it loses many times over: its warp's lanes are
// at different vertices, on different materials, and the SM's warps, at
// different places of a kernel that its instruction cache does not hold, fetch
// each other's code away.  Which kernel: render_grid (hk_host.cpp).
//
// Every warp starts with the chunk of its own number, so that the warps of an SM
// shade neighbouring pixels and share the instruction cache, which bounds this
// kernel (a warp runs the traversal and the BSDFs of its lanes one after another);
// claimed in order of arrival, smooth materials took 2510 instead of 2414 us at 2^16 paths.
// An ended path is splatted when its lane takes the next one, and where none is left all
// of a warp's together: at each path's own end the filter's taps ran once for every
// path length in the warp (Cornell box 378 -> 346 us at 2^14 paths, smooth
// materials 983 -> 905).
template <int kAccel, bool kTex, bool kRounds>
__global__ void __launch_bounds__(kRounds ? kRoundThreads : kRenderThreads, kRounds ? 1 : kRenderBlocks)
    render_pathmis_kernel(DevScene S, RenderLaunch P) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t pixels = (uint64_t)S.width * S.height, total = pixels * (uint64_t)P.spp;
    PathCounters pc{0, 0, TravStats()};
    uint32_t dropped = 0;
    Path p;
    BumpFrames bf;
    // few paths: fewer lanes of each warp take part, so that more warps do
    bool have = false, ended = false, exhausted = lane >= P.lanes;
    // warp-uniform: undealt paths of the warp's chunk; the paths of all warps' first chunks
    uint64_t next = (blockIdx.x * (uint64_t)(blockDim.x / 32) + threadIdx.x / 32) * P.lanes, end = next + P.lanes;
    const uint64_t first = gridDim.x * (uint64_t)(blockDim.x / 32) * P.lanes;
    auto splat = [&] {
        if (is_valid(p.L)) splat_film(S, P.film, (int)S.width, (int)S.height, p.px, p.py, p.L);
        else ++dropped;   // ImageBlock::Put (src/core/Block.cpp:97)
    };
    for (;;) {
        unsigned want = __ballot_sync(0xffffffffu, !have && !exhausted);
        if constexpr (kRounds)
            if (__any_sync(0xffffffffu, have)) want = 0u;
        if (want) {
            // warps that find no path leave, and the barrier with them
            if constexpr (kRounds) __syncthreads();
            const unsigned k = __popc(want), rank = __popc(want & ((1u << lane) - 1u));
            const unsigned avail = (unsigned)(end - next);
            uint64_t i = next + rank;
            if (k > avail) {   // claim the next chunk for the lanes past the old one
                unsigned long long base = 0;
                if ((int)lane == __ffs(want) - 1) base = atomicAdd(P.work_counter, (unsigned long long)P.lanes);
                base = __shfl_sync(0xffffffffu, base, __ffs(want) - 1) + first;
                if (rank >= avail) i = base + (rank - avail);
                next = base + (k - avail);
                end = base + P.lanes;
            } else {
                next += k;
            }
            if (want >> lane & 1u) {
                if (i < total) {
                    if (ended) splat();
                    ended = false;
                    // path -> sample, row of tiles, tile, pixel (tiles at the right and bottom edges are smaller)
                    const uint64_t s = i / pixels;
                    const uint32_t q = (uint32_t)(i - s * pixels);
                    const uint32_t strip = q / (S.width * kTile), r = q - strip * (S.width * kTile);
                    const uint32_t th = min((uint32_t)kTile, S.height - strip * kTile);
                    const uint32_t tx = r / (th * kTile), t = r - tx * (th * kTile);
                    const uint32_t tw = min((uint32_t)kTile, S.width - tx * kTile);
                    const uint32_t x = tx * kTile + t % tw, y = strip * kTile + t / tw;
                    p.rng.seed(mix_seed(P.seed, (uint64_t)P.sample_offset + s),
                               (uint64_t)y * S.width + x + (uint64_t)P.image_index * S.width * S.height);
                    p.px = (float)x + p.rng.nextf();
                    p.py = (float)y + p.rng.nextf();
                    p.ray = camera_ray(S, p.px, p.py);
                    p.L = v3(0, 0, 0);
                    p.beta = v3(1, 1, 1);
                    p.w_mats = 1.0f;
                    p.depth = 0;
                    p.force_mats = false;
                    have = true;
                } else {
                    exhausted = true;
                }
            }
        }
        if (!__any_sync(0xffffffffu, have)) break;
        if (have && !(P.depth > 0 && path_vertex<kAccel, kTex>(S, p, bf, P.depth, P.rr_start, pc))) {
            have = false;
            ended = true;
        }
    }
    if (ended) splat();
    // per-warp counter reduction (64-bit: node counts of one thread can pass 2^32)
    unsigned long long r = pc.rays, sh = pc.shadow, dr = dropped, nv = pc.trav.nodes, nt = pc.trav.tris;
    for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_down_sync(0xffffffffu, r, o);
        sh += __shfl_down_sync(0xffffffffu, sh, o);
        dr += __shfl_down_sync(0xffffffffu, dr, o);
        nv += __shfl_down_sync(0xffffffffu, nv, o);
        nt += __shfl_down_sync(0xffffffffu, nt, o);
    }
    if ((threadIdx.x & 31) == 0 && P.counters) {
        atomicAdd(P.counters + 0, r);
        atomicAdd(P.counters + 1, sh);
        atomicAdd(P.counters + 2, dr);
        atomicAdd(P.counters + 3, nv);
        atomicAdd(P.counters + 4, nt);
    }
}

template <int kAccel, bool kTex, bool kRounds>
cudaError_t launch_render_t(const DevScene &S, const RenderLaunch &P, int grid, cudaStream_t st) {
    render_pathmis_kernel<kAccel, kTex, kRounds><<<grid, P.threads, 0, st>>>(S, P);
    return cudaGetLastError();
}
template <int kAccel, bool kTex>
int render_occupancy_t() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, render_pathmis_kernel<kAccel, kTex, false>, kRenderThreads, 0);
    return n;
}

}  // namespace hk
