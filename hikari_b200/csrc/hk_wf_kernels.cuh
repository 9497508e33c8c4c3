// Wavefront pathMIS kernels shared by the wavefront translation units: the
// queue helpers and the shade kernel template.  hk_wavefront.cu holds regen
// and the launches of an iteration; hk_wf_trace_*.cu instantiate the traversal kernels
// (hk_wf_trace.cuh) per tree kind and hk_wf_shade_*.cu the shade kernels per
// queue, so they compile in parallel.
#pragma once
#include "hk_shading.cuh"
#include "hk_wavefront.h"

namespace hk {

// ------------------------------------------------------------ helpers
__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

// Warp-aggregated append to a queue counter: one atomic per warp.
__device__ __forceinline__ unsigned warp_append(unsigned *counter) {
    unsigned mask = __activemask();
    int leader = __ffs(mask) - 1;
    unsigned rank = __popc(mask & ((1u << lane_id()) - 1u));
    unsigned base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(counter, (unsigned)__popc(mask));
    base = __shfl_sync(mask, base, leader);
    return base + rank;
}
// Append grouped by key (lanes with equal keys share one atomic).
__device__ __forceinline__ unsigned warp_append_keyed(unsigned *counters, int key) {
    unsigned mask = __activemask();
    unsigned peers = __match_any_sync(mask, key);
    int leader = __ffs(peers) - 1;
    unsigned rank = __popc(peers & ((1u << lane_id()) - 1u));
    unsigned base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(counters + key, (unsigned)__popc(peers));
    base = __shfl_sync(peers, base, leader);
    return base + rank;
}
__device__ __forceinline__ float4 f4(V3 v, float w) { return make_float4(v.x, v.y, v.z, w); }

// PerspectiveCamera::SampleRay (src/camera/PerspectiveCamera.cpp:71) at the
// job's resolution and pose; field of view and clip planes are the scene's.
__device__ __forceinline__ Ray camera_ray_job(const DevScene &S, const WfJob &J, float px, float py) {
    const float *M = J.cam;
    float u = px * (1.0f / (float)J.width), v = py * (1.0f / (float)J.height);
    V3 np = v3(S.cam_near * (1.0f - 2.0f * u) / S.cam_cot, S.cam_near * (1.0f - 2.0f * v) / (J.cam_aspect * S.cam_cot),
               S.cam_near);
    V3 dir = normalize(np);
    float invz = 1.0f / dir.z;
    Ray r;
    r.o = v3(M[3], M[7], M[11]);
    r.d = v3(M[0] * dir.x + M[1] * dir.y + M[2] * dir.z, M[4] * dir.x + M[5] * dir.y + M[6] * dir.z,
             M[8] * dir.x + M[9] * dir.y + M[10] * dir.z);
    r.tmin = S.cam_near * invz;
    r.tmax = S.cam_far * invz;
    return r;
}

// Piece of the current plan that holds plan item w (pieces are sorted by plan_begin).
__device__ __forceinline__ int find_seg(const WfState &W, uint64_t w, int nseg) {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (W.segs[mid].plan_begin <= w) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// ------------------------------------------------------------ shade
__device__ __forceinline__ void finish(const WfState &W, int slot) { W.fq[warp_append(&W.ctr->fq_count)] = slot; }

// Register budgets: the kernels of untextured materials are held to three
// resident blocks of 256 threads (80 registers; left to itself the compiler
// takes up to 122 for the coating, and the shade phase of the 64-sphere scene
// 16.1 instead of 15.4 ms), the others, whose calls need 128 anyway, are left
// alone.  kLeanShade asks for four blocks (64 registers, more spilling: 15.0 ms
// there, but 13.2 instead of 12.5 on the Cornell box); only queues 0-5 have it.
constexpr int kLeanShade = 4;
template <int kType, int kMinBlocks = kType < kWfTexturedQueue0 ? 3 : 0>
__global__ void __launch_bounds__(256, kMinBlocks) wf_shade_kernel(DevScene S, WfState W, int nxt) {
    const int n = (int)W.ctr->sq_count[kType];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int slot = W.sq[kType][i];
        const float4 o4 = W.ray_o[slot], d4 = W.ray_d[slot];
        const V3 ro = v3(o4.x, o4.y, o4.z), rd = v3(d4.x, d4.y, d4.z);
        float4 b4 = W.beta[slot];
        V3 beta = v3(b4.x, b4.y, b4.z);
        float w_mats = b4.w;
        float4 p4 = W.pix[slot];
        const uint32_t dflags = (uint32_t)__float_as_int(p4.w);
        int depth = (int)(dflags & 0xffffu);
        uint32_t flags = dflags >> 16;
        const WfJob &J = W.jobs[__float_as_int(p4.z)];
        // radiance terms go to the path's accumulator with vector reductions
        // (as the unoccluded next-event terms do): shade neither reads nor
        // rewrites it
        if constexpr (kType == 0) {
            // miss (PathMISIntegrator.cpp:35-66); a new path's accumulator is zero
            V3 Le = v3(0, 0, 0);
            if (S.env_index >= 0 && (depth > 0 || !S.force_background)) Le = beta * env_eval(S, rd);
            else if (depth == 0) Le = ld3(S.background);
            if (!all_zero(Le)) red_add_v4(W.lacc + slot, Le.x, Le.y, Le.z, 0.0f);
            finish(W, slot);
            continue;
        } else {
            // queue -> top-level BSDF type (run-time dispatch for the generic
            // queue) and whether texture lookups are compiled in
            // kBumpQ: a bumpMap / normalMap over the type BT (the
            // records move through the perturbed frame, the nested BSDF is
            // evaluated with its type compiled in)
            constexpr bool kBumpQ = kType >= kWfBumpQueue0 && kType != kWfGenericQueue;
            constexpr int BT = kType == kWfGenericQueue
                                   ? -1
                                   : (kBumpQ ? kType - kWfBumpQueue0
                                             : (kType >= kWfTexturedQueue0 ? kType - kWfTexturedQueue0 : kType - 1));
            constexpr bool kTexQ = kType >= kWfTexturedQueue0;
            uint4 rs = W.rng[slot];
            Pcg32 rng;
            rng.state = (uint64_t)rs.x | ((uint64_t)rs.y << 32);
            rng.inc = (uint64_t)rs.z | ((uint64_t)rs.w << 32);
            float4 h4 = W.hit[slot];
            Hit h;
            h.t = h4.x; h.u = h4.y; h.v = h4.z; h.tri = __float_as_int(h4.w);
            Isect it;
            post_intersect(S, h, it);
            const DevMesh &m = S.meshes[it.mesh];
            const int bsdf = m.bsdf;
            if (m.emitter >= 0) {
                const DevAreaLight &AL = S.area_lights[__ldg(S.emitter_area + m.emitter)];
                ERec er;
                er.ref = ro; er.p = it.p; er.n = it.sh.n;
                V3 wi = er.p - er.ref; er.dist = norm(wi); er.wi = wi / er.dist;
                if (depth > 0) {
                    // MIS weight of the BSDF-sampled hit (PathMISIntegrator.cpp:122-140)
                    if (flags & kWfFlagForceMats) {
                        w_mats = 1.0f;
                    } else {
                        const float plm = area_pdf(AL, er);
                        const float pbm = W.prev_pdf[slot];   // taken when the BSDF sampled
                        if (pbm + plm != 0.0f) w_mats = pbm / (pbm + plm);
                    }
                }
                const V3 Le = (beta * w_mats) * area_eval(AL, er);
                if (!all_zero(Le)) red_add_v4(W.lacc + slot, Le.x, Le.y, Le.z, 0.0f);
            }
            // screen-space partials of a camera ray's first hit (textured
            // materials only: Intersection::ComputeScreenSpacePartial)
            float4 duv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            BumpFrames bf;   // a bumpMap / normalMap vertex's frames (the bump queues and the generic one)
            if constexpr (BT < 0) {
                if (is_bump(S.bsdfs[bsdf])) bf = perturbed_frames(S, h, it, S.bsdfs[bsdf]);
            } else if constexpr (kBumpQ) {
                bf = perturbed_frames(S, h, it, S.bsdfs[bsdf]);
            }
            // what wireframe / curvature textures read at this vertex
            float3 geo = make_float3(INFINITY, 0.0f, 0.0f);
            if constexpr (kTexQ) {
                if (depth == 0 && S.ray_diff) {
                    V3 rx, ry;
                    camera_diff(S, J.cam, J.width, J.height, J.cam_aspect, p4.x, p4.y, rx, ry);
                    duv = screen_partials(S, h, it, ro, rx, ry);
                }
                if (S.bsdfs[bsdf].geo_tex) geo = tex_geometry(S, h, it);
            }
            // next-event estimation over every emitter (PathMISIntegrator.cpp:83-109)
            const V3 wi_local = to_local(it.sh, rd * -1.0f);
            BsdfVertex bv;   // the typed kernels'
            TexVals looked;  // the typed kernels' of textured materials
            if constexpr (BT >= 0) {
                BRec br;
                br.wi = wi_local;
                br.tex = kTexQ;
                br.tu = it.u;
                br.tv = it.v;
                if constexpr (kTexQ) {
                    br.duv = duv;
                    br.geo = geo;
                    tex_look_up<BT>(S.bsdfs, kBumpQ ? S.bsdfs[bsdf].nested : bsdf, br, looked);
                    br.looked = &looked;
                }
                if constexpr (kBumpQ) bv = bump_vertex_t<BT>(S.bsdfs, bsdf, br, bf);
                else bv = bsdf_vertex_t<BT>(S.bsdfs, bsdf, br);
            }
            for (int e = 0; e < S.nemitters; ++e) {
                ERec er;
                er.ref = it.p;
                er.dist = 0.0f;
                er.pdf = 0.0f;
                float u1 = rng.nextf();
                float ux = rng.nextf(), uy = rng.nextf();
                V3 ld = emitter_sample(S, e, er, ux, uy, u1);
                if (is_zero(ld)) continue;
                BRec br;
                br.wi = wi_local;
                br.wo = to_local(it.sh, er.wi);
                br.measure = kMeasureSolidAngle;
                br.eta = 0.0f;
                br.tex = kTexQ;   // lookups only in the kernels of textured materials
                br.tu = it.u;
                br.tv = it.v;
                if constexpr (kTexQ) {   // unread where lookups are compiled out
                    br.duv = duv;
                    br.geo = geo;
                    if constexpr (BT >= 0) br.looked = &looked;
                }
                float pl = er.pdf;
                float pb;
                V3 f;
                if constexpr (BT < 0) {
                    pb = bsdf_pdf_b(S.bsdfs, bsdf, br, bf);
                    f = bsdf_eval_b(S.bsdfs, bsdf, br, bf);
                } else if constexpr (kBumpQ) {
                    f = bump_eval_pdf_t<BT>(S.bsdfs, bsdf, br, bf, bv, pb);
                } else {
                    f = bsdf_eval_pdf_t<BT>(S.bsdfs, bsdf, br, bv, pb);
                }
                float w = (pl + pb != 0.0f) ? pl / (pl + pb) : 1.0f;
                float c = fabsf(br.wo.z);
                V3 contrib = v3((((beta.x * f.x) * c) * ld.x) * w, (((beta.y * f.y) * c) * ld.y) * w,
                                (((beta.z * f.z) * c) * ld.z) * w);
                if (all_zero(contrib)) continue;   // adds nothing whether occluded or not
                unsigned q = warp_append(&W.ctr->shadow_count);
                if (q < (unsigned)W.max_shadow) {
                    W.sh_o[q] = f4(it.p, __int_as_float(slot));
                    W.sh_d[q] = f4(er.p - it.p, 0.0f);
                    W.sh_c[q] = f4(contrib, 0.0f);
                }
            }
            // BSDF sampling (PathMISIntegrator.cpp:111-120)
            BRec br;
            br.wi = wi_local;
            br.wo = v3(0, 0, 0);
            br.measure = kMeasureUnknown;
            br.eta = 0.0f;
            br.tex = kTexQ;
            br.tu = it.u;
            br.tv = it.v;
            if constexpr (kTexQ) {
                br.duv = duv;
                br.geo = geo;
                if constexpr (BT >= 0) br.looked = &looked;
            }
            float sx = rng.nextf(), sy = rng.nextf();
            float u1 = needs_u1(S.bsdfs, bsdf) ? rng.nextf() : 0.0f;
            V3 F;
            float spdf = 0.0f;   // the typed kernels' pdf of the sampled direction
            if constexpr (BT < 0) F = bsdf_sample_b(S.bsdfs, bsdf, br, sx, sy, u1, bf);
            else if constexpr (kBumpQ) F = bump_sample_t<BT>(S.bsdfs, bsdf, br, sx, sy, u1, bf);
            else F = bsdf_sample_pdf_t<BT>(S.bsdfs, bsdf, br, sx, sy, u1, bv, S.narea != 0, spdf);
            beta = beta * F;
            bool alive = !is_zero(beta);
            if (alive) {
                flags = (br.measure == kMeasureDiscrete) ? kWfFlagForceMats : 0u;
                if (flags) w_mats = 1.0f;
                // Russian roulette (PathMISIntegrator.cpp:142-151)
                if (depth >= J.rr_start) {
                    if (rng.nextf() < 0.95f) beta = beta * (1.0f / 0.95f);
                    else alive = false;
                }
                ++depth;
                if (depth >= J.depth) alive = false;   // the next hit would not be shaded
            }
            if (!alive) {
                finish(W, slot);
                continue;
            }
            W.ray_o[slot] = f4(it.p, kRayEps);
            W.ray_d[slot] = f4(to_world(it.sh, br.wo), __int_as_float(0x7f800000));
            W.beta[slot] = f4(beta, w_mats);
            W.pix[slot] = make_float4(p4.x, p4.y, p4.z, __int_as_float((int)((flags << 16) | (uint32_t)depth)));
            // the MIS weight at an emitter hit next needs this BSDF's pdf of the
            // sampled direction (PathMISIntegrator.cpp:128).  It is taken here,
            // where the BSDF's type is compiled in, and kept as one float: an
            // emitter hit that evaluated the previous vertex's BSDF instead
            // dispatched over every type at run time, which put the calls and
            // registers of all of them into each of these kernels (128
            // registers, 22% of the warps resident; now 77-97) and the previous
            // record's two directions into the path state.  Shade phase of the
            // 64-sphere scene, 1024^2 x 32 spp: 27.9 -> 22.8 ms.
            if (S.narea && !(flags & kWfFlagForceMats)) {
                BRec pr = br;
                pr.eta = 0.0f;
                if constexpr (BT < 0) W.prev_pdf[slot] = bsdf_pdf_b(S.bsdfs, bsdf, pr, bf);
                else if constexpr (kBumpQ) W.prev_pdf[slot] = bump_pdf_t<BT>(S.bsdfs, bsdf, pr, bf);
                else W.prev_pdf[slot] = spdf;
            }
            W.rng[slot] = make_uint4((uint32_t)rng.state, (uint32_t)(rng.state >> 32), (uint32_t)rng.inc,
                                     (uint32_t)(rng.inc >> 32));
            W.eq[nxt][warp_append(&W.ctr->eq_count[nxt])] = slot;
        }
    }
}

// ------------------------------------------------------------ launchers
template <int kType>
cudaError_t wf_launch_shade_t(const DevScene &S, const WfState &W, const WfLaunchConfig &C, int nxt, cudaStream_t st) {
    if constexpr (kType <= 5) {
        if (C.lean_shade) {
            wf_shade_kernel<kType, kLeanShade><<<C.blocks_shade[kType], C.threads_shade, 0, st>>>(S, W, nxt);
            return cudaGetLastError();
        }
    }
    wf_shade_kernel<kType><<<C.blocks_shade[kType], C.threads_shade, 0, st>>>(S, W, nxt);
    return cudaGetLastError();
}
template <int kType>
int wf_shade_occupancy_t(int threads, bool lean) {
    int n = 0;
    if constexpr (kType <= 5) {
        if (lean) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wf_shade_kernel<kType, kLeanShade>, threads, 0);
            return n;
        }
    }
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wf_shade_kernel<kType>, threads, 0);
    return n;
}

}  // namespace hk
