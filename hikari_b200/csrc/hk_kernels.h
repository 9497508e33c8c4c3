// Launch interface between the host library (hk_host.cpp) and the kernels.
#pragma once
#include <cuda_runtime.h>

#include "hk_device.h"

namespace hk {

constexpr int kTile = 16;             // the megakernel numbers paths tile by tile: 16 x 16 pixels
constexpr int kRenderThreads = 128;
// Resident blocks per SM that the megakernel's register budget allows: two, the
// 198 registers that it asks for.  With 128 for four blocks it spills 480 B, and
// more warps per scheduler only take turns in the instruction cache (us at 2 / 3 / 4
// blocks: Cornell box 346 / 354 / 384 at 2^14 paths, 892 / 903 / 1067 at 2^17;
// smooth materials 905 / 922 / 981 and 4025 / 4194 / 4583; a mesh 787 / 812 / 874 at 2^16).
// Many paths of the smallest scenes would want four (Cornell box 8.9 / 7.1 ms with two / four
// at 2^21 paths, smooth materials 52.8 / 52.8, 64 spheres 81.7 / 86.4), but so many come here only from
// captures and hk_render_image_static: the wavefront renders them otherwise.
constexpr int kRenderBlocks = 2;
constexpr int kRoundThreads = 256;    // the most threads of a block that deals its paths in rounds

struct RenderLaunch {
    float *film;                          // (H+2B) x (W+2B) x 4 floats, accumulated
    unsigned long long *work_counter;     // paths dealt past the warps' first chunks; zeroed before launch
    unsigned long long *counters;         // [rays, shadow rays, dropped samples, node visits, triangle tests]
    uint64_t seed;
    int spp;                              // samples per pixel in this launch
    int sample_offset;                    // first sample index (progressive rendering)
    int depth, rr_start;
    int image_index;
    unsigned lanes;                       // lanes of each warp that take paths (1 to 32)
    unsigned threads;                     // of a block
    bool rounds;                          // a block's paths start together
};

// Static scratch of hk_render_image_static: a 256-byte header ([0] work
// counter, [1..5] ray/sample counters) followed by the film accumulator, sized
// for films of up to 512 x 512 pixels with a filter border of up to 4.
constexpr size_t kStaticHeaderWords = 32;
constexpr size_t kStaticFilmFloats = 4ull * 520 * 520;
constexpr size_t kStaticScratchWords = kStaticHeaderWords + kStaticFilmFloats / 2;
constexpr int kStaticMaxDevices = 64;
// Device address of the static scratch on the current device (looked up once
// per device with cudaGetSymbolAddress, then cached).
cudaError_t static_render_scratch(void **out);

cudaError_t launch_render(const DevScene &S, const RenderLaunch &P, int grid, cudaStream_t st);
cudaError_t launch_resolve(const float *film, float *rgb, int W, int H, int B, cudaStream_t st);
cudaError_t launch_trace(const DevScene &S, uint64_t n, const float *rays, int32_t *tri, float *t, float *u, float *v,
                         int any_hit, unsigned long long *visits, cudaStream_t st);
// type: top-level BSDF type of id `bsdf` (HK_BSDF_*)
cudaError_t launch_bsdf_batch(const DevScene &S, int bsdf, int type, uint64_t n, const float *wi, const float *u2,
                              const float *u1, const float *wo, const float *uv, const float *duv, float *s_wo, float *s_w,
                              float *s_pdf, int32_t *s_m, float *e_rgb, float *p_pdf, cudaStream_t st);
cudaError_t launch_texture_eval(const DevScene &S, const DevTexture *T, int tex, uint64_t n, const float *uv,
                                const float *duv, float *out, cudaStream_t st);
cudaError_t launch_emitter_sample(const DevScene &S, int e, uint64_t n, const float *in, float *out, cudaStream_t st);
cudaError_t launch_camera_rays(const DevScene &S, uint64_t n, const float *pos, float *out, cudaStream_t st);
cudaError_t launch_env_eval(const DevScene &S, uint64_t n, const float *wi, float *out, float *pdf, cudaStream_t st);
int render_occupancy(int accel, bool textured);

// Per-instantiation launchers behind the functions above, each compiled in its
// own translation unit (megakernel: hk_render_*.cu; BSDF batch: hk_batch_*.cu).
template <int kAccel, bool kTex, bool kRounds>
cudaError_t launch_render_t(const DevScene &S, const RenderLaunch &P, int grid, cudaStream_t st);
template <int kAccel, bool kTex>
int render_occupancy_t();
template <int BT>
cudaError_t launch_bsdf_batch_t(const DevScene &S, int bsdf, uint64_t n, const float *wi, const float *u2, const float *u1,
                                const float *wo, const float *uv, const float *duv, float *s_wo, float *s_w, float *s_pdf,
                                int32_t *s_m, float *e_rgb, float *p_pdf, int grid, cudaStream_t st);

}  // namespace hk
