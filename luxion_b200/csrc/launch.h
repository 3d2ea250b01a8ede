// launch.h -- host-callable launchers of the kernels (defined in trace.cu, shade.cu, sort.cu).
#pragma once

#include <algorithm>
#include <cuda_runtime.h>
#include "device_scene.h"

namespace lux {

constexpr int kTraceBlock = 128;
constexpr int kShadeBlock = 384;  // three blocks per SM; both measured, see k_shade
constexpr int kShadeOcc = 3;
constexpr int kCameraBlock = 128;
constexpr int kPathBlock = 128;  // three blocks per SM; see k_paths
constexpr int kPathOcc = 3;

// persistent traversal grid of `mode` for the two-level or the single-level layout
int trace_grid_blocks(int mode, bool single = false);
int shade_grid_blocks();

// persistent trace of bounce `bounce`: mode 0 radiance (queues shadow rays when nee != 0:
// 1 DL, 2 env), 1 DL shadow rays, 2 env occlusion rays
// grid > 0 overrides the persistent grid (blocks), for the job engine's autotuner
cudaError_t launch_trace(const DevScene& S, const DevWave& W, int bounce, int mode, int nee, cudaStream_t st,
                         int grid = 0);
// the same over several (lane, bounce) segments of waves in flight, in one launch
cudaError_t launch_trace_segs(const DevScene& S, const DevWave& W, const Segs& G, int mode, int nee, cudaStream_t st,
                              int grid = 0);
// trace caller rays (device buffers), n * 8 floats -> n * 5 words; fetch is a zeroed int, err a
// zeroed int (page-locked, so that the host can read it, or on the device): nonzero after a
// traversal stack overflow
cudaError_t launch_trace_ext(const DevScene& S, const DevWave& W, const float* rays, uint32_t* hits, int n, int mode,
                             int iter, int* fetch, int* err, cudaStream_t st);

// the fixed scratch of lux_trace_rays_static on `device` (trace_static.cu), which must be the
// current device on the first call for it: cursor and error word, then LUX_TRACE_STATIC_MAX_RAYS rays
// and hits
struct TraceScratch {
    int* cursor;  // cursor[1]: the error word where there is no page-locked one
    float* rays;
    uint32_t* hits;
};
cudaError_t trace_static_scratch(int device, TraceScratch& out);
size_t trace_static_scratch_bytes();

// camera rays for paths [0, n) of a wave in lane `lane` (+ NEE sample of bounce 0), queue 0 =
// identity; wave_iter: the wave's first iteration and sample count (device)
cudaError_t launch_camera(const DevScene& S, const DevWave& W, const DevOptions& O, const DevCamera& cam, int n,
                          int lane, const int* wave_iter, cudaStream_t st);
// the paths of the segments to their end (`depth` bounces; job engine: each job's trace depth) in
// one launch, paths.cu. It does nothing when they are more than `limit`; when it does run, later
// wavefront launches of those lanes find them finished.
cudaError_t launch_paths(const DevScene& S, const DevWave& W, const DevOptions& O, const Segs& G, int depth, int limit,
                         cudaStream_t st);
int path_grid_blocks();
// Waves of at most kWholePerLane paths per lane of the whole-path kernel's grid (284k on 148 SMs)
// run in it from the camera on. Above, the wavefront's full warps win. One sample, depth 8, both light
// samplings (the box: emitters), ms a wave as a wavefront and whole (medians of 41):
//   paths            150k        200k        250k        284k        350k        450k
//   Cornell box   0.60 0.41   0.61 0.48   0.66 0.55   0.66 0.60   0.71 0.71   0.81 0.88
//   50k triangles 0.72 0.46   0.79 0.54   0.83 0.63   0.85 0.68   0.90 0.79   0.98 0.96
//   400k          1.16 0.81   1.25 0.97   1.34 1.11   1.38 1.24   1.44 1.42   1.56 1.72
//   1M            1.48 1.29   1.60 1.56   1.70 1.84   1.75 2.03   1.92 2.42   2.18 2.99
// At 284k it still wins by 9 to 20 % up to 400k triangles and loses 16 % at 1M, where the two meet at
// 210k; without light sampling the figures stand alike (284k: 0.35 0.34, 0.51 0.43, 0.89 0.81, 1.08 1.30).
// A larger wave hands over before one of the bounces 1 to kTailLast once at most kTailPerLane paths per
// lane are left (114k) and two bounces or more are to come: a frame of 2.07M paths, 1M triangles, depth 12
// took 4.18 ms instead of 5.34 when it came, while handing over at twice that many took 5 to 20 %
// longer in 700k-triangle scenes. An attempt that finds more paths left costs an empty launch.
constexpr int kWholePerLane = 5;
constexpr int kTailPerLane = 2;
constexpr int kTailLast = 3;
inline int path_limit(int per_lane) { return per_lane * path_grid_blocks() * kPathBlock; }
inline int tail_attempts(int depth) { return std::max(0, std::min(kTailLast, depth - 2)); }
inline bool try_tail(int bounce, int depth) { return bounce >= 1 && bounce <= kTailLast && bounce + 2 <= depth; }

// shade bounce `bounce` (depth = bounce + 1 after the increment of src/pathtrace.cu:264)
cudaError_t launch_shade(const DevScene& S, const DevWave& W, const DevOptions& O, int bounce, int compact,
                         cudaStream_t st);
// the same over several (lane, bounce) segments of waves in flight, in one launch
cudaError_t launch_shade_segs(const DevScene& S, const DevWave& W, const DevOptions& O, const Segs& G,
                              cudaStream_t st);
// job engine: camera rays of the wave's segments (W.segs, counts read from W.wave_hdr) into lane
// `lane`, and the per-job accumulation of that lane's segments in sample order
cudaError_t launch_camera_jobs(const DevWave& W, const DevOptions& O, int max_paths, int lane, cudaStream_t st);
cudaError_t launch_accumulate_jobs(const DevWave& W, int compensated, int lane, cudaStream_t st);
// image[p] (+comp) += radiance of every sample of the wave in lane `lane`, in sample order
cudaError_t launch_accumulate(const DevWave& W, int lane, float* image, float* comp, int nsamples, int compensated,
                              cudaStream_t st);
cudaError_t launch_tonemap(const float* image, uint8_t* rgba, int npix, float iter, int color_mode, cudaStream_t st);

// n texel channels at src (device) of format fmt (LUX_TEX_RGBA8/16/32F) to float (c / 255,
// c / 65535) or, with to_half, to binary16 at dst (device); texconv.cu
cudaError_t launch_convert_texels(const void* src, int fmt, int to_half, void* dst, size_t n, cudaStream_t st);

// Morton keys of the bounce's queue and a stable LSD radix sort of the queue by key
cudaError_t launch_morton_sort(const DevScene& S, DevWave& W, int bounce, void* temp, size_t temp_bytes,
                               cudaStream_t st);
size_t morton_sort_temp_bytes(int max_paths);
constexpr int kSortLaunches = 5;  // of one launch_morton_sort
// before the first bounce of a wave: the sort's counters start at zero
cudaError_t clear_sort_counters(void* temp, cudaStream_t st);
cudaError_t launch_morton_ext(const DevScene& S, const float* rays, uint32_t* keys, int n, cudaStream_t st);

// kernel-level parity entry points (device buffers)
cudaError_t launch_shade_ext(const DevScene& S, const DevOptions& O, float* paths, const uint32_t* hits, int n,
                             int iter, int depth, int compact, int* survivors, int* n_out, cudaStream_t st);
cudaError_t launch_light_ext(const DevScene& S, const DevOptions& O, int iter, int depth, const int* pixels, int n,
                             float* out, cudaStream_t st);
cudaError_t launch_rng_ext(int iter, int index, int depth, int n, float* out, cudaStream_t st);
cudaError_t launch_tex_ext(unsigned long long tex, const float* uv, int n, float* out, cudaStream_t st);

}  // namespace lux
