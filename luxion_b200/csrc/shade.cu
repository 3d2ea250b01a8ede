// shade.cu -- camera generation, shading, light sampling, accumulation and tonemapping.
//
// Compiled with --fmad=false: every float multiply and add is rounded on its own, in the
// order the reference writes it, so these kernels agree with the reference's host build
// except where CUDA's transcendental functions differ from the host's by an ulp.
//
//   k_camera      generateRayFromCamera (src/kernels/generate_ray_from_camera.cu:8-39) and the
//                 bounce-0 sampleDirectLight (src/kernels/sample_direct_light.cu:9-101)
//   k_shade       shadePath (src/kernels/shade_path.cu:94-364) with the uber-shader
//                 (src/shaders/cook_torrance.cu), material queries (src/material_queries.cu),
//                 throughput/RR (src/update_throughput_materials.cu:23-67), the warp-aggregated
//                 survivor append (:355-363) and, fused behind it, the next bounce's
//                 sampleDirectLight: that kernel seeds its RNG with the pre-increment depth,
//                 which equals the post-increment depth this shade just used
//                 (src/pathtrace.cu:193,264,299), so the stream is the same.
//   k_accumulate  finalGather (src/kernels/image_kernels.cu:49-60), samples added in order
//   k_tonemap     sendImageToPBO (src/kernels/image_kernels.cu:6-46, src/tonemapping.cu)

#include "shade_core.cuh"

#include <algorithm>
#include <map>
#include <mutex>

namespace lux {
namespace {

// The fields shade_one reads on entry.
LUX_DI PathState load_path(const DevWave& W, int pid) {
    float4 b = ld_stream(&W.s1[pid]), c = ld_stream(&W.s2[pid]);
    PathState p;
    p.d = mk(b.x, b.y, b.z);
    p.spec = (__float_as_int(b.w) & 1) != 0;
    p.thr = mk(c.x, c.y, c.z);
    p.pixel = __float_as_int(c.w);
    p.iter = __float_as_int(ld_stream(&W.s3[pid]).w);
    return p;
}

// Pixel of the t-th path of a sample: 8x4 pixel tiles in row-major tile order, so that a warp's
// 32 camera rays (and, through the order-preserving survivor queue, their later bounces) start
// from one compact patch of the image rather than a 32x1 strip. Pixels outside the whole tiles
// (a right margin of W % 8 columns and a bottom margin of H % 4 rows) follow in row order.
LUX_HDI int tiled_pixel(int t, int W, int H) {
    const int W8 = W - W % 8, H4 = H - H % 4;
    const int a = W8 * H4;
    if (t < a) {
        const int tile = t >> 5, k = t & 31, tpr = W8 >> 3;
        return ((tile / tpr) * 4 + (k >> 3)) * W + (tile % tpr) * 8 + (k & 7);
    }
    t -= a;
    const int rw = W - W8;
    if (t < rw * H4) return (t / rw) * W + W8 + t % rw;
    t -= rw * H4;
    return (H4 + t / W) * W + t % W;
}

// Paths [0, n) of a wave in lane `lane`: path ids and queue slots from lane * lane_stride on.
__global__ void __launch_bounds__(kCameraBlock, 16) k_camera(DevScene S, DevWave W, DevOptions O, DevCamera C, int n,
                                                            int lane, const int* wave_iter) {
    const int first_iter = wave_iter[0];
    const bool nee = O.dl || O.env;
    const int base = lane * W.lane_stride;
    for (int local = blockIdx.x * blockDim.x + threadIdx.x; local < n; local += gridDim.x * blockDim.x) {
        const int pid = base + local;
        int s = local / W.npix, index = tiled_pixel(local - s * W.npix, C.width, C.height);
        int iter = first_iter + s;
        int x = index % C.width, y = index / C.width;
        Rng rng = Rng::seeded(iter, index, O.trace_depth);
        float x1 = rng.u01() - 0.5f;
        float x2 = rng.u01() - 0.5f;
        float pX = (float(x) + x1 + 0.5f) - float(C.width) * 0.5f;
        float pY = (float(y) + x2 + 0.5f) - float(C.height) * 0.5f;
        f3 view = ld3(C.view), right = ld3(C.right), up = ld3(C.up);
        f3 d = normalize(view - (right * C.pixel_length[0] * pX) - (up * C.pixel_length[1] * pY));
        st_stream(&W.s0[pid], make_float4(C.pos[0], C.pos[1], C.pos[2], -1.0f));
        st_stream(&W.s1[pid], make_float4(d.x, d.y, d.z, __int_as_float(0)));
        st_stream(&W.s2[pid], make_float4(1.0f, 1.0f, 1.0f, __int_as_float(index)));
        st_stream(&W.s3[pid], make_float4(0.0f, 0.0f, 0.0f, __int_as_float(iter)));
        if (nee) {
            f3 ed;
            f3 dl = light_sample(S, O, iter, index, 0, ed, !O.env);
            f3 v = O.env ? ed : dl;
            st_stream(&W.s4[pid], make_float4(v.x, v.y, v.z, 0.0f));
        }
        st_stream(&W.queue[0][pid], pid);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) (W.ctr + lane)->count[0] = n;
}

// JOBS: the shared wavefront of the job engine; each path shades against its job's scene
// (lights, environment) and stops compacting at its job's trace depth.
// The code of one path is some 5000 instructions with little reuse, far more than an SM's
// instruction caches hold, so warps that run at their own pace starve on instruction fetch (with
// 16 free-running 128-thread blocks per SM: 14.0 of 31 stall cycles per issue, bounce 1 of the
// 1M-triangle 1080p scene). Here the warps of a block walk the phases of shade_one in step and
// share each fetched line: 0.3 stall cycles, and what is left is waiting for loads (12 of 24).
// Shade time of that scene's 16-spp step: 12.95 ms free-running; in step with 128-thread blocks
// 13.7, 256 x 8 per SM 13.0, 512 x 4 12.2, 512 x 3 (40 registers) 11.0, 384 x 3 (56) 10.7,
// 256 x 4 (64) 11.0, 512 x 2 (64) 11.8, 1024 x 1 11.9. Values that wait for a later phase do so in
// shared memory (35 KB a block) instead of being spilled: 10.7 -> 10.5, and a path whose radiance
// does not change is not written; 384 x 4 (40 registers) 10.7, 512 x 3 10.8, 512 x 2 10.6. Prefetching
// the next item's state to L2 or L1 took 11.2.
// G: the (lane, bounce) segments of waves in flight this launch shades; the paths of segment k
// are its lane's queue at its bounce, and its survivors go to the lane's next queue.
template <bool JOBS, bool MATDBG, int NEE>
__global__ void __launch_bounds__(kShadeBlock, kShadeOcc) k_shade(const __grid_constant__ DevScene S0, DevWave W, DevOptions O,
                                                       const __grid_constant__ Segs G) {
    __shared__ int seg_first[kMaxSegs + 1];
    __shared__ float parked[kParked][kShadeBlock];
    if (threadIdx.x == 0) {
        int t = 0;
        seg_first[0] = 0;
        for (int k = 0; k < kMaxSegs; ++k) {
            if (k < G.n && *(volatile const int*)&(W.ctr + G.lane[k])->finished == 0)
                t += *(volatile const int*)&(W.ctr + G.lane[k])->count[G.bounce[k]];
            seg_first[k + 1] = t;
        }
    }
    __syncthreads();
    const int n = seg_first[kMaxSegs];
    const bool nee = nee_dl<NEE>(O) || nee_env<NEE>(O);
    const int lane = threadIdx.x & 31;
    // A launch of fewer paths than the grid has threads gives every block its share, in whole
    // warps, so that they reach all SMs.
    const int chunk = min(kShadeBlock, ((n + int(gridDim.x) - 1) / int(gridDim.x) + 31) & ~31);
    const int stride = int(gridDim.x) * chunk;
    // uniform trip count across the block: the phases run in step
    for (int base = blockIdx.x * chunk; base < n; base += stride) {
        const int item = base + threadIdx.x;
        const bool on = int(threadIdx.x) < chunk && item < n;
        bool alive = false;
        int pid = 0, k = 0, depth = 0, job_compact = 0;
        const DevScene* sp = &S0;
        PathState p{};
        float4 h = make_float4(-1.0f, 0.0f, 0.0f, __int_as_float(-1));
        int prim = 0, si = -1, spr = -1;
        float sh_t = -1.0f, su = 0.0f, sv = 0.0f;
        if (on) {
            while (k + 1 < G.n && item >= seg_first[k + 1]) ++k;
            const int slot = G.lane[k] * W.lane_stride + (item - seg_first[k]);
            depth = G.bounce[k] + 1;
            pid = ld_stream(&W.queue[G.bounce[k] & 1][slot]);
            job_compact = G.compact[k];
            if (JOBS) {
                const DevJob& J = W.jobs[W.path_job[pid]];
                sp = &W.scenes[J.scene];
                job_compact = depth < J.trace_depth;
            }
            p = load_path(W, pid);
            h = ld_stream(&W.hit[slot]);
            prim = ld_stream(&W.hit_prim[slot]);
            if (nee && __float_as_int(h.w) >= 0) {
                float4 sh = ld_stream(&W.sh_hit[slot]);
                sh_t = sh.x;
                if (!nee_env<NEE>(O)) {
                    su = sh.y;
                    sv = sh.z;
                    si = __float_as_int(sh.w);
                    spr = ld_stream(&W.sh_prim[slot]);
                }
            }
        }
        const DevScene& S = *sp;
        SharedPark K{&parked[0][threadIdx.x]};
        alive = shade_one<MATDBG, NEE, false, !MATDBG>(S, O, depth, p, WavePathIn{W, pid}, K, h.x, __float_as_int(h.w), prim,
                                                      h.y, h.z, sh_t, si, spr, su, sv, on) &&
                job_compact;
        if (alive) {
            st_stream(&W.s0[pid], make_float4(p.o.x, p.o.y, p.o.z, p.last_pdf));
            st_stream(&W.s1[pid], make_float4(p.d.x, p.d.y, p.d.z, __int_as_float(p.spec ? 1 : 0)));
            st_stream(&W.s2[pid], make_float4(p.thr.x, p.thr.y, p.thr.z, K.get(kPkPixel)));
            if (nee) {
                f3 ed;
                f3 dl = light_sample<NEE>(S, O, __float_as_int(K.get(kPkIter)), __float_as_int(K.get(kPkPixel)), depth, ed, !nee_env<NEE>(O));
                f3 v = nee_env<NEE>(O) ? ed : dl;
                st_stream(&W.s4[pid], make_float4(v.x, v.y, v.z, 0.0f));
            }
        }
        // warp-aggregated survivor append (src/kernels/shade_path.cu:355-363), one atomic per
        // segment present in the warp
        const unsigned am = __ballot_sync(0xffffffffu, alive);
        if (am) {
            const unsigned grp = __match_any_sync(0xffffffffu, alive ? k : -1);
            if (alive) {
                const int lk = G.lane[k], nb = G.bounce[k] + 1;
                const int leader = __ffs(grp) - 1;
                int b = 0;
                if (lane == leader) b = atomicAdd(&(W.ctr + lk)->count[nb], __popc(grp));
                b = __shfl_sync(grp, b, leader);
                st_stream(&W.queue[nb & 1][lk * W.lane_stride + b + __popc(grp & ((1u << lane) - 1u))], pid);
            }
        }
    }
}

// Path t of every sample of the wave is pixel tiled_pixel(t) (k_camera).
__global__ void k_accumulate(const float4* __restrict__ s3, float* __restrict__ image, float* __restrict__ comp,
                             int width, int height, int nsamples, int compensated) {
    const int npix = width * height;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < npix; t += gridDim.x * blockDim.x) {
        const int p = tiled_pixel(t, width, height);
        float r = image[p * 3], g = image[p * 3 + 1], b = image[p * 3 + 2];
        if (compensated) {
            // Kahan-compensated running sum (precision form)
            float cr = comp[p * 3], cg = comp[p * 3 + 1], cb = comp[p * 3 + 2];
            for (int s = 0; s < nsamples; ++s) {
                float4 c = ld_stream(&s3[size_t(s) * npix + t]);
                float yr = c.x - cr, tr = r + yr;
                cr = (tr - r) - yr;
                r = tr;
                float yg = c.y - cg, tg = g + yg;
                cg = (tg - g) - yg;
                g = tg;
                float yb = c.z - cb, tb = b + yb;
                cb = (tb - b) - yb;
                b = tb;
            }
            comp[p * 3] = cr;
            comp[p * 3 + 1] = cg;
            comp[p * 3 + 2] = cb;
        } else {
            for (int s = 0; s < nsamples; ++s) {
                float4 c = ld_stream(&s3[size_t(s) * npix + t]);
                r += c.x;
                g += c.y;
                b += c.z;
            }
        }
        image[p * 3] = r;
        image[p * 3 + 1] = g;
        image[p * 3 + 2] = b;
    }
}

// Segment of the wave holding index v of a prefix array (path0 or pix0), by binary search
// over the segment table staged in shared memory.
template <int FIELD>
LUX_DI int find_segment(const DevSegment* segs, int nsegs, int v) {
    int lo = 0, hi = nsegs - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        int start = FIELD == 0 ? segs[mid].path0 : segs[mid].pix0;
        if (start <= v) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Camera rays of a job-engine wave (generateRayFromCamera, src/kernels/generate_ray_from_camera.cu:8-39,
// per job): path pid belongs to the segment covering it; its sample s and pixel index give the
// job-local iteration and pixel that seed the RNG, exactly as a single-job render would.
// W.segs and W.wave_hdr are the wave's own tables; its paths go to lane `lane`.
__global__ void __launch_bounds__(kCameraBlock) k_camera_jobs(DevWave W, DevOptions O, int lane) {
    __shared__ DevSegment segs[kMaxSegments];
    const int nsegs = W.wave_hdr[0], n = min(W.wave_hdr[1], W.lane_stride);
    for (int k = threadIdx.x; k < nsegs; k += blockDim.x) segs[k] = W.segs[k];
    __syncthreads();
    const bool nee = O.dl || O.env;
    const int base = lane * W.lane_stride;
    for (int local = blockIdx.x * blockDim.x + threadIdx.x; local < n; local += gridDim.x * blockDim.x) {
        const int pid = base + local;
        const DevSegment& g = segs[find_segment<0>(segs, nsegs, local)];
        const DevJob& J = W.jobs[g.job];
        int off = local - g.path0;
        int s = off / J.npix, index = off - s * J.npix;
        int iter = J.first_iter + g.sample0 + s;
        int x = index % J.width, y = index / J.width;
        Rng rng = Rng::seeded(iter, index, J.trace_depth);
        float x1 = rng.u01() - 0.5f;
        float x2 = rng.u01() - 0.5f;
        float pX = (float(x) + x1 + 0.5f) - float(J.width) * 0.5f;
        float pY = (float(y) + x2 + 0.5f) - float(J.height) * 0.5f;
        f3 view = ld3(J.view), right = ld3(J.right), up = ld3(J.up);
        f3 d = normalize(view - (right * J.pixel_length[0] * pX) - (up * J.pixel_length[1] * pY));
        W.s0[pid] = make_float4(J.pos[0], J.pos[1], J.pos[2], -1.0f);
        W.s1[pid] = make_float4(d.x, d.y, d.z, __int_as_float(0));
        W.s2[pid] = make_float4(1.0f, 1.0f, 1.0f, __int_as_float(index));
        W.s3[pid] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(iter));
        if (nee) {
            f3 ed;
            f3 dl = light_sample(W.scenes[J.scene], O, iter, index, 0, ed, !O.env);
            f3 v = O.env ? ed : dl;
            W.s4[pid] = make_float4(v.x, v.y, v.z, 0.0f);
        }
        W.path_job[pid] = g.job;
        W.queue[0][pid] = pid;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) (W.ctr + lane)->count[0] = n;
}

// image[job pixel] (+comp) += radiance of the segment's samples, in sample order, so that a
// job's image is the same bit for bit however its samples were split into waves.
__global__ void k_accumulate_jobs(DevWave W, int compensated, int lane) {
    __shared__ DevSegment segs[kMaxSegments];
    const int nsegs = W.wave_hdr[0], total = W.wave_hdr[2];
    const float4* __restrict__ s3 = W.s3 + size_t(lane) * W.lane_stride;
    for (int k = threadIdx.x; k < nsegs; k += blockDim.x) segs[k] = W.segs[k];
    __syncthreads();
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < total; q += gridDim.x * blockDim.x) {
        const DevSegment& g = segs[find_segment<1>(segs, nsegs, q)];
        const DevJob& J = W.jobs[g.job];
        const int p = q - g.pix0;
        const size_t o = size_t(p) * 3;
        float* __restrict__ image = J.image;
        float* __restrict__ comp = J.comp;
        float r = image[o], gr = image[o + 1], b = image[o + 2];
        if (compensated) {
            float cr = comp[o], cg = comp[o + 1], cb = comp[o + 2];
            for (int s = 0; s < g.nsamples; ++s) {
                float4 c = ld_stream(&s3[size_t(g.path0) + size_t(s) * J.npix + p]);
                float yr = c.x - cr, tr = r + yr;
                cr = (tr - r) - yr;
                r = tr;
                float yg = c.y - cg, tg = gr + yg;
                cg = (tg - gr) - yg;
                gr = tg;
                float yb = c.z - cb, tb = b + yb;
                cb = (tb - b) - yb;
                b = tb;
            }
            comp[o] = cr;
            comp[o + 1] = cg;
            comp[o + 2] = cb;
        } else {
            for (int s = 0; s < g.nsamples; ++s) {
                float4 c = ld_stream(&s3[size_t(g.path0) + size_t(s) * J.npix + p]);
                r += c.x;
                gr += c.y;
                b += c.z;
            }
        }
        image[o] = r;
        image[o + 1] = gr;
        image[o + 2] = b;
    }
}

LUX_DI f3 aces(f3 x) {  // src/tonemapping.cu:3-11
    const float a = 2.51f, b = 0.03f, c = 2.43f, d = 0.59f, e = 0.14f;
    f3 num = x * (a * x + mk(b, b, b));
    f3 den = x * (c * x + mk(d, d, d)) + mk(e, e, e);
    return mk(gclamp(num.x / den.x, 0.0f, 1.0f), gclamp(num.y / den.y, 0.0f, 1.0f), gclamp(num.z / den.z, 0.0f, 1.0f));
}
LUX_DI f3 agx(f3 v) {  // src/tonemapping.cu:13-30
    float c[3] = {v.x, v.y, v.z};
    for (int i = 0; i < 3; ++i) {
        c[i] = gmax(c[i], 1e-6f);
        c[i] = (log2f(c[i]) + 10.0f) / 16.0f;
        c[i] = gclamp(c[i], 0.0f, 1.0f);
        float x2 = c[i] * c[i], x4 = x2 * x2;
        c[i] = 15.5f * x4 * c[i] - 40.14f * x4 + 31.96f * x2 * c[i] - 6.86f * x2 + 0.429f * c[i] + 0.0322f;
    }
    float r = c[0] * 1.1968790f - c[1] * 0.0980208f - c[2] * 0.0990297f;
    float g = -c[0] * 0.0528968f + c[1] * 1.1519031f - c[2] * 0.0989611f;
    float b = -c[0] * 0.0529716f - c[1] * 0.0980434f + c[2] * 1.1510736f;
    return mk(gclamp(r, 0.0f, 1.0f), gclamp(g, 0.0f, 1.0f), gclamp(b, 0.0f, 1.0f));
}

__global__ void k_tonemap(const float* __restrict__ image, uchar4* __restrict__ out, int npix, float iter, int mode) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
        float inv = __frcp_rn(iter);
        f3 p = mk(image[i * 3], image[i * 3 + 1], image[i * 3 + 2]) * inv;
        if (mode >= 0) {  // mode < 0: material debug view, shown without tone map or gamma
            if (mode == 0) p = mk(p.x / (p.x + 1.0f), p.y / (p.y + 1.0f), p.z / (p.z + 1.0f));
            else if (mode == 1) p = agx(p);
            else p = aces(p);
            p = vpow(p, 0.45f);
        }
        out[i] = make_uchar4((unsigned char)gclampi(int(double(p.x) * 255.0), 0, 255),
                             (unsigned char)gclampi(int(double(p.y) * 255.0), 0, 255),
                             (unsigned char)gclampi(int(double(p.z) * 255.0), 0, 255), 0);
    }
}

// ---- kernel-level parity entry points ------------------------------------------------
// Path rows of 24 floats: origin 0-2, direction 3-5, radiance 6-8, throughput 9-11, DL point
// 12-14, env direction 15-17, pixel 18, killed 19, specular 20, pdf 21.
struct RowPathIn {
    float* f;
    bool env;
    LUX_DI f3 origin() const { return mk(f[0], f[1], f[2]); }
    LUX_DI float last_pdf() const { return f[21]; }
    LUX_DI f3 color0() const { return mk(f[6], f[7], f[8]); }
    LUX_DI f3 nee() const { return env ? mk(f[15], f[16], f[17]) : mk(f[12], f[13], f[14]); }
    LUX_DI void set_color(f3 c, int) const {
        f[6] = c.x;
        f[7] = c.y;
        f[8] = c.z;
    }
};

__global__ void k_shade_ext(DevScene S, DevOptions O, float* paths, const uint32_t* hits, int n, int iter, int depth,
                            int compact, int* survivors, int* n_out) {
    const int lane = threadIdx.x & 31;
    for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        int i = base + threadIdx.x;
        bool alive = false;
        if (i < n) {
            float* f = paths + size_t(i) * 24;
            PathState p;
            p.o = mk(f[0], f[1], f[2]);
            p.d = mk(f[3], f[4], f[5]);
            p.thr = mk(f[9], f[10], f[11]);
            p.pixel = __float_as_int(f[18]);
            p.spec = f[20] != 0.0f;
            p.last_pdf = f[21];
            p.iter = iter;
            const uint32_t* h = hits + size_t(i) * 10;
            float t = __uint_as_float(h[0]);
            int inst = int(h[1]), prim = int(h[2]);
            float su = __uint_as_float(h[8]), sv = __uint_as_float(h[9]);
            int si = int(h[6]), spr = int(h[7]);
            if (O.env) si = -1;
            RegisterPark K;
            bool survived = shade_one<true, -1, true, false>(S, O, depth, p, RowPathIn{f, O.env != 0}, K, t, inst, prim,
                                                __uint_as_float(h[3]), __uint_as_float(h[4]), __uint_as_float(h[5]), si,
                                                spr, su, sv);
            alive = survived && compact;
            f[0] = p.o.x; f[1] = p.o.y; f[2] = p.o.z;
            f[3] = p.d.x; f[4] = p.d.y; f[5] = p.d.z;
            f[9] = p.thr.x; f[10] = p.thr.y; f[11] = p.thr.z;
            f[19] = survived ? 0.0f : 1.0f;
            f[20] = p.spec ? 1.0f : 0.0f;
            f[21] = p.last_pdf;
        }
        unsigned am = __ballot_sync(0xffffffffu, alive);
        if (am) {
            int b = 0, leader = __ffs(am) - 1;
            if (lane == leader) b = atomicAdd(n_out, __popc(am));
            b = __shfl_sync(0xffffffffu, b, leader);
            if (alive) survivors[b + __popc(am & ((1u << lane) - 1u))] = i;
        }
    }
}

__global__ void k_light_ext(DevScene S, DevOptions O, int iter, int depth, const int* pixels, int n, float* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        f3 ed;
        f3 dl = light_sample(S, O, iter, pixels[i], depth, ed);
        float* o = out + size_t(i) * 6;
        o[0] = dl.x; o[1] = dl.y; o[2] = dl.z;
        o[3] = ed.x; o[4] = ed.y; o[5] = ed.z;
    }
}

__global__ void k_rng_ext(int iter, int index, int depth, int n, float* out) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        Rng r = Rng::seeded(iter, index, depth);
        for (int i = 0; i < n; ++i) out[i] = r.u01();
    }
}

__global__ void k_tex_ext(unsigned long long t, const float* uv, int n, float* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 v = tex(t, uv[i * 2], uv[i * 2 + 1]);
        out[i * 4] = v.x; out[i * 4 + 1] = v.y; out[i * 4 + 2] = v.z; out[i * 4 + 3] = v.w;
    }
}

}  // namespace

// Grid of the shading kernels: SMs x resident blocks per SM, cached per device ordinal under a
// lock, as trace_grid_blocks is.
int shade_grid_blocks() {
    static std::mutex mu;
    static std::map<int, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    int& cached = cache[dev];
    if (cached == 0) {
        int sms = 0, per = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        int per_jobs = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_shade<false, false, 2>, kShadeBlock, 0);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_jobs, k_shade<true, false, 2>, kShadeBlock, 0);
        per = std::min(per, per_jobs);
        cached = sms * (per > 0 ? per : 1);
    }
    return cached;
}

// Grid cap of the camera kernels: two rounds of sixteen blocks on every SM (the shading grid is
// three blocks an SM)
static int camera_grid_blocks() { return shade_grid_blocks() / kShadeOcc * 32; }

cudaError_t launch_camera(const DevScene& S, const DevWave& W, const DevOptions& O, const DevCamera& C, int n,
                          int lane, const int* wave_iter, cudaStream_t st) {
    if (n > W.lane_stride || lane < 0) return cudaErrorInvalidValue;
    int grid = std::min((n + kCameraBlock - 1) / kCameraBlock, camera_grid_blocks());
    if (grid < 1) grid = 1;
    k_camera<<<grid, kCameraBlock, 0, st>>>(S, W, O, C, n, lane, wave_iter);
    return cudaGetLastError();
}

cudaError_t launch_shade(const DevScene& S, const DevWave& W, const DevOptions& O, int bounce, int compact,
                         cudaStream_t st) {
    return launch_shade_segs(S, W, O, one_seg(bounce, compact), st);
}

cudaError_t launch_shade_segs(const DevScene& S, const DevWave& W, const DevOptions& O, const Segs& G,
                              cudaStream_t st) {
    if (G.n < 1 || G.n > kMaxSegs) return cudaErrorInvalidValue;
    const int g = shade_grid_blocks(), mode = nee_mode_of(O);
    if (O.material_debug && !W.path_job) {
        k_shade<false, true, -1><<<g, kShadeBlock, 0, st>>>(S, W, O, G);
    } else if (W.path_job) {
        if (mode == 2) k_shade<true, false, 2><<<g, kShadeBlock, 0, st>>>(S, W, O, G);
        else if (mode == 1) k_shade<true, false, 1><<<g, kShadeBlock, 0, st>>>(S, W, O, G);
        else k_shade<true, false, 0><<<g, kShadeBlock, 0, st>>>(S, W, O, G);
    } else {
        if (mode == 2) k_shade<false, false, 2><<<g, kShadeBlock, 0, st>>>(S, W, O, G);
        else if (mode == 1) k_shade<false, false, 1><<<g, kShadeBlock, 0, st>>>(S, W, O, G);
        else k_shade<false, false, 0><<<g, kShadeBlock, 0, st>>>(S, W, O, G);
    }
    return cudaGetLastError();
}

cudaError_t launch_camera_jobs(const DevWave& W, const DevOptions& O, int max_paths, int lane, cudaStream_t st) {
    if (lane < 0) return cudaErrorInvalidValue;
    int grid = std::min((max_paths + kCameraBlock - 1) / kCameraBlock, camera_grid_blocks());
    if (grid < 1) grid = 1;
    k_camera_jobs<<<grid, kCameraBlock, 0, st>>>(W, O, lane);
    return cudaGetLastError();
}

cudaError_t launch_accumulate_jobs(const DevWave& W, int compensated, int lane, cudaStream_t st) {
    if (lane < 0) return cudaErrorInvalidValue;
    k_accumulate_jobs<<<148 * 8, 256, 0, st>>>(W, compensated, lane);
    return cudaGetLastError();
}

cudaError_t launch_accumulate(const DevWave& W, int lane, float* image, float* comp, int nsamples, int compensated,
                              cudaStream_t st) {
    if (lane < 0 || size_t(nsamples) * size_t(W.npix) > size_t(W.lane_stride)) return cudaErrorInvalidValue;
    int grid = std::min((W.npix + 255) / 256, 148 * 8);
    if (grid < 1) grid = 1;
    if (W.width * W.height != W.npix) return cudaErrorInvalidValue;
    k_accumulate<<<grid, 256, 0, st>>>(W.s3 + size_t(lane) * W.lane_stride, image, comp, W.width, W.height, nsamples,
                                       compensated);
    return cudaGetLastError();
}

cudaError_t launch_tonemap(const float* image, uint8_t* rgba, int npix, float iter, int color_mode, cudaStream_t st) {
    int grid = std::min((npix + 255) / 256, 148 * 8);
    if (grid < 1) grid = 1;
    k_tonemap<<<grid, 256, 0, st>>>(image, reinterpret_cast<uchar4*>(rgba), npix, iter, color_mode);
    return cudaGetLastError();
}

cudaError_t launch_shade_ext(const DevScene& S, const DevOptions& O, float* paths, const uint32_t* hits, int n,
                             int iter, int depth, int compact, int* survivors, int* n_out, cudaStream_t st) {
    int grid = std::max(1, std::min((n + 127) / 128, 1024));
    k_shade_ext<<<grid, 128, 0, st>>>(S, O, paths, hits, n, iter, depth, compact, survivors, n_out);
    return cudaGetLastError();
}

cudaError_t launch_light_ext(const DevScene& S, const DevOptions& O, int iter, int depth, const int* pixels, int n,
                             float* out, cudaStream_t st) {
    int grid = std::max(1, std::min((n + 127) / 128, 1024));
    k_light_ext<<<grid, 128, 0, st>>>(S, O, iter, depth, pixels, n, out);
    return cudaGetLastError();
}

cudaError_t launch_rng_ext(int iter, int index, int depth, int n, float* out, cudaStream_t st) {
    k_rng_ext<<<1, 32, 0, st>>>(iter, index, depth, n, out);
    return cudaGetLastError();
}

cudaError_t launch_tex_ext(unsigned long long t, const float* uv, int n, float* out, cudaStream_t st) {
    int grid = std::max(1, std::min((n + 127) / 128, 1024));
    k_tex_ext<<<grid, 128, 0, st>>>(t, uv, n, out);
    return cudaGetLastError();
}

}  // namespace lux
