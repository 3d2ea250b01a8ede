// paths.cu -- the rest of a path in one launch: traversal, shadow ray, shading and the next
// bounce's light sample in a loop over the bounces, path state in registers.
//
// The wavefront (trace.cu, shade.cu) runs each bounce as launches over all paths. That pays for
// many paths: rays of one kind fill the warps and warps fetch the next ray as one ends. With few
// paths a launch takes as long as its slowest ray plus the cold start of its code, 20 to 60 us
// however few rays it has, three launches a bounce. Here only the lanes of a block wait for one
// another between the bounces, and a 256x256 frame of depth 8 takes one launch instead of 24.
// Every path is computed as the wavefront computes it (same functions, same order of its own
// operations) and paths do not depend on one another, so images and counts are the same bit for
// bit.
//
// Compiled with --fmad=false, as shade.cu is.

#include "path_segs.h"
#include "trace_core.cuh"
#include "shade_core.cuh"

#include <algorithm>
#include <map>
#include <mutex>

namespace lux {
namespace {

// Pixel and iteration of a path in registers (alpha-blend hash).
struct PathKey {
    const PathState& p;
    LUX_DI void operator()(int, int& pixel, int& iter) const {
        pixel = p.pixel;
        iter = p.iter;
    }
};

// The path fields shade_one reads late. The radiance so far stays in the wave's s3.
struct RegPathIn {
    const DevWave& W;
    int pid;
    f3 o, ns;
    float pdf;
    LUX_DI f3 origin() const { return o; }
    LUX_DI float last_pdf() const { return pdf; }
    LUX_DI f3 color0() const {
        float4 a = W.s3[pid];
        return mk(a.x, a.y, a.z);
    }
    LUX_DI f3 nee() const { return ns; }
    LUX_DI void set_color(f3 c, int iter) const { W.s3[pid] = make_float4(c.x, c.y, c.z, __int_as_float(iter)); }
};

struct PathArgs {
    DevScene S;
    DevWave W;
    DevOptions O;
    Segs G;      // the (lane, bounce) segments whose paths the launch finishes
    int depth;   // bounces of a path (job engine: each job's own)
    int limit;   // do nothing when the segments hold more paths than this
};

// What bounds it is latency and instruction fetch, not throughput: the shading's code exceeds the
// instruction caches, so the block's warps shade in step (k_shade), and one copy of the traversal
// serves both kinds of ray. 256x256 Cornell box, depth 8 (65536 paths): 0.53 ms as a wavefront; here
// 0.76 with warps shading at their own pace and four blocks per SM (0.59 with three, 0.55 with two),
// in step 0.38 with four blocks, 0.35 with three and two. With today's traversal and shading 0.32
// (150 registers), as with 256 x 2; 0.33 with 64 x 6 and 256 x 1. 29302 paths, 50k triangles: 0.48 as
// a wavefront, 0.15 here (0.17 with 256 x 2).
template <bool JOBS, int NEE, bool SINGLE>
__global__ void __launch_bounds__(kPathBlock, kPathOcc) k_paths(const __grid_constant__ PathArgs A) {
    __shared__ uint2 stack[kShStack][kPathBlock];
    __shared__ float4 hits[kPathBlock];
    __shared__ unsigned char lut[2048];
    fill_key_table(lut);  // read after the barrier below
    __shared__ PathSegs segs;
    // this block's share of the counters: survivors entering each bounce and shadow rays
    __shared__ int n_path[kMaxSegs][kMaxDepth + 1], n_shadow[kMaxSegs][kMaxDepth];
    if (threadIdx.x == 0) segs = path_segments(A.W.ctr, A.G);
    for (int i = threadIdx.x; i < kMaxSegs * (kMaxDepth + 1); i += kPathBlock) (&n_path[0][0])[i] = 0;
    for (int i = threadIdx.x; i < kMaxSegs * kMaxDepth; i += kPathBlock) (&n_shadow[0][0])[i] = 0;
    __syncthreads();
    const int total = segs.first[kMaxSegs];
    if (total == 0 || total > A.limit) return;
    if (blockIdx.x == 0 && int(threadIdx.x) < A.G.n) mark_segment(A.W.ctr, A.G, threadIdx.x);

    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    // Fewer paths than lanes: every warp gets the same share, so that a path waits for few others.
    const int warps = int(gridDim.x) * (kPathBlock / 32);
    const int cap = min(32, (total + warps - 1) / warps);
    int* cursor = &(A.W.ctr + segs.lane)->fetch_p;
    int* err = &(A.W.ctr + segs.lane)->error;
    bool first = true, exhausted = false;  // warp-uniform
    bool has = false;
    PathState p{};
    f3 ns = mk(0.0f, 0.0f, 0.0f);
    int pid = 0, seg = 0, depth = 0, last = 0;  // depth of the bounce being computed, last depth
    const DevScene* sp = &A.S;
    uint32_t root = A.S.tlas_root;
    while (true) {
        const unsigned need = __ballot_sync(FULL, !has && lane < cap);
        if (need && !exhausted) {
            // the first paths of every warp are assigned by its place, the rest by the cursor
            int base = 0;
            if (first) {
                base = (int(threadIdx.x >> 5) * int(gridDim.x) + int(blockIdx.x)) * cap;
                first = false;
                if (cap < 32) exhausted = true;
            } else {
                if (lane == 0) base = atomicAdd(cursor, __popc(need));
                base = __shfl_sync(FULL, base, 0) + warps * 32;
            }
            if (base + __popc(need) >= total) exhausted = true;
            const int r = base + __popc(need & ((1u << lane) - 1u));
            if (!has && lane < cap && r < total) {
                seg = 0;
                while (seg + 1 < A.G.n && r >= segs.first[seg + 1]) ++seg;
                const int b = A.G.bounce[seg];
                pid = ld_stream(&A.W.queue[b & 1][A.G.lane[seg] * A.W.lane_stride + (r - segs.first[seg])]);
                depth = b + 1;
                last = A.depth;
                if (JOBS) {
                    const DevJob& J = A.W.jobs[A.W.path_job[pid]];
                    sp = &A.W.scenes[J.scene];
                    root = J.tlas_root;
                    last = J.trace_depth;
                }
                const float4 s0 = ld_stream(&A.W.s0[pid]), s1 = ld_stream(&A.W.s1[pid]), s2 = ld_stream(&A.W.s2[pid]);
                p.o = mk(s0.x, s0.y, s0.z);
                p.last_pdf = s0.w;
                p.d = mk(s1.x, s1.y, s1.z);
                p.spec = (__float_as_int(s1.w) & 1) != 0;
                p.thr = mk(s2.x, s2.y, s2.z);
                p.pixel = __float_as_int(s2.w);
                p.iter = __float_as_int(A.W.s3[pid].w);
                if (NEE) {
                    const float4 s4 = ld_stream(&A.W.s4[pid]);
                    ns = mk(s4.x, s4.y, s4.z);
                }
                has = true;
            }
        }
        if (!__syncthreads_or(has)) break;
        const unsigned hm = __ballot_sync(FULL, has);
        // postponement as in the traversal kernel, for the rays this warp holds
        const int postpone = (__popc(hm) * kPostpone) >> 5;
        // radiance ray, then shadow ray: one copy of the traversal's code
        Best best, sh;
        best.inst = sh.inst = -1;
        best.t = sh.t = -1.0f;
        best.prim = sh.prim = -1;
        best.u = best.v = sh.u = sh.v = 0.0f;
        bool hit = false;
#pragma unroll 1
        for (int k = 0; k < (NEE ? 2 : 1); ++k) {
            Tracer<NEE == 2 ? -1 : 0, SINGLE, kPathBlock, PathKey> T{A.S, stack, hits, lut, {}, int(threadIdx.x), err, PathKey{p}, k == 1};
            Lane L;
            bool active = has;
            if (k == 0) {
                if (has) T.start(L, p.o, p.d, 1e16f, root);
            } else {
                active = hit;
                if (hit) {
                    f3 so, sd;
                    float tmax;
                    shadow_ray(A.S, best, p.o, p.d, ns, NEE == 2, so, sd, tmax);
                    T.start(L, so, sd, tmax, root);
                    atomicAdd(&n_shadow[seg][depth - 1], 1);
                }
            }
            const bool on = active;
            while (__any_sync(FULL, active))
                if (T.step(L, active, postpone)) active = false;
            if (on && k == 0) {
                best = T.best(L);
                hit = best.inst >= 0;
            } else if (on) {
                sh = T.best(L);
            }
        }
        if (NEE == 2 && hit) sh.t = sh.inst >= 0 ? 1.0f : -1.0f;
        // shading, the block's warps in step (see k_shade)
        phase<true>();
        const RegPathIn in{A.W, pid, p.o, ns, p.last_pdf};
        RegisterPark K;
        const bool alive = shade_one<false, NEE, false, true>(*sp, A.O, depth, p, in, K, hit ? best.t : -1.0f, best.inst, best.prim,
                                                              best.u, best.v, sh.t, NEE == 2 ? -1 : sh.inst, sh.prim, sh.u,
                                                              sh.v, has) &&
                           depth < last;
        if (has) {
            if (alive) {
                if (NEE) {
                    f3 ed;
                    f3 dl = light_sample<NEE>(*sp, A.O, p.iter, p.pixel, depth, ed, NEE != 2);
                    ns = NEE == 2 ? ed : dl;
                }
                atomicAdd(&n_path[seg][depth], 1);
                ++depth;
            } else {
                has = false;
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < A.G.n * (kMaxDepth + 1); i += kPathBlock) {
        const int k = i / (kMaxDepth + 1), b = i % (kMaxDepth + 1);
        WaveCounters* c = A.W.ctr + A.G.lane[k];
        if (const int v = n_path[k][b]) atomicAdd(&c->count[b], v);
        if (b < kMaxDepth)
            if (const int v = n_shadow[k][b]) atomicAdd(&c->shadow[b], v);
    }
}

template <class F>
int blocks_per_sm(F f) {
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, kPathBlock, 0);
    return per > 0 ? per : 1;
}

}  // namespace

// Persistent grid of the whole-path kernel, cached per device as trace_grid_blocks is.
int path_grid_blocks() {
    static std::mutex mu;
    static std::map<int, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    int& cached = cache[dev];
    if (cached == 0) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cached = sms * std::min(blocks_per_sm(k_paths<false, 2, true>), blocks_per_sm(k_paths<false, 1, false>));
    }
    return cached;
}

cudaError_t launch_paths(const DevScene& S, const DevWave& W, const DevOptions& O, const Segs& G, int depth, int limit,
                         cudaStream_t st) {
    if (G.n < 1 || G.n > kMaxSegs || depth > kMaxDepth) return cudaErrorInvalidValue;
    const PathArgs A{S, W, O, G, depth, limit};
    const int grid = path_grid_blocks(), nee = O.env ? 2 : (O.dl ? 1 : 0);
    const bool single = S.single_level != 0, jobs = W.path_job != nullptr;
#define LUX_PATHS(J, N, B) k_paths<J, N, B><<<grid, kPathBlock, 0, st>>>(A)
#define LUX_PATHS_NEE(J, B)              \
    do {                                 \
        if (nee == 2) LUX_PATHS(J, 2, B); \
        else if (nee == 1) LUX_PATHS(J, 1, B); \
        else LUX_PATHS(J, 0, B);         \
    } while (0)
    if (jobs) {
        if (single) LUX_PATHS_NEE(true, true);
        else LUX_PATHS_NEE(true, false);
    } else {
        if (single) LUX_PATHS_NEE(false, true);
        else LUX_PATHS_NEE(false, false);
    }
#undef LUX_PATHS_NEE
#undef LUX_PATHS
    return cudaGetLastError();
}

}  // namespace lux
