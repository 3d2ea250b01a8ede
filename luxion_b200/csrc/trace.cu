// trace.cu -- ray traversal of the compressed 8-wide BVH, of two levels or one, on sm_100a.
//
// Replaces the reference's OptiX launch (src/pathtrace.cu:238-258, device programs in
// src/optixshaders/optix_triangle.cu:52-366) and its disabled software path
// (src/kernels/compute_intersections.cu:6-87, src/intersections/mesh_isect.cu:6-149).
//
// Design:
//  * persistent warps: lanes without a ray take the next ones from a global cursor with one
//    atomicAdd per warp (ballot/popc), and a warp leaves its inner loop to refill as soon as
//    fewer than kRefill lanes are still traversing (Aila & Laine's while-while with dynamic
//    fetch);
//  * the traversal stack keeps its top kShStack entries in shared memory (one column per
//    thread, conflict-free) and spills deeper entries to local memory;
//  * node groups / triangle groups as in Ylitie et al. 2017: a stack entry is a node's
//    remaining internal-child hits (ordered by ray octant) or a set of leaf records;
//  * two-level layout: the TLAS is traversed with the world ray; a TLAS leaf pushes a marker and
//    continues in the instance's BLAS with the object-space ray the reference uses
//    (inverseTransform * (o,1), (d,0), src/intersections/mesh_isect.cu:15-16);
//  * the triangle test is the reference's Moller-Trumbore (mesh_isect.cu:78-137) with every
//    operation rounded on its own, so t, u, v and the hit triangle match the CPU oracle bit
//    for bit on the same rays; equal t is resolved toward the lowest (instance, primitive);
//  * alpha mask / blend any-hit (optix_triangle.cu:317-366) is evaluated on candidate hits of
//    instances whose material is not opaque.
// Box tests are conservative: child boxes are quantised outward at build time and a child is
// entered while tnear <= tfar * (1 + 2^-17), so no triangle the exact test accepts is skipped.

#include "trace_core.cuh"

#include <array>
#include <map>
#include <mutex>

namespace lux {

namespace {

struct TraceArgs {
    DevScene S;
    DevWave W;
    Segs G;      // the (lane, bounce) segments of the launch
    int mode;    // 0 radiance, 1 DL shadow, 2 env shadow, 3 BVH heatmap of radiance rays
    int nee;     // radiance pass: 0 none, 1 DL, 2 env
    const float* ext_rays;  // lux_trace_rays: rays given directly (n * 8 floats)
    uint32_t* ext_hits;     // and hits written directly (n * 5 words)
    int ext_n;
    int ext_iter;
    int* ext_fetch;
    int* ext_err;           // and its error word, page-locked or on the device
};


// The segment of a slot: the one that holds the slot's lane.
LUX_DI int seg_of_slot(const TraceArgs& A, int slot) {
    int k = 0;
    if (A.G.n > 1) {
        const int ln = slot / A.W.lane_stride;
        while (k + 1 < A.G.n && A.G.lane[k] != ln) ++k;
    }
    return k;
}

// The key of a ray's alpha-blend hash: of wave rays (item: the radiance ray's slot) the path's
// pixel and iteration, of rays given directly the pixel that came with the ray.
template <bool EXT>
struct RayKey {
    const TraceArgs& A;  // the launch's arguments, in parameter space like the scene
    LUX_DI void operator()(int item, int& pixel, int& iter) const {
        if (EXT) {
            pixel = __float_as_int(A.ext_rays[size_t(item) * 8 + 7]);
            iter = A.ext_iter;
            return;
        }
        const int pid = A.W.queue[A.G.bounce[seg_of_slot(A, item)] & 1][item];
        pixel = __float_as_int(A.W.s2[pid].w);
        iter = __float_as_int(A.W.s3[pid].w);
    }
};

// Rays given directly are spread over the warps up to this many per warp: 20,000 rays (5 a warp)
// 251 -> 237 us a call, 100 rays 81 -> 68, but 65,536 rays (16 a warp) 438 -> 482.
constexpr int kSpread = 8;

// EXT: rays given directly (lux_trace_rays); else the rays of waves.
template <int MODE, bool SINGLE, bool EXT>
// The arguments stay in parameter space (__grid_constant__): the tracer reads the scene
// through a reference to them, which would otherwise copy the struct to local memory.
// Seven 128-thread blocks per SM (72 registers) measured faster than six (80) and eight (64, with
// spills): 32.9, 35.1 and 35.1 ms of traversal per 16-spp step of the 1M-triangle 1080p scene.
// The loop is bound by instruction issue and the latency of dependent loads (bounce 1 of that
// scene: 64 % issue, ALU pipe 54 %, L1 hit 61 %, 3.4 of 10.5 stall cycles on loads), so what counts
// is instructions: 324 per thread and ray after the following, 421 before. Traversal per step:
// 36.4 ms; 35.7 with the closest hit in shared memory, one limit register and the sign-bit slab
// test; 33.9 with the plane distances two to an instruction (fma.rn.f32x2, which lost before the
// registers were freed); 32.9 without the two-level layout's marker test in the single-level pop;
// 32.7 with the key order from a table; 32.2 without its instance phase. Tried on top: the node's
// own constants two to an instruction (35.1, spills), plane bytes by dp4a instead of byte permutes
// (32.2), prefetching the next node before the triangle tests (33.1).
__global__ void __launch_bounds__(kTraceBlock, SINGLE ? 7 : 6) k_trace(const __grid_constant__ TraceArgs A) {
    __shared__ uint2 stack[kShStack][kTraceBlock];
    __shared__ float4 hits[kTraceBlock];
    __shared__ unsigned char lut[2048];
    fill_key_table(lut);  // read after the barrier below
    // work of segment k: items [seg_first[k], seg_first[k + 1]) of the launch's list
    __shared__ int seg_first[kMaxSegs + 1];
    if (threadIdx.x == 0) {
        int t = 0;
        seg_first[0] = 0;
        for (int k = 0; k < kMaxSegs; ++k) {
            if (!EXT && k < A.G.n) {
                const WaveCounters* c = A.W.ctr + A.G.lane[k];
                if (*(volatile const int*)&c->finished == 0)
                    t += (MODE == 0 || MODE == 3) ? *(volatile const int*)&c->count[A.G.bounce[k]]
                                                  : *(volatile const int*)&c->shadow[A.G.bounce[k]];
            }
            seg_first[k + 1] = t;
        }
    }
    __syncthreads();
    Tracer<MODE, SINGLE, kTraceBlock, RayKey<EXT>> T{A.S, stack, hits, lut, {}, int(threadIdx.x), EXT ? A.ext_err : &(A.W.ctr + A.G.lane[0])->error,
                                        RayKey<EXT>{A}, MODE == 2};
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int total;
    int* cursor;
    // the cursor of the first segment's (lane, bounce) serves the whole launch: no other
    // launch of this kind covers that lane at that bounce
    if (EXT) {
        total = A.ext_n;
        cursor = A.ext_fetch;
    } else if (MODE == 0 || MODE == 3) {
        total = seg_first[kMaxSegs];
        cursor = &(A.W.ctr + A.G.lane[0])->fetch_r[A.G.bounce[0]];
    } else {
        total = seg_first[kMaxSegs];
        cursor = &(A.W.ctr + A.G.lane[0])->fetch_s[A.G.bounce[0]];
    }
    // Rays given directly that are fewer than the grid's lanes are spread over all its warps: `cap`
    // lanes of each take one, by the warp's place. A ray's time is its chain of dependent node
    // visits, and rays of one warp wait for one another's phases; the postponement threshold shrinks
    // with the warp's rays, or no triangle would be tested (and no limit shortened) before every
    // lane had run out of nodes. (The waves' launches leave few rays to the whole-path kernel, and
    // the two thresholds in registers cost their loop 1 to 2 %.)
    const int warps = int(gridDim.x) * (kTraceBlock / 32);
    int cap = 32;
    if (EXT && total <= kSpread * warps) cap = (total + warps - 1) / warps;
    const int postpone = EXT ? (cap * kPostpone) >> 5 : kPostpone;
    const int refill = cap < 32 ? 0 : (MODE == 2 ? kRefillOcclusion : kRefill);
    Lane L;
    bool active = false;
    bool exhausted = false;  // warp-uniform: the cursor has passed the end of the work list
    bool pending = false;    // the lane's ray is done and its result not yet written
    L.item = 0;
    while (true) {
        // Results of the rays that finished, written by all such lanes of the warp together
        // (at least 32 - kRefill of them, or the last ones): a lane that finishes keeps its
        // ray state untouched until the refill below replaces it.
        if (pending) {
            pending = false;
            const Best best = T.best(L);
            const int item = L.item;
            if (EXT) {
                uint32_t* h = A.ext_hits + size_t(item) * 5;
                if (MODE == 2) {
                    h[0] = __float_as_uint(best.inst >= 0 ? 1.0f : -1.0f);
                    h[1] = h[2] = 0xffffffffu;
                    h[3] = h[4] = 0u;
                } else if (MODE == 3) {
                    h[0] = __float_as_uint(best.t);
                    h[1] = uint32_t(best.inst);
                    h[2] = uint32_t(best.prim);
                    h[3] = uint32_t(L.work);
                    h[4] = 0u;
                } else {
                    h[0] = __float_as_uint(best.t);
                    h[1] = uint32_t(best.inst);
                    h[2] = uint32_t(best.prim);
                    h[3] = __float_as_uint(best.u);
                    h[4] = __float_as_uint(best.v);
                }
            } else if (MODE == 0) {
                bool hit = best.inst >= 0;
                st_stream(&A.W.hit[item], make_float4(best.t, best.u, best.v, __int_as_float(best.inst)));
                st_stream(&A.W.hit_prim[item], best.prim);
                if (hit && A.nee) {
                    const int k = seg_of_slot(A, item);
                    const int bk = A.G.bounce[k], lk = A.G.lane[k];
                    int pid = ld_stream(&A.W.queue[bk & 1][item]);
                    float4 ns = ld_stream(&A.W.s4[pid]);
                    f3 so, sd;
                    float tmax;
                    shadow_ray(A.S, best, T.world_o(L), T.world_d(L), mk(ns.x, ns.y, ns.z), A.nee == 2, so, sd, tmax);
                    // append to the lane's shadow queue, aggregated over the lanes of the
                    // warp that append to the same one; the ray is stored at its queue
                    // position, beside the slot it belongs to, so the occlusion launch reads
                    // rays contiguously and without first reading the slot
                    const unsigned am = __match_any_sync(__activemask(), lk);
                    int leader = __ffs(am) - 1;
                    int b2 = 0;
                    if (lane == leader) b2 = atomicAdd(&(A.W.ctr + lk)->shadow[bk], __popc(am));
                    b2 = __shfl_sync(am, b2, leader);
                    const size_t q = size_t(lk) * A.W.lane_stride + b2 + __popc(am & ((1u << lane) - 1u));
                    st_stream(&A.W.sh_o[q], make_float4(so.x, so.y, so.z, tmax));
                    st_stream(&A.W.sh_d[q], make_float4(sd.x, sd.y, sd.z, 0.0f));
                    st_stream(&A.W.sh_queue[q], item);
                }
            } else if (MODE == 1) {
                bool hit = best.inst >= 0;
                st_stream(&A.W.sh_hit[item], make_float4(best.t, best.u, best.v, __int_as_float(best.inst)));
                st_stream(&A.W.sh_prim[item], best.prim);
            } else if (MODE == 3) {
                // drawBVH (src/kernels/draw_bvh.cu:33): color += count * 0.001 on every channel
                int pid = A.W.queue[A.G.bounce[0] & 1][item];  // the heatmap traces one wave
                float4 c = A.W.s3[pid];
                const float h = float(L.work) * 0.001f;
                A.W.s3[pid] = make_float4(c.x + h, c.y + h, c.z + h, c.w);
            } else {
                st_stream(&A.W.sh_hit[item], make_float4(best.inst >= 0 ? 1.0f : -1.0f, 0.0f, 0.0f, __int_as_float(-1)));
            }
        }
        unsigned need = __ballot_sync(FULL, !active && lane < cap);
        if (need && !exhausted) {
            int base = 0;
            if (EXT && cap < 32) {  // blocks apart, so that a few rays reach many SMs
                base = (int(threadIdx.x >> 5) * int(gridDim.x) + int(blockIdx.x)) * cap;
                exhausted = true;
            } else {
                if (lane == 0) base = atomicAdd(cursor, __popc(need));
                base = __shfl_sync(FULL, base, 0);
                if (base + __popc(need) >= total) exhausted = true;
            }
            if (!active && lane < cap) {
                int r = base + __popc(need & ((1u << lane) - 1u));
                if (r < total) {
                    int item = r;
                    f3 o, d;
                    float tmax;
                    uint32_t root = A.S.tlas_root;
                    if (EXT) {
                        const float* ry = A.ext_rays + size_t(r) * 8;
                        o = mk(ry[0], ry[1], ry[2]);
                        d = mk(ry[4], ry[5], ry[6]);
                        tmax = MODE == 1 ? ry[3] : 1e16f;
                    } else if (MODE == 0 || MODE == 3) {
                        int k = 0;
                        while (k + 1 < A.G.n && r >= seg_first[k + 1]) ++k;
                        item = A.G.lane[k] * A.W.lane_stride + (r - seg_first[k]);  // absolute slot
                        int pid = ld_stream(&A.W.queue[A.G.bounce[k] & 1][item]);
                        float4 a = ld_stream(&A.W.s0[pid]), b = ld_stream(&A.W.s1[pid]);
                        o = mk(a.x, a.y, a.z);
                        d = mk(b.x, b.y, b.z);
                        tmax = 1e16f;
                        if (A.W.path_job) root = A.W.jobs[A.W.path_job[pid]].tlas_root;
                    } else {
                        int k = 0;
                        while (k + 1 < A.G.n && r >= seg_first[k + 1]) ++k;
                        const size_t q = size_t(A.G.lane[k]) * A.W.lane_stride + (r - seg_first[k]);
                        int slot = ld_stream(&A.W.sh_queue[q]);
                        item = slot;
                        float4 a = ld_stream(&A.W.sh_o[q]), b = ld_stream(&A.W.sh_d[q]);
                        o = mk(a.x, a.y, a.z);
                        d = mk(b.x, b.y, b.z);
                        tmax = a.w;
                        if (A.W.path_job) {
                            const int pid = ld_stream(&A.W.queue[A.G.bounce[k] & 1][slot]);
                            root = A.W.jobs[A.W.path_job[pid]].tlas_root;
                        }
                    }
                    L.item = item;
                    T.start(L, o, d, tmax, root);
                    active = true;
                }
            }
        }
        if (!__any_sync(FULL, active)) break;
        while (true) {
            if (T.step(L, active, postpone)) {
                active = false;
                pending = true;
            }
            const unsigned am = __ballot_sync(FULL, active);
            if (!am) break;
            if (__popc(am) < refill && !exhausted) break;
        }
    }
}

// resident blocks per SM that both the waves' kernel and the direct rays' reach
template <int MODE, bool SINGLE>
int blocks_per_sm() {
    int a = 0, b = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_trace<MODE, SINGLE, false>, kTraceBlock, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_trace<MODE, SINGLE, true>, kTraceBlock, 0);
    return a < b ? a : b;
}

}  // namespace

// Persistent grid of each traversal kind: SMs x resident blocks per SM. The answer depends on
// the device, so it is cached per device ordinal, under a lock (contexts on several devices and
// several host threads ask for it).
int trace_grid_blocks(int mode, bool single) {
    static std::mutex mu;
    static std::map<int, std::array<int, 8>> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    int& cached = cache[dev][mode * 2 + (single ? 1 : 0)];
    if (cached == 0) {
        int sms = 0, per = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        switch (mode * 2 + (single ? 1 : 0)) {
            case 0: per = blocks_per_sm<0, false>(); break;
            case 1: per = blocks_per_sm<0, true>(); break;
            case 2: per = blocks_per_sm<1, false>(); break;
            case 3: per = blocks_per_sm<1, true>(); break;
            case 4: per = blocks_per_sm<2, false>(); break;
            case 5: per = blocks_per_sm<2, true>(); break;
            case 6: per = blocks_per_sm<3, false>(); break;
            default: per = blocks_per_sm<3, true>(); break;
        }
        cached = sms * (per > 0 ? per : 1);
    }
    return cached;
}

namespace {
template <bool SINGLE, bool EXT>
void launch_mode(int mode, int grid, cudaStream_t st, const TraceArgs& A) {
    if (mode == 0) k_trace<0, SINGLE, EXT><<<grid, kTraceBlock, 0, st>>>(A);
    else if (mode == 1) k_trace<1, SINGLE, EXT><<<grid, kTraceBlock, 0, st>>>(A);
    else if (mode == 2) k_trace<2, SINGLE, EXT><<<grid, kTraceBlock, 0, st>>>(A);
    else k_trace<3, SINGLE, EXT><<<grid, kTraceBlock, 0, st>>>(A);
}
}  // namespace

cudaError_t launch_trace(const DevScene& S, const DevWave& W, int bounce, int mode, int nee, cudaStream_t st,
                         int grid) {
    return launch_trace_segs(S, W, one_seg(bounce), mode, nee, st, grid);
}

cudaError_t launch_trace_segs(const DevScene& S, const DevWave& W, const Segs& G, int mode, int nee, cudaStream_t st,
                              int grid) {
    if (G.n < 1 || G.n > kMaxSegs) return cudaErrorInvalidValue;
    TraceArgs A{S, W, G, mode, nee, nullptr, nullptr, 0, 0, nullptr, nullptr};
    const bool single = S.single_level != 0;
    if (grid <= 0) grid = trace_grid_blocks(mode, single);
    if (single) launch_mode<true, false>(mode, grid, st, A);
    else launch_mode<false, false>(mode, grid, st, A);
    return cudaGetLastError();
}

cudaError_t launch_trace_ext(const DevScene& S, const DevWave& W, const float* rays, uint32_t* hits, int n, int mode,
                             int iter, int* fetch, int* err, cudaStream_t st) {
    TraceArgs A{S, W, one_seg(0), mode, 0, rays, hits, n, iter, fetch, err};
    const bool single = S.single_level != 0;
    const int grid = trace_grid_blocks(mode, single);
    if (single) launch_mode<true, true>(mode, grid, st, A);
    else launch_mode<false, true>(mode, grid, st, A);
    return cudaGetLastError();
}

}  // namespace lux
