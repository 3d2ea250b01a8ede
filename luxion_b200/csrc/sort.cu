// sort.cu -- Morton-keyed ray sorting of a bounce's queue (RAY_SORTING, include/config.h:4).
//
// Keys follow intersectionPrecompute (src/kernels/intersection_precompute.cu:6-33) and
// rayMortonCode / morton3D (src/morton_codes.cu:13-24, include/morton_codes.h:12-38): the
// ray in the first instance's object space, the reference slab test against the Morton box
// (src/mesh/bounding_box.cu:7-40), 0xFFFFFFFF on a miss, else the 30-bit code of the midpoint
// of o and o+d normalised by the box diagonal. Every float operation is rounded on its own,
// so keys are bit-exact with the CPU oracle.
// The reference sorts with thrust::sort_by_key (src/pathtrace.cu:182); here a stable LSD
// radix sort (4 passes of 8 bits) whose length is read from the device counter, so the
// whole bounce stays free of host round trips. Each pass is one sweep over the items with
// decoupled look-back (Merrill and Garland, "Single-pass Parallel Prefix Scan with Decoupled
// Look-back", 2016; Adinets and Merrill, "Onesweep", 2022), after one kernel that computes the
// keys and the digit histograms of all passes.

#include "device_scene.h"
#include "device_math.cuh"
#include "launch.h"

#include <algorithm>

namespace lux {
namespace {

constexpr int kSortThreads = 256;             // one thread per bin of an 8-bit digit
constexpr int kWarps = kSortThreads / 32;
constexpr int kItems = 16;
constexpr int kTile = kSortThreads * kItems;  // items of one tile
constexpr int kWarpItems = 32 * kItems;       // a warp's consecutive items of a tile
constexpr int kPasses = 4;

// Look-back state of a sort, in the caller's scratch. Two sets of counters by bounce parity: a
// bounce's last pass clears the other parity's set for the next bounce (clear_sort_counters
// clears both before a wave), so no memset runs between the bounces.
struct SortCounters {
    int hist[kPasses][256];  // items per digit value
    int tile[kPasses];       // next tile of the pass
    int pad[4];
};
// One word per (pass, tile, digit): bits 62-63 the state (0 not yet, 1 the tile's own count,
// 2 the count of this and all earlier tiles), the count below.
using SortWord = unsigned long long;
constexpr SortWord kOwn = SortWord(1) << 62, kPrefix = SortWord(2) << 62, kCount = kOwn - 1;
// Polls of one word before a look-back gives up (error bit 1 of the wave's counters): tiles are
// taken in order by running blocks, so a word appears within the time of a tile.
constexpr int kPollLimit = 1 << 22;
constexpr int kErrSort = 2;

LUX_DI uint32_t expand_bits(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

LUX_DI uint32_t morton3d(float x, float y, float z) {
    x = fminf(fmaxf(__fmul_rn(x, 1024.0f), 0.0f), 1023.0f);
    y = fminf(fmaxf(__fmul_rn(y, 1024.0f), 0.0f), 1023.0f);
    z = fminf(fmaxf(__fmul_rn(z, 1024.0f), 0.0f), 1023.0f);
    return (expand_bits(uint32_t(x)) << 2) | (expand_bits(uint32_t(y)) << 1) | expand_bits(uint32_t(z));
}

LUX_DI uint32_t morton_key(const DevScene& S, f3 o, f3 d) {
    const DevInstance& I = S.insts[0];
    f3 ro = xform(I.Minv, o, 1.0f);
    f3 rd = xform(I.Minv, d, 0.0f);
    f3 inv = mk(__frcp_rn(rd.x), __frcp_rn(rd.y), __frcp_rn(rd.z));
    int sx = inv.x < 0.0f, sy = inv.y < 0.0f, sz = inv.z < 0.0f;
    const float bx[2] = {S.morton_bmin[0], S.morton_bmax[0]};
    const float by[2] = {S.morton_bmin[1], S.morton_bmax[1]};
    const float bz[2] = {S.morton_bmin[2], S.morton_bmax[2]};
    float tmin = __fmul_rn(__fsub_rn(bx[sx], ro.x), inv.x);
    float tmax = __fmul_rn(__fsub_rn(bx[1 - sx], ro.x), inv.x);
    float tymin = __fmul_rn(__fsub_rn(by[sy], ro.y), inv.y);
    float tymax = __fmul_rn(__fsub_rn(by[1 - sy], ro.y), inv.y);
    if (tmin > tymax || tymin > tmax) return 0xFFFFFFFFu;
    tmin = gmax(tmin, tymin);
    tmax = gmin(tmax, tymax);
    float tzmin = __fmul_rn(__fsub_rn(bz[sz], ro.z), inv.z);
    float tzmax = __fmul_rn(__fsub_rn(bz[1 - sz], ro.z), inv.z);
    if (tmin > tzmax || tzmin > tmax) return 0xFFFFFFFFu;
    tmin = gmax(tmin, tzmin);
    if (tmax < 0.0f) return 0xFFFFFFFFu;
    if (!(tmin < tmax)) return 0xFFFFFFFFu;
    f3 ext3 = mk(__fsub_rn(bx[1], bx[0]), __fsub_rn(by[1], by[0]), __fsub_rn(bz[1], bz[0]));
    float ext = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(ext3.x, ext3.x), __fmul_rn(ext3.y, ext3.y)), __fmul_rn(ext3.z, ext3.z)));
    float two = __fmul_rn(2.0f, ext);
    f3 far = mk(__fadd_rn(ro.x, __fmul_rn(rd.x, 1.0f)), __fadd_rn(ro.y, __fmul_rn(rd.y, 1.0f)), __fadd_rn(ro.z, __fmul_rn(rd.z, 1.0f)));
    float p0x = __fdiv_rn(__fadd_rn(ro.x, ext), two), p0y = __fdiv_rn(__fadd_rn(ro.y, ext), two), p0z = __fdiv_rn(__fadd_rn(ro.z, ext), two);
    float p1x = __fdiv_rn(__fadd_rn(far.x, ext), two), p1y = __fdiv_rn(__fadd_rn(far.y, ext), two), p1z = __fdiv_rn(__fadd_rn(far.z, ext), two);
    return morton3d(__fmul_rn(0.5f, __fadd_rn(p0x, p1x)), __fmul_rn(0.5f, __fadd_rn(p0y, p1y)), __fmul_rn(0.5f, __fadd_rn(p0z, p1z)));
}

// Keys of the bounce's queue, the digit histograms of all passes, and cleared look-back words
// for the tiles the passes will use.
__global__ void __launch_bounds__(kSortThreads) k_keys(DevScene S, DevWave W, int bounce, SortCounters* C,
                                                       SortWord* words, int max_tiles) {
    __shared__ int h[kPasses][256];
    const int n = *(volatile int*)&W.ctr->count[bounce];
    const int stride = gridDim.x * kSortThreads, first = blockIdx.x * kSortThreads + threadIdx.x;
    const int tiles = (n + kTile - 1) / kTile;
    for (int p = 0; p < kPasses; ++p) {
        h[p][threadIdx.x] = 0;
        for (int64_t i = first; i < int64_t(tiles) * 256; i += stride) words[size_t(p) * max_tiles * 256 + i] = 0;
    }
    __syncthreads();
    const int* q = W.queue[bounce & 1];
    for (int64_t i = first; i < n; i += stride) {
        int pid = q[i];
        float4 a = W.s0[pid], b = W.s1[pid];
        const uint32_t key = morton_key(S, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z));
        W.keys[i] = key;
        for (int p = 0; p < kPasses; ++p) {
            // lanes of one digit value add together: the keys of a tile share their upper digits
            // (the lanes that are together here: with rounds of whole warps and a digit of its own for
            // lanes past the end, the sorting of an 800x600, 4 spp, depth 8 render took 0.574 instead of
            // 0.557 ms)
            const int dg = (key >> (8 * p)) & 0xff;
            const unsigned peers = __match_any_sync(__activemask(), dg);
            if (__ffs(peers) - 1 == int(threadIdx.x & 31)) atomicAdd(&h[p][dg], __popc(peers));
        }
    }
    __syncthreads();
    for (int p = 0; p < kPasses; ++p)
        if (const int c = h[p][threadIdx.x]) atomicAdd(&C->hist[p][threadIdx.x], c);
}

__global__ void k_keys_ext(DevScene S, const float* rays, uint32_t* keys, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* r = rays + size_t(i) * 8;
        keys[i] = morton_key(S, mk(r[0], r[1], r[2]), mk(r[4], r[5], r[6]));
    }
}

// exclusive sum over the block's 256 threads; ws: kWarps words
LUX_DI int block_exclusive(int v, int* ws) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    int base = 0;
    for (int w = 0; w < warp; ++w) base += ws[w];
    __syncthreads();
    return base + x - v;
}

// One pass of the radix sort: each tile's items ranked in shared memory, the counts of earlier
// tiles found by look-back (one thread per digit), the tile written out digit by digit.
// The pass is latency bound at these sizes (2M items move 32 MB a pass, 5 us at the measured
// copy rate), so it is one launch: a histogram, a scan of the tile table and a scatter as three
// launches, with the scan in one block, took 1.22 ms of a pass on 1.92M items. An 800x600, 4 spp,
// depth 8 render with sorting went from 10.12 to 3.18 ms (sorting alone 7.9 ms before).
__global__ void __launch_bounds__(kSortThreads) k_pass(const uint32_t* keys, const int* vals, uint32_t* okeys,
                                                       int* ovals, const int* nptr, int pass, SortCounters* C,
                                                       SortCounters* next, SortWord* words, int* err) {
    __shared__ int wh[kWarps][256];   // a warp's items per digit, then the first local place of each
    __shared__ int out0[256];         // place of local item 0 if it had the digit: out = out0 + local
    __shared__ uint32_t sk[kTile];
    __shared__ int sv[kTile];
    __shared__ int ws[kWarps];
    __shared__ int s_tile;
    const int n = *(volatile const int*)nptr;
    const int tiles = (n + kTile - 1) / kTile;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int shift = 8 * pass;
    if (pass == kPasses - 1 && blockIdx.x == 0) {
        for (int p = 0; p < kPasses; ++p) next->hist[p][tid] = 0;
        if (tid < kPasses) next->tile[tid] = 0;
    }
    if (int(blockIdx.x) >= tiles) return;
    const int digit0 = block_exclusive(C->hist[pass][tid], ws);  // first place of digit tid
    while (true) {
        if (tid == 0) s_tile = atomicAdd(&C->tile[pass], 1);
        for (int w = 0; w < kWarps; ++w) wh[w][tid] = 0;
        __syncthreads();
        const int tile = s_tile;
        if (tile >= tiles) break;
        const int64_t t0 = int64_t(tile) * kTile;
        const int count = int(min(int64_t(kTile), int64_t(n) - t0));
        uint32_t key[kItems];
        int val[kItems];
        int rank[kItems];
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const int k = warp * kWarpItems + j * 32 + lane;
            key[j] = k < count ? keys[t0 + k] : 0u;
            val[j] = k < count ? vals[t0 + k] : 0;
        }
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const bool ok = warp * kWarpItems + j * 32 + lane < count;
            const int dg = (key[j] >> shift) & 0xff;
            const unsigned peers = __match_any_sync(0xffffffffu, ok ? dg : 256);
            const int leader = __ffs(peers) - 1;
            int b = 0;
            if (ok && lane == leader) {
                b = wh[warp][dg];
                wh[warp][dg] = b + __popc(peers);
            }
            rank[j] = __shfl_sync(0xffffffffu, b, leader) + __popc(peers & lt);
            __syncwarp();
        }
        __syncthreads();
        // thread = digit: the tile's count, and each warp's first rank within it
        int total = 0;
        for (int w = 0; w < kWarps; ++w) {
            const int c = wh[w][tid];
            wh[w][tid] = total;
            total += c;
        }
        volatile SortWord* mine = words + size_t(tile) * 256 + tid;
        *mine = (tile == 0 ? kPrefix : kOwn) | SortWord(total);
        const int local0 = block_exclusive(total, ws);
        for (int w = 0; w < kWarps; ++w) wh[w][tid] += local0;
        SortWord before = 0;
        for (int t = tile - 1; t >= 0; --t) {
            volatile const SortWord* p = words + size_t(t) * 256 + tid;
            SortWord v = *p;
            for (int polls = 0; !(v & (kOwn | kPrefix)) && polls < kPollLimit; ++polls) v = *p;
            if (!(v & (kOwn | kPrefix))) atomicOr(err, kErrSort);
            before += v & kCount;
            if ((v & kPrefix) || !(v & kOwn)) break;
        }
        if (tile) *mine = kPrefix | (before + SortWord(total));
        out0[tid] = digit0 + int(before) - local0;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            if (warp * kWarpItems + j * 32 + lane < count) {
                const int at = wh[warp][(key[j] >> shift) & 0xff] + rank[j];
                sk[at] = key[j];
                sv[at] = val[j];
            }
        }
        __syncthreads();
        for (int k = tid; k < count; k += kSortThreads) {
            const uint32_t ky = sk[k];
            const int64_t o = out0[(ky >> shift) & 0xff] + k;
            if (o >= 0 && o < n) {  // always, unless a look-back gave up
                okeys[o] = ky;
                ovals[o] = sv[k];
            }
        }
        __syncthreads();
    }
}

}  // namespace

size_t morton_sort_temp_bytes(int max_paths) {
    const size_t tiles = (size_t(max_paths) + kTile - 1) / kTile;
    return 2 * sizeof(SortCounters) + tiles * kPasses * 256 * sizeof(SortWord);
}

cudaError_t clear_sort_counters(void* temp, cudaStream_t st) {
    return cudaMemsetAsync(temp, 0, 2 * sizeof(SortCounters), st);
}

cudaError_t launch_morton_sort(const DevScene& S, DevWave& W, int bounce, void* temp, size_t temp_bytes,
                               cudaStream_t st) {
    const int max_tiles = int((size_t(W.max_paths) + kTile - 1) / kTile);
    if (temp_bytes < morton_sort_temp_bytes(W.max_paths)) return cudaErrorInvalidValue;
    SortCounters* sets = static_cast<SortCounters*>(temp);
    SortCounters *C = sets + (bounce & 1), *next = sets + (1 - (bounce & 1));
    SortWord* words = reinterpret_cast<SortWord*>(sets + 2);
    const int* nptr = &W.ctr->count[bounce];
    int* err = &W.ctr->error;
    k_keys<<<148 * 4, kSortThreads, 0, st>>>(S, W, bounce, C, words, max_tiles);
    uint32_t* ka = W.keys;
    uint32_t* kb = W.keys_alt;
    int* va = W.queue[bounce & 1];
    int* vb = W.queue_alt;
    const int grid = std::max(1, std::min(max_tiles, 148 * 4));
    for (int pass = 0; pass < kPasses; ++pass) {
        k_pass<<<grid, kSortThreads, 0, st>>>(ka, va, kb, vb, nptr, pass, C, next,
                                              words + size_t(pass) * max_tiles * 256, err);
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    // four passes: the sorted queue is back in queue[bounce & 1]
    return cudaGetLastError();
}

cudaError_t launch_morton_ext(const DevScene& S, const float* rays, uint32_t* keys, int n, cudaStream_t st) {
    int grid = std::max(1, std::min((n + 255) / 256, 1184));
    k_keys_ext<<<grid, 256, 0, st>>>(S, rays, keys, n);
    return cudaGetLastError();
}

}  // namespace lux
