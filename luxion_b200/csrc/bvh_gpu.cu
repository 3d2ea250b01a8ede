// bvh_gpu.cu -- device build of the compressed 8-wide BVH (bvh_gpu.h).
//
// Binary stage (binned SAH, one primitive per leaf), over all trees at once:
//   * nodes of more than kMedium primitives are split level by level: their ranges are cut into
//     chunks of kChunk primitives, one block per chunk; a pass reduces each node's box and
//     centroid bounds, a pass bins the centroids (32 bins per live axis, shared-memory bins
//     merged into the node's bins with atomic min/max on order-preserving integer keys), one
//     thread per node sweeps the bins in double, and a stable two-pass scatter partitions the
//     node's range;
//   * a node of kSmall + 1 .. kMedium primitives is handed to one block, which splits it and its
//     descendants down to kSmall primitives in shared memory;
//   * a node of 2..kSmall primitives is handed to one warp, which builds its whole subtree with
//     one primitive per lane, shuffles for the reductions and the sweep, and a ballot for the
//     stable partition.
// Collapse stage, level by level over the 8-wide levels of all trees at once: eight lanes per
// 8-wide node open the child of largest area until 8 slots are filled, assign slots by child
// centroid octant and quantise the child boxes; a look-back over the level's tiles gives every
// node's children and leaf records their places, breadth first within its tree, trees one after
// another.
// Every floating-point step is the host builder's (bvh_build.cpp), rounded the same way, and
// every tie is broken the same way, so the nodes are identical to the host build's.

#include "bvh_gpu.h"
#include "host_common.h"

#include <cfloat>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>

namespace lux {

// Scratch of the device builds comes from one memory pool per device, owned by the library:
// allocations and frees are stream-ordered (no device-wide synchronisation, as cudaFree has),
// and up to kPoolKeep bytes of freed scratch stay reserved for the next build.
namespace {
constexpr uint64_t kPoolKeep = uint64_t(4) << 30;
std::mutex g_pool_mu;
std::map<int, cudaMemPool_t> g_pools;
}  // namespace

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t st) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaMemPool_t pool;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        auto it = g_pools.find(dev);
        if (it == g_pools.end()) {
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            if ((e = cudaMemPoolCreate(&pool, &props)) != cudaSuccess) return e;
            uint64_t keep = kPoolKeep;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
            g_pools[dev] = pool;
        } else {
            pool = it->second;
        }
    }
    cudaError_t r = cudaMallocFromPoolAsync(p, bytes, pool, st);
    if (r == cudaSuccess) note_device_alloc();
    return r;
}

void scratch_free(void* p, cudaStream_t st) {
    if (p) cudaFreeAsync(p, st);
}

namespace {

constexpr int kBins = 32;
constexpr int kSmall = 32;      // nodes of at most this many primitives: one warp per subtree
constexpr int kMedium = 1024;   // nodes of at most this many: one block down to kSmall
constexpr int kChunk = 2048;    // primitives per block in the large-node passes
constexpr int kBlock = 256;
constexpr int kPerThread = kChunk / kBlock;
constexpr unsigned FULL = 0xffffffffu;

struct BinNode {
    float lo[3], hi[3];
    int left, right;  // children (-1 for a leaf)
    int begin, count;
};

// Order-preserving map of floats to unsigned keys, for atomic min / max.
__device__ __forceinline__ unsigned fkey(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fval(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

__device__ __forceinline__ float cen(float lo, float hi) { return __fmul_rn(0.5f, __fadd_rn(lo, hi)); }

// bin of centroid coordinate c: int((double(c) - lo) * k1), clamped to the bins
__device__ __forceinline__ int bin_of(float c, float lo, double k1) {
    const int b = __double2int_rz(__dmul_rn(__dsub_rn(double(c), double(lo)), k1));
    return min(kBins - 1, max(0, b));
}

// surface area of a float box in double: 2 (dx dy + dy dz + dz dx), extents clamped at 0
__device__ __forceinline__ double area(const float* lo, const float* hi) {
    double d[3];
    for (int a = 0; a < 3; ++a) {
        const double x = __dsub_rn(double(hi[a]), double(lo[a]));
        d[a] = 0.0 < x ? x : 0.0;
    }
    return __dmul_rn(2.0, __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[1]), __dmul_rn(d[1], d[2])), __dmul_rn(d[2], d[0])));
}

// SAH cost area(L) nL + area(R) nR
__device__ __forceinline__ double sah(double al, int nl, double ar, int nr) {
    return __dadd_rn(__dmul_rn(al, double(nl)), __dmul_rn(ar, double(nr)));
}

__device__ __forceinline__ int ceil_log2(double x) {
    int k = 0;
    const double m = frexp(x, &k);
    return m == 0.5 ? k - 1 : k;
}

// ---------------------------------------------------------------------------------------------
// binary stage: set-up
// ---------------------------------------------------------------------------------------------

// Roots: node t is tree t's root; identity order; lists of large, medium and small roots; single-
// primitive trees are leaves at once.
__global__ void k_roots(const float* boxes, const int* tree_begin, int num_trees, BinNode* bn, int* ord0, int* ord_fin,
                        int* large, int* n_large, unsigned* medium, int* n_medium, int* small, int* n_small) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < num_trees; t += gridDim.x * blockDim.x) {
        const int b = tree_begin[t], n = tree_begin[t + 1] - b;
        BinNode& r = bn[t];
        r.begin = b;
        r.count = n;
        r.left = r.right = -1;
        if (n == 1) {
            for (int a = 0; a < 3; ++a) {
                r.lo[a] = boxes[size_t(b) * 6 + a];
                r.hi[a] = boxes[size_t(b) * 6 + 3 + a];
            }
            ord_fin[b] = b;
        } else if (n <= kSmall) {
            for (int i = 0; i < n; ++i) ord_fin[b + i] = b + i;
            small[atomicAdd(n_small, 1)] = t;
        } else if (n <= kMedium) {
            medium[atomicAdd(n_medium, 1)] = unsigned(t);  // its order is in buffer 0
        } else {
            large[atomicAdd(n_large, 1)] = t;
        }
    }
}

__global__ void k_iota(int* ord, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) ord[i] = i;
}

// ---------------------------------------------------------------------------------------------
// binary stage: one level of large nodes
// ---------------------------------------------------------------------------------------------

// Per-level-slot state of a large node.
struct Slot {
    unsigned red[12];     // keys: box lo[3], box hi[3], centroid lo[3], centroid hi[3]
    double k1[3];         // bins per unit of centroid extent, 0 for a dead axis
    float clo[3];         // centroid bounds minimum
    int live;             // bit a: axis a has a centroid extent
    int axis, split;      // chosen split: axis and last bin on the left; axis -1: halve by position
    int nl;               // primitives going left
    int chunk0, nchunk;   // the node's chunks in the level's chunk table
};

// Chunk table of the level: chunk c covers [chunk_start[c], +kChunk) of slot chunk_slot[c]'s
// range. One block: per-slot chunk counts, a block-wide exclusive scan, then the entries.
__global__ void __launch_bounds__(1024) k_chunks(const int* level, const int* n_level_ptr, const BinNode* bn,
                                                 Slot* slots, int* chunk_slot, int* chunk_start, int* n_chunks) {
    __shared__ int part[1024];
    const int n_level = *n_level_ptr;
    const int per = (n_level + 1023) / 1024;
    const int s0 = min(n_level, int(threadIdx.x) * per), s1 = min(n_level, s0 + per);
    int sum = 0;
    for (int s = s0; s < s1; ++s) sum += (bn[level[s]].count + kChunk - 1) / kChunk;
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const int v = threadIdx.x >= unsigned(off) ? part[threadIdx.x - off] : 0;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    int c = part[threadIdx.x] - sum;
    for (int s = s0; s < s1; ++s) {
        const BinNode& nd = bn[level[s]];
        const int k = (nd.count + kChunk - 1) / kChunk;
        slots[s].chunk0 = c;
        slots[s].nchunk = k;
        for (int r = 0; r < 12; ++r) slots[s].red[r] = (r < 3 || (r >= 6 && r < 9)) ? 0xffffffffu : 0u;
        for (int j = 0; j < k; ++j) {
            chunk_slot[c + j] = s;
            chunk_start[c + j] = nd.begin + j * kChunk;
        }
        c += k;
    }
    if (threadIdx.x == 1023) *n_chunks = part[1023];
}

__device__ __forceinline__ void load_prim(const float* boxes, int p, float* lo, float* hi) {
    const float* b = boxes + size_t(p) * 6;
    lo[0] = b[0], lo[1] = b[1], lo[2] = b[2];
    hi[0] = b[3], hi[1] = b[4], hi[2] = b[5];
}

// Box and centroid bounds of each large node, merged over its chunks.
__global__ void __launch_bounds__(kBlock) k_reduce(const float* boxes, const int* ord, const int* level, const BinNode* bn,
                                                   Slot* slots, const int* chunk_slot, const int* chunk_start,
                                                   const int* n_chunks) {
    __shared__ unsigned sh[12];
    const int nc = *n_chunks;
    for (int c = blockIdx.x; c < nc; c += gridDim.x) {
        const int s = chunk_slot[c];
        const BinNode& nd = bn[level[s]];
        const int p0 = chunk_start[c], p1 = min(nd.begin + nd.count, p0 + kChunk);
        unsigned r[12];
        for (int k = 0; k < 12; ++k) r[k] = (k < 3 || (k >= 6 && k < 9)) ? 0xffffffffu : 0u;
        for (int i = p0 + threadIdx.x; i < p1; i += kBlock) {
            float lo[3], hi[3];
            load_prim(boxes, ord[i], lo, hi);
            for (int a = 0; a < 3; ++a) {
                const float c3 = cen(lo[a], hi[a]);
                r[a] = min(r[a], fkey(lo[a]));
                r[3 + a] = max(r[3 + a], fkey(hi[a]));
                r[6 + a] = min(r[6 + a], fkey(c3));
                r[9 + a] = max(r[9 + a], fkey(c3));
            }
        }
        for (int k = 0; k < 12; ++k) {
            for (int off = 16; off > 0; off >>= 1) {
                const unsigned o = __shfl_xor_sync(FULL, r[k], off);
                r[k] = (k < 3 || (k >= 6 && k < 9)) ? min(r[k], o) : max(r[k], o);
            }
        }
        if (threadIdx.x < 12) sh[threadIdx.x] = (threadIdx.x < 3 || (threadIdx.x >= 6 && threadIdx.x < 9)) ? 0xffffffffu : 0u;
        __syncthreads();
        if ((threadIdx.x & 31) == 0)
            for (int k = 0; k < 12; ++k) {
                if (k < 3 || (k >= 6 && k < 9)) atomicMin(&sh[k], r[k]);
                else atomicMax(&sh[k], r[k]);
            }
        __syncthreads();
        if (threadIdx.x < 12) {
            const int k = threadIdx.x;
            if (k < 3 || (k >= 6 && k < 9)) atomicMin(&slots[s].red[k], sh[k]);
            else atomicMax(&slots[s].red[k], sh[k]);
        }
        __syncthreads();
    }
}

// Node boxes from the reductions; live axes and bin scales.
__global__ void k_bin_setup(const int* level, const int* n_level_ptr, BinNode* bn, Slot* slots) {
    const int n_level = *n_level_ptr;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n_level; s += gridDim.x * blockDim.x) {
        Slot& S = slots[s];
        BinNode& nd = bn[level[s]];
        S.live = 0;
        for (int a = 0; a < 3; ++a) {
            nd.lo[a] = fval(S.red[a]);
            nd.hi[a] = fval(S.red[3 + a]);
            const float clo = fval(S.red[6 + a]), chi = fval(S.red[9 + a]);
            const double ext = __dsub_rn(double(chi), double(clo));
            S.clo[a] = clo;
            if (ext > 0.0) {
                S.live |= 1 << a;
                S.k1[a] = __ddiv_rn(double(kBins), ext);
            } else {
                S.k1[a] = 0.0;
            }
        }
    }
}

// Bins of each large node: counts and boxes per live axis, merged over its chunks.
__global__ void __launch_bounds__(kBlock) k_bin(const float* boxes, const int* ord, const int* level, const BinNode* bn,
                                                const Slot* slots, const int* chunk_slot, const int* chunk_start,
                                                const int* n_chunks, unsigned* bin_cnt, unsigned* bin_lo,
                                                unsigned* bin_hi) {
    __shared__ unsigned cnt[3 * kBins];
    __shared__ unsigned blo[3 * kBins * 3], bhi[3 * kBins * 3];
    const int nc = *n_chunks;
    for (int c = blockIdx.x; c < nc; c += gridDim.x) {
        const int s = chunk_slot[c];
        const Slot& S = slots[s];
        const BinNode& nd = bn[level[s]];
        const int p0 = chunk_start[c], p1 = min(nd.begin + nd.count, p0 + kChunk);
        for (int b = threadIdx.x; b < 3 * kBins; b += kBlock) {
            cnt[b] = 0;
            for (int d = 0; d < 3; ++d) {
                blo[b * 3 + d] = 0xffffffffu;
                bhi[b * 3 + d] = 0u;
            }
        }
        __syncthreads();
        for (int i = p0 + threadIdx.x; i < p1; i += kBlock) {
            float lo[3], hi[3];
            load_prim(boxes, ord[i], lo, hi);
            for (int a = 0; a < 3; ++a) {
                if (!((S.live >> a) & 1)) continue;
                const int b = a * kBins + bin_of(cen(lo[a], hi[a]), S.clo[a], S.k1[a]);
                atomicAdd(&cnt[b], 1u);
                for (int d = 0; d < 3; ++d) {
                    atomicMin(&blo[b * 3 + d], fkey(lo[d]));
                    atomicMax(&bhi[b * 3 + d], fkey(hi[d]));
                }
            }
        }
        __syncthreads();
        for (int b = threadIdx.x; b < 3 * kBins; b += kBlock) {
            if (cnt[b] == 0) continue;
            const size_t g = size_t(s) * 3 * kBins + b;
            atomicAdd(&bin_cnt[g], cnt[b]);
            for (int d = 0; d < 3; ++d) {
                atomicMin(&bin_lo[g * 3 + d], blo[b * 3 + d]);
                atomicMax(&bin_hi[g * 3 + d], bhi[b * 3 + d]);
            }
        }
        __syncthreads();
    }
}

// The host builder's sweep over the non-empty bins of each live axis: the first split of
// lowest cost in (axis, bin) order; no live axis (or a one-sided split) halves the range.
// One warp per node, lane b = bin b: the box and count left of a split after bin b are a
// prefix union over lanes 0..b, those right of it a suffix union over lanes b+1..31 (empty
// bins contribute nothing), so every candidate's cost is the host's value exactly.
constexpr int kSplitWarps = 4;

// The sweep of one axis: lane b holds bin b's count n and box; (best, bsp, bnl) take the lane's
// split if it is the axis's candidate of lower cost than best. Whole warps call it.
__device__ __forceinline__ void sweep_axis(int a, int n, const float* lo, const float* hi, double& best, int& bax,
                                           int& bsp, int& bnl) {
    const int lane = threadIdx.x & 31;
    // inclusive prefix (left side) and inclusive suffix unions over the lanes
    float pl[3], ph[3], ql[3], qh[3];
    int pc = n, qc = n;
    for (int d = 0; d < 3; ++d) {
        pl[d] = ql[d] = lo[d];
        ph[d] = qh[d] = hi[d];
    }
    for (int off = 1; off < 32; off <<= 1) {
        const int uc = __shfl_up_sync(FULL, pc, off), dc = __shfl_down_sync(FULL, qc, off);
        float ul[3], uh[3], dl[3], dh[3];
        for (int d = 0; d < 3; ++d) {
            ul[d] = __shfl_up_sync(FULL, pl[d], off);
            uh[d] = __shfl_up_sync(FULL, ph[d], off);
            dl[d] = __shfl_down_sync(FULL, ql[d], off);
            dh[d] = __shfl_down_sync(FULL, qh[d], off);
        }
        if (lane >= off) {
            pc += uc;
            for (int d = 0; d < 3; ++d) {
                pl[d] = fminf(pl[d], ul[d]);
                ph[d] = fmaxf(ph[d], uh[d]);
            }
        }
        if (lane + off < 32) {
            qc += dc;
            for (int d = 0; d < 3; ++d) {
                ql[d] = fminf(ql[d], dl[d]);
                qh[d] = fmaxf(qh[d], dh[d]);
            }
        }
    }
    // right side of a split after bin b: the suffix from b + 1
    int rc = __shfl_down_sync(FULL, qc, 1);
    float rl[3], rh[3];
    for (int d = 0; d < 3; ++d) {
        rl[d] = __shfl_down_sync(FULL, ql[d], 1);
        rh[d] = __shfl_down_sync(FULL, qh[d], 1);
    }
    if (lane == 31) rc = 0;
    if (n > 0 && rc > 0) {
        const double c = sah(area(pl, ph), pc, area(rl, rh), rc);
        if (c < best) {  // axes ascend, so an earlier axis keeps a tie
            best = c;
            bax = a;
            bsp = lane;
            bnl = pc;
        }
    }
}

// Of all lanes' candidates the lowest (cost, axis, bin), in every lane.
__device__ __forceinline__ void best_split(double& best, int& bax, int& bsp, int& bnl) {
    for (int off = 16; off > 0; off >>= 1) {
        const double ob = __shfl_xor_sync(FULL, best, off);
        const int oa = __shfl_xor_sync(FULL, bax, off);
        const int os = __shfl_xor_sync(FULL, bsp, off);
        const int on = __shfl_xor_sync(FULL, bnl, off);
        if (ob < best || (ob == best && (oa < bax || (oa == bax && os < bsp)))) {
            best = ob;
            bax = oa;
            bsp = os;
            bnl = on;
        }
    }
}

__global__ void __launch_bounds__(32 * kSplitWarps) k_split(const int* level, const int* n_level_ptr, const BinNode* bn,
                                                             Slot* slots, const unsigned* bin_cnt,
                                                             const unsigned* bin_lo, const unsigned* bin_hi) {
    const int n_level = *n_level_ptr;
    const int lane = threadIdx.x & 31;
    for (int s = blockIdx.x * kSplitWarps + (threadIdx.x >> 5); s < n_level; s += gridDim.x * kSplitWarps) {
        Slot& S = slots[s];
        const BinNode& nd = bn[level[s]];
        double best = DBL_MAX;
        int bax = 3, bsp = kBins, bnl = 0;
        for (int a = 0; a < 3; ++a) {
            if (!((S.live >> a) & 1)) continue;
            const size_t g = size_t(s) * 3 * kBins + size_t(a) * kBins + lane;
            const int n = int(bin_cnt[g]);
            float lo[3], hi[3];
            for (int d = 0; d < 3; ++d) {
                lo[d] = n ? fval(bin_lo[g * 3 + d]) : FLT_MAX;
                hi[d] = n ? fval(bin_hi[g * 3 + d]) : -FLT_MAX;
            }
            sweep_axis(a, n, lo, hi, best, bax, bsp, bnl);
        }
        best_split(best, bax, bsp, bnl);
        if (lane == 0) {
            int axis = bax < 3 ? bax : -1;
            if (axis >= 0 && (bnl <= 0 || bnl >= nd.count)) axis = -1;
            S.axis = axis;
            S.split = axis >= 0 ? bsp : -1;
            S.nl = axis >= 0 ? bnl : nd.count / 2;
        }
    }
}

__device__ __forceinline__ bool goes_left(const Slot& S, const float* boxes, int p, int rel) {
    if (S.axis < 0) return rel < S.nl;
    const float* b = boxes + size_t(p) * 6;
    const int a = S.axis;
    return bin_of(cen(b[a], b[3 + a]), S.clo[a], S.k1[a]) <= S.split;
}

__global__ void __launch_bounds__(kBlock) k_count_left(const float* boxes, const int* ord, const int* level,
                                                       const BinNode* bn, const Slot* slots, const int* chunk_slot,
                                                       const int* chunk_start, const int* n_chunks, int* chunk_left) {
    __shared__ int sh[kBlock / 32];
    const int nc = *n_chunks;
    for (int c = blockIdx.x; c < nc; c += gridDim.x) {
        const int s = chunk_slot[c];
        const Slot& S = slots[s];
        const BinNode& nd = bn[level[s]];
        const int p0 = chunk_start[c], p1 = min(nd.begin + nd.count, p0 + kChunk);
        int k = 0;
        for (int i = p0 + threadIdx.x; i < p1; i += kBlock) k += goes_left(S, boxes, ord[i], i - nd.begin) ? 1 : 0;
        for (int off = 16; off > 0; off >>= 1) k += __shfl_xor_sync(FULL, k, off);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = k;
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
            for (int w = 0; w < kBlock / 32; ++w) t += sh[w];
            chunk_left[c] = t;
        }
        __syncthreads();
    }
}

// Exclusive prefix of the left counts over each node's chunks.
__global__ void k_chunk_base(const int* n_level_ptr, const Slot* slots, const int* chunk_left, int* chunk_lbase) {
    const int n_level = *n_level_ptr;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n_level; s += gridDim.x * blockDim.x) {
        int run = 0;
        for (int j = 0; j < slots[s].nchunk; ++j) {
            chunk_lbase[slots[s].chunk0 + j] = run;
            run += chunk_left[slots[s].chunk0 + j];
        }
    }
}

// Empty bins of the level's nodes: count 0, minimum keys all ones, maximum keys zero.
__global__ void k_bin_clear(const int* n_level_ptr, unsigned* bin_cnt, unsigned* bin_lo, unsigned* bin_hi) {
    const size_t n = size_t(*n_level_ptr) * 3 * kBins;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        bin_cnt[i] = 0u;
        for (int d = 0; d < 3; ++d) {
            bin_lo[i * 3 + d] = 0xffffffffu;
            bin_hi[i * 3 + d] = 0u;
        }
    }
}

// After a level: the next binary ids start past its children, and its list count is cleared
// for the level after next (the two lists alternate).
__global__ void k_level_advance(int* n_level_cur, int* next_id) {
    *next_id += 2 * *n_level_cur;
    *n_level_cur = 0;
}

// Stable partition: each chunk's primitives, in order, to the left or right part of the range.
__global__ void __launch_bounds__(kBlock) k_scatter(const float* boxes, const int* ord, int* ord_next, const int* level,
                                                    const BinNode* bn, const Slot* slots, const int* chunk_slot,
                                                    const int* chunk_start, const int* n_chunks,
                                                    const int* chunk_lbase) {
    __shared__ int sh[kBlock / 32];
    const int nc = *n_chunks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = blockIdx.x; c < nc; c += gridDim.x) {
        const int s = chunk_slot[c];
        const Slot& S = slots[s];
        const BinNode& nd = bn[level[s]];
        const int p0 = chunk_start[c], p1 = min(nd.begin + nd.count, p0 + kChunk);
        // thread t owns positions p0 + t*kPerThread .. + kPerThread - 1 (in order)
        int prim[kPerThread];
        bool left[kPerThread];
        int mine = 0;
        for (int k = 0; k < kPerThread; ++k) {
            const int i = p0 + int(threadIdx.x) * kPerThread + k;
            prim[k] = i < p1 ? ord[i] : -1;
            left[k] = i < p1 && goes_left(S, boxes, prim[k], i - nd.begin);
            mine += left[k] ? 1 : 0;
        }
        int incl = mine;
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(FULL, incl, off);
            if (lane >= off) incl += v;
        }
        if (lane == 31) sh[warp] = incl;
        __syncthreads();
        int wbase = 0;
        for (int w = 0; w < warp; ++w) wbase += sh[w];
        int lrank = chunk_lbase[c] + wbase + incl - mine;   // lefts before this thread's first
        int pos_in_chunk = int(threadIdx.x) * kPerThread;
        const int chunk_rel = p0 - nd.begin;
        for (int k = 0; k < kPerThread; ++k) {
            const int i = p0 + pos_in_chunk + k;
            if (i >= p1) break;
            if (left[k]) {
                ord_next[nd.begin + lrank] = prim[k];
                ++lrank;
            } else {
                const int rrank = (chunk_rel + pos_in_chunk + k) - lrank;  // rights before it in the node
                ord_next[nd.begin + S.nl + rrank] = prim[k];
            }
        }
        __syncthreads();
    }
}

// Children of the level's nodes: ids next_id + 2 s and + 1; leaves take their primitive's box
// at once, small children go to the warp list (their range copied to the final order), medium ones
// to the block list (with the order buffer their range stays in), large children to the next level.
// Child ids continue from *next_id (k_level_advance moves it on); ids past bn_cap set *err
// and the level stops there.
__global__ void k_children(const float* boxes, const int* ord_next, int* ord_fin, const int* level,
                           const int* n_level_ptr, BinNode* bn, const Slot* slots, const int* next_id_ptr,
                           int bn_cap, int* err, int* large_next, int* n_large_next, unsigned* medium, int* n_medium,
                           unsigned buffer, int* small, int* n_small) {
    const int n_level = *n_level_ptr, next_id = *next_id_ptr;
    if (n_level > 0 && next_id + 2 * n_level > bn_cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *err = 1;
        return;
    }
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n_level; s += gridDim.x * blockDim.x) {
        BinNode& nd = bn[level[s]];
        const int nl = slots[s].nl;
        const int ids[2] = {next_id + 2 * s, next_id + 2 * s + 1};
        const int beg[2] = {nd.begin, nd.begin + nl};
        const int cnt[2] = {nl, nd.count - nl};
        nd.left = ids[0];
        nd.right = ids[1];
        for (int k = 0; k < 2; ++k) {
            BinNode& ch = bn[ids[k]];
            ch.begin = beg[k];
            ch.count = cnt[k];
            ch.left = ch.right = -1;
            if (cnt[k] == 1) {
                const int p = ord_next[beg[k]];
                load_prim(boxes, p, ch.lo, ch.hi);
                ord_fin[beg[k]] = p;
            } else if (cnt[k] <= kSmall) {
                for (int i = 0; i < cnt[k]; ++i) ord_fin[beg[k] + i] = ord_next[beg[k] + i];
                small[atomicAdd(n_small, 1)] = ids[k];
            } else if (cnt[k] <= kMedium) {
                medium[atomicAdd(n_medium, 1)] = unsigned(ids[k]) | buffer << 31;
            } else {
                large_next[atomicAdd(n_large_next, 1)] = ids[k];
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// binary stage: subtrees of at most kMedium primitives down to kSmall, one block each
// ---------------------------------------------------------------------------------------------

// The passes of one level of large nodes (bounds, bins, sweep, stable partition) on a node in
// shared memory, node after node: below kMedium primitives the levels' eleven launches each, with
// a few us of work, were the larger part of the binary stage (1M triangles: 9 of its 25 levels and
// 4.0 ms of kernels; now 16 levels, 2.1 ms, and 0.59 ms here).
// 31 KB of shared memory, so seven blocks share an SM and hide one another's barriers.
__global__ void __launch_bounds__(kBlock) k_medium(const float* boxes, const int* ord0, const int* ord1,
                                                   const unsigned* medium, const int* n_medium_ptr, BinNode* bn,
                                                   int bn_cap, int* next_id, int* err, int* ord_fin, int* small,
                                                   int* n_small) {
    constexpr int kPer = kMedium / kBlock;
    constexpr int kWarps = kBlock / 32;
    __shared__ float sb[6][kMedium];
    __shared__ int sid[kMedium];
    __shared__ unsigned cnt[3 * kBins], blo[3 * kBins * 3], bhi[3 * kBins * 3];
    __shared__ unsigned red[12];
    __shared__ double s_cost[3], k1[3];
    __shared__ float clo[3];
    __shared__ int s_bin[3], s_nl[3], live[3], wsum[kWarps], s_ids;
    // nodes to split: the smaller child is taken first, so few wait
    __shared__ int st_node[16], st_at[16], st_n[16];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_medium = *n_medium_ptr;
    for (int w = blockIdx.x; w < n_medium; w += gridDim.x) {
        const int root = int(medium[w] & 0x7fffffffu);
        const int* ord = (medium[w] >> 31) ? ord1 : ord0;
        const int base = bn[root].begin, n0 = min(bn[root].count, kMedium);
        for (int i = tid; i < n0; i += kBlock) {
            const int p = ord[base + i];
            float lo[3], hi[3];
            load_prim(boxes, p, lo, hi);
            sid[i] = p;
            for (int a = 0; a < 3; ++a) {
                sb[a][i] = lo[a];
                sb[3 + a][i] = hi[a];
            }
        }
        int sp = 1;
        if (tid == 0) {
            st_node[0] = root;
            st_at[0] = 0;
            st_n[0] = n0;
        }
        __syncthreads();
        while (sp > 0) {
            --sp;
            const int node = st_node[sp], at = st_at[sp], n = st_n[sp];
            // bounds
            if (tid < 12) red[tid] = (tid < 3 || (tid >= 6 && tid < 9)) ? 0xffffffffu : 0u;
            for (int b = tid; b < 3 * kBins; b += kBlock) {
                cnt[b] = 0;
                for (int d = 0; d < 3; ++d) {
                    blo[b * 3 + d] = 0xffffffffu;
                    bhi[b * 3 + d] = 0u;
                }
            }
            unsigned r[12];
            for (int k = 0; k < 12; ++k) r[k] = (k < 3 || (k >= 6 && k < 9)) ? 0xffffffffu : 0u;
            for (int i = tid; i < n; i += kBlock)
                for (int a = 0; a < 3; ++a) {
                    const float l = sb[a][at + i], h = sb[3 + a][at + i], c = cen(l, h);
                    r[a] = min(r[a], fkey(l));
                    r[3 + a] = max(r[3 + a], fkey(h));
                    r[6 + a] = min(r[6 + a], fkey(c));
                    r[9 + a] = max(r[9 + a], fkey(c));
                }
            __syncthreads();
            if (warp * 32 < n) {
                for (int k = 0; k < 12; ++k) {
                    const bool mn = k < 3 || (k >= 6 && k < 9);
                    r[k] = mn ? __reduce_min_sync(FULL, r[k]) : __reduce_max_sync(FULL, r[k]);
                    if (lane == 0) {
                        if (mn) atomicMin(&red[k], r[k]);
                        else atomicMax(&red[k], r[k]);
                    }
                }
            }
            __syncthreads();
            if (tid < 3) {
                bn[node].lo[tid] = fval(red[tid]);
                bn[node].hi[tid] = fval(red[3 + tid]);
                const float cl = fval(red[6 + tid]), ch = fval(red[9 + tid]);
                const double ext = __dsub_rn(double(ch), double(cl));
                clo[tid] = cl;
                live[tid] = ext > 0.0;
                k1[tid] = ext > 0.0 ? __ddiv_rn(double(kBins), ext) : 0.0;
            }
            __syncthreads();
            // bins
            for (int i = tid; i < n; i += kBlock) {
                unsigned lk[3], hk[3];
                for (int d = 0; d < 3; ++d) {
                    lk[d] = fkey(sb[d][at + i]);
                    hk[d] = fkey(sb[3 + d][at + i]);
                }
                for (int a = 0; a < 3; ++a) {
                    if (!live[a]) continue;
                    const int b = a * kBins + bin_of(cen(sb[a][at + i], sb[3 + a][at + i]), clo[a], k1[a]);
                    atomicAdd(&cnt[b], 1u);
                    for (int d = 0; d < 3; ++d) {
                        atomicMin(&blo[b * 3 + d], lk[d]);
                        atomicMax(&bhi[b * 3 + d], hk[d]);
                    }
                }
            }
            __syncthreads();
            // sweep: one warp per axis, lane = bin
            if (warp < 3) {
                double best = DBL_MAX;
                int bax = 3, bsp = kBins, bnl = 0;
                if (live[warp]) {
                    const int g = warp * kBins + lane;
                    const int c = int(cnt[g]);
                    float lo[3], hi[3];
                    for (int d = 0; d < 3; ++d) {
                        lo[d] = c ? fval(blo[g * 3 + d]) : FLT_MAX;
                        hi[d] = c ? fval(bhi[g * 3 + d]) : -FLT_MAX;
                    }
                    sweep_axis(warp, c, lo, hi, best, bax, bsp, bnl);
                    best_split(best, bax, bsp, bnl);
                }
                if (lane == 0) {
                    s_cost[warp] = bax < 3 ? best : DBL_MAX;
                    s_bin[warp] = bax < 3 ? bsp : -1;
                    s_nl[warp] = bnl;
                }
            }
            if (tid == 96) s_ids = atomicAdd(next_id, 2);
            __syncthreads();
            int axis = -1;
            for (int a = 0; a < 3; ++a)
                if (s_bin[a] >= 0 && (axis < 0 || s_cost[a] < s_cost[axis])) axis = a;
            if (axis >= 0 && (s_nl[axis] <= 0 || s_nl[axis] >= n)) axis = -1;
            const int split = axis >= 0 ? s_bin[axis] : -1;
            const int nl = axis >= 0 ? s_nl[axis] : n / 2;
            const int id = s_ids;
            if (id + 2 > bn_cap) {
                if (tid == 0) *err = 1;
                break;
            }
            // stable partition: thread t owns positions t * per .. t * per + per - 1, in registers
            const int per = (n + kBlock - 1) / kBlock;
            float pb[kPer][6];
            int pp[kPer];
            unsigned lmask = 0;
            int mine = 0;
            for (int k = 0; k < kPer; ++k) {
                const int i = tid * per + k;
                if (k >= per || i >= n) break;
                pp[k] = sid[at + i];
                for (int d = 0; d < 6; ++d) pb[k][d] = sb[d][at + i];
                const bool left = axis < 0 ? i < nl : bin_of(cen(sb[axis][at + i], sb[3 + axis][at + i]), clo[axis], k1[axis]) <= split;
                if (left) {
                    lmask |= 1u << k;
                    ++mine;
                }
            }
            int incl = mine;
            for (int off = 1; off < 32; off <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, off);
                if (lane >= off) incl += v;
            }
            if (lane == 31) wsum[warp] = incl;
            __syncthreads();
            int lrank = incl - mine;
            for (int v = 0; v < warp; ++v) lrank += wsum[v];
            for (int k = 0; k < kPer; ++k) {
                const int i = tid * per + k;
                if (k >= per || i >= n) break;
                const bool left = (lmask >> k) & 1u;
                const int to = at + (left ? lrank : nl + (i - lrank));
                lrank += left ? 1 : 0;
                sid[to] = pp[k];
                for (int d = 0; d < 6; ++d) sb[d][to] = pb[k][d];
            }
            __syncthreads();
            // children: leaves and small subtrees leave the block, the others wait here
            if (tid == 0) {
                bn[node].left = id;
                bn[node].right = id + 1;
            }
            const int first = nl > n - nl ? 0 : 1;  // the larger child waits below the smaller
            for (int j = 0; j < 2; ++j) {
                const int k = j == 0 ? first : 1 - first;
                const int cat = k ? at + nl : at, cn = k ? n - nl : nl;
                if (tid == 0) {
                    BinNode& ch = bn[id + k];
                    ch.begin = base + cat;
                    ch.count = cn;
                    ch.left = ch.right = -1;
                    if (cn == 1)
                        for (int a = 0; a < 3; ++a) {
                            ch.lo[a] = sb[a][cat];
                            ch.hi[a] = sb[3 + a][cat];
                        }
                    else if (cn <= kSmall) small[atomicAdd(n_small, 1)] = id + k;
                }
                if (cn <= kSmall) {
                    if (tid < cn) ord_fin[base + cat + tid] = sid[cat + tid];
                } else if (sp < 16) {
                    if (tid == 0) {
                        st_node[sp] = id + k;
                        st_at[sp] = cat;
                        st_n[sp] = cn;
                    }
                    ++sp;
                } else if (tid == 0) {
                    *err = 1;  // cannot be: each waiting node is at least as large as all above it
                }
            }
            __syncthreads();
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------
// binary stage: subtrees of at most kSmall primitives, one warp each
// ---------------------------------------------------------------------------------------------

constexpr int kSmallWarps = 4;

__device__ __forceinline__ float wmin(float v) {
    for (int off = 16; off > 0; off >>= 1) v = fminf(v, __shfl_xor_sync(FULL, v, off));
    return v;
}
__device__ __forceinline__ float wmax(float v) {
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(FULL, v, off));
    return v;
}

// All nodes of one depth of the subtree are split together: lanes lb .. lb + n - 1 hold a node's
// primitives in order, so every step is a segmented warp operation, and a subtree takes its depth
// in steps instead of its node count (1M triangles: 1.15 ms node by node, 0.48 so).
__global__ void __launch_bounds__(32 * kSmallWarps) k_small(const float* boxes, const int* small, const int* n_small_ptr,
                                                            BinNode* bn, int* ord_fin, int* bn_next) {
    __shared__ int perm[kSmallWarps][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int n_small = *n_small_ptr;
    const unsigned lt = (1u << lane) - 1u;
    for (int w = blockIdx.x * kSmallWarps + wib; w < n_small; w += gridDim.x * kSmallWarps) {
        int node = small[w];  // the node of this lane's segment
        const int begin0 = bn[node].begin, cnt0 = min(bn[node].count, kSmall);   // 2 .. kSmall
        int pid = -1;
        float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX}, c[3] = {0.f, 0.f, 0.f};
        int lb = 0, n = cnt0;  // the lane's segment; lanes past the subtree are segments of their own
        if (lane < cnt0) {
            pid = ord_fin[begin0 + lane];
            load_prim(boxes, pid, lo, hi);
            for (int a = 0; a < 3; ++a) c[a] = cen(lo[a], hi[a]);
        } else {
            lb = lane;
            n = 1;
        }
        int next = 0;
        if (lane == 0) next = atomicAdd(bn_next, 2 * cnt0 - 2);
        next = __shfl_sync(FULL, next, 0);
        while (true) {
            const bool in = n > 1;
            if (!__any_sync(FULL, in)) break;
            const bool leader = in && lane == lb;
            const int end = lb + n - 1;  // last lane of the segment
            // box and centroid bounds: segmented inclusive scans, then the last lane's value
            float nlo[3], nhi[3], clo[3], chi[3];
            for (int a = 0; a < 3; ++a) {
                nlo[a] = lo[a];
                nhi[a] = hi[a];
                clo[a] = chi[a] = c[a];
                for (int off = 1; off < 32; off <<= 1) {
                    const float x0 = __shfl_up_sync(FULL, nlo[a], off), x1 = __shfl_up_sync(FULL, nhi[a], off);
                    const float x2 = __shfl_up_sync(FULL, clo[a], off), x3 = __shfl_up_sync(FULL, chi[a], off);
                    if (lane - off >= lb) {
                        nlo[a] = fminf(nlo[a], x0);
                        nhi[a] = fmaxf(nhi[a], x1);
                        clo[a] = fminf(clo[a], x2);
                        chi[a] = fmaxf(chi[a], x3);
                    }
                }
                nlo[a] = __shfl_sync(FULL, nlo[a], end);
                nhi[a] = __shfl_sync(FULL, nhi[a], end);
                clo[a] = __shfl_sync(FULL, clo[a], end);
                chi[a] = __shfl_sync(FULL, chi[a], end);
            }
            if (leader)
                for (int a = 0; a < 3; ++a) {
                    bn[node].lo[a] = nlo[a];
                    bn[node].hi[a] = nhi[a];
                }
            int newpos = lane;      // position after the partition
            int mid = lb + n / 2;   // coincident centroids: halve by position
            // two primitives: the first axis with a centroid extent decides, the smaller centroid
            // goes left
            bool swap = false, decided = false;
            for (int a = 0; a < 3; ++a) {
                const float c0 = __shfl_sync(FULL, c[a], lb), c1 = __shfl_sync(FULL, c[a], end);
                if (!decided && __dsub_rn(double(chi[a]), double(clo[a])) > 0.0) {
                    swap = c1 < c0;
                    decided = true;
                }
            }
            if (n == 2) {
                if (swap) newpos = lane == lb ? lb + 1 : lb;
                mid = lb + 1;
            }
            const bool sahn = n > 2;
            if (__any_sync(FULL, sahn)) {
                const int longest = __reduce_max_sync(FULL, sahn ? n : 0);
                int bin[3] = {0, 0, 0};
                int live = 0;
                for (int a = 0; a < 3; ++a) {
                    const double ext = __dsub_rn(double(chi[a]), double(clo[a]));
                    if (sahn && ext > 0.0) {
                        live |= 1 << a;
                        bin[a] = bin_of(c[a], clo[a], __ddiv_rn(double(kBins), ext));
                    }
                }
                // each lane evaluates the split after its own bin on every live axis
                double best = DBL_MAX;
                int bax = 3, bsp = kBins, bnl = 0;
                bool any = false;
                for (int a = 0; a < 3; ++a) {
                    if (!__any_sync(FULL, (live >> a) & 1)) continue;
                    float l_lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, l_hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
                    float r_lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, r_hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
                    int nl = 0, nr = 0;
                    for (int t = 0; t < longest; ++t) {
                        const int m = min(lb + t, end);
                        const int bm = __shfl_sync(FULL, bin[a], m);
                        float mlo[3], mhi[3];
                        for (int d = 0; d < 3; ++d) {
                            mlo[d] = __shfl_sync(FULL, lo[d], m);
                            mhi[d] = __shfl_sync(FULL, hi[d], m);
                        }
                        if (t >= n) continue;
                        if (bm <= bin[a]) {
                            for (int d = 0; d < 3; ++d) {
                                l_lo[d] = fminf(l_lo[d], mlo[d]);
                                l_hi[d] = fmaxf(l_hi[d], mhi[d]);
                            }
                            ++nl;
                        } else {
                            for (int d = 0; d < 3; ++d) {
                                r_lo[d] = fminf(r_lo[d], mlo[d]);
                                r_hi[d] = fmaxf(r_hi[d], mhi[d]);
                            }
                            ++nr;
                        }
                    }
                    if (((live >> a) & 1) && nr > 0) {
                        const double cst = sah(area(l_lo, l_hi), nl, area(r_lo, r_hi), nr);
                        if (!any || cst < best) {  // axes ascend, so the first wins ties
                            best = cst;
                            bax = a;
                            bsp = bin[a];
                            bnl = nl;
                            any = true;
                        }
                    }
                }
                // the segment's lowest (cost, axis, bin)
                for (int off = 1; off < 32; off <<= 1) {
                    const double ob = __shfl_up_sync(FULL, best, off);
                    const int oa = __shfl_up_sync(FULL, bax, off);
                    const int os = __shfl_up_sync(FULL, bsp, off);
                    const int on = __shfl_up_sync(FULL, bnl, off);
                    if (lane - off >= lb && (ob < best || (ob == best && (oa < bax || (oa == bax && os < bsp))))) {
                        best = ob;
                        bax = oa;
                        bsp = os;
                        bnl = on;
                    }
                }
                bax = __shfl_sync(FULL, bax, end);
                bsp = __shfl_sync(FULL, bsp, end);
                bnl = __shfl_sync(FULL, bnl, end);
                const bool part = sahn && bax < 3 && bnl > 0 && bnl < n;
                const int mybin = bax == 0 ? bin[0] : (bax == 1 ? bin[1] : bin[2]);
                const unsigned lm = __ballot_sync(FULL, part && mybin <= bsp);
                if (part) {
                    const unsigned seg = (n == 32 ? FULL : (1u << n) - 1u) << lb;
                    const int nl = __popc(lm & seg);
                    newpos = (lm >> lane) & 1u ? lb + __popc(lm & seg & lt) : lb + nl + __popc(~lm & seg & lt);
                    mid = lb + nl;
                }
            }
            // apply the permutation (lanes move to newpos)
            perm[wib][newpos] = lane;
            __syncwarp();
            const int src = perm[wib][lane];
            __syncwarp();
            pid = __shfl_sync(FULL, pid, src);
            for (int a = 0; a < 3; ++a) {
                lo[a] = __shfl_sync(FULL, lo[a], src);
                hi[a] = __shfl_sync(FULL, hi[a], src);
                c[a] = __shfl_sync(FULL, c[a], src);
            }
            // children: two ids per segment
            const unsigned leaders = __ballot_sync(FULL, leader);
            const int id = next + 2 * __popc(leaders & ((1u << lb) - 1u));
            next += 2 * __popc(leaders);
            if (in) {
                const bool right = lane >= mid;
                if (leader) {
                    bn[node].left = id;
                    bn[node].right = id + 1;
                }
                const int e = lb + n;
                lb = right ? mid : lb;
                n = right ? e - mid : mid - lb;
                node = id + (right ? 1 : 0);
                if (lane == lb) {
                    BinNode& ch = bn[node];
                    ch.begin = begin0 + lb;
                    ch.count = n;
                    ch.left = ch.right = -1;
                    if (n == 1) {
                        for (int a = 0; a < 3; ++a) {
                            ch.lo[a] = lo[a];
                            ch.hi[a] = hi[a];
                        }
                        ord_fin[begin0 + lane] = pid;
                    }
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// collapse stage
// ---------------------------------------------------------------------------------------------

struct Item {
    int bnode;
    int tree;
};

// Look-back words of the collapse: bits 62-63 the state (0 not yet, 1 the tile's own counts, 2 those
// of it and all earlier tiles of the level), then the leaf and internal children, 31 bits each.
using TileWord = unsigned long long;
constexpr TileWord kOwn = TileWord(1) << 62, kPrefix = TileWord(2) << 62, kCounts = kOwn - 1;
constexpr TileWord kIntMask = (TileWord(1) << 31) - 1;
// Polls of a word before a look-back gives up (err): tiles are taken in order by running blocks.
constexpr int kPollLimit = 1 << 22;
constexpr int kMaxLevels = 120;  // 8-wide levels
constexpr int kColThreads = 256;
constexpr int kColItems = kColThreads / 8;  // items of a tile, eight lanes each

// One level of 8-wide nodes: level l of the table (lvl[2 l]: offset of its items, lvl[2 l + 1]: their
// number). Per item: its children, slots and quantised boxes (child_base and tri_base are placed
// later) and the primitives of its leaf slots in slot order; cs and ls: internal children and leaf
// slots of the level's earlier items; the next level's items, in order, right after this level's,
// and its entry in the table. Past the capacity it is left empty and err is set.
// Eight lanes hold an item's children, one each: a thread per item kept them in local memory and
// took about 100 us a level however few items it had, and the places took eight more launches
// (1M triangles, 11 levels: 1.08 ms and 88 launches of 0.4 ms; 0.46 ms so).
__global__ void __launch_bounds__(kColThreads) k_collapse(int* lvl, int l, Item* items_all, const BinNode* bn,
                                                          const int* ord_fin, BVH8Node* tmp_all, int* n_leaf_all,
                                                          int* cs_all, int* ls_all, int* leaf_prim_all,
                                                          TileWord* words_all, int* tile_ctr, long long cap, int* err) {
    __shared__ BVH8Node s_node[kColItems];
    __shared__ TileWord s_count[kColItems];
    __shared__ int s_tile;
    const int o = lvl[2 * l], n_items = lvl[2 * l + 1];
    const int tiles = (n_items + kColItems - 1) / kColItems;
    const Item* items = items_all + o;
    TileWord* words = words_all + o / kColItems + l;
    const int lane = threadIdx.x & 31, j = threadIdx.x & 7, g = threadIdx.x >> 3, g0 = lane & ~7;
    while (true) {
        if (threadIdx.x == 0) s_tile = atomicAdd(tile_ctr + l, 1);
        __syncthreads();
        const int tile = s_tile;
        if (tile >= tiles) break;
        const int it = tile * kColItems + g;
        const bool on = it < n_items;
        const Item item = on ? items[it] : Item{0, 0};
        const BinNode b = bn[item.bnode];
        // children: lane j holds child j
        int nch = 1, id = -1;
        bool open = false;
        if (b.left < 0 || b.count <= kMaxLeafPrims) {
            if (j == 0) id = item.bnode;
        } else {
            nch = 2;
            if (j < 2) id = j == 0 ? b.left : b.right;
            open = true;
        }
        BinNode c = bn[id < 0 ? 0 : id];
        for (int round = 0; round < 6; ++round) {  // two children at first, eight at most
            // the child of largest area that is no leaf, the first of equals
            double pa = -1.0;
            int pick = -1;
            if (open && j < nch && c.left >= 0 && c.count > kMaxLeafPrims) {
                const double a = area(c.lo, c.hi);
                if (a > pa) {
                    pa = a;
                    pick = j;
                }
            }
            for (int off = 1; off < 8; off <<= 1) {
                const double oa = __shfl_xor_sync(FULL, pa, off);
                const int op = __shfl_xor_sync(FULL, pick, off);
                if (oa > pa || (oa == pa && op >= 0 && (pick < 0 || op < pick))) {
                    pa = oa;
                    pick = op;
                }
            }
            pick = __shfl_sync(FULL, pick, g0);
            open = open && pick >= 0;
            const int from = g0 + (pick < 0 ? 0 : pick);
            const int cl = __shfl_sync(FULL, c.left, from), cr = __shfl_sync(FULL, c.right, from);
            if (open) {
                if (j == pick || j == nch) {
                    id = j == pick ? cl : cr;
                    c = bn[id];
                }
                ++nch;
            }
            if (!__any_sync(FULL, open)) break;
        }
        // slots by centroid octant around the node centre, cheapest (child, slot) pairs first
        const bool child = j < nch;
        double d[3], cost[8];
        for (int a = 0; a < 3; ++a)
            d[a] = __dsub_rn(__dmul_rn(0.5, __dadd_rn(double(c.lo[a]), double(c.hi[a]))), double(cen(b.lo[a], b.hi[a])));
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            double v = 0.0;
            for (int a = 0; a < 3; ++a) v = __dadd_rn(v, ((s >> a) & 1) ? -d[a] : d[a]);
            cost[s] = v;
        }
        unsigned used = 0;
        int slot = -1;
        const int rounds = __reduce_max_sync(FULL, nch);
        for (int round = 0; round < rounds; ++round) {
            double best = 0.0;
            int bs = -1;
            if (child && slot < 0) {
#pragma unroll
                for (int s = 0; s < 8; ++s)
                    if (!((used >> s) & 1u) && (bs < 0 || cost[s] < best)) {
                        best = cost[s];
                        bs = s;
                    }
            }
            int bk = bs >= 0 ? j : -1;
            for (int off = 1; off < 8; off <<= 1) {
                const double oc = __shfl_xor_sync(FULL, best, off);
                const int ok = __shfl_xor_sync(FULL, bk, off), os = __shfl_xor_sync(FULL, bs, off);
                if (ok >= 0 && (bk < 0 || oc < best || (oc == best && ok < bk))) {
                    best = oc;
                    bk = ok;
                    bs = os;
                }
            }
            // one lane's answer for the group, whatever the comparisons did on values not ordered
            bk = __shfl_sync(FULL, bk, g0);
            bs = __shfl_sync(FULL, bs, g0);
            if (bk >= 0) {
                used |= 1u << bs;
                if (j == bk) slot = bs;
            }
        }
        if (!child) {  // the empty slots, in order
            int k = j - nch;
            for (int s = 0; s < 8; ++s)
                if (!((used >> s) & 1u) && k-- == 0) slot = s;
        }
        // quantisation (encode_node of the host builder)
        double mext = 0.0, mabs = 0.0;
        for (int a = 0; a < 3; ++a) {
            mext = fmax(mext, __dsub_rn(double(b.hi[a]), double(b.lo[a])));
            mabs = fmax(mabs, fmax(fabs(double(b.lo[a])), fabs(double(b.hi[a]))));
        }
        const double pad = __dadd_rn(__dadd_rn(__dmul_rn(1e-4, mext), __dmul_rn(1e-7, mabs)), 1e-30);
        BVH8Node& N = s_node[g];
        for (int a = 0; a < 3; ++a) {
            const double lo_d = __dsub_rn(double(b.lo[a]), pad);
            const double hi_d = __dadd_rn(double(b.hi[a]), pad);
            float pf = __double2float_rn(lo_d);
            if (double(pf) > lo_d) pf = nextafterf(pf, -FLT_MAX);
            const double ext = __dsub_rn(hi_d, double(pf));
            int e = -126;
            if (ext > 0.0) e = ceil_log2(__ddiv_rn(ext, 255.0));
            e = max(-126, min(127, e));
            while (ldexp(255.0, e) < ext && e < 127) ++e;
            uint8_t ql = 0xff, qh = 0x00;
            if (child) {
                const double scale = ldexp(1.0, e);
                const double lq = floor(__dsub_rn(__ddiv_rn(__dsub_rn(double(c.lo[a]), double(pf)), scale), 0.01));
                const double hq = ceil(__dadd_rn(__ddiv_rn(__dsub_rn(double(c.hi[a]), double(pf)), scale), 0.01));
                ql = uint8_t(fmax(0.0, fmin(255.0, lq)));
                qh = uint8_t(fmax(0.0, fmin(255.0, hq)));
            }
            (a == 0 ? N.qlox : a == 1 ? N.qloy : N.qloz)[slot] = ql;
            (a == 0 ? N.qhix : a == 1 ? N.qhiy : N.qhiz)[slot] = qh;
            if (j == 0) {
                N.p[a] = pf;
                N.e[a] = uint8_t(e + 127);
            }
        }
        const bool leaf = child && (c.left < 0 || c.count <= kMaxLeafPrims);
        unsigned lm = leaf ? 1u << slot : 0u, im = child && !leaf ? 1u << slot : 0u;
        for (int off = 1; off < 8; off <<= 1) {
            lm |= __shfl_xor_sync(FULL, lm, off);
            im |= __shfl_xor_sync(FULL, im, off);
        }
        const int ni = __popc(im), nl = __popc(lm);
        if (j == 0) {
            N.imask = uint8_t(im);
            N.child_base = N.tri_base = 0u;
            N.meta[0] = uint8_t(lm);
            for (int k = 1; k < 8; ++k) N.meta[k] = 0;
            s_count[g] = on ? (TileWord(nl) << 31 | TileWord(ni)) : 0;
        }
        __syncthreads();
        if (threadIdx.x < 32) {  // places of the tile's items
            const TileWord mine = lane < kColItems ? s_count[lane] : 0;
            TileWord incl = mine;
            for (int off = 1; off < 32; off <<= 1) {
                const TileWord v = __shfl_up_sync(FULL, incl, off);
                if (lane >= off) incl += v;
            }
            const TileWord total = __shfl_sync(FULL, incl, 31);
            volatile TileWord* own = words + tile;
            if (lane == 0) *own = (tile == 0 ? kPrefix : kOwn) | total;
            TileWord before = 0;
            for (int t = tile - 1; t >= 0; t -= 32) {
                TileWord v = kPrefix;
                if (t - lane >= 0) {
                    volatile const TileWord* p = words + (t - lane);
                    v = *p;
                    for (int polls = 0; !(v & (kOwn | kPrefix)) && polls < kPollLimit; ++polls) v = *p;
                    if (!(v & (kOwn | kPrefix))) {
                        *err = 1;
                        v = kPrefix;
                    }
                }
                const unsigned done = __ballot_sync(FULL, (v & kPrefix) != 0);
                const int stop = done ? __ffs(done) - 1 : 31;
                TileWord x = lane <= stop ? (v & kCounts) : 0;
                for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(FULL, x, off);
                before += x;
                if (done) break;
            }
            if (lane == 0 && tile) *own = kPrefix | (before + total);
            if (lane < kColItems) s_count[lane] = before + incl - mine;
            if (lane == 0 && tile == tiles - 1) {  // the next level
                const long long start = (long long)o + n_items;
                const long long n = (long long)((before + total) & kIntMask);
                lvl[2 * (l + 1)] = int(start);
                lvl[2 * (l + 1) + 1] = start + n > cap ? 0 : int(n);
                if (start + n > cap) *err = 1;
            }
        }
        __syncthreads();
        if (on) {
            const int cs = int(s_count[g] & kIntMask), ls = int(s_count[g] >> 31);
            const size_t at = size_t(o) + it;
            if (leaf) leaf_prim_all[at * 8 + __popc(lm & ((1u << slot) - 1u))] = ord_fin[c.begin];
            else if (child) {
                const long long to = (long long)o + n_items + cs + __popc(im & ((1u << slot) - 1u));
                if (to < cap) items_all[to] = Item{id, item.tree};
            }
            if (j < 5) reinterpret_cast<uint4*>(tmp_all + at)[j] = reinterpret_cast<const uint4*>(&N)[j];
            if (j == 5) n_leaf_all[at] = nl;
            if (j == 6) cs_all[at] = cs;
            if (j == 7) ls_all[at] = ls;
        }
        __syncthreads();
    }
}

// The levels of the table in shared memory, for kernels over the items of all levels.
struct Levels {
    int off[kMaxLevels + 1];
    int n;
    __device__ void load(const int* lvl, int num_levels) {
        for (int l = threadIdx.x; l <= num_levels; l += blockDim.x) off[l] = l < num_levels ? lvl[2 * l] : 0;
        if (threadIdx.x == 0) {
            // an empty level past the last has no offset of its own
            int k = 1;
            while (k < num_levels && lvl[2 * k + 1] > 0) ++k;
            n = k;
        }
        __syncthreads();
        if (threadIdx.x == 0) off[n] = lvl[2 * (n - 1)] + lvl[2 * (n - 1) + 1];
        __syncthreads();
    }
    __device__ int total() const { return off[n]; }
    __device__ int of(int at) const {
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (off[mid] <= at) lo = mid;
            else hi = mid - 1;
        }
        return lo;
    }
};

// Where each tree's items of each level start and end, from the level's start.
__global__ void k_bounds(const int* lvl, int num_levels, const Item* items, int num_trees, int* first, int* last) {
    __shared__ Levels V;
    V.load(lvl, num_levels);
    for (int at = blockIdx.x * blockDim.x + threadIdx.x; at < V.total(); at += gridDim.x * blockDim.x) {
        const int L = V.of(at), it = at - V.off[L], n = V.off[L + 1] - V.off[L];
        const int t = items[at].tree;
        if (it == 0 || items[at - 1].tree != t) first[size_t(L) * num_trees + t] = it;
        if (it == n - 1 || items[at + 1].tree != t) last[size_t(L) * num_trees + t] = it;
    }
}

// Per tree: nodes and leaf records per level -> offsets of each level (nodes absolute, leaf
// records relative to the tree), total nodes and depth. One thread per tree after a scan of the
// trees' node totals (single block).
__global__ void __launch_bounds__(1024) k_tree_offsets(int num_trees, int num_levels, const int* first, const int* last,
                                                       const int* lvl, const int* ls, const int* n_leaf,
                                                       uint32_t node_base, uint32_t* node_off, uint32_t* leaf_off,
                                                       uint32_t* tree_nodes, int* tree_depth, uint32_t* tree_root) {
    __shared__ uint32_t part[1024];
    const int per = (num_trees + 1023) / 1024;
    const int t0 = min(num_trees, int(threadIdx.x) * per), t1 = min(num_trees, t0 + per);
    uint32_t sum = 0;
    for (int t = t0; t < t1; ++t) {
        uint32_t cnt = 0;
        int depth = 0;
        for (int L = 0; L < num_levels; ++L) {
            const int f = first[size_t(L) * num_trees + t];
            if (f < 0 || last[size_t(L) * num_trees + t] < f) continue;
            cnt += uint32_t(last[size_t(L) * num_trees + t] - f + 1);
            depth = L + 1;
        }
        tree_nodes[t] = cnt;
        tree_depth[t] = depth;
        sum += cnt;
    }
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const uint32_t v = threadIdx.x >= unsigned(off) ? part[threadIdx.x - off] : 0u;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    uint32_t run = node_base + part[threadIdx.x] - sum;
    for (int t = t0; t < t1; ++t) {
        tree_root[t] = run;
        uint32_t lrun = 0;
        for (int L = 0; L <= num_levels; ++L) {
            node_off[size_t(L) * num_trees + t] = run;
            leaf_off[size_t(L) * num_trees + t] = lrun;
            if (L == num_levels) break;
            const int f = first[size_t(L) * num_trees + t];
            if (f < 0) continue;
            const int l = last[size_t(L) * num_trees + t];
            if (l < f) continue;
            run += uint32_t(l - f + 1);
            const int o = lvl[2 * L];
            lrun += uint32_t(ls[o + l] + n_leaf[o + l] - ls[o + f]);
        }
    }
}

// Final nodes and their leaf records.
__global__ void k_place(const int* lvl, int num_levels, const Item* items, int num_trees, const BVH8Node* tmp,
                        const int* cs, const int* ls, const int* n_leaf, const int* leaf_prim, const int* first,
                        const uint32_t* node_off, const uint32_t* leaf_off, const int* tree_begin, bool global_tri,
                        uint32_t node_base, uint32_t node_cap, BVH8Node* nodes, uint32_t* leaf_out) {
    __shared__ Levels V;
    V.load(lvl, num_levels);
    for (int at = blockIdx.x * blockDim.x + threadIdx.x; at < V.total(); at += gridDim.x * blockDim.x) {
        const int L = V.of(at), o = V.off[L];
        const int t = items[at].tree;
        const int f = first[size_t(L) * num_trees + t];
        const uint32_t idx = node_off[size_t(L) * num_trees + t] + uint32_t(at - o - f);
        BVH8Node N = tmp[at];
        N.child_base = node_off[size_t(L + 1) * num_trees + t] + uint32_t(cs[at] - cs[o + f]);
        const uint32_t rec = leaf_off[size_t(L) * num_trees + t] + uint32_t(ls[at] - ls[o + f]);
        N.tri_base = rec + (global_tri ? uint32_t(tree_begin[t]) : 0u);
        if (idx - node_base < node_cap) nodes[idx - node_base] = N;
        for (int k = 0; k < n_leaf[at]; ++k) {
            const size_t r = size_t(tree_begin[t]) + rec + k;
            if (r < size_t(tree_begin[t + 1])) leaf_out[r] = uint32_t(leaf_prim[size_t(at) * 8 + k]);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// scene geometry
// ---------------------------------------------------------------------------------------------

__global__ void k_fill_mesh_ids(const uint32_t* tri_off, int num_meshes, int* prim_mesh) {
    for (int m = blockIdx.x; m < num_meshes; m += gridDim.x)
        for (uint32_t p = tri_off[m] + threadIdx.x; p < tri_off[m + 1]; p += blockDim.x) prim_mesh[p] = m;
}

__global__ void k_tri_boxes(const float* pos, const uint32_t* idx, const int* prim_mesh, const uint32_t* vert_off, int n,
                            float* boxes) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t vb = vert_off[prim_mesh[p]];
        float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        for (int c = 0; c < 3; ++c) {
            const float* v = pos + size_t(vb + idx[size_t(p) * 3 + c]) * 3;
            for (int a = 0; a < 3; ++a) {
                lo[a] = fminf(lo[a], v[a]);
                hi[a] = fmaxf(hi[a], v[a]);
            }
        }
        float* b = boxes + size_t(p) * 6;
        for (int a = 0; a < 3; ++a) {
            const float pad = __fadd_rn(__fmul_rn(1e-6f, fmaxf(fabsf(lo[a]), fabsf(hi[a]))), 1e-9f);
            b[a] = __fsub_rn(lo[a], pad);
            b[3 + a] = __fadd_rn(hi[a], pad);
        }
    }
}

__global__ void k_tri_records(const uint32_t* leaf_prim, int n, const int* prim_mesh, const uint32_t* tri_off,
                              const uint32_t* vert_off, const float* pos, const uint32_t* idx, float4* out) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const uint32_t p = min(leaf_prim[r], uint32_t(n - 1));
        const int m = prim_mesh[p];
        const uint32_t vb = vert_off[m];
        const float* v0 = pos + size_t(vb + idx[size_t(p) * 3 + 0]) * 3;
        const float* v1 = pos + size_t(vb + idx[size_t(p) * 3 + 1]) * 3;
        const float* v2 = pos + size_t(vb + idx[size_t(p) * 3 + 2]) * 3;
        const int local = int(p - tri_off[m]);
        out[size_t(r) * 3 + 0] = make_float4(v0[0], v0[1], v0[2], __int_as_float(local));
        out[size_t(r) * 3 + 1] = make_float4(__fsub_rn(v1[0], v0[0]), __fsub_rn(v1[1], v0[1]), __fsub_rn(v1[2], v0[2]), 0.0f);
        out[size_t(r) * 3 + 2] = make_float4(__fsub_rn(v2[0], v0[0]), __fsub_rn(v2[1], v0[1]), __fsub_rn(v2[2], v0[2]), 0.0f);
    }
}

__global__ void k_mesh_boxes(const float* pos, const uint32_t* vert_off, int num_meshes, float* boxes) {
    __shared__ float sh[6][32];
    for (int m = blockIdx.x; m < num_meshes; m += gridDim.x) {
        float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        for (uint32_t v = vert_off[m] + threadIdx.x; v < vert_off[m + 1]; v += blockDim.x)
            for (int a = 0; a < 3; ++a) {
                lo[a] = fminf(lo[a], pos[size_t(v) * 3 + a]);
                hi[a] = fmaxf(hi[a], pos[size_t(v) * 3 + a]);
            }
        for (int a = 0; a < 3; ++a) {
            lo[a] = wmin(lo[a]);
            hi[a] = wmax(hi[a]);
        }
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
        if (lane == 0)
            for (int a = 0; a < 3; ++a) {
                sh[a][w] = lo[a];
                sh[3 + a][w] = hi[a];
            }
        __syncthreads();
        if (threadIdx.x < 6) {
            float r = threadIdx.x < 3 ? FLT_MAX : -FLT_MAX;
            for (int k = 0; k < nw; ++k) r = threadIdx.x < 3 ? fminf(r, sh[threadIdx.x][k]) : fmaxf(r, sh[threadIdx.x][k]);
            boxes[size_t(m) * 6 + threadIdx.x] = r;
        }
        __syncthreads();
    }
}

__device__ __forceinline__ double dmin_w(double v) {
    for (int off = 16; off > 0; off >>= 1) v = fmin(v, __shfl_xor_sync(FULL, v, off));
    return v;
}
__device__ __forceinline__ double dmax_w(double v) {
    for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(FULL, v, off));
    return v;
}

__global__ void k_inst_boxes(const float* M, const int* inst_mesh, int num_insts, const float* pos, const uint32_t* vert_off,
                             const float* mesh_box, int exact, float* boxes) {
    __shared__ double sh[6][32];
    for (int i = blockIdx.x; i < num_insts; i += gridDim.x) {
        const float* T = M + size_t(i) * 12;
        const int m = inst_mesh[i];
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        auto grow = [&](double x, double y, double z) {
            for (int a = 0; a < 3; ++a) {
                const double w = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(double(T[0 * 3 + a]), x), __dmul_rn(double(T[1 * 3 + a]), y)),
                                                     __dmul_rn(double(T[2 * 3 + a]), z)),
                                           double(T[3 * 3 + a]));
                lo[a] = fmin(lo[a], w);
                hi[a] = fmax(hi[a], w);
            }
        };
        if (exact) {
            for (uint32_t v = vert_off[m] + threadIdx.x; v < vert_off[m + 1]; v += blockDim.x)
                grow(pos[size_t(v) * 3], pos[size_t(v) * 3 + 1], pos[size_t(v) * 3 + 2]);
        } else if (threadIdx.x < 8) {
            const float* mb = mesh_box + size_t(m) * 6;
            const int c = threadIdx.x;
            grow((c & 1) ? mb[3] : mb[0], (c & 2) ? mb[4] : mb[1], (c & 4) ? mb[5] : mb[2]);
        }
        for (int a = 0; a < 3; ++a) {
            lo[a] = dmin_w(lo[a]);
            hi[a] = dmax_w(hi[a]);
        }
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
        if (lane == 0)
            for (int a = 0; a < 3; ++a) {
                sh[a][w] = lo[a];
                sh[3 + a][w] = hi[a];
            }
        __syncthreads();
        if (threadIdx.x == 0) {
            double L[3], H[3];
            for (int a = 0; a < 3; ++a) {
                L[a] = 1e300;
                H[a] = -1e300;
                for (int k = 0; k < nw; ++k) {
                    L[a] = fmin(L[a], sh[a][k]);
                    H[a] = fmax(H[a], sh[3 + a][k]);
                }
            }
            double mext = 0, mabs = 0;
            for (int a = 0; a < 3; ++a) {
                mext = fmax(mext, __dsub_rn(H[a], L[a]));
                mabs = fmax(mabs, fmax(fabs(L[a]), fabs(H[a])));
            }
            const double pad = __dadd_rn(__dadd_rn(__dmul_rn(1e-5, mext), __dmul_rn(1e-6, mabs)), 1e-12);
            for (int a = 0; a < 3; ++a) {
                boxes[size_t(i) * 6 + a] = __double2float_rn(__dsub_rn(L[a], pad));
                boxes[size_t(i) * 6 + 3 + a] = __double2float_rn(__dadd_rn(H[a], pad));
            }
        }
        __syncthreads();
    }
}

// World boxes of instanced triangles for the single-level layout: flat primitive f is
// triangle k = f - inst_tri_off[i] of instance i = flat_inst[f]. The box of the triangle's
// vertices transformed in double is padded by 1e-5 of the instance's world extent plus 1e-5 of
// its largest coordinate (ibox: the instance's padded world box): the object-space triangle
// test sees the ray through the instance's float inverse, whose point error grows with the
// coordinates' magnitude, and the pad covers it for condition numbers up to about 20.
__global__ void k_flat_boxes(const float* M, const int* inst_mesh, const uint32_t* inst_tri_off, const int* flat_inst,
                             int n, const float* ibox, const float* pos, const uint32_t* idx, const uint32_t* tri_off,
                             const uint32_t* vert_off, float* boxes) {
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < n; f += gridDim.x * blockDim.x) {
        const int i = flat_inst[f];
        const int m = inst_mesh[i];
        const uint32_t p = tri_off[m] + (uint32_t(f) - inst_tri_off[i]);
        const float* T = M + size_t(i) * 12;
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        for (int c = 0; c < 3; ++c) {
            const float* v = pos + size_t(vert_off[m] + idx[size_t(p) * 3 + c]) * 3;
            for (int a = 0; a < 3; ++a) {
                const double w = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(double(T[0 * 3 + a]), double(v[0])),
                                                               __dmul_rn(double(T[1 * 3 + a]), double(v[1]))),
                                                     __dmul_rn(double(T[2 * 3 + a]), double(v[2]))),
                                           double(T[3 * 3 + a]));
                lo[a] = fmin(lo[a], w);
                hi[a] = fmax(hi[a], w);
            }
        }
        const float* ib = ibox + size_t(i) * 6;
        double mext = 0.0, mabs = 0.0;
        for (int a = 0; a < 3; ++a) {
            mext = fmax(mext, __dsub_rn(double(ib[3 + a]), double(ib[a])));
            mabs = fmax(mabs, fmax(fabs(double(ib[a])), fabs(double(ib[3 + a]))));
        }
        const double pad = __dadd_rn(__dmul_rn(1e-5, __dadd_rn(mext, mabs)), 1e-12);
        for (int a = 0; a < 3; ++a) {
            boxes[size_t(f) * 6 + a] = __double2float_rd(__dsub_rn(lo[a], pad));
            boxes[size_t(f) * 6 + 3 + a] = __double2float_ru(__dadd_rn(hi[a], pad));
        }
    }
}

// Single-level triangle records in leaf order: v0 with the mesh-local triangle index in w,
// e1 with the instance index in w, e2 -- object-space values, exactly those of the two-level
// records, so the triangle test is the same.
__global__ void k_flat_records(const uint32_t* leaf_prim, int n, const int* flat_inst, const uint32_t* inst_tri_off,
                               const int* inst_mesh, const uint32_t* tri_off, const uint32_t* vert_off, const float* pos,
                               const uint32_t* idx, float4* out) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const uint32_t f = min(leaf_prim[r], uint32_t(n - 1));
        const int i = flat_inst[f];
        const int m = inst_mesh[i];
        const uint32_t k = f - inst_tri_off[i];
        const uint32_t p = tri_off[m] + k;
        const uint32_t vb = vert_off[m];
        const float* v0 = pos + size_t(vb + idx[size_t(p) * 3 + 0]) * 3;
        const float* v1 = pos + size_t(vb + idx[size_t(p) * 3 + 1]) * 3;
        const float* v2 = pos + size_t(vb + idx[size_t(p) * 3 + 2]) * 3;
        out[size_t(r) * 3 + 0] = make_float4(v0[0], v0[1], v0[2], __int_as_float(int(k)));
        out[size_t(r) * 3 + 1] = make_float4(__fsub_rn(v1[0], v0[0]), __fsub_rn(v1[1], v0[1]), __fsub_rn(v1[2], v0[2]),
                                             __int_as_float(i));
        out[size_t(r) * 3 + 2] = make_float4(__fsub_rn(v2[0], v0[0]), __fsub_rn(v2[1], v0[1]), __fsub_rn(v2[2], v0[2]), 0.0f);
    }
}

// device buffers of one build, freed together: carved from one block of the expected size (an
// allocation is a driver call of 30 to 100 us while other threads of a scene build make theirs)
struct Bufs {
    cudaStream_t st;
    std::vector<void*> p;
    char* at = nullptr;
    size_t left = 0;
    Bufs(cudaStream_t s, size_t expected) : st(s) {
        at = raw(expected);
        left = at ? expected : 0;
    }
    Bufs(const Bufs&) = delete;
    Bufs& operator=(const Bufs&) = delete;
    ~Bufs() {
        for (void* q : p) scratch_free(q, st);
    }
    char* raw(size_t bytes) {
        void* q = nullptr;
        if (scratch_alloc(&q, bytes, st) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        p.push_back(q);
        return static_cast<char*>(q);
    }
    template <class T>
    T* get(size_t n) {
        const size_t bytes = (std::max<size_t>(n, 1) * sizeof(T) + 255) & ~size_t(255);
        if (bytes > left) return reinterpret_cast<T*>(raw(bytes));
        T* q = reinterpret_cast<T*>(at);
        at += bytes;
        left -= bytes;
        return q;
    }
};

int grid_for(int n, int per_block, int cap) { return std::max(1, std::min(cap, (n + per_block - 1) / per_block)); }

}  // namespace

void DeviceBvh8::release() {
    scratch_free(nodes, stream);
    scratch_free(leaf_prim, stream);
    nodes = nullptr;
    leaf_prim = nullptr;
    num_nodes = 0;
}

namespace {

// One build. levels: binary levels of large nodes that are launched; *unfinished is set when nodes
// of more than kMedium primitives are left after them.
//
// Everything is enqueued without reading a size back: every kernel takes its level's counts from
// the device (the two large lists alternate, binary ids continue from ctr[3], and a level past the
// last has no nodes, so its kernels do nothing), buffers have room for the most there can be, and
// one wait ends the build. Launches and read-backs in turn cost more than the kernels: while the
// texture thread of a scene build copies from pageable memory, a driver call of this thread can
// wait 1 to 3 ms (1M triangles: 4.0 ms of kernels took 7.3 ms with a read-back per stage, 5.9 so).
int build_attempt(const float* d_boxes, const std::vector<int>& tree_begin, uint32_t node_base, bool global_tri,
                  cudaStream_t st, int levels, DeviceBvh8& out, bool* unfinished) {
    const int G = int(tree_begin.size()) - 1;
    const int N = tree_begin[G];
    const size_t bn_cap = size_t(2) * N;
    const int large_cap = N / (kMedium + 1) + 1;
    const int medium_cap = N / (kSmall + 1) + 1;
    const int chunk_cap = large_cap + N / kChunk + 1;
    const size_t item_cap = size_t(N) + G;
    const size_t words_n = item_cap / kColItems + kMaxLevels + 2;
    int max_tree = 1;
    for (int t = 0; t < G; ++t) max_tree = std::max(max_tree, tree_begin[t + 1] - tree_begin[t]);
    // 8-wide levels a tree of the largest size usually has (about one per three binary levels of a
    // binary depth near 1.5 log2 n), and two more
    const int wide0 = std::min(kMaxLevels, int(std::ceil(0.5 * std::log2(double(max_tree) + 1.0))) + 3);
    const size_t expected = size_t(N) * (12 + 2 * sizeof(BinNode) + 4) + size_t(medium_cap) * 4 +
                            size_t(large_cap) * (sizeof(Slot) + 8 + 3 * kBins * 28) + size_t(chunk_cap) * 16 +
                            item_cap * (sizeof(Item) + sizeof(BVH8Node) + 12 + 32) + words_n * 8 +
                            size_t(G) * (size_t(wide0) * 16 + 32) + 40 * 256 + 8192;
    Bufs B(st, expected);
    int* d_tb = B.get<int>(G + 1);
    int* ord[2] = {B.get<int>(N), B.get<int>(N)};
    int* ord_fin = B.get<int>(N);
    BinNode* bn = B.get<BinNode>(bn_cap);
    int* large[2] = {B.get<int>(large_cap), B.get<int>(large_cap)};
    unsigned* medium = B.get<unsigned>(medium_cap);
    int* small = B.get<int>(N / 2 + 1);
    Slot* slots = B.get<Slot>(large_cap);
    unsigned* bin_cnt = B.get<unsigned>(size_t(large_cap) * 3 * kBins);
    unsigned* bin_lo = B.get<unsigned>(size_t(large_cap) * 3 * kBins * 3);
    unsigned* bin_hi = B.get<unsigned>(size_t(large_cap) * 3 * kBins * 3);
    int* chunk_slot = B.get<int>(chunk_cap);
    int* chunk_start = B.get<int>(chunk_cap);
    int* chunk_left = B.get<int>(chunk_cap);
    int* chunk_lbase = B.get<int>(chunk_cap);
    Item* items = B.get<Item>(item_cap);
    BVH8Node* tmp = B.get<BVH8Node>(item_cap);
    int* n_leaf = B.get<int>(item_cap);
    int* cs = B.get<int>(item_cap);
    int* ls = B.get<int>(item_cap);
    int* leafp = B.get<int>(item_cap * 8);
    // Words that start at zero, one block: ctr (0,1: large list sizes; 2: small list size; 3: next
    // binary id; 4: chunks; 5: medium list size; 7: capacity error), the level table (offset and
    // count per 8-wide level, then an error word), tile counters, look-back words.
    constexpr int kLvl = 8, kErr = kLvl + 2 * kMaxLevels + 2, kTiles = kErr + 2, kWords = kTiles + kMaxLevels + 2;
    static_assert(kWords % 2 == 0, "look-back words are 8 bytes");
    const size_t zero_n = size_t(kWords) + 2 * words_n;
    int* zero = B.get<int>(zero_n);
    if (!d_tb || !ord[0] || !ord[1] || !ord_fin || !bn || !large[0] || !large[1] || !medium || !small || !slots ||
        !bin_cnt || !bin_lo || !bin_hi || !chunk_slot || !chunk_start || !chunk_left || !chunk_lbase || !items || !tmp ||
        !n_leaf || !cs || !ls || !leafp || !zero)
        return fail(LUX_ERR_OOM, "BVH build: device scratch allocation failed");
    int *ctr = zero, *lvl = zero + kLvl, *err = zero + kErr, *tile_ctr = zero + kTiles;
    TileWord* words = reinterpret_cast<TileWord*>(zero + kWords);
    out.stream = st;
    if (scratch_alloc(reinterpret_cast<void**>(&out.nodes), sizeof(BVH8Node) * item_cap, st) != cudaSuccess ||
        scratch_alloc(reinterpret_cast<void**>(&out.leaf_prim), sizeof(uint32_t) * size_t(N), st) != cudaSuccess) {
        cudaGetLastError();
        out.release();
        return fail(LUX_ERR_OOM, "BVH build: node allocation failed");
    }
    // page-locked: tree starts, roots and the start of the level table go up, the tables and the
    // trees' results come down
    const size_t host_n = size_t(kTiles) + size_t(G + 1) + 2 * size_t(G) + 3 * size_t(G) + 8;
    struct HostBlock {  // back to the pool once no copy can still use it
        int* p;
        size_t bytes;
        cudaStream_t st;
        ~HostBlock() {
            cudaStreamSynchronize(st);
            pinned_put(p, bytes);
        }
    } hb{static_cast<int*>(pinned_get(host_n * sizeof(int))), host_n * sizeof(int), st};
    if (!hb.p) return fail(LUX_ERR_OOM, "BVH build: page-locked host allocation failed");
    int* h_zero = hb.p;
    int* h_tb = h_zero + kTiles;
    Item* h_roots = reinterpret_cast<Item*>(h_tb + G + 1);
    int* h_out = h_tb + G + 1 + 2 * G;
    std::memcpy(h_tb, tree_begin.data(), sizeof(int) * (G + 1));
    for (int t = 0; t < G; ++t) h_roots[t] = Item{t, t};
    std::memset(h_zero, 0, sizeof(int) * kTiles);
    h_zero[3] = G;          // binary ids after the roots'
    h_zero[kLvl + 1] = G;   // level 0: the roots
    LUX_CUDA(cudaMemcpyAsync(d_tb, h_tb, sizeof(int) * (G + 1), cudaMemcpyHostToDevice, st));
    LUX_CUDA(cudaMemcpyAsync(items, h_roots, sizeof(Item) * G, cudaMemcpyHostToDevice, st));
    LUX_CUDA(cudaMemsetAsync(zero, 0, sizeof(int) * zero_n, st));
    LUX_CUDA(cudaMemcpyAsync(zero, h_zero, sizeof(int) * kTiles, cudaMemcpyHostToDevice, st));
    // every index array starts in range, so no read can leave its buffer whatever is computed
    LUX_CUDA(cudaMemsetAsync(ord[1], 0, sizeof(int) * size_t(N), st));
    LUX_CUDA(cudaMemsetAsync(ord_fin, 0, sizeof(int) * size_t(N), st));
    LUX_CUDA(cudaMemsetAsync(bn, 0, sizeof(BinNode) * bn_cap, st));
    LUX_CUDA(cudaMemsetAsync(out.leaf_prim, 0, sizeof(uint32_t) * size_t(N), st));
    k_iota<<<grid_for(N, 256, 4096), 256, 0, st>>>(ord[0], N);
    k_roots<<<grid_for(G, 128, 1024), 128, 0, st>>>(d_boxes, d_tb, G, bn, ord[0], ord_fin, large[0], ctr + 0, medium,
                                                   ctr + 5, small, ctr + 2);
    // ---- binary levels of large nodes ----
    const int grid_s = grid_for(large_cap, 128, 4096);
    const int grid_sp = grid_for(large_cap, kSplitWarps, 4096);
    const int grid_clear = grid_for(large_cap * 3 * kBins, 256, 148 * 16);
    const int grid_c = std::min(chunk_cap, 148 * 8);
    int cur = 0;
    for (int b = 0; b < levels; ++b) {
        const int nxt = cur ^ 1;
        k_chunks<<<1, 1024, 0, st>>>(large[cur], ctr + cur, bn, slots, chunk_slot, chunk_start, ctr + 4);
        k_bin_clear<<<grid_clear, 256, 0, st>>>(ctr + cur, bin_cnt, bin_lo, bin_hi);
        k_reduce<<<grid_c, kBlock, 0, st>>>(d_boxes, ord[cur], large[cur], bn, slots, chunk_slot, chunk_start, ctr + 4);
        k_bin_setup<<<grid_s, 128, 0, st>>>(large[cur], ctr + cur, bn, slots);
        k_bin<<<grid_c, kBlock, 0, st>>>(d_boxes, ord[cur], large[cur], bn, slots, chunk_slot, chunk_start, ctr + 4,
                                          bin_cnt, bin_lo, bin_hi);
        k_split<<<grid_sp, 32 * kSplitWarps, 0, st>>>(large[cur], ctr + cur, bn, slots, bin_cnt, bin_lo, bin_hi);
        k_count_left<<<grid_c, kBlock, 0, st>>>(d_boxes, ord[cur], large[cur], bn, slots, chunk_slot, chunk_start,
                                                 ctr + 4, chunk_left);
        k_chunk_base<<<grid_s, 128, 0, st>>>(ctr + cur, slots, chunk_left, chunk_lbase);
        k_scatter<<<grid_c, kBlock, 0, st>>>(d_boxes, ord[cur], ord[nxt], large[cur], bn, slots, chunk_slot,
                                              chunk_start, ctr + 4, chunk_lbase);
        k_children<<<grid_s, 128, 0, st>>>(d_boxes, ord[nxt], ord_fin, large[cur], ctr + cur, bn, slots, ctr + 3,
                                           int(bn_cap), ctr + 7, large[nxt], ctr + nxt, medium, ctr + 5,
                                           unsigned(nxt), small, ctr + 2);
        k_level_advance<<<1, 1, 0, st>>>(ctr + cur, ctr + 3);
        LUX_CUDA(cudaGetLastError());
        cur = nxt;
    }
    // ---- medium and small subtrees, from the lists' device counts: binary ids continue in ctr[3] ----
    k_medium<<<grid_for(medium_cap, 1, 148 * 7), kBlock, 0, st>>>(d_boxes, ord[0], ord[1], medium, ctr + 5, bn, int(bn_cap),
                                                                  ctr + 3, ctr + 7, ord_fin, small, ctr + 2);
    k_small<<<grid_for(N / 2 + 1, kSmallWarps, 148 * 16), 32 * kSmallWarps, 0, st>>>(d_boxes, small, ctr + 2, bn, ord_fin,
                                                                                     ctr + 3);
    LUX_CUDA(cudaGetLastError());
    // ---- collapse level by level, then the placement over all levels ----
    const int grid_items = grid_for(int(item_cap), kColItems, 148 * 4);
    const int grid_place = grid_for(int(item_cap), 128, 148 * 16);
    int launched = 0, batch = wide0;
    while (true) {
        for (int l = launched; l < launched + batch; ++l)
            k_collapse<<<grid_items, kColThreads, 0, st>>>(lvl, l, items, bn, ord_fin, tmp, n_leaf, cs, ls, leafp, words,
                                                           tile_ctr, (long long)item_cap, err);
        launched += batch;
        const size_t lg = size_t(launched) * G;
        int* first = B.get<int>(2 * lg);
        uint32_t* node_off = B.get<uint32_t>(2 * (lg + G));
        uint32_t* tree_out = B.get<uint32_t>(3 * size_t(G));  // roots, node counts, depths
        if (!first || !node_off || !tree_out) return fail(LUX_ERR_OOM, "BVH build: device scratch allocation failed");
        int* last = first + lg;
        uint32_t* leaf_off = node_off + lg + G;
        LUX_CUDA(cudaMemsetAsync(first, 0xff, 2 * sizeof(int) * lg, st));
        k_bounds<<<grid_place, 128, 0, st>>>(lvl, launched, items, G, first, last);
        k_tree_offsets<<<1, 1024, 0, st>>>(G, launched, first, last, lvl, ls, n_leaf, node_base, node_off, leaf_off,
                                           tree_out + G, reinterpret_cast<int*>(tree_out + 2 * G), tree_out);
        k_place<<<grid_place, 128, 0, st>>>(lvl, launched, items, G, tmp, cs, ls, n_leaf, leafp, first, node_off, leaf_off,
                                            d_tb, global_tri, node_base, uint32_t(item_cap), out.nodes, out.leaf_prim);
        LUX_CUDA(cudaGetLastError());
        LUX_CUDA(cudaMemcpyAsync(h_zero, zero, sizeof(int) * kTiles, cudaMemcpyDeviceToHost, st));
        LUX_CUDA(cudaMemcpyAsync(h_out, tree_out, 3 * sizeof(uint32_t) * G, cudaMemcpyDeviceToHost, st));
        LUX_CUDA(cudaStreamSynchronize(st));
        if (h_zero[7]) return fail(LUX_ERR_UNSUPPORTED, "BVH build: binary node capacity");
        if (h_zero[cur]) {
            *unfinished = true;
            return LUX_OK;
        }
        if (h_zero[kErr]) return fail(LUX_ERR_UNSUPPORTED, "BVH build: 8-wide node capacity");
        if (h_zero[kLvl + 2 * launched + 1] == 0) break;  // no level after the launched ones
        batch = std::min(8, kMaxLevels - launched);
        if (batch <= 0) return fail(LUX_ERR_UNSUPPORTED, "BVH build: too many 8-wide levels");
    }
    uint32_t total = 0;
    for (int l = 0; l < launched; ++l) total += uint32_t(h_zero[kLvl + 2 * l + 1]);
    out.root.assign(reinterpret_cast<uint32_t*>(h_out), reinterpret_cast<uint32_t*>(h_out) + G);
    out.count.assign(reinterpret_cast<uint32_t*>(h_out) + G, reinterpret_cast<uint32_t*>(h_out) + 2 * G);
    out.depth.assign(h_out + 2 * G, h_out + 3 * G);
    out.num_nodes = total;
    *unfinished = false;
    return LUX_OK;
}

}  // namespace

int build_bvh8_device(const float* d_boxes, const std::vector<int>& tree_begin, uint32_t node_base, bool global_tri,
                      cudaStream_t st, DeviceBvh8& out) {
    out.release();
    const int G = int(tree_begin.size()) - 1;
    if (G <= 0) return fail(LUX_ERR_INVALID, "BVH build without trees");
    int max_tree = 1;
    for (int t = 0; t < G; ++t) {
        if (tree_begin[t + 1] <= tree_begin[t]) return fail(LUX_ERR_INVALID, "BVH build: a tree without primitives");
        max_tree = std::max(max_tree, tree_begin[t + 1] - tree_begin[t]);
    }
    // Halving reaches kMedium in log2(max_tree / kMedium) levels; SAH splits of real scenes take a
    // few more (16 instead of 10 for 1M triangles). Primitives that peel off a few at a time can take
    // any number: the build is then repeated with four times the levels.
    int levels = max_tree <= kMedium ? 0 : int(std::ceil(std::log2(double(max_tree) / kMedium))) + 8;
    while (true) {
        bool unfinished = false;
        if (int rc = build_attempt(d_boxes, tree_begin, node_base, global_tri, st, levels, out, &unfinished)) {
            out.release();
            return rc;
        }
        if (!unfinished) return LUX_OK;
        out.release();
        if (levels > 4 * (64 + max_tree / kMedium)) return fail(LUX_ERR_UNSUPPORTED, "BVH build did not converge");
        levels *= 4;
    }
}

cudaError_t launch_fill_mesh_ids(const uint32_t* tri_off, int num_meshes, int* prim_mesh, cudaStream_t st) {
    if (num_meshes <= 0) return cudaSuccess;
    k_fill_mesh_ids<<<std::min(num_meshes, 4096), 256, 0, st>>>(tri_off, num_meshes, prim_mesh);
    return cudaGetLastError();
}

cudaError_t launch_tri_boxes(const float* pos, const uint32_t* idx, const int* prim_mesh, const uint32_t* vert_off, int n,
                             float* boxes, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_tri_boxes<<<grid_for(n, 256, 148 * 16), 256, 0, st>>>(pos, idx, prim_mesh, vert_off, n, boxes);
    return cudaGetLastError();
}

cudaError_t launch_tri_records(const uint32_t* leaf_prim, int n, const int* prim_mesh, const uint32_t* tri_off,
                               const uint32_t* vert_off, const float* pos, const uint32_t* idx, float4* prims,
                               cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_tri_records<<<grid_for(n, 256, 148 * 16), 256, 0, st>>>(leaf_prim, n, prim_mesh, tri_off, vert_off, pos, idx, prims);
    return cudaGetLastError();
}

cudaError_t launch_flat_boxes(const float* M, const int* inst_mesh, const uint32_t* inst_tri_off, const int* flat_inst,
                              int n, const float* ibox, const float* pos, const uint32_t* idx, const uint32_t* tri_off,
                              const uint32_t* vert_off, float* boxes, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_flat_boxes<<<grid_for(n, 256, 148 * 16), 256, 0, st>>>(M, inst_mesh, inst_tri_off, flat_inst, n, ibox, pos, idx,
                                                             tri_off, vert_off, boxes);
    return cudaGetLastError();
}

cudaError_t launch_flat_records(const uint32_t* leaf_prim, int n, const int* flat_inst, const uint32_t* inst_tri_off,
                                const int* inst_mesh, const uint32_t* tri_off, const uint32_t* vert_off, const float* pos,
                                const uint32_t* idx, float4* prims, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_flat_records<<<grid_for(n, 256, 148 * 16), 256, 0, st>>>(leaf_prim, n, flat_inst, inst_tri_off, inst_mesh, tri_off,
                                                               vert_off, pos, idx, prims);
    return cudaGetLastError();
}

cudaError_t launch_mesh_boxes(const float* pos, const uint32_t* vert_off, int num_meshes, float* boxes, cudaStream_t st) {
    if (num_meshes <= 0) return cudaSuccess;
    k_mesh_boxes<<<std::min(num_meshes, 4096), 256, 0, st>>>(pos, vert_off, num_meshes, boxes);
    return cudaGetLastError();
}

cudaError_t launch_inst_boxes(const float* M, const int* inst_mesh, int num_insts, const float* pos,
                              const uint32_t* vert_off, const float* mesh_box, int exact, float* boxes,
                              cudaStream_t st) {
    if (num_insts <= 0) return cudaSuccess;
    k_inst_boxes<<<std::min(num_insts, 4096), 256, 0, st>>>(M, inst_mesh, num_insts, pos, vert_off, mesh_box, exact,
                                                            boxes);
    return cudaGetLastError();
}

}  // namespace lux
