// trace_core.cuh -- ray traversal of the compressed 8-wide BVH, one warp at a time: what the
// traversal kernels (trace.cu) and the whole-path kernel (paths.cu) share. Every operation whose
// rounding a result depends on is written with its rounding, so the code computes the same in
// units compiled with and without contraction.
#pragma once

#include "device_scene.h"
#include "device_math.cuh"
#include "bvh8.h"
#include "launch.h"

namespace lux {
namespace {

// stack entries in shared memory; 6 to 16 measured alike (the rest of a deep stack is in local memory)
constexpr int kShStack = 12;
constexpr int kLocStack = 52;
static_assert(kShStack + kLocStack == kTraversalStack, "the scene build bounds the stack by kTraversalStack");
constexpr int kRefill = 20;
// environment occlusion rays (any hit, mode 2) refill below this many traversing lanes
constexpr int kRefillOcclusion = 24;
constexpr uint32_t kTagMask = 3u << 30;
constexpr uint32_t kTagNode = 0u;
constexpr uint32_t kTagTri = 1u << 30;
constexpr uint32_t kTagInst = 2u << 30;
constexpr uint32_t kTagMarker = 3u << 30;
constexpr uint32_t kRecMask = 0xffu;
// fewer lanes than this with triangles to test: push the triangle groups and keep
// traversing nodes (the postponement of Ylitie et al. 2017); 6 and a refill threshold of 20
// lanes were the fastest of the values tried on the 1M-triangle 1080p workload (3 to 8, 10 to 12 and
// 16; 16 to 18, 20, 22 to 24 and 28), and 24 for the occlusion rays (16, 20, 24, 28 and 32)
constexpr int kPostpone = 6;
// Slab acceptance tnear <= tfar * kWiden (tnear >= 0): a relative margin of 2^-17, far above
// the few-ulp rounding of the plane distances.
constexpr float kWiden = 1.0f + 1.0f / 131072.0f;
// Boxes that end behind the origin are skipped; the bound lies a hair below 0, so that a far plane
// at -0 still counts as at the origin when the sign bit of tf * kWiden - tn decides.
constexpr float kBehind = -1e-30f;
static_assert(kMaxLeafPrims == 1, "visit_node marks one triangle per leaf slot");

struct TRay {
    f3 o, d, idir;
    uint32_t oct;
};

// Reciprocal for the box tests only (the triangle test uses the direction itself): the
// hardware approximation, at most 1 ulp off, scales both slab distances of an axis by the same
// factor within 2^-23 of 1, far inside the 2^-17 acceptance margin.
// A component below 2^-66 in magnitude (zero and subnormals included) is raised to 2^-66 with
// its sign. An exact zero would give an infinite reciprocal, that axis's slab distances would
// then be NaN, and fminf / fmaxf drop NaN operands: the axis would stop culling, and in a
// world-space tree the ray would sweep a whole slab of the scene (a camera on an axis-aligned
// plane makes such rays, one pixel column of them). With 2^-66 the axis culls every box that
// does not hold the origin's coordinate to within 2^-66 * tmax, and keeps every box that holds
// it with a margin m for t up to m * 2^66: boxes are padded by far more than the 2^-66 * t a
// ray this close to the axis plane drifts within the scene.
LUX_DI float rcp_box(float x) {
    const float c = copysignf(fmaxf(fabsf(x), 1.35525271560688054e-20f), x);  // 2^-66
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(c));
    return r;
}

LUX_DI TRay make_ray(f3 o, f3 d) {
    TRay r;
    r.o = o;
    r.d = d;
    r.idir = mk(rcp_box(d.x), rcp_box(d.y), rcp_box(d.z));
    r.oct = (__float_as_uint(r.idir.x) >> 31) | ((__float_as_uint(r.idir.y) >> 31) << 1) |
            ((__float_as_uint(r.idir.z) >> 31) << 2);
    return r;
}

// Byte s of w as the float 2^23 + 256 * byte: one byte permute builds 0x4B00bb00. The 2^23
// bias is folded into the per-node plane constant (visit_node), so no add removes it.
LUX_DI float ubyte_biased(uint32_t w, int s) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7504u | (uint32_t(s) << 4))); }

// Three-operand max / min (sm_100 and later): one instruction where two fmaxf / fminf would
// be, with their NaN rule (a NaN operand is dropped).
LUX_DI float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
LUX_DI float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

LUX_DI unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
// Distances of planes b and b + 1 of word w: two lanes of one fma (sm_100), each rounded as fmaf.
LUX_DI float2 planes(uint32_t w, int b, unsigned long long a, unsigned long long c) {
    unsigned long long q = pack2(ubyte_biased(w, b), ubyte_biased(w, b + 1)), r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(q), "l"(a), "l"(c));
    float2 o;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
    return o;
}

// missed << 1 | whether the slab test misses. The sign of tf * kWiden - tn decides, one multiply-add
// and a funnel shift for a multiply, a compare and a bit.
LUX_DI uint32_t miss_bit(uint32_t missed, float tnx, float tny, float tnz, float tfx, float tfy, float tfz, float tmax) {
    const float tn = max3f(tnx, tny, fmaxf(tnz, kBehind));
    const float tf = min3f(tfx, tfy, fminf(tfz, tmax));
    return __funnelshift_l(__float_as_uint(fmaf(tf, kWiden, -tn)), missed, 1);
}

// Table of the slot masks in key order: bit s of lut[oct << 8 | mask] is bit s ^ oct of mask.
LUX_DI void fill_key_table(unsigned char* lut) {
    for (int i = threadIdx.x; i < 2048; i += blockDim.x) {
        uint32_t m = i & 255;
        const int oct = i >> 8;
        if (oct & 1) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
        if (oct & 2) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
        if (oct & 4) m = ((m & 0x0Fu) << 4) | ((m >> 4) & 0x0Fu);
        lut[i] = (unsigned char)m;
    }
}

// Intersect the 8 child boxes of node ni. Returns internal-child hits as a key mask
// (bit slot ^ oct), leaf hits as a slot mask, the node's leaf-slot mask, child_base and
// tri_base.
LUX_DI void visit_node(const uint4* __restrict__ nodes, uint32_t ni, const TRay& r, float tmax, uint32_t& keys,
                       uint32_t& imask, uint32_t& child_base, uint32_t& tri_base, uint32_t& trimask,
                       uint32_t& leafmask, const unsigned char* lut) {
    const uint4* n = nodes + size_t(ni) * 5;
    uint4 w0 = __ldg(n + 0), w1 = __ldg(n + 1), w2 = __ldg(n + 2), w3 = __ldg(n + 3), w4 = __ldg(n + 4);
    float px = __uint_as_float(w0.x), py = __uint_as_float(w0.y), pz = __uint_as_float(w0.z);
    float sx = __uint_as_float((w0.w & 0xffu) << 23);
    float sy = __uint_as_float(((w0.w >> 8) & 0xffu) << 23);
    float sz = __uint_as_float(((w0.w >> 16) & 0xffu) << 23);
    imask = w0.w >> 24;
    child_base = w1.x;
    tri_base = w1.y;
    // plane q of an axis lies at t = q * a + b with a = scale * idir, b = (p - o) * idir.
    // It is evaluated as fma(2^23 + 256 q, a / 256, b - 2^15 a): a / 256 is exact, and the
    // rounding of the folded constant adds at most 2^-9 of a quantisation step (the host pads
    // every plane by at least 1 % of a step).
    float ax = sx * r.idir.x * 0.00390625f, ay = sy * r.idir.y * 0.00390625f, az = sz * r.idir.z * 0.00390625f;
    float bx = (px - r.o.x) * r.idir.x, by = (py - r.o.y) * r.idir.y, bz = (pz - r.o.z) * r.idir.z;
    bx = fmaf(-8388608.0f, ax, bx);
    by = fmaf(-8388608.0f, ay, by);
    bz = fmaf(-8388608.0f, az, bz);
    // near/far quantised planes per axis, by ray octant
    const bool fx = r.oct & 1, fy = r.oct & 2, fz = r.oct & 4;
    uint32_t nx0 = fx ? w3.z : w2.x, nx1 = fx ? w3.w : w2.y, fx0 = fx ? w2.x : w3.z, fx1 = fx ? w2.y : w3.w;
    uint32_t ny0 = fy ? w4.x : w2.z, ny1 = fy ? w4.y : w2.w, fy0 = fy ? w2.z : w4.x, fy1 = fy ? w2.w : w4.y;
    uint32_t nz0 = fz ? w4.z : w3.x, nz1 = fz ? w4.w : w3.y, fz0 = fz ? w3.x : w4.z, fz1 = fz ? w3.y : w4.w;
    uint32_t missed = 0;
    const unsigned long long ax2 = pack2(ax, ax), ay2 = pack2(ay, ay), az2 = pack2(az, az);
    const unsigned long long bx2 = pack2(bx, bx), by2 = pack2(by, by), bz2 = pack2(bz, bz);
#pragma unroll
    for (int s = 6; s >= 0; s -= 2) {
        const int b = s & 3;
        uint32_t wnx = s < 4 ? nx0 : nx1, wny = s < 4 ? ny0 : ny1, wnz = s < 4 ? nz0 : nz1;
        uint32_t wfx = s < 4 ? fx0 : fx1, wfy = s < 4 ? fy0 : fy1, wfz = s < 4 ? fz0 : fz1;
        float2 tnx = planes(wnx, b, ax2, bx2), tny = planes(wny, b, ay2, by2), tnz = planes(wnz, b, az2, bz2);
        float2 tfx = planes(wfx, b, ax2, bx2), tfy = planes(wfy, b, ay2, by2), tfz = planes(wfz, b, az2, bz2);
        missed = miss_bit(missed, tnx.y, tny.y, tnz.y, tfx.y, tfy.y, tfz.y, tmax);
        missed = miss_bit(missed, tnx.x, tny.x, tnz.x, tfx.x, tfy.x, tfz.x, tmax);
    }
    leafmask = w1.z & 0xffu;
    const uint32_t hits = ~missed & (imask | leafmask);
    trimask = hits & leafmask;
    keys = lut[(r.oct << 8) | (hits & imask)];
}

// A ray's closest hit; inst -1: none.
struct Best {
    float t;
    int inst, prim;
    float u, v;
};

// Moller-Trumbore exactly as src/intersections/mesh_isect.cu:78-115, single-rounded ops, on a
// triangle record (v0 with the triangle index in w, e1, e2) and the ray (ro, d) of the
// triangle's object space.
LUX_DI bool mt_core(float4 a4, float4 e14, float4 e24, f3 ro, f3 d, float& t, float& u, float& v, int& prim) {
    prim = __float_as_int(a4.w);
    const f3 e1 = mk(e14.x, e14.y, e14.z), e2 = mk(e24.x, e24.y, e24.z);
    // cross(d, e2) = (d.y*e2.z - e2.y*d.z, d.z*e2.x - e2.z*d.x, d.x*e2.y - e2.x*d.y)
    f3 c = mk(__fsub_rn(__fmul_rn(d.y, e2.z), __fmul_rn(e2.y, d.z)), __fsub_rn(__fmul_rn(d.z, e2.x), __fmul_rn(e2.z, d.x)),
              __fsub_rn(__fmul_rn(d.x, e2.y), __fmul_rn(e2.x, d.y)));
    float det = __fadd_rn(__fadd_rn(__fmul_rn(e1.x, c.x), __fmul_rn(e1.y, c.y)), __fmul_rn(e1.z, c.z));
    if (det > -kMT_EPS && det < kMT_EPS) return false;
    float inv = __frcp_rn(det);
    f3 a = mk(__fsub_rn(ro.x, a4.x), __fsub_rn(ro.y, a4.y), __fsub_rn(ro.z, a4.z));
    u = __fmul_rn(inv, __fadd_rn(__fadd_rn(__fmul_rn(a.x, c.x), __fmul_rn(a.y, c.y)), __fmul_rn(a.z, c.z)));
    if (u < -kMT_EPS || u > 1.0f + kMT_EPS) return false;
    // cross(a, e1)
    c = mk(__fsub_rn(__fmul_rn(a.y, e1.z), __fmul_rn(e1.y, a.z)), __fsub_rn(__fmul_rn(a.z, e1.x), __fmul_rn(e1.z, a.x)),
           __fsub_rn(__fmul_rn(a.x, e1.y), __fmul_rn(e1.x, a.y)));
    v = __fmul_rn(inv, __fadd_rn(__fadd_rn(__fmul_rn(d.x, c.x), __fmul_rn(d.y, c.y)), __fmul_rn(d.z, c.z)));
    float uv = __fadd_rn(u, v);
    if ((v < 0.0f && fabsf(v) > kMT_EPS) || (uv > 1.0f && fabsf(__fsub_rn(uv, 1.0f)) > kMT_EPS)) return false;
    t = __fmul_rn(inv, __fadd_rn(__fadd_rn(__fmul_rn(e2.x, c.x), __fmul_rn(e2.y, c.y)), __fmul_rn(e2.z, c.z)));
    return t > kMT_EPS;
}

LUX_DI bool mt_test(const float4* __restrict__ prims, uint32_t rec, const TRay& r, float& t, float& u, float& v,
                    int& prim) {
    const float4* q = prims + size_t(rec) * 3;
    return mt_core(__ldg(q), __ldg(q + 1), __ldg(q + 2), r.o, r.d, t, u, v, prim);
}

// Any-hit program (src/optixshaders/optix_triangle.cu:317-366): true = accept the hit. The
// multiply-adds are written out, so that every kernel decides alike whatever its unit's
// contraction setting.
LUX_DI bool alpha_accept(const DevScene& S, const DevInstance& I, int inst, int prim, float bu, float bv, f3 wdir,
                         int pixel, int iter) {
    const DevMaterial& m = S.mats[I.material];
    if (m.alpha_mode == 0) return true;
    float alpha = m.alpha;
    if (m.flags & kMatAlbedoTex) {
        float ux = 0.0f, uy = 0.0f;
        if (I.flags & kInstHasUVs) {
            const uint32_t* id = S.idx + (size_t(I.idx_base) + prim) * 3;
            uint32_t i0 = I.vert_base + id[0], i1 = I.vert_base + id[1], i2 = I.vert_base + id[2];
            const float bA = __fsub_rn(__fsub_rn(1.0f, bu), bv);
            ux = __fmaf_rn(bv, S.uv[i2 * 2], __fmaf_rn(bA, S.uv[i0 * 2], __fmul_rn(bu, S.uv[i1 * 2])));
            uy = __fmaf_rn(bv, S.uv[i2 * 2 + 1], __fmaf_rn(bA, S.uv[i0 * 2 + 1], __fmul_rn(bu, S.uv[i1 * 2 + 1])));
        }
        ux = __fmul_rn(ux, m.albedo_tt.scale[0]);
        uy = __fmul_rn(uy, m.albedo_tt.scale[1]);
        if (m.albedo_tt.rotation != 0.0f) {
            const float c = cosf(m.albedo_tt.rotation), s = sinf(m.albedo_tt.rotation);
            const float nx = __fmaf_rn(c, ux, -__fmul_rn(s, uy)), ny = __fmaf_rn(c, uy, __fmul_rn(s, ux));
            ux = nx;
            uy = ny;
        }
        ux = __fadd_rn(ux, m.albedo_tt.offset[0]);
        uy = __fadd_rn(uy, m.albedo_tt.offset[1]);
        float4 tx = tex2D<float4>(cudaTextureObject_t(m.albedo_tex), ux, uy);
        alpha *= tx.w;
    }
    if (m.alpha_mode == 1) return !(alpha < m.alpha_cutoff);
    uint32_t h = hash_u32(uint32_t(pixel) ^ hash_u32(uint32_t(iter)));
    h = hash_u32(h ^ __float_as_uint(wdir.x));
    h = hash_u32(h ^ __float_as_uint(wdir.y));
    h = hash_u32(h ^ __float_as_uint(wdir.z));
    h = hash_u32(h ^ uint32_t(I.key));  // the instance's index within its own scene
    h = hash_u32(h ^ uint32_t(prim));
    float rnd = float(h >> 8) * (1.0f / 16777216.0f);
    return !(rnd >= alpha);
}

// Traversal state of one lane. Two-level layout: wo, wd hold the world ray (its reciprocals are
// recomputed when the traversal leaves an instance) and cur the ray of the current level.
// Single-level layout: cur is the world ray throughout, and wo, wd hold the object-space ray of
// the instance `inst` whose triangles were tested last.
struct Lane {
    f3 wo, wd;          // world ray (two-level) / object ray of `inst` (single-level)
    TRay cur;           // ray of the current level (world in the TLAS, object space in a BLAS)
    float tlim;         // the ray's limit: tmax until a hit, then the closest hit's t
    uint2 g;            // node group: x = first internal child, y = imask << 8 | remaining hit keys
    uint2 t;            // leaf group: x = first record, y = tag (kTagTri / kTagInst) | leaf-slot
                        // mask << 8 | remaining hit slots
    int sp;             // stack depth
    int inst;           // current instance (-1 in the TLAS)
    int inst_flags;
    uint32_t inst_prim_base;
    int item;           // the ray's work item, from which the alpha-blend hash key is found when an
                        // alpha-blended instance is tested
    int work;           // BVH heatmap (mode 3): node visits + triangle tests
    bool done;
};

// MODE: 0 radiance, 1 DL shadow, 2 env occlusion (any hit), 3 BVH heatmap; -1: `any` says at run
// time whether any hit ends the ray (one copy of the code for both kinds of ray).
// KEY: gives the pixel and iteration that key a ray's alpha-blend hash, from Lane::item.
template <int MODE, bool SINGLE, int BLOCK, class KEY>
struct Tracer {
    const DevScene& S;
    uint2 (*sh)[BLOCK];  // shared stack [kShStack][block]
    float4* hits;              // shared, per thread: the closest hit's u, v, instance, prim (int bits)
    const unsigned char* lut;  // shared, fill_key_table
    uint2 loc[kLocStack];
    int tid;
    int* err;
    KEY keys;
    bool any;

    LUX_DI bool any_hit() const { return MODE == 2 || (MODE < 0 && any); }

    LUX_DI void push(Lane& L, uint2 e) {
        if (L.sp < kShStack) sh[L.sp][tid] = e;
        else if (L.sp < kShStack + kLocStack) loc[L.sp - kShStack] = e;
        else {
            atomicOr(err, 1);
            return;
        }
        ++L.sp;
    }
    LUX_DI uint2 pop(Lane& L) {
        --L.sp;
        return L.sp < kShStack ? sh[L.sp][tid] : loc[L.sp - kShStack];
    }

    LUX_DI void start(Lane& L, f3 o, f3 d, float tmax, uint32_t root) {
        L.wo = o;
        L.wd = d;
        L.cur = make_ray(o, d);
        L.tlim = tmax;
        hits[tid] = make_float4(0.0f, 0.0f, __int_as_float(-1), __int_as_float(-1));
        L.sp = 0;
        L.inst = -1;
        L.inst_flags = 0;
        L.inst_prim_base = 0;
        L.done = false;
        L.work = 0;
        // root group: a single internal child (slot 0) = the TLAS root, at key oct
        L.g = make_uint2(root, (1u << 8) | (1u << L.cur.oct));
        L.t = make_uint2(0u, 0u);
    }

    LUX_DI Best best(const Lane& L) const {
        const float4 h = hits[tid];
        Best b;
        b.u = h.x;
        b.v = h.y;
        b.inst = __float_as_int(h.z);
        b.prim = __float_as_int(h.w);
        b.t = b.inst >= 0 ? L.tlim : -1.0f;
        return b;
    }
    static LUX_DI f3 world_o(const Lane& L) { return SINGLE ? L.cur.o : L.wo; }
    static LUX_DI f3 world_d(const Lane& L) { return SINGLE ? L.cur.d : L.wd; }

    // Node phase: visit the nearest remaining child of the node group.
    LUX_DI void visit(Lane& L) {
        uint32_t keys = L.g.y & 0xffu;
        uint32_t key = __ffs(keys) - 1;
        keys &= keys - 1;
        uint32_t slot = key ^ L.cur.oct;
        uint32_t imask = L.g.y >> 8;
        uint32_t child = L.g.x + __popc(imask & ((1u << slot) - 1u));
        if (keys) push(L, make_uint2(L.g.x, (imask << 8) | keys));
        uint32_t nkeys, nimask, cbase, tbase, tmask, lmask;
        visit_node(S.nodes, child, L.cur, L.tlim, nkeys, nimask, cbase, tbase, tmask, lmask, lut);
        if (MODE == 3) ++L.work;
        L.g = make_uint2(cbase, (nimask << 8) | nkeys);
        if (tmask) {
            if (SINGLE) L.t = make_uint2(tbase, kTagTri | (lmask << 8) | tmask);
            else if (L.inst >= 0) L.t = make_uint2(L.inst_prim_base + tbase, kTagTri | (lmask << 8) | tmask);
            else L.t = make_uint2(tbase, kTagInst | (lmask << 8) | tmask);
        }
    }

    // Triangle phase: test the lowest triangle of the leaf group.
    LUX_DI void test_one(Lane& L) {
        uint32_t m = L.t.y & kRecMask;
        const uint32_t lm = (L.t.y >> 8) & 0xffu;
        int k = __ffs(m) - 1;
        m &= m - 1;
        L.t.y = m ? (kTagTri | (lm << 8) | m) : 0u;
        k = __popc(lm & ((1u << k) - 1u));  // the slot's record: its rank among the leaf slots
        float t, u, v;
        int prim;
        if (MODE == 3) ++L.work;
        if (SINGLE) {
            // the record names its instance; the object-space ray is rebuilt when it changes,
            // exactly as entering the instance from a TLAS leaf builds it
            const float4* q = S.prims + size_t(L.t.x + uint32_t(k)) * 3;
            const float4 a4 = __ldg(q), e14 = __ldg(q + 1), e24 = __ldg(q + 2);
            const int inst = __float_as_int(e14.w);
            if (inst != L.inst) {
                const DevInstance& I = S.insts[inst];
                const float4* mq = reinterpret_cast<const float4*>(I.Minv);
                const float4 m0 = __ldg(mq), m1 = __ldg(mq + 1), m2 = __ldg(mq + 2);
                const float Minv[12] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w, m2.x, m2.y, m2.z, m2.w};
                L.wo = xform(Minv, L.cur.o, 1.0f);
                L.wd = xform(Minv, L.cur.d, 0.0f);
                L.inst = inst;
                L.inst_flags = __ldg(&I.flags);
            }
            if (!mt_core(a4, e14, e24, L.wo, L.wd, t, u, v, prim)) return;
        } else {
            if (!mt_test(S.prims, L.t.x + uint32_t(k), L.cur, t, u, v, prim)) return;
        }
        if (!(t <= L.tlim)) return;
        if (!any_hit() && t == L.tlim) {  // a tie with a hit goes to the lowest (instance, prim)
            const float4 h = hits[tid];
            const int bi = __float_as_int(h.z), bp = __float_as_int(h.w);
            if (bi >= 0 && !(L.inst < bi || (L.inst == bi && prim < bp))) return;
        }
        if (L.inst_flags & kInstAnyHit) {
            int pixel, iter;
            keys(L.item, pixel, iter);
            if (!alpha_accept(S, S.insts[L.inst], L.inst, prim, u, v, world_d(L), pixel, iter)) return;
        }
        L.tlim = t;
        hits[tid] = make_float4(u, v, __int_as_float(L.inst), __int_as_float(prim));
        if (any_hit()) L.done = true;
    }

    // Instance phase: enter the lowest instance of a TLAS leaf group. The world-level node
    // group and the rest of the leaf group wait on the stack under a marker.
    LUX_DI void enter(Lane& L) {
        uint32_t m = L.t.y & kRecMask;
        const uint32_t lm = (L.t.y >> 8) & 0xffu;
        int k = __ffs(m) - 1;
        m &= m - 1;
        const int slot_k = k;
        k = __popc(lm & ((1u << slot_k) - 1u));
        // the instance's leaf record: transform and BLAS root in one dependent 64-byte load
        const float4* q = S.tlas_leaf + size_t(L.t.x + uint32_t(k)) * 4;
        const float4 r0 = __ldg(q), r1 = __ldg(q + 1), r2 = __ldg(q + 2);
        const uint4 e = __ldg(reinterpret_cast<const uint4*>(q + 3));
        if (L.g.y & 0xffu) push(L, L.g);
        if (m) push(L, make_uint2(L.t.x, kTagInst | (lm << 8) | m));
        push(L, make_uint2(0u, kTagMarker));
        const float Minv[12] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, r2.x, r2.y, r2.z, r2.w};
        L.cur = make_ray(xform(Minv, L.wo, 1.0f), xform(Minv, L.wd, 0.0f));
        L.inst = int(e.w);
        L.inst_flags = int(e.z);
        L.inst_prim_base = e.y;
        L.g = make_uint2(e.x, (1u << 8) | (1u << L.cur.oct));
        L.t = make_uint2(0u, 0u);
    }

    // Pop phase: take the next group from the stack; the ray is done when it is empty.
    LUX_DI void next(Lane& L) {
        while (true) {
            if (L.sp == 0) {
                L.done = true;
                return;
            }
            uint2 e = pop(L);
            uint32_t tag = e.y & kTagMask;
            if (!SINGLE && tag == kTagMarker) {
                L.cur = make_ray(L.wo, L.wd);
                L.inst = -1;
                L.inst_flags = 0;
                continue;
            }
            if (tag == kTagNode) L.g = e;
            else L.t = e;
            return;
        }
    }

    // One iteration of a warp's traversal loop. Every lane of the warp runs every phase (lanes
    // without a ray or without work for a phase are predicated off), so the ballots see the
    // whole warp. Returns true in the lanes whose ray is done.
    LUX_DI bool step(Lane& L, bool active, int postpone) {
        const unsigned FULL = 0xffffffffu;
        // node phase
        if (active && (L.g.y & 0xffu)) visit(L);
        // triangle phase, postponed while too few lanes have triangles and others nodes
        while (true) {
            const bool want = active && (SINGLE ? L.t.y != 0u : (L.t.y & kTagMask) == kTagTri);
            const unsigned wm = __ballot_sync(FULL, want);
            if (!wm) break;
            const bool nodes = active && (L.g.y & 0xffu);
            if (__popc(wm) < postpone && __any_sync(FULL, nodes)) {
                // lanes with nodes left push their triangles; the others keep them
                if (want && nodes) {
                    push(L, L.t);
                    L.t = make_uint2(0u, 0u);
                }
                break;
            }
            if (want) test_one(L);
            if (any_hit() && want && L.done) {
                L.t = make_uint2(0u, 0u);
                L.g = make_uint2(0u, 0u);
            }
        }
        // instance phase
        if (!SINGLE && active && !L.done && (L.t.y & kTagMask) == kTagInst) enter(L);
        // pop phase
        if (active && !L.done && !(L.g.y & 0xffu) && !(L.t.y & kRecMask)) next(L);
        return active && L.done;
    }
};

// World normal of a radiance hit as the closest-hit program computes it
// (src/optixshaders/optix_triangle.cu:170-192,224): interpolated vertex normals when the
// mesh has them, else the geometric normal, then the normal transform of the instance.
LUX_DI f3 hit_world_normal(const DevScene& S, int inst, int prim, float bu, float bv) {
    const DevInstance& I = S.insts[inst];
    const uint32_t* id = S.idx + (size_t(I.idx_base) + prim) * 3;
    uint32_t i0 = I.vert_base + __ldg(id), i1 = I.vert_base + __ldg(id + 1), i2 = I.vert_base + __ldg(id + 2);
    f3 n;
    if (I.flags & kInstHasNormals) {
        float bA = __fsub_rn(__fsub_rn(1.0f, bu), bv);
        f3 nA = ld3(S.nrm + i0 * 3), nB = ld3(S.nrm + i1 * 3), nC = ld3(S.nrm + i2 * 3);
        f3 s = mk(__fadd_rn(__fadd_rn(__fmul_rn(bA, nA.x), __fmul_rn(bu, nB.x)), __fmul_rn(bv, nC.x)),
                  __fadd_rn(__fadd_rn(__fmul_rn(bA, nA.y), __fmul_rn(bu, nB.y)), __fmul_rn(bv, nC.y)),
                  __fadd_rn(__fadd_rn(__fmul_rn(bA, nA.z), __fmul_rn(bu, nB.z)), __fmul_rn(bv, nC.z)));
        float l2 = __fadd_rn(__fadd_rn(__fmul_rn(s.x, s.x), __fmul_rn(s.y, s.y)), __fmul_rn(s.z, s.z));
        float il = __fdiv_rn(1.0f, __fsqrt_rn(l2));
        n = mk(__fmul_rn(s.x, il), __fmul_rn(s.y, il), __fmul_rn(s.z, il));
    } else {
        f3 A = ld3(S.pos + i0 * 3), B = ld3(S.pos + i1 * 3), C = ld3(S.pos + i2 * 3);
        f3 e1 = mk(__fsub_rn(B.x, A.x), __fsub_rn(B.y, A.y), __fsub_rn(B.z, A.z));
        f3 e2 = mk(__fsub_rn(C.x, A.x), __fsub_rn(C.y, A.y), __fsub_rn(C.z, A.z));
        f3 c = mk(__fsub_rn(__fmul_rn(e1.y, e2.z), __fmul_rn(e2.y, e1.z)), __fsub_rn(__fmul_rn(e1.z, e2.x), __fmul_rn(e2.z, e1.x)),
                  __fsub_rn(__fmul_rn(e1.x, e2.y), __fmul_rn(e2.x, e1.y)));
        float l2 = __fadd_rn(__fadd_rn(__fmul_rn(c.x, c.x), __fmul_rn(c.y, c.y)), __fmul_rn(c.z, c.z));
        float il = __fdiv_rn(1.0f, __fsqrt_rn(l2));
        n = mk(__fmul_rn(c.x, il), __fmul_rn(c.y, il), __fmul_rn(c.z, il));
    }
    f3 w = xform(I.MinvT, n, 0.0f);
    float l2 = __fadd_rn(__fadd_rn(__fmul_rn(w.x, w.x), __fmul_rn(w.y, w.y)), __fmul_rn(w.z, w.z));
    float il = __fdiv_rn(1.0f, __fsqrt_rn(l2));
    return mk(__fmul_rn(w.x, il), __fmul_rn(w.y, il), __fmul_rn(w.z, il));
}

// The shadow ray of a radiance hit (raygen program, src/optixshaders/optix_triangle.cu:82-132):
// from the hit point, off the surface by the unflipped normal, toward the NEE sample ns (an
// emitter point, or with ENV an environment direction).
LUX_DI void shadow_ray(const DevScene& S, const Best& best, f3 wo, f3 wd, f3 ns, bool env, f3& so, f3& sd, float& tmax) {
    f3 n = hit_world_normal(S, best.inst, best.prim, best.u, best.v);
    f3 hp = mk(__fadd_rn(wo.x, __fmul_rn(best.t, wd.x)), __fadd_rn(wo.y, __fmul_rn(best.t, wd.y)),
               __fadd_rn(wo.z, __fmul_rn(best.t, wd.z)));
    so = mk(__fadd_rn(hp.x, __fmul_rn(n.x, 1e-4f)), __fadd_rn(hp.y, __fmul_rn(n.y, 1e-4f)),
            __fadd_rn(hp.z, __fmul_rn(n.z, 1e-4f)));
    if (env) {
        sd = ns;
        tmax = 1e16f;
    } else {
        f3 ld = mk(__fsub_rn(ns.x, so.x), __fsub_rn(ns.y, so.y), __fsub_rn(ns.z, so.z));
        float dl = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(ld.x, ld.x), __fmul_rn(ld.y, ld.y)), __fmul_rn(ld.z, ld.z)));
        float il = __fdiv_rn(1.0f, dl);
        sd = mk(__fmul_rn(ld.x, il), __fmul_rn(ld.y, il), __fmul_rn(ld.z, il));
        tmax = __fadd_rn(__fmul_rn(dl, 1.0001f), 1e-4f);
    }
}

}  // namespace
}  // namespace lux
