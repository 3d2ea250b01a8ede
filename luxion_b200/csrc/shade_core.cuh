// shade_core.cuh -- shading and light sampling of one path: what the wavefront's kernels (shade.cu)
// and the whole-path kernel (paths.cu) share.
//
// For units compiled with --fmad=false: every float multiply and add is rounded on its own, in
// the order the reference writes it (see shade.cu).
#pragma once

#include "device_scene.h"
#include "device_math.cuh"
#include "launch.h"

namespace lux {
namespace {

// A closest hit as the shading reads it. The tangent frame is only read under a normal map,
// so it is rebuilt there from the hit (hit_tangent) instead of for every hit.
struct Isect {
    float t;
    f3 normal;
    int inst, prim;
    int material;
    float u, v;
};

LUX_DI float4 tex(unsigned long long t, float u, float v) { return tex2D<float4>(cudaTextureObject_t(t), u, v); }

// The rotation of a texture transform, out of line: few transforms rotate, and a sine and cosine
// at every texture fetch are a good part of the shading's code (see k_shade on why that matters).
__device__ __noinline__ float2 tt_rotate(float u, float v, float rotation) {
    float c = cosf(rotation), s = sinf(rotation);
    return make_float2(c * u - s * v, s * u + c * v);
}
LUX_DI void tt_apply(const DevTexTransform& tt, float& u, float& v) {  // src/material_queries.cu:3-17
    u *= tt.scale[0];
    v *= tt.scale[1];
    if (tt.rotation != 0.0f) {
        const float2 r = tt_rotate(u, v, tt.rotation);
        u = r.x;
        v = r.y;
    }
    u = u + tt.offset[0];
    v = v + tt.offset[1];
}

LUX_DI void mesh_tri(const DevScene& S, const DevInstance& I, int prim, uint32_t& i0, uint32_t& i1, uint32_t& i2) {
    const uint32_t* id = S.idx + (size_t(I.idx_base) + prim) * 3;
    i0 = I.vert_base + __ldg(id);
    i1 = I.vert_base + __ldg(id + 1);
    i2 = I.vert_base + __ldg(id + 2);
}

// closest-hit program (src/optixshaders/optix_triangle.cu:156-243); its tangent is hit_tangent
LUX_DI Isect ch_radiance(const DevScene& S, float t, int inst, int prim, float bu, float bv) {
    Isect r;
    const DevInstance& I = S.insts[inst];
    uint32_t i0, i1, i2;
    mesh_tri(S, I, prim, i0, i1, i2);
    f3 n;
    float bA = 1.0f - bu - bv;
    if (I.flags & kInstHasNormals) {
        f3 nA = ld3(S.nrm + i0 * 3), nB = ld3(S.nrm + i1 * 3), nC = ld3(S.nrm + i2 * 3);
        n = normalize(bA * nA + bu * nB + bv * nC);
    } else {
        f3 A = ld3(S.pos + i0 * 3), B = ld3(S.pos + i1 * 3), C = ld3(S.pos + i2 * 3);
        n = normalize(cross(B - A, C - A));
    }
    float uu = 0.0f, vv = 0.0f;
    if (I.flags & kInstHasUVs) {
        float ax = S.uv[i0 * 2], ay = S.uv[i0 * 2 + 1], bx = S.uv[i1 * 2], by = S.uv[i1 * 2 + 1];
        float cx = S.uv[i2 * 2], cy = S.uv[i2 * 2 + 1];
        uu = bA * ax + bu * bx + bv * cx;
        vv = bA * ay + bu * by + bv * cy;
    }
    r.t = t;
    r.normal = normalize(xform(I.MinvT, n, 0.0f));
    r.inst = inst;
    r.prim = prim;
    r.material = I.material;
    r.u = uu;
    r.v = vv;
    return r;
}

// The closest-hit program's world tangent (optix_triangle.cu:194-223): the object-space
// tangent from the uv deltas, transformed by the instance, then made orthogonal to the world
// normal n (the hit's is.normal).
LUX_DI f3 hit_tangent(const DevScene& S, int inst, int prim, f3 n) {
    const DevInstance& I = S.insts[inst];
    uint32_t i0, i1, i2;
    mesh_tri(S, I, prim, i0, i1, i2);
    f3 tg = mk(1.0f, 0.0f, 0.0f);
    if (I.flags & kInstHasUVs) {
        f3 A = ld3(S.pos + i0 * 3), B = ld3(S.pos + i1 * 3), C = ld3(S.pos + i2 * 3);
        f3 e1 = B - A, e2 = C - A;
        float ax = S.uv[i0 * 2], ay = S.uv[i0 * 2 + 1], bx = S.uv[i1 * 2], by = S.uv[i1 * 2 + 1];
        float cx = S.uv[i2 * 2], cy = S.uv[i2 * 2 + 1];
        float d1x = bx - ax, d1y = by - ay, d2x = cx - ax, d2y = cy - ay;
        float det = d1x * d2y - d2x * d1y;
        float f = (fabsf(det) < 1e-10f) ? 0.0f : 1.0f / det;
        if (f != 0.0f) {
            tg.x = f * (d2y * e1.x - d1y * e2.x);
            tg.y = f * (d2y * e1.y - d1y * e2.y);
            tg.z = f * (d2y * e1.z - d1y * e2.z);
        }
    }
    tg = normalize(xform(I.M, tg, 0.0f));
    f3 T = tg - dot(tg, n) * n;
    float l2 = dot(T, T);
    if (l2 > 1e-10f) {
        tg = T * (1.0f / sqrtf(l2));
    } else {
        tg = (fabsf(n.x) > 0.9f) ? mk(0.0f, 1.0f, 0.0f) : mk(1.0f, 0.0f, 0.0f);
        tg = normalize(cross(tg, n));
    }
    return tg;
}

// direct-light closest-hit program (src/optixshaders/optix_triangle.cu:259-305)
LUX_DI Isect ch_direct_light(const DevScene& S, float t, int inst, int prim, float bu, float bv) {
    Isect r;
    const DevInstance& I = S.insts[inst];
    uint32_t i0, i1, i2;
    mesh_tri(S, I, prim, i0, i1, i2);
    float bA = 1.0f - bu - bv;
    f3 n;
    if (I.flags & kInstHasNormals) {
        n = normalize(bA * ld3(S.nrm + i0 * 3) + bu * ld3(S.nrm + i1 * 3) + bv * ld3(S.nrm + i2 * 3));
    } else {
        f3 A = ld3(S.pos + i0 * 3), B = ld3(S.pos + i1 * 3), C = ld3(S.pos + i2 * 3);
        n = normalize(cross(B - A, C - A));
    }
    float uu = 0.0f, vv = 0.0f;
    if (I.flags & kInstHasUVs) {
        uu = bA * S.uv[i0 * 2] + bu * S.uv[i1 * 2] + bv * S.uv[i2 * 2];
        vv = bA * S.uv[i0 * 2 + 1] + bu * S.uv[i1 * 2 + 1] + bv * S.uv[i2 * 2 + 1];
    }
    r.t = t;
    r.normal = normalize(xform(I.MinvT, n, 0.0f));
    r.inst = inst;
    r.prim = prim;
    r.material = I.material;
    r.u = uu;
    r.v = vv;
    return r;
}

// vpow in one copy of powf's code, run three times (see k_shade on why code size matters)
LUX_DI f3 vpow_loop(f3 v, float e) {
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
        const float r = powf(v.x, e);
        v.x = v.y;
        v.y = v.z;
        v.z = r;
    }
    return v;
}

// ---- material queries (src/material_queries.cu:19-117)
LUX_DI f3 get_albedo(const DevMaterial& m, float u, float v) {
    if (m.flags & kMatAlbedoTex) {
        tt_apply(m.albedo_tt, u, v);
        float4 t = tex(m.albedo_tex, u, v);
        return vpow_loop(mk(t.x, t.y, t.z), 2.2f);
    }
    return mk(m.color[0], m.color[1], m.color[2]);
}
LUX_DI f3 get_normal(const DevScene& S, const DevMaterial& m, const Isect& is) {
    if (m.flags & kMatNormalTex) {
        float u = is.u, v = is.v;
        tt_apply(m.normal_tt, u, v);
        float4 t = tex(m.normal_tex, u, v);
        f3 ln = mk(t.x * 2.0f - 1.0f, t.y * 2.0f - 1.0f, t.z * 2.0f - 1.0f);
        const f3 N = is.normal;
        if (!(dot(ln, ln) > 1e-12f)) return N;
        const f3 tangent = hit_tangent(S, is.inst, is.prim, N);
        f3 T = tangent - dot(tangent, N) * N;
        float t2 = dot(T, T);
        if (!(t2 > 1e-12f)) return N;
        T = T * (1.0f / sqrtf(t2));
        f3 Bt = cross(N, T);
        f3 mp = mk(T.x * ln.x + Bt.x * ln.y + N.x * ln.z, T.y * ln.x + Bt.y * ln.y + N.y * ln.z,
                   T.z * ln.x + Bt.z * ln.y + N.z * ln.z);
        float m2 = dot(mp, mp);
        if (!(m2 > 1e-12f)) return N;
        mp = mp * (1.0f / sqrtf(m2));
        if (!(dot(mp, N) > 1e-4f)) return N;
        return mp;
    }
    return is.normal;
}
LUX_DI void get_mr(const DevMaterial& m, float u, float v, float& rough, float& metal) {
    rough = m.roughness;
    metal = m.metallic;
    if (m.flags & kMatMRTex) {
        tt_apply(m.mr_tt, u, v);
        float4 t = tex(m.mr_tex, u, v);
        rough *= t.y;
        metal *= t.z;
    }
}
LUX_DI f3 get_emission(const DevMaterial& m, float u, float v) {
    f3 e = mk(m.emission[0], m.emission[1], m.emission[2]);
    if (m.flags & kMatEmissiveTex) {
        tt_apply(m.emissive_tt, u, v);
        float4 t = tex(m.emissive_tex, u, v);
        e = e * vpow_loop(mk(t.x, t.y, t.z), 2.2f);
    }
    return e;
}

// The normal-map texel get_normal reads (src/material_queries.cu:32-40), or (0.5, 0.5, 1)
// without a normal texture.
LUX_DI f3 normal_map_texel(const DevMaterial& m, float u, float v) {
    if (!(m.flags & kMatNormalTex)) return mk(0.5f, 0.5f, 1.0f);
    tt_apply(m.normal_tt, u, v);
    float4 t = tex(m.normal_tex, u, v);
    return mk(t.x, t.y, t.z);
}
// get_alpha (src/material_queries.cu:119-137)
LUX_DI float get_alpha(const DevMaterial& m, float u, float v) {
    if (m.alpha_mode == 0) return 1.0f;
    float alpha = m.alpha;
    if (m.flags & kMatAlbedoTex) {
        tt_apply(m.albedo_tt, u, v);
        alpha *= tex(m.albedo_tex, u, v).w;
    }
    if (m.alpha_mode == 1) return alpha >= m.alpha_cutoff ? 1.0f : 0.0f;
    return alpha;
}
// render_material_debug_mode (src/material_debug_render.cu:3-26)
LUX_DI f3 material_debug_color(int mode, f3 mc, f3 normal, f3 nmap, float rough, float metal, float alpha) {
    switch (mode) {
        case 1: return mc;
        case 2: return normal * 0.5f + mk(0.5f, 0.5f, 0.5f);
        case 3: return nmap;
        case 4: return mk(rough, rough, rough);
        case 5: return mk(metal, metal, metal);
        case 6: return mk(alpha, alpha, alpha);
    }
    return mk(0.0f, 0.0f, 0.0f);
}

// ---- Cook-Torrance (src/shaders/cook_torrance.cu:8-331)
LUX_DI float D_GGX(f3 h, f3 n, float alpha) {
    float ndh = dot(n, h);
    if (ndh <= 0.0f) return 0.0f;
    float a2 = alpha * alpha;
    float ndh2 = ndh * ndh;
    float dc = (ndh2 * a2) + (1.0f - ndh2);
    float den = dc * dc * kPI;
    return a2 / gmax(den, kEPS_CT);
}
LUX_DI f3 F_schlick(float vdh, f3 f0) {
    float m = 1.0f - vdh;
    float m2 = m * m;
    return f0 + ((mk(1.0f, 1.0f, 1.0f) - f0) * (m2 * m2 * m));
}
LUX_DI float F_dielectric(float ci, float etaI, float etaT) {
    ci = gclamp(ci, 0.0f, 1.0f);
    float si = sqrtf(gmax(0.0f, 1.0f - ci * ci));
    float st = (etaI / etaT) * si;
    if (st >= 1.0f) return 1.0f;
    float ct = sqrtf(gmax(0.0f, 1.0f - st * st));
    float rpa = ((etaT * ci) - (etaI * ct)) / ((etaT * ci) + (etaI * ct));
    float rpe = ((etaI * ci) - (etaT * ct)) / ((etaI * ci) + (etaT * ct));
    return (rpa * rpa + rpe * rpe) / 2.0f;
}
LUX_DI f3 half_t(f3 wo, f3 wi, float etaI, float etaT) { return normalize(-(etaI * wo + etaT * wi)); }
LUX_DI float smith(f3 w, f3 n, float alpha) {
    float a2 = alpha * alpha;
    float nw = gmax(dot(n, w), 0.0f);
    float num = 2.0f * nw;
    float us = a2 + (1.0f - a2) * (nw * nw);
    float den = nw + sqrtf(us);
    return num / gmax(den, kEPS_CT);
}
LUX_DI f3 fresnel(float c, f3 albedo, float metal, float etaI, float etaT) {
    float d = F_dielectric(c, etaI, etaT);
    return vmix(mk(d, d, d), F_schlick(c, albedo), metal);
}
LUX_DI f3 BRDF(f3 v, f3 n, f3 l, f3 albedo, float rough, float metal, float ior, float trans) {
    ior = gmax(ior, 1.0001f);
    bool enter = dot(v, n) > 0.0f;
    f3 nf = enter ? n : -n;
    float etaI = enter ? 1.0f : ior, etaT = enter ? ior : 1.0f;
    f3 h = normalize(v + l);
    rough = gclamp(rough, 0.0001f, 1.0f);
    float alpha = rough * rough;
    float D = D_GGX(h, nf, alpha);
    f3 F = fresnel(gmax(dot(v, h), 0.0f), albedo, metal, etaI, etaT);
    float G = smith(v, nf, alpha) * smith(l, nf, alpha);
    f3 num = D * F * G;
    float den = 4.0f * gmax(dot(nf, v), 0.0f) * gmax(dot(nf, l), 0.0f);
    f3 spec = num / gmax(den, kEPS_CT);
    f3 kD = (1.0f - metal) * (mk(1.0f, 1.0f, 1.0f) - F) * (1.0f - trans);
    f3 diffuse = kD * albedo * kINV_PI;
    return diffuse + spec;
}
LUX_DI f3 BTDF(f3 wo, f3 n, f3 wi, f3 albedo, float rough, float metal, float ior, float trans) {
    bool enter = dot(wo, n) > 0.0f;
    float etaI = enter ? 1.0f : ior, etaT = enter ? ior : 1.0f;
    f3 ht = half_t(wo, wi, etaI, etaT);
    float jd = (etaT * dot(wi, ht) + etaI * dot(wo, ht));
    float jac = (etaI * etaI) / gmax(jd * jd, kEPS_CT);
    float cnum = fabsf(dot(wi, ht)) * fabsf(dot(wo, ht));
    float cden = fabsf(dot(wi, n)) * fabsf(dot(wo, n));
    rough = gclamp(rough, 0.0001f, 1.0f);
    float alpha = rough * rough;
    float D = D_GGX(ht, n, alpha);
    float F = F_dielectric(fabsf(dot(wo, ht)), etaI, etaT);
    bool gv = dot(wi, ht) * dot(wi, n) > 0.0f && dot(wo, ht) * dot(wo, n) > 0.0f;
    float G = gv ? smith(dot(wi, n) > 0.0f ? wi : -wi, n, alpha) * smith(dot(wo, n) > 0.0f ? wo : -wo, n, alpha) : 0.0f;
    float DFG = D * G * (1.0f - F);
    return albedo * (trans * (1.0f - metal) * (cnum / cden) * jac * DFG);
}
LUX_DI void lobe_probs(f3 wo, f3 n, float metal, f3 color, float ior, float trans, float& pR, float& pD, float& pS) {
    bool enter = dot(wo, n) > 0.0f;
    float etaI = enter ? 1.0f : ior, etaT = enter ? ior : 1.0f;
    float cm = fabsf(dot(wo, n));
    f3 Fa = fresnel(cm, color, metal, etaI, etaT);
    float sr = gclamp((Fa.x + Fa.y + Fa.z) / 3.0f, 0.01f, 0.99f);
    float Fm = F_dielectric(cm, etaI, etaT);
    pR = trans * (1.0f - metal) * (1.0f - Fm);
    pD = (1.0f - pR) * (1.0f - sr) * (1.0f - metal);
    pS = 1.0f - pR - pD;
}
// The lobe probabilities depend on the outgoing direction and the material only, so one
// evaluation serves the direction sampling and every pdf of a shading point (the reference
// evaluates them in each call, with the same operands).
struct Lobes {
    float pR, pD, pS;
};
LUX_DI Lobes lobes_of(f3 wo, f3 n, float metal, f3 color, float ior, float trans) {
    Lobes L;
    lobe_probs(wo, n, metal, color, gmax(ior, 1.0001f), trans, L.pR, L.pD, L.pS);
    return L;
}
// sampleCookTorrance (src/shaders/cook_torrance.cu:156-224) with the diffuse lobe's
// calculateRandomDirectionInHemisphere (src/interactions.cu:7-45); L = lobes_of(wo, n, metal,
// color, ior, trans), ior at least 1.0001. Both lobes take their angle around the axis from the
// third draw, so one sine and cosine serve both.
LUX_DI f3 sample_ct(f3 wo, f3 n, float rough, Rng& rng, float ior, const Lobes& L) {
    const float r = rng.u01();
    const float x1 = rng.u01(), x2 = rng.u01();
    rough = gclamp(rough, 0.0001f, 1.0f);
    float alpha = rough * rough;
    bool enter = dot(wo, n) > 0.0f;
    f3 nf = enter ? n : -n;
    const float pD = L.pD, pS = L.pS;
    static_assert(2.0f * kPI == kTWO_PI, "the lobes' angles around the axis");
    float sp, cp;
    sincosf(x2 * kTWO_PI, &sp, &cp);
    if (r > pS && r <= pS + pD) {
        float up = sqrtf(x1);
        float over = sqrtf(1.0f - up * up);
        f3 dnn;
        if (fabsf(nf.x) < kSQRT13) dnn = mk(1.0f, 0.0f, 0.0f);
        else if (fabsf(nf.y) < kSQRT13) dnn = mk(0.0f, 1.0f, 0.0f);
        else dnn = mk(0.0f, 0.0f, 1.0f);
        f3 p1 = normalize(cross(nf, dnn));
        f3 p2 = normalize(cross(nf, p1));
        return up * nf + cp * over * p1 + sp * over * p2;
    }
    float etaI = enter ? 1.0f : ior, etaT = enter ? ior : 1.0f;
    float th = atanf((alpha * sqrtf(x1)) / sqrtf(1.0f - x1));
    float st, ct;
    sincosf(th, &st, &ct);
    f3 h = normalize(mk(1.0f * st * cp, 1.0f * st * sp, 1.0f * ct));
    f3 t = normalize(fabsf(nf.z) < 0.999f ? cross(mk(0.0f, 0.0f, 1.0f), nf) : cross(mk(1.0f, 0.0f, 0.0f), nf));
    f3 b = cross(nf, t);
    f3 hw = h.x * t + h.y * b + h.z * nf;
    if (r <= pS) {
        f3 wi = reflect(-wo, hw);
        if (dot(wi, nf) <= 0.0f) return mk(0.0f, 0.0f, 0.0f);
        return normalize(wi);
    }
    f3 wi = refract(-wo, hw, etaI / etaT);
    if (dot(wi, wi) < kEPS_CT || isnan(wi.x) || isnan(wi.y) || isnan(wi.z) || dot(wi, nf) >= 0.0f)
        return mk(0.0f, 0.0f, 0.0f);
    return normalize(wi);
}
LUX_DI float pdf_ggx(f3 wo, f3 wi, f3 n, float rough) {
    f3 h = normalize(wo + wi);
    rough = gclamp(rough, 0.0001f, 1.0f);
    float alpha = rough * rough;
    float ph = D_GGX(h, n, alpha) * dot(n, h);
    return ph / gmax((4.0f * fabsf(dot(wo, h))), kEPS_CT);
}
LUX_DI float pdf_ggx_t(f3 wo, f3 wi, f3 n, float rough, float ior) {
    bool enter = dot(wo, n) > 0.0f;
    float etaI = enter ? 1.0f : ior, etaT = enter ? ior : 1.0f;
    f3 ht = half_t(wo, wi, etaI, etaT);
    rough = gclamp(rough, 0.0001f, 1.0f);
    float alpha = rough * rough;
    float den = etaT * dot(wi, ht) + etaI * dot(wo, ht);
    float ph = D_GGX(ht, n, alpha) * fabsf(dot(n, ht));
    return ph * (etaT * etaT * fabsf(dot(wi, ht))) / gmax(den * den, kEPS_CT);
}
// L = lobes_of(wo, n, metal, color, ior, trans)
LUX_DI float PDF(f3 wo, f3 wi, f3 n, float rough, float ior, const Lobes& L) {
    ior = gmax(ior, 1.0001f);
    f3 nf = dot(wo, n) < 0.0f ? -n : n;
    float pdfD = fmaxf(0.0f, dot(wi, nf)) * kINV_PI;
    float pdfS = pdf_ggx(wo, wi, nf, rough);
    float pdfR = pdf_ggx_t(wo, wi, n, rough, ior);
    bool refr = (dot(wi, n) * dot(wo, n)) < 0.0f;
    float pdf = refr ? L.pR * pdfR : L.pD * pdfD + L.pS * pdfS;
    return gmax(pdf, kPDF_CLAMP);
}

// ---- environment (src/kernels/shade_path.cu:27-42, :207-215)
// Spherical coordinates of a direction, as both the pdf and the lookup take them.
LUX_DI void env_angles(f3 d, float& phi, float& theta) {
    phi = atan2f(d.z, d.x);
    theta = acosf(gclamp(d.y, -1.0f, 1.0f));
}
LUX_DI float envmap_pdf(const DevScene& S, float phi, float theta) {
    const int W = S.env_w, H = S.env_h;
    float u = (phi + kPI) / (2.0f * kPI);
    float v = theta / kPI;
    int col = gclampi(int(u * float(W)), 0, W - 1);
    int row = gclampi(int(v * float(H)), 0, H - 1);
    float pm = (__ldg(S.marginal + row) - (row == 0 ? 0.0f : __ldg(S.marginal + row - 1))) * float(H);
    const float* cr = S.conditional + size_t(row) * W;
    float pc = (__ldg(cr + col) - (col == 0 ? 0.0f : __ldg(cr + col - 1))) * float(W);
    float st = sinf(theta);
    return (st > 1e-6f) ? (pm * pc) / (2.0f * kPI * kPI * st) : 0.0f;
}
LUX_DI f3 env_lookup(const DevScene& S, float phi, float theta, float intensity) {
    float u = float((double(phi) + kM_PI_SHADE) * (double(1.0f) / (double(2.0f) * kM_PI_SHADE)));
    float v = float(double(theta) * (double(1.0f) / kM_PI_SHADE));
    float4 e = tex(S.env_tex, u, v);
    return mk(e.x, e.y, e.z) * intensity;
}

// NEE mode of a kernel instantiation: -1 = read from the options at run time, 0 = none,
// 1 = emitter sampling only (-dmis), 2 = environment sampling (-emis, with or without -dmis;
// the reference's shading then takes the environment branch, src/kernels/shade_path.cu:166-249).
template <int NEE> LUX_DI bool nee_env(const DevOptions& O) { return NEE < 0 ? O.env != 0 : NEE == 2; }
template <int NEE> LUX_DI bool nee_dl(const DevOptions& O) {
    return NEE < 0 ? O.dl != 0 : (NEE == 1 || (NEE == 2 && O.dl != 0));
}
inline int nee_mode_of(const DevOptions& O) { return O.env ? 2 : (O.dl ? 1 : 0); }

// sampleDirectLight for one path (src/kernels/sample_direct_light.cu:31-100). With both -dmis
// and -emis the reference draws the emitter point and then keeps only the environment
// direction (the shading reads one of the two); want_dl = false skips the emitter point's CDF
// searches and vertex loads and only advances the random stream past its three draws.
template <int NEE = -1>
LUX_DI f3 light_sample(const DevScene& S, const DevOptions& O, int iter, int pixel, int depth, f3& env_dir,
                       bool want_dl = true) {
    Rng rng = Rng::seeded(iter, pixel, depth);
    f3 dl = mk(0.0f, 0.0f, 0.0f);
    env_dir = mk(0.0f, 0.0f, 0.0f);
    const bool dl_on = nee_dl<NEE>(O);
    if (dl_on && !want_dl) {
        rng.skip3();
    } else if (dl_on) {
        float rnd = rng.u01();
        int sel = select_from_cdf(S.emissive_prefix, S.num_emissive, rnd);
        int ii = __ldg(S.emissive_inst + sel);
        const DevInstance& I = S.insts[ii];
        float lower = (sel == 0) ? 0.0f : __ldg(S.emissive_prefix + sel - 1);
        float upper = __ldg(S.emissive_prefix + sel);
        float den = upper - lower;
        float off = (den > 1e-10f) ? (rnd - lower) / den : 0.0f;
        off = gclamp(off, 0.0f, 1.0f);
        int ts = select_from_cdf(S.tri_prefix + __ldg(S.tri_prefix_off + sel), I.num_tris, off);
        uint32_t i0, i1, i2;
        mesh_tri(S, I, ts, i0, i1, i2);
        f3 v0 = ld3(S.pos + i0 * 3), v1 = ld3(S.pos + i1 * 3), v2 = ld3(S.pos + i2 * 3);
        float r1 = sqrtf(rng.u01());
        float r2 = rng.u01();
        float u = 1.0f - r1, v = r2 * r1;
        f3 lp = u * v0 + v * v1 + (1.0f - u - v) * v2;
        dl = xform(I.M, lp, 1.0f);
    }
    if (nee_env<NEE>(O)) {
        float rnd = rng.u01();
        const int H = S.env_h, W = S.env_w;
        int mg = select_from_cdf_guided(S.marginal, S.marginal_guide, S.guide_marg, rnd);
        float lower = (mg == 0) ? 0.0f : __ldg(S.marginal + mg - 1);
        float upper = __ldg(S.marginal + mg);
        float den = upper - lower;
        float off = (den > 1e-10f) ? (rnd - lower) / den : 0.0f;
        off = gclamp(off, 0.0f, 1.0f);
        int cn = select_from_cdf_guided(S.conditional + size_t(mg) * W,
                                        S.conditional_guide + size_t(mg) * (S.guide_cond + 1), S.guide_cond, off);
        float u = (float(cn) + 0.5f) / float(W);
        float v = (float(mg) + 0.5f) / float(H);
        float phi = float(double(u) * 2.0 * double(kPI) - double(kPI));
        float st, ct, sp, cp;
        sincosf(v * kPI, &st, &ct);
        sincosf(phi, &sp, &cp);
        env_dir = mk(st * cp, ct, st * sp);
    }
    return dl;
}

// A path as shade_one sees it. d, thr, spec, pixel and iter are read on entry; the other
// fields are outputs: the new origin and pdf of a surviving path.
struct PathState {
    f3 o, d, thr;
    float last_pdf;
    bool spec;
    int pixel, iter;
};

// The path fields shade_one reads late, loaded where they are used instead of being held in
// registers across the shading (origin, radiance so far, pdf of the last bounce, NEE sample), and
// the radiance, written where it is known (a path without a radiance term keeps it).
struct WavePathIn {
    const DevWave& W;
    int pid;
    LUX_DI f3 origin() const { float4 a = ld_stream(&W.s0[pid]); return mk(a.x, a.y, a.z); }
    LUX_DI float last_pdf() const { return ld_stream(&W.s0[pid]).w; }
    LUX_DI f3 color0() const { float4 a = ld_stream(&W.s3[pid]); return mk(a.x, a.y, a.z); }
    LUX_DI f3 nee() const { float4 a = ld_stream(&W.s4[pid]); return mk(a.x, a.y, a.z); }
    LUX_DI void set_color(f3 c, int iter) const { st_stream(&W.s3[pid], make_float4(c.x, c.y, c.z, __int_as_float(iter))); }
};

// Values that wait from one phase to a later one. In the wavefront's kernel they wait in shared
// memory (a phase's barrier makes the compiler read them back), in the others in registers.
enum Parked {
    kPkAlbedo = 0, kPkNormal = 3, kPkN0 = 6, kPkRough = 9, kPkMetal = 10, kPkIor = 11, kPkTrans = 12, kPkThr = 13,
    kPkLight = 16, kPkPdf = 19, kPkCos = 20, kPkPixel = 21, kPkIter = 22, kParked = 23
};
struct SharedPark {
    float* at;  // [kParked][kShadeBlock], this thread's column
    LUX_DI void put(int i, float v) { at[i * kShadeBlock] = v; }
    LUX_DI float get(int i) const { return at[i * kShadeBlock]; }
};
struct RegisterPark {
    float v[kParked];
    LUX_DI void put(int i, float x) { v[i] = x; }
    LUX_DI float get(int i) const { return v[i]; }
};
template <class PARK> LUX_DI void put3(PARK& K, int i, f3 v) {
    K.put(i, v.x);
    K.put(i + 1, v.y);
    K.put(i + 2, v.z);
}
template <class PARK> LUX_DI f3 get3(const PARK& K, int i) { return mk(K.get(i), K.get(i + 1), K.get(i + 2)); }

// A phase boundary of the shading: the block's warps meet, so that they fetch the next phase's
// instructions together (k_shade).
template <bool PHASED> LUX_DI void phase() {
    if (PHASED) __syncthreads();
}

// shadePath for one path; returns true if the path survives (is not killed).
// sh_t: DL shadow hit t (or env occlusion); sh_* the DL shadow hit record.
// MATDBG: the instantiation that also renders the material debug views (O.material_debug).
// NEE: as for light_sample. At most one radiance term is added per call (emission, the NEE
// contribution or the environment on a miss).
// SPAWN_KILLED: also sample the next direction and spawn the ray of a path that an emitter
// hit kills, as the reference does (its result is then unused; the parity entry reports it).
// The NEE terms draw no random numbers, so sampling the direction after them leaves the
// random stream as the reference's (sample first, then Russian roulette).
//
// The shading runs in steps that every path of the warp takes part in, hit or miss, each step in
// one copy of its code: surface, light (emission, shadow result, environment), then the BSDF for
// the light's direction and for the sampled one. Paths that end in the environment share the
// environment step with the hits that sample it, and the two BSDF evaluations of a hit share
// theirs. on: false for a lane that only takes part in the phases (PHASED needs every thread of
// the block; the results of such a lane are not read).
template <bool MATDBG, int NEE, bool SPAWN_KILLED, bool PHASED, class In, class PARK>
LUX_DI bool shade_one(const DevScene& S, const DevOptions& O, int depth, PathState& p, const In& in, PARK& K, float t,
                      int inst, int prim, float bu, float bv, float sh_t, int sh_inst, int sh_prim, float sh_u, float sh_v,
                      bool on = true) {
    Rng rng = Rng::seeded(p.iter, p.pixel, depth);
    K.put(kPkPixel, __int_as_float(p.pixel));
    K.put(kPkIter, __int_as_float(p.iter));
    put3(K, kPkThr, p.thr);
    const bool has_exr = S.has_env != 0;
    const bool hit = on && inst >= 0 && t > 0.0f;
    const bool miss = on && !hit;
    bool emissive = false;
    // ---- surface
    if (hit) {
        const Isect is = ch_radiance(S, t, inst, prim, bu, bv);
        const DevMaterial& m = S.mats[is.material];
        const f3 mc = get_albedo(m, is.u, is.v);
        const f3 normal = get_normal(S, m, is);
        float rough, metal;
        get_mr(m, is.u, is.v, rough, metal);
        if (MATDBG && O.material_debug) {
            // the debug view replaces the colour and ends the path (shade_path.cu:154-164)
            in.set_color(material_debug_color(O.material_debug, mc, normal, normal_map_texel(m, is.u, is.v), rough, metal,
                                              get_alpha(m, is.u, is.v)),
                         p.iter);
            return false;
        }
        const f3 emission = get_emission(m, is.u, is.v);
        emissive = length(emission) > kEPS_UTIL;
        put3(K, kPkAlbedo, mc);
        put3(K, kPkNormal, normal);
        put3(K, kPkN0, is.normal);
        K.put(kPkRough, rough);
        K.put(kPkMetal, metal);
        K.put(kPkIor, gmax(m.ior, 1.0001f));
        K.put(kPkTrans, m.transmission);
        put3(K, kPkLight, emission);
    }
    phase<PHASED>();
    // ---- light: the sample of a hit that sees it (lit), emission, environment
    // MIS applies to the light a BSDF sample found (not for camera rays and specular bounces)
    const bool mis = depth > 1 && !p.spec;
    bool lit = false;
    f3 wl = mk(0.0f, 0.0f, 0.0f);
    {
        float pl = 0.0f;
        float w = 1.0f;  // MIS weight of emission or the environment found by the BSDF
        if (nee_env<NEE>(O)) {
            if (hit && !emissive && sh_t < 0.0f && !(K.get(kPkRough) < kSPEC_ROUGH) && has_exr) {
                const f3 normal = get3(K, kPkNormal);
                wl = in.nee();
                const float cs = dot(dot(-p.d, normal) < 0.0f ? -normal : normal, wl);
                lit = cs > 0.0f;  // a sample below the horizon contributes nothing
                K.put(kPkCos, cs);
            }
        }
        if (has_exr && (miss || (hit && nee_env<NEE>(O)))) {
            f3 d = lit ? wl : hit ? p.d : normalize(p.d);
            bool pdf = lit || (nee_env<NEE>(O) && mis && (miss || emissive));
            bool look = miss && !pdf;
            // a hit's sample takes the pdf of its direction and the radiance of the normalised one;
            // a miss takes both of one direction
            if (pdf || look) {
#pragma unroll 1
                while (true) {
                    float phi, theta;
                    env_angles(d, phi, theta);
                    if (pdf) {
                        pl = envmap_pdf(S, phi, theta);
                        pdf = false;
                        if (lit && pl > 1e-8f) {
                            d = normalize(wl);
                            look = true;
                            continue;
                        }
                        look = miss;
                    }
                    if (look) put3(K, kPkLight, env_lookup(S, phi, theta, O.env_intensity));
                    break;
                }
            }
            if (lit) {
                lit = pl > 1e-8f;
                K.put(kPkPdf, pl);
            } else if (mis && nee_env<NEE>(O) && (miss || emissive)) {
                const float pb = in.last_pdf();
                w = (pb * pb) / (pb * pb + pl * pl);
            }
        }
        if (nee_dl<NEE>(O) && !nee_env<NEE>(O) && hit) {
            if (emissive) {
                if (mis) {
                    float pb = in.last_pdf();
                    float dsq = t * t;
                    float cl = dot(get3(K, kPkN0), -p.d);
                    if (cl > 0.0001f) {
                        float pa = 1.0f / S.total_area;
                        float ps = pa * (dsq / cl);
                        w = (pb * pb) / (pb * pb + ps * ps);
                    } else {
                        w = 0.0f;
                    }
                }
            } else if (sh_inst >= 0 && sh_t > 0.0f && !(K.get(kPkRough) < kSPEC_ROUGH)) {
                Isect dli = ch_direct_light(S, sh_t, sh_inst, sh_prim, sh_u, sh_v);
                f3 sp = t * p.d + in.origin();
                f3 lv = in.nee() - sp;
                float dsq = dot(lv, lv);
                float dist = sqrtf(dsq);
                wl = lv / dist;
                const f3 normal = get3(K, kPkNormal);
                const float cs = dot(dot(-p.d, normal) < 0.0f ? -normal : normal, wl);
                float cl = dot(dli.normal, -wl);
                if (cs > 0.0f && cl > 0.0f) {
                    float pa = 1.0f / S.total_area;
                    const DevMaterial& lm = S.mats[dli.material];
                    K.put(kPkCos, cs);
                    K.put(kPkPdf, pa * (dsq / cl));
                    put3(K, kPkLight, get_emission(lm, dli.u, dli.v));
                    lit = true;
                }
            }
        }
        // radiance a path without a BSDF step ends with (at most one term is added per call)
        if (miss ? has_exr : emissive) {
            const f3 thr = get3(K, kPkThr), le = get3(K, kPkLight);
            const f3 add = miss ? thr * le * w : (nee_env<NEE>(O) || nee_dl<NEE>(O)) ? thr * (w * le) : thr * le;
            in.set_color(in.color0() + add, __float_as_int(K.get(kPkIter)));
        }
    }
    phase<PHASED>();
    bool kill = emissive;
    const bool done = !hit || (emissive && !SPAWN_KILLED);  // no BSDF step
    // ---- BSDF: k = 0 for the light's direction, k = 1 for the sampled one
    f3 sd = mk(0.0f, 0.0f, 0.0f);
    {
        f3 normal = mk(0.0f, 0.0f, 1.0f), mc = normal;
        float rough = 1.0f, metal = 0.0f, ior = 1.5f, trans = 0.0f;
        Lobes L;
        L.pR = L.pD = L.pS = 0.0f;
        const f3 wo = -p.d;
        if (!done) {
            mc = get3(K, kPkAlbedo);
            normal = get3(K, kPkNormal);
            rough = K.get(kPkRough);
            metal = K.get(kPkMetal);
            ior = K.get(kPkIor);
            trans = K.get(kPkTrans);
            L = lobes_of(wo, normal, metal, mc, ior, trans);
        }
#pragma unroll 1
        for (int k = NEE == 0 ? 1 : 0; k < 2; ++k) {
            if (k == 1) {
                if (!done) sd = sample_ct(wo, normal, rough, rng, ior, L);
                phase<PHASED>();
            }
            if (!(done || (k == 0 ? !lit : kill))) {
                const f3 wi = k == 0 ? wl : sd;
                const bool refr = (dot(wi, normal) * dot(wo, normal)) < 0.0f;
                const float pdf = PDF(wo, wi, normal, rough, ior, L);
                const f3 f = (k == 1 && refr) ? BTDF(wo, normal, wi, mc, rough, metal, ior, trans)
                                              : BRDF(wo, normal, wi, mc, rough, metal, ior, trans);
                const f3 thr = get3(K, kPkThr);
                if (k == 0) {
                    const float pl = K.get(kPkPdf), cs = K.get(kPkCos);
                    const float wt = (pl * pl) / (pl * pl + pdf * pdf);
                    f3 contrib = (get3(K, kPkLight) * f * cs) / pl;
                    in.set_color(in.color0() + thr * contrib * wt, __float_as_int(K.get(kPkIter)));
                } else {
                    p.thr = thr * ((f * fabsf(dot(wi, normal))) / pdf);
                    p.last_pdf = pdf;
                    p.spec = rough < kSPEC_ROUGH || refr;
                    if (depth >= kRR_MIN_DEPTH) {
                        float mx = gmax(p.thr.x, gmax(p.thr.y, p.thr.z));
                        float surv = gclamp(mx, 0.0f, 1.0f);
                        if (rng.u01() >= surv) kill = true;
                        else p.thr = p.thr / surv;
                    }
                }
            }
            phase<PHASED>();
        }
    }
    if (done) return false;
    // ray spawn (shade_path.cu:333-353), run for paths killed above as well
    const f3 n0 = get3(K, kPkN0);
    f3 hp = in.origin() + (t - .0001f) * normalize(p.d);
    float sl2 = dot(sd, sd);
    if (!(sl2 > 1e-12f) || !isfinite(sl2)) return false;
    p.d = sd;
    if (dot(p.d, n0) > 0.0f) p.o = hp + (n0 * kGLASS_EPS);
    else p.o = hp - (n0 * kGLASS_EPS);
    return !kill;
}

}  // namespace
}  // namespace lux
