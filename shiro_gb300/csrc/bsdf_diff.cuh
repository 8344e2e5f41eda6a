// bsdf_diff.cuh - material gradients of EvaluateBsdf.
//
// bsdf_grad differentiates EvaluateBsdf (src/backend/cpu/CpuPathTracer.cpp:
// 1275-1354) with respect to the differentiable material parameters - base
// colour (r, g, b), specular roughness and metalness - and contracts the
// derivative with the caller's coefficient per colour channel.  Clamps and
// max / min propagate the derivative of the branch they select (zero when a
// bound is selected); the coat lobe, the tints and the cosines depend on none
// of the parameters.
//
// A channel of the BSDF depends on its own channel of the base colour only,
// the GGX terms on the roughness only, Fresnel terms and diffuse colour on
// base colour and metalness only, so three derivatives per quantity at most
// are carried (dual numbers with all five spent most of their operations on
// zeros).
#pragma once

#include "bsdf.cuh"

namespace shiro_gpu {

// d(coef . f) / d parameters.
struct MatGrad {
    float base[3], rough, metal;
};

// A quantity of one channel: value and derivatives by base colour channel
// and metalness.
struct DualBM {
    float v, b, m;
};
// A quantity of the roughness alone.
struct DualR {
    float v, r;
};

__device__ __forceinline__ DualBM operator+(const DualBM& a, const DualBM& b) { return {a.v + b.v, a.b + b.b, a.m + b.m}; }
__device__ __forceinline__ DualBM operator*(const DualBM& a, float s) { return {a.v * s, a.b * s, a.m * s}; }
__device__ __forceinline__ DualBM operator*(const DualBM& a, const DualBM& b) {
    return {a.v * b.v, a.b * b.v + a.v * b.b, a.m * b.v + a.v * b.m};
}

__device__ __forceinline__ float schlick_weight(float x) {  // (1 - x)^5 of a clamped cosine
    const float c = sclamp(1.0f - x, 0.0f, 1.0f);
    return c * c * c * c * c;
}
// f0 + (1 - f0) f
__device__ __forceinline__ DualBM schlick_d(const DualBM& f0, float f) {
    return {f0.v + (1.0f - f0.v) * f, f0.b - f0.b * f, f0.m - f0.m * f};
}
__device__ __forceinline__ DualR ggx_lambda_d(float x, const DualR& a2) {
    const float c = smax(x, 1.0e-6f);
    const float cc = c * c;
    const float root = sqrtf(1.0f + a2.v * (1.0f - cc) / cc);
    const float k = root > 0.0f ? 0.5f / root : 0.0f;
    return {(-1.0f + root) * 0.5f, k * (a2.r * (1.0f - cc) / cc) * 0.5f};
}
// Distribution x visibility / (4 nv nl) and its roughness derivative.
__device__ __forceinline__ DualR ggx_scale_d(float nh, float nv, float nl, const DualR& r) {
    const float rr = r.v * r.v;
    const DualR a{smax(0.02f, rr), 0.02f < rr ? r.r * r.v + r.v * r.r : 0.0f};
    const DualR a2{a.v * a.v, a.r * a.v + a.v * a.r};
    const DualR t{nh * nh * (a2.v - 1.0f) + 1.0f, nh * nh * a2.r};
    const float tt = t.v * t.v;
    const DualR x{kPi * smax(1.0e-6f, tt), 1.0e-6f < tt ? kPi * (t.r * t.v + t.v * t.r) : 0.0f};
    const DualR d{a2.v / x.v, (a2.r * x.v - a2.v * x.r) * (1.0f / (x.v * x.v))};
    const DualR lv = ggx_lambda_d(nv, a2), ll = ggx_lambda_d(nl, a2);
    const float den = 1.0f + lv.v + ll.v;
    const DualR g{1.0f / den, -1.0f / (den * den) * (lv.r + ll.r)};
    const float norm = smax(4.0f * nv * nl, 1.0e-6f);
    return {d.v * g.v / norm, (d.r * g.v + d.v * g.r) / norm};
}

// Gradient of coef . EvaluateBsdf(n, cn, v, l).
static __device__ __noinline__ MatGrad bsdf_grad(const Mat& m, const V3 n, const V3 cn, const V3 v, const V3 l,
                                                 const V3 coef) {
    MatGrad out{{0.0f, 0.0f, 0.0f}, 0.0f, 0.0f};
    const float nv = sclamp(dot(n, v), 0.0f, 1.0f);
    const float nl = sclamp(dot(n, l), 0.0f, 1.0f);
    if (nv <= 0.0f || nl <= 0.0f) return out;
    const float metal = sclamp(m.metallic, 0.0f, 1.0f);
    const float dMetal = (m.metallic < 0.0f || 1.0f < m.metallic) ? 0.0f : 1.0f;
    const V3 underCoat = coat_tint(m) * layer_transmittance(coat_f0(m), dot(cn, v), dot(cn, l));
    // diffuse lobe: Oren-Nayar term and the colour's scale (base weight, metalness, transmission)
    const float sigma = sclamp(m.diffuse_roughness, 0.0f, 1.0f);
    const float radius = sclamp(maxc(ld3(m.subsurface_radius)) / 3.0f, 0.0f, 1.0f);
    const float wrap = sclamp(m.subsurface * m.subsurface_scale *
                                  (0.35f + 0.15f * sclamp(m.subsurface_anisotropy, -1.0f, 1.0f) + 0.1f * radius),
                              0.0f, 0.9f);
    const float wrapped = sclamp((nl + wrap) / (1.0f + wrap), 0.0f, 1.0f);
    float term = wrapped / smax(nl, 1.0e-6f);
    if (sigma != 0.0f) term = oren_nayar(sigma, n, v, l, nv, nl) * term;
    const float trans = sclamp(m.transmission, 0.0f, 1.0f);
    const float sss = sclamp(m.subsurface, 0.0f, 1.0f);
    const float weight = sclamp(m.base_weight, 0.0f, 1.0f);
    const float colorScale = weight * (1.0f - metal) * (1.0f - trans);
    const float dColorScale = weight * -dMetal * (1.0f - trans);
    // base specular lobe
    const V3 h = safe_normalized(v + l, n);
    const float nh = sclamp(dot(n, h), 0.0f, 1.0f);
    const float vh = sclamp(dot(v, h), 0.0f, 1.0f);
    const float rough = m.roughness + m.coat_affect_roughness * m.coat_weight * m.coat_roughness;
    DualR r{sclamp(rough, 0.0f, 1.0f), (rough < 0.0f || 1.0f < rough) ? 0.0f : 1.0f};
    {
        const float ca = sclamp(m.specular_anisotropy, -0.95f, 0.95f);
        const float k = 1.0f - 0.35f * ca * (ca != 0.0f ? aniso_phase(m.specular_rotation, m, n, v, l) : 0.0f);
        const float x = r.v * k;
        r = DualR{sclamp(x, 0.02f, 1.0f), (x < 0.02f || 1.0f < x) ? 0.0f : r.r * k};
    }
    const DualR scale = ggx_scale_d(nh, nv, nl, r);
    V3 film{1.0f, 1.0f, 1.0f};
    if (m.thin_film_thickness > 0.0f) film = film_color(m.thin_film_thickness, m.thin_film_ior, vh);
    // sheen scales the layer transmittance
    const float sw = sclamp(m.sheen, 0.0f, 1.0f);
    V3 sheen{0.0f, 0.0f, 0.0f};
    if (sw != 0.0f)
        sheen = ld3(m.sheen_color) * sw * (sheen_factor(l, h) * (1.0f - 0.5f * sclamp(m.sheen_roughness, 0.0f, 1.0f))) *
                underCoat;
    const float fv = schlick_weight(nv), fl = schlick_weight(nl), fh = schlick_weight(vh);
    const float specWeight = sclamp(m.specular_weight, 0.0f, 1.0f) * f0_dielectric(m.ior);
    const float uc[3] = {underCoat.x, underCoat.y, underCoat.z}, fc[3] = {film.x, film.y, film.z},
                sh[3] = {sheen.x, sheen.y, sheen.z}, cf[3] = {coef.x, coef.y, coef.z};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float b = m.base_color[c], d = m.specular_color[c] * specWeight;
        const DualBM f0{d * (1.0f - metal) + b * metal, metal, d * -dMetal + b * dMetal};
        // 1 - (schlick(nv) + schlick(nl)) / 2, clamped
        const DualBM s = (schlick_d(f0, fv) + schlick_d(f0, fl)) * 0.5f;
        const float u = 1.0f - s.v;
        const bool in = !(u < 0.0f || 1.0f < u);
        const DualBM under{sclamp(u, 0.0f, 1.0f), in ? -s.b : 0.0f, in ? -s.m : 0.0f};
        // DiffuseColor: lerp(base, lerp(base, subsurface colour, radius), sss) x scale
        const float tint = b * (1.0f - radius) + m.subsurface_color[c] * radius;
        const float color = b * (1.0f - sss) + tint * sss;
        const float dColor = (1.0f - sss) + (1.0f - radius) * sss;
        const DualBM dc{color * colorScale, dColor * colorScale, color * dColorScale};
        const DualBM diffuse = dc * uc[c] * under * (kInvPi * term);
        const DualBM fres = schlick_d(f0, fh) * (fc[c] * uc[c]);
        out.base[c] = cf[c] * (diffuse.b + fres.b * scale.v + sh[c] * under.b);
        out.metal += cf[c] * (diffuse.m + fres.m * scale.v + sh[c] * under.m);
        out.rough += cf[c] * (fres.v * scale.r);
    }
    return out;
}

}  // namespace shiro_gpu
