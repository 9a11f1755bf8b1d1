// Forward-mode derivatives of the material functions with respect to their
// parameters, for the path-replay adjoint.  A Dual<K> carries a value and its
// derivatives with respect to K parameters; the functions below restate the
// BRDF and Fresnel code of omv_device.cuh (same formulas and operation order
// for the value part) on duals.
#pragma once

#include "omv_device.cuh"

namespace omv {

template <int K>
struct Dual {
    float v;
    float d[K];
};

template <int K>
__device__ __forceinline__ Dual<K> dconst(float v)
{
    Dual<K> r;
    r.v = v;
#pragma unroll
    for (int i = 0; i < K; ++i) r.d[i] = 0.0f;
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> dvar(float v, int i)
{
    Dual<K> r = dconst<K>(v);
    r.d[i] = 1.0f;
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> operator+(Dual<K> a, Dual<K> b)
{
    Dual<K> r;
    r.v = a.v + b.v;
#pragma unroll
    for (int i = 0; i < K; ++i) r.d[i] = a.d[i] + b.d[i];
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> operator-(Dual<K> a, Dual<K> b)
{
    Dual<K> r;
    r.v = a.v - b.v;
#pragma unroll
    for (int i = 0; i < K; ++i) r.d[i] = a.d[i] - b.d[i];
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> operator-(Dual<K> a)
{
    Dual<K> r;
    r.v = -a.v;
#pragma unroll
    for (int i = 0; i < K; ++i) r.d[i] = -a.d[i];
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> operator*(Dual<K> a, Dual<K> b)
{
    Dual<K> r;
    r.v = a.v * b.v;
#pragma unroll
    for (int i = 0; i < K; ++i) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> operator*(Dual<K> a, float s)
{
    Dual<K> r;
    r.v = a.v * s;
#pragma unroll
    for (int i = 0; i < K; ++i) r.d[i] = a.d[i] * s;
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> operator*(float s, Dual<K> a)
{
    Dual<K> r;
    r.v = s * a.v;
#pragma unroll
    for (int i = 0; i < K; ++i) r.d[i] = s * a.d[i];
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> operator/(Dual<K> a, Dual<K> b)
{
    Dual<K> r;
    r.v = a.v / b.v;
    const float ib = 1.0f / b.v;
#pragma unroll
    for (int i = 0; i < K; ++i) r.d[i] = (a.d[i] - r.v * b.d[i]) * ib;
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> operator/(Dual<K> a, float s)
{
    Dual<K> r;
    r.v = a.v / s;
#pragma unroll
    for (int i = 0; i < K; ++i) r.d[i] = a.d[i] / s;
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> operator/(float s, Dual<K> b)
{
    return dconst<K>(s) / b;
}
template <int K>
__device__ __forceinline__ Dual<K> operator+(Dual<K> a, float s)
{
    a.v = a.v + s;
    return a;
}
template <int K>
__device__ __forceinline__ Dual<K> operator+(float s, Dual<K> a)
{
    a.v = s + a.v;
    return a;
}
template <int K>
__device__ __forceinline__ Dual<K> operator-(Dual<K> a, float s)
{
    a.v = a.v - s;
    return a;
}
template <int K>
__device__ __forceinline__ Dual<K> operator-(float s, Dual<K> a)
{
    return dconst<K>(s) - a;
}
template <int K>
__device__ __forceinline__ Dual<K> dsqrt(Dual<K> a)
{
    Dual<K> r;
    r.v = sqrtf(a.v);
    const float g = r.v > 0.0f ? 0.5f / r.v : 0.0f;
#pragma unroll
    for (int i = 0; i < K; ++i) r.d[i] = a.d[i] * g;
    return r;
}
template <int K>
__device__ __forceinline__ Dual<K> dabs(Dual<K> a)
{
    return a.v < 0.0f ? -a : a;
}
// clamp: the derivative is zero where the value is clamped
template <int K>
__device__ __forceinline__ Dual<K> dclamp(Dual<K> a, float lo, float hi)
{
    if (a.v < lo) return dconst<K>(lo);
    if (a.v > hi) return dconst<K>(hi);
    return a;
}
// lerp(lo, up, v) = (up - lo) * v + lo, as lerpf
template <int K>
__device__ __forceinline__ Dual<K> dlerp(Dual<K> lo, Dual<K> up, Dual<K> v)
{
    return (up - lo) * v + lo;
}

// ----------------------------------------------------------- GGX / Smith ---
template <int K>
__device__ __forceinline__ Dual<K> d_ggx_pdf(float c, Dual<K> alpha)
{
    const float c2 = c * c;
    const Dual<K> a2 = alpha * alpha;
    const Dual<K> l = dlerp(dconst<K>(1.0f), a2, dconst<K>(c2));
    return a2 / ((l * l) * kPi);
}
template <int K>
__device__ __forceinline__ Dual<K> d_smith_g1(float c, Dual<K> alpha)
{
    if (!(alpha.v > 0.0f || c < 0.99f)) return dconst<K>(1.0f);
    const float s = sqrtf(1.0f - c * c);
    if (!(s > 0.0f)) return dconst<K>(1.0f);  // c = 1: the float code's limit (a infinite, G1 = 1)
    const Dual<K> a = c / (alpha * s);
    const Dual<K> lam = (dsqrt(1.0f + 1.0f / (a * a)) - 1.0f) * 0.5f;
    return 1.0f / (1.0f + lam);
}
template <int K>
__device__ __forceinline__ Dual<K> d_smith_g2(Dual<K> s, Dual<K> m)
{
    const Dual<K> p = s * m;
    return p / (s + m - p);
}

// The two PBR functions on duals, one colour channel at a time: a channel
// depends on its own colour (slot 0), the GGX alpha (1) and the metallic factor
// (2).  What the channels share is computed once, and the caller's loop over
// them is not unrolled: the derivative code is long, and instruction fetch is
// what bounds the launches that run it (see bsdf_evaluate).
__device__ __forceinline__ Dual<1> d_smith_g(float VdotN, float LdotN, float alpha)
{
    Dual<1> g = dconst<1>(0.0f), s = g;
#pragma unroll 1
    for (int j = 0; j < 2; ++j) {
        s = g;
        g = d_smith_g1(j == 0 ? VdotN : LdotN, dvar<1>(alpha, 0));
    }
    return d_smith_g2(s, g);
}
__device__ __forceinline__ Dual<3> alpha_dual(Dual<1> x)
{
    Dual<3> r = dconst<3>(x.v);
    r.d[1] = x.d[0];
    return r;
}

// bsdf_evaluate on duals (directions fixed)
struct DualEvaluate {
    int kind;
    float VdotN, LdotN, P, k;
    Dual<1> G;
};
__device__ __forceinline__ DualEvaluate d_bsdf_evaluate(V3 vIn, V3 vOut, V3 norm, float alpha, int kind, V3 Hext, float p)
{
    DualEvaluate e;
    e.kind = kind;
    const V3 H = kind == 2 ? Hext : normalize(vOut - vIn);
    e.VdotN = clampf(fabsf(dot(vIn, norm)), 0.0001f, 1.0f);
    e.LdotN = clampf(fabsf(dot(vOut, norm)), 0.0001f, 1.0f);
    const float NdotH = fabsf(dot(norm, H));
    const float VdotH = fabsf(dot(vIn, H));
    const float LdotH = fabsf(dot(vOut, H));
    e.P = pow5(clamp01(1.0f - VdotH));
    if (kind == 0) {
        e.G = dconst<1>(0.0f);
        e.k = kPi / e.LdotN / p;
    } else {
        e.G = d_smith_g(e.VdotN, e.LdotN, alpha);
        e.k = 4.0f * LdotH * e.VdotN / NdotH / e.LdotN / (kind == 1 ? (1.0f - p) : p);
    }
    return e;
}
__device__ __forceinline__ Dual<3> d_evaluate_channel(const DualEvaluate& e, float color, float metal)
{
    const Dual<3> c = dvar<3>(color, 0), m = dvar<3>(metal, 2);
    const Dual<3> F0 = dlerp(dconst<3>(0.04f), c, m);
    const Dual<3> F = dlerp(dconst<3>(e.P), dconst<3>(1.0f), F0);
    if (e.kind == 0) {
        const Dual<3> cd = (1.0f - m) * c;
        return ((1.0f - F) * cd / kPi) * e.k;
    }
    const Dual<3> fs =
        dclamp((0.25f * (e.kind == 2 ? 1.0f - F : F) * alpha_dual(e.G)) / (e.VdotN * e.LdotN), 0.0f, kFltMax);
    return fs * e.k;
}

// bsdf_eval_direct on duals
struct DualDirect {
    bool lit;
    float VdotN, LdotN, P;
    Dual<1> D, G;
};
__device__ __forceinline__ DualDirect d_bsdf_eval_direct(V3 I, V3 O, V3 N, float alpha)
{
    DualDirect e;
    e.VdotN = -dot(I, N);
    e.LdotN = dot(O, N);
    e.lit = e.VdotN > 0.0f && e.LdotN > 0.0f;
    e.P = 0.0f;
    e.D = e.G = dconst<1>(0.0f);
    if (!e.lit) return e;
    const V3 H = normalize(O - I);
    const float VdotH = fabsf(dot(I, H));
    const float NdotH = fabsf(dot(N, H));
    e.P = pow5(clamp01(1.0f - VdotH));
    e.D = d_ggx_pdf(clamp01(NdotH), dvar<1>(alpha, 0));
    e.G = d_smith_g(e.VdotN, e.LdotN, alpha);
    return e;
}
__device__ __forceinline__ Dual<3> d_direct_channel(const DualDirect& e, float color, float metal)
{
    if (!e.lit) return dconst<3>(0.0f);
    const Dual<3> c = dvar<3>(color, 0), m = dvar<3>(metal, 2);
    const Dual<3> F0 = dlerp(dconst<3>(0.04f), c, m);
    const Dual<3> F = dlerp(dconst<3>(e.P), dconst<3>(1.0f), F0);
    const Dual<3> cd = (1.0f - m) * c;
    const Dual<3> fd = (1.0f - F) * cd / kPi;
    const Dual<3> fs =
        dclamp((0.25f * F * alpha_dual(e.D) * alpha_dual(e.G)) / (e.VdotN * e.LdotN), 0.0f, kFltMax);
    return fd + fs;
}

// d/dalpha of log D_alpha(c) for the GGX half-vector density the sampler draws
// from (RandomSampler::GGXHemisphere): the score of a GGX-sampled direction
__device__ __forceinline__ float ggx_log_pdf_dalpha(float c, float alpha)
{
    const float c2 = c * c, a2 = alpha * alpha;
    const float l = (a2 - 1.0f) * c2 + 1.0f;
    return 2.0f / alpha - 4.0f * alpha * c2 / l;
}

// --------------------------------------------------- OpenMATERIAL Fresnel ---
struct DC {
    Dual<2> re, im;
};
__device__ __forceinline__ DC dcmul(DC a, DC b) { return DC{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ Dual<2> dselect(bool c, Dual<2> a, Dual<2> b)
{
    return Dual<2>{c ? a.v : b.v, {c ? a.d[0] : b.d[0], c ? a.d[1] : b.d[1]}};
}
__device__ __forceinline__ DC dcdiv(DC a, DC b)  // as cdiv
{
    const bool big = fabsf(b.re.v) >= fabsf(b.im.v);
    const Dual<2> x = dselect(big, b.re, b.im), y = dselect(big, b.im, b.re);
    const Dual<2> p = dselect(big, a.re, a.im), q = dselect(big, a.im, a.re);
    const Dual<2> r = y / x, den = x + y * r, pr = p * r;
    return DC{(p + q * r) / den, (dselect(big, q, pr) - dselect(big, pr, q)) / den};
}
__device__ __forceinline__ DC dcsqrt(DC z)
{
    const Dual<2> m = dsqrt(z.re * z.re + z.im * z.im);
    if (m.v == 0.0f) return DC{dconst<2>(0.0f), z.im};
    const Dual<2> t = dsqrt((m + dabs(z.re)) * 0.5f);
    if (z.re.v >= 0.0f) return DC{t, (z.im * 0.5f) / t};
    return DC{(dabs(z.im) * 0.5f) / t, z.im.v < 0.0f ? -t : t};
}
// om_channel with n (slot 0) and k (slot 1) as duals
__device__ __forceinline__ Dual<2> d_om_channel(float n, float k, float cosTheta)
{
    const DC N{dvar<2>(n, 0), dvar<2>(k, 1)};
    const DC N2 = dcmul(N, N);
    const float c = fabsf(cosTheta);
    const float s2 = 1.0f - c * c;
    const DC root = dcsqrt(DC{N2.re - s2, N2.im});
    const DC N2c{N2.re * c, N2.im * c};
    const DC rp = dcdiv(DC{N2c.re - root.re, N2c.im - root.im}, DC{N2c.re + root.re, N2c.im + root.im});
    const DC rs = dcdiv(DC{c - root.re, -root.im}, DC{c + root.re, root.im});
    const Dual<2> P = rp.re * rp.re + rp.im * rp.im;
    const Dual<2> S = rs.re * rs.re + rs.im * rs.im;
    return dlerp(P, S, dconst<2>(0.5f)) / fabsf(cosTheta);
}

}  // namespace omv
