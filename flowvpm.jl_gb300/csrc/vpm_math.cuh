// vpm_math.cuh -- device-side regularizing-kernel math for the UJ and Estr
// kernels.
//
// Two forms are provided:
//
//  * FP64: the functions of src/FLOWVPM_kernel.jl:45-84 to FP64 rounding, used by the plain
//    FP64 kernels.  Gaussian-erf is evaluated without the reference's cancellation at small rho,
//    and for rho > 9, where erf(rho/sqrt2)-1 and sqrt(2/pi)*rho*exp(-rho^2/2) are below 2^-56,
//    as g = 1, dg = 0.
//
//  * FP32, a regular reformulation used by the mixed kernels.  With
//    s = rho^2 = r^2/sigma^2 the pair terms of src/FLOWVPM_fmm.jl:130-160 are
//        g/r^3                          = G(s) / sigma^3
//        dg/(sigma r^4) - 3 g / r^5     = H(s) / sigma^5
//    with G(s) = g(rho)/rho^3 and H(s) = (rho g'(rho) - 3 g(rho)) / rho^5.
//    G and H are smooth at s = 0, so the cancellation of erf(rho/sqrt2) against
//    sqrt(2/pi)*rho*exp(-rho^2/2) that the literal formula suffers for small
//    rho in FP32 never happens.  For the Gaussian-erf kernel G and H come from
//    their series of positive terms for s < 2 (< 1e-8 relative), from
//    e^{-s/2} and a fit of erfcx for 2 <= s <= 50 (no erf call), and from the
//    singular form G = s^-1.5, H = -3 s^-2.5 for s > 50 (rho > 7.07), where the
//    neglected terms are below 2e-9 relative (gerf_GQ below).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace vpm {

// src/FLOWVPM.jl:62-66
constexpr double C1 = 0.063493635934240969;   // 1/(2*pi)^1.5
constexpr double C2 = 0.79788456080286541;    // sqrt(2/pi)
constexpr double C3 = 0.23873241463784300;    // 3/(4*pi)
constexpr double C4 = 0.079577471545947673;   // 1/(4*pi)

enum : int { K_SING = 0, K_GAUS = 1, K_GAUSERF = 2, K_WNKLMNS = 3 };

// Normalisation of zeta per kernel: zeta(rho) = ZNORM * zhat(s).
__host__ __device__ constexpr double zeta_norm(int K)
{
    return K == K_GAUS ? C3 : K == K_GAUSERF ? C1 : K == K_WNKLMNS ? C4 * 7.5 : 1.0;
}

// ------------------------------------------------------------------ FP64
// The FP64 pipe runs at 1/64 of the FP32 rate and bounds every FP64 kernel, so the forms below
// count its instructions: an exponential from a table (11 of them), Gaussian-erf from that one
// exponential and a polynomial (no erf call, no square root), Winckelmans from one rsqrt (no
// division).

// e^x for x <= 0 by Tang's table method (P. T. P. Tang, "Table-driven implementation of the
// exponential function in IEEE floating-point arithmetic", ACM TOMS 15, 1989): x = (k/64) ln 2 + r,
// e^x = 2^(k div 64) T[k mod 64] (1 + p(r)), |r| <= ln 2/128, p the Taylor polynomial of degree 5
// (3.5e-17 relative).  T: 2^(j/64), j < 64, in shared memory (exp_table).  Results below
// 2^-1021 and non-finite x take the library's exp.
__device__ __forceinline__ void exp_table(double* T)
{
    for (int j = threadIdx.x; j < 64; j += blockDim.x) T[j] = exp2(j * (1.0 / 64.0));
}
__device__ __forceinline__ double exp_neg(double x, const double* T)
{
    if ((unsigned)__double2hiint(x) >= 0xC0862000u) return exp(x);     // x <= -708, -inf
    constexpr double magic = 6755399441055744.0;                       // 1.5 2^52
    double kd = fma(x, 92.33248261689366, magic);                      // 64/ln 2
    const int k = __double2loint(kd);
    kd -= magic;
    double r = fma(kd, -0.010830424695086549, x);                      // ln 2/64: 33 bits, and the rest
    r = fma(kd, -1.162596423439437e-12, r);
    double p = fma(r, 1.0 / 120.0, 1.0 / 24.0);
    p = fma(p, r, 1.0 / 6.0);
    p = fma(p, r, 0.5);
    p = fma(p * r, r, r);
    const double t = T[k & 63];
    const double ts = __hiloint2double(__double2hiint(t) + ((k >> 6) << 20), __double2loint(t));
    return fma(ts, p, ts);
}

// Gaussian-erf below s = 2: g = c2 e rho^3 K(s) and -H/3 = c2 e S2(s) with K = 1/3 + s S2 the
// Kummer series sum s^m/(2m+3)!! (positive terms: none of the cancellation of erf against
// sqrt(2/pi) rho e); S2 by its degree-11 Chebyshev fit on [0, 2] (2e-17).
__device__ __forceinline__ double gerf_S2_f64(double s)
{
    double p = 7.117914962008134e-15;
    p = fma(p, s, 1.12787989755004e-13);
    p = fma(p, s, 3.2049748194948006e-12);
    p = fma(p, s, 7.26474696490197e-11);
    p = fma(p, s, 1.5274561118204643e-09);
    p = fma(p, s, 2.9019546056094325e-08);
    p = fma(p, s, 4.933338773525617e-07);
    p = fma(p, s, 7.400007382107342e-06);
    p = fma(p, s, 9.620009620382055e-05);
    p = fma(p, s, 0.0010582010582006584);
    p = fma(p, s, 0.00952380952380954);
    p = fma(p, s, 0.06666666666666667);
    return p;
}
// ... and from s = 2 to rho = 9: g = 1 - e h, h = erfcx(rho/sqrt2) + c2 rho, with
// erfcx(rho/sqrt2) = t P(w), t = 1/(1 + rho/2), w = A t + B, P a degree-16 Chebyshev fit (3e-17).
__device__ __forceinline__ double gerf_h_f64(double rho)
{
    const double d = fma(0.5, rho, 1.0);
    double t;                                   // 1/d: the approximate reciprocal and two Newton steps
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(t) : "d"(d));
    double e = fma(-d, t, 1.0);
    t = fma(t, e, t);
    e = fma(-d, t, 1.0);
    t = fma(t, e, t);
    const double w = fma(t, 4.950884063887905, -1.9001607388887100);
    double p = -1.5660591337542868e-11;
    p = fma(p, w, 5.63460752287977e-11);
    p = fma(p, w, 5.1974104520460814e-11);
    p = fma(p, w, -9.507498606778384e-10);
    p = fma(p, w, 2.8308353212461513e-09);
    p = fma(p, w, 3.3164182614796496e-09);
    p = fma(p, w, -5.620367325865092e-08);
    p = fma(p, w, 1.4651970275804292e-07);
    p = fma(p, w, 4.7370926853939187e-07);
    p = fma(p, w, -4.228927081890189e-06);
    p = fma(p, w, 2.9494713884413277e-06);
    p = fma(p, w, 8.528834233914718e-05);
    p = fma(p, w, -0.0002486943660856597);
    p = fma(p, w, -0.002127601067365253);
    p = fma(p, w, 0.008702997368809272);
    p = fma(p, w, 0.12611846511040975);
    p = fma(p, w, 0.5974010771326975);
    return fma(C2, rho, p * t);
}

// zeta(rho)/ZNORM as a function of s = rho^2 (src/FLOWVPM_kernel.jl)
template <int K>
__device__ __forceinline__ double zhat_f64(double s, const double* T)
{
    if constexpr (K == K_SING) return s == 0.0 ? 1.0 : 0.0;
    else if constexpr (K == K_GAUS) return exp_neg(-s * sqrt(s), T);
    else if constexpr (K == K_GAUSERF) return exp_neg(-0.5 * s, T);
    else {
        const double t = rsqrt(s + 1.0), t2 = t * t, t4 = t2 * t2;
        return t4 * t2 * t;
    }
}

// ------------------------------------------------------------------ FP32
constexpr float F_C2 = 0.7978845608028654f;
constexpr float F_C4 = 0.07957747154594767f;   // 1/(4 pi)
constexpr float S_SERIES = 2.0f;      // positive series below this s (Gaussian-erf, gerf_GQ)
constexpr float S_FAR_GERF = 50.0f;   // singular form above this s (rho > 7.07)
constexpr float S_FAR_GAUS = 8.0f;    // singular form above this s (rho^3 > 22.6)

#ifndef VPM_FTZ_UNARY
#define VPM_FTZ_UNARY 1
#endif
// 1/sqrt(x), 2^x and 1/x of the FP32 pair forms: the hardware approximations with
// subnormal arguments and results flushed to zero (PTX rsqrt.approx.ftz.f32,
// ex2.approx.ftz.f32, rcp.approx.ftz.f32).  The arguments on the pair paths are
// normal numbers (s, r^2 and 1 + s are at least 1e-30, or the pair is masked out),
// and a 2^x flushed below 2^-126 is far under the FP32 resolution of the sums; the
// forms that keep subnormals guard every call.  0 selects rsqrtf, exp2f, __frcp_rn.
__device__ __forceinline__ float frsqrt(float x)
{
#if VPM_FTZ_UNARY
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return rsqrtf(x);
#endif
}
__device__ __forceinline__ float fexp2(float x)
{
#if VPM_FTZ_UNARY
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return exp2f(x);
#endif
}
__device__ __forceinline__ float frcp(float x)
{
#if VPM_FTZ_UNARY
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return __frcp_rn(x);
#endif
}

// Gaussian kernel, t = rho^3: G = (1 - e^-t)/t = sum (-t)^k/(k+1)!,
// H = 3 rho sum_{k>=2} (-1)^(k+1) (k-1)/k! t^(k-2).
__device__ __forceinline__ float gaus_G_series(float t)
{
    float p = -2.08767569878681e-09f;
    p = fmaf(p, t, 2.505210838544172e-08f);
    p = fmaf(p, t, -2.755731922398589e-07f);
    p = fmaf(p, t, 2.7557319223985893e-06f);
    p = fmaf(p, t, -2.48015873015873e-05f);
    p = fmaf(p, t, 0.0001984126984126984f);
    p = fmaf(p, t, -0.001388888888888889f);
    p = fmaf(p, t, 0.008333333333333333f);
    p = fmaf(p, t, -0.041666666666666664f);
    p = fmaf(p, t, 0.16666666666666666f);
    p = fmaf(p, t, -0.5f);
    p = fmaf(p, t, 1.0f);
    return p;
}
__device__ __forceinline__ float gaus_H_series(float t)
{
    float p = 1.9270852604185937e-09f;
    p = fmaf(p, t, -2.296443268665491e-08f);
    p = fmaf(p, t, 2.505210838544172e-07f);
    p = fmaf(p, t, -2.48015873015873e-06f);
    p = fmaf(p, t, 2.2045855379188714e-05f);
    p = fmaf(p, t, -0.00017361111111111112f);
    p = fmaf(p, t, 0.0011904761904761906f);
    p = fmaf(p, t, -0.006944444444444444f);
    p = fmaf(p, t, 0.03333333333333333f);
    p = fmaf(p, t, -0.125f);
    p = fmaf(p, t, 0.3333333333333333f);
    p = fmaf(p, t, -0.5f);
    return p;
}

// The mixed kernels accumulate, per pair,
//     U += G c,   W += G gam,   J' += Q c_i dx_j,
// with c = dx x gam, gam = -Gamma/(4 pi sigma^3), and Q = -H/(3 sigma^2), so
// that J = -3 J' + (Kronecker term from W) once per target.  In the singular
// (far) form Q = G / r^2.

// s above which the kernel equals its singular form to FP32 resolution; 0 for
// the singular kernel (every pair with r > 0), +inf for Winckelmans (never).
template <int K>
__host__ __device__ constexpr float s_far()
{
    return K == K_SING ? 0.0f : K == K_GAUSERF ? S_FAR_GERF : K == K_GAUS ? S_FAR_GAUS : 3.0e38f;
}

// Singular form: G = s^-1.5, Q = G / r^2 = G s^-1 / sigma^2.
__device__ __forceinline__ void far_GQ(float s, float isig2, float& G, float& Q)
{
    const float rs = frsqrt(s);
    const float rs2 = rs * rs;
    G = rs * rs2;
    Q = G * (rs2 * isig2);
}

// ---------------------------------------------------------- packed FP32 pairs
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { return fma2(b, pk(-1.f, -1.f), a); }
// G = g/rho^3 of Gaussian-erf for s >= 2 from the erfcx fit, given e = e^{-s/2}, rs = s^-1/2
__device__ __forceinline__ float gerf_G_erfcx(float s, float e, float rs)
{
    const float rho = s * rs;
    const float t = __fdividef(1.0f, fmaf(0.5f, fminf(rho, 10.0f), 1.0f));
    const float w = fmaf(4.77190564267067f, t, -1.795317607111778f);
    float p = -5.1560079373370265e-06f;
    p = fmaf(p, w, 5.998428003101994e-06f);
    p = fmaf(p, w, 0.00010125038777505872f);
    p = fmaf(p, w, -0.00030713426402493693f);
    p = fmaf(p, w, -0.0023330098304451836f);
    p = fmaf(p, w, 0.009623567049071946f);
    p = fmaf(p, w, 0.13016216050000662f);
    p = fmaf(p, w, 0.5926831417002281f);
    const float h = fmaf(F_C2, rho, p * t);
    return fmaf(-e, h, 1.0f) * rs * (rs * rs);
}

// Gaussian-erf G and Q = -H/(3 sigma^2) of one lane at any s >= 0, with
// e = e^{-s/2} (coefficients from fit_gerf.py):
//   s < 2:  G = c2 e (1/3 + s S2(s)), -H/3 = c2 e S2(s), S2(s) = sum_m s^m/(2m+5)!!
//           (Kummer's series of erf: positive terms, no cancellation);
//   s >= 2: g = 1 - e (erfcx(rho/sqrt2) + c2 rho) with erfcx(rho/sqrt2) = P(w) t,
//           t = 1/(1 + rho/2), w = A t + B, P of degree 7 (rho capped at 10, beyond
//           which e < 2e-22 and G is its singular form s^-1.5); G = g/rho^3,
//           -H/3 = (G - c2 e/3)/s.
// No erf call.  FAR adds a third branch, the singular form beyond s = 50, for
// callers whose near groups hold many lanes past the kernel's reach (the
// all-pairs kernels); without it those lanes take the s >= 2 form, which is
// valid there.
template <bool FAR>
__device__ __forceinline__ void gerf_GQ(float s, float isig2, float& G, float& Q)
{
    if (FAR && s > S_FAR_GERF) {
        far_GQ(s, isig2, G, Q);
        return;
    }
    const float e = fexp2(s * -0.72134752044448170f);
    if (s < S_SERIES) {
        float p = 3.1622138893727926e-12f;
        p = fmaf(p, s, 7.273091945557423e-11f);
        p = fmaf(p, s, 1.5273493085670588e-09f);
        p = fmaf(p, s, 2.901963686277412e-08f);
        p = fmaf(p, s, 4.9333382666716e-07f);
        p = fmaf(p, s, 7.4000074000074e-06f);
        p = fmaf(p, s, 9.62000962000962e-05f);
        p = fmaf(p, s, 0.0010582010582010583f);
        p = fmaf(p, s, 0.009523809523809525f);
        p = fmaf(p, s, 0.06666666666666667f);
        const float ce = F_C2 * e;
        G = ce * fmaf(s, p, 0.33333333333333333f);
        Q = ce * p * isig2;
    } else {
        const float rs = frsqrt(s);
        const float rs2 = rs * rs;
        G = gerf_G_erfcx(s, e, rs);
        Q = fmaf(F_C2 * -0.33333333333333333f, e, G) * rs2 * isig2;
    }
}

// Full form of kernel K for one lane (any s > 0); FAR as in gerf_GQ.
template <int K, bool FAR = true>
__device__ __forceinline__ void near_GQ(float s, float isig2, float& G, float& Q)
{
    if constexpr (K == K_WNKLMNS) {
        // g/rho^3 = (s+2.5)(s+1)^-2.5 ; -H/3 = (s+3.5)(s+1)^-3.5
        const float q = s + 1.0f;
        const float t = frcp(q);
        const float t2u = t * t * frsqrt(q);
        G = (s + 2.5f) * t2u;
        Q = (s + 3.5f) * t * t2u * isig2;
    } else if constexpr (K == K_SING) {
        // J of a singular cloud is a handful of its nearest pairs, and Q = r^-5 carries five
        // times the error of rsqrt.approx: one Newton step (not where r^2 overflows: infinity times zero)
        float rs = frsqrt(s);
        if (s < INFINITY) rs = fmaf(0.5f * rs, fmaf(-s * rs, rs, 1.0f), rs);
        const float rs2 = rs * rs;
        G = rs * rs2;
        Q = G * (rs2 * isig2);
    } else if constexpr (K == K_GAUSERF) {
        gerf_GQ<FAR>(s, isig2, G, Q);
    } else {  // Gaussian
        if (s > S_FAR_GAUS) {
            far_GQ(s, isig2, G, Q);
        } else {
            const float rs = frsqrt(s);
            const float rho = s * rs;
            const float t = s * rho;
            if (t < 1.0f) {
                G = gaus_G_series(t);
                Q = -rho * gaus_H_series(t) * isig2;
            } else {
                const float e = expf(-t);
                G = (1.0f - e) * frcp(t);
                const float rs2 = rs * rs;
                Q = fmaf(-t, e, 1.0f - e) * rs2 * rs2 * rs * isig2;   // -H/3 = (1 - e - t e)/rho^5
            }
        }
    }
}

// near_GQ of N pairs of f32x2, without the singular branches.  Gaussian-erf: the s >= 2 form (valid at
// any s > 0), replaced by the series where s < 2 when `series` says that one may be.
template <int K, int N>
__device__ __forceinline__ void near_GQ2(const f32x2 (&s)[N], const f32x2 (&isig2)[N], bool series, f32x2 (&G)[N],
                                         f32x2 (&Q)[N])
{
    auto both = [](float v) { return pk(v, v); };
    if constexpr (K == K_GAUSERF) {
        constexpr float P[8] = {5.1560079373370265e-06f, -5.998428003101994e-06f, -0.00010125038777505872f,
                                0.00030713426402493693f, 0.0023330098304451836f, -0.009623567049071946f,
                                -0.13016216050000662f, -0.5926831417002281f};   // minus gerf_G_erfcx's
        constexpr float S2[10] = {3.1622138893727926e-12f, 7.273091945557423e-11f, 1.5273493085670588e-09f,
                                  2.901963686277412e-08f, 4.9333382666716e-07f, 7.4000074000074e-06f,
                                  9.62000962000962e-05f, 0.0010582010582010583f, 0.009523809523809525f,
                                  0.06666666666666667f};
        f32x2 e[N];
#pragma unroll
        for (int q = 0; q < N; q++) {
            float v0, v1;
            upk(s[q], v0, v1);
            const f32x2 rs = pk(frsqrt(v0), frsqrt(v1));
            upk(mul2(s[q], both(-0.72134752044448170f)), v0, v1);
            e[q] = pk(fexp2(v0), fexp2(v1));
            const f32x2 rho = mul2(s[q], rs);
            upk(fma2(rho, both(0.5f), both(1.f)), v0, v1);
            const f32x2 t = pk(frcp(v0), frcp(v1));
            const f32x2 w = fma2(t, both(4.77190564267067f), both(-1.795317607111778f));
            f32x2 p = both(P[0]);
#pragma unroll
            for (int k = 1; k < 8; k++) p = fma2(p, w, both(P[k]));
            const f32x2 nh = fma2(rho, both(-F_C2), mul2(p, t));
            const f32x2 g = fma2(e[q], nh, both(1.f)), rs2 = mul2(rs, rs);
            G[q] = mul2(mul2(g, rs), rs2);
            Q[q] = mul2(mul2(fma2(e[q], both(F_C2 * -0.33333333333333333f), G[q]), rs2), isig2[q]);
        }
        if (series) {
#pragma unroll
            for (int q = 0; q < N; q++) {
                f32x2 p = both(S2[0]);
#pragma unroll
                for (int k = 1; k < 10; k++) p = fma2(p, s[q], both(S2[k]));
                const f32x2 ce = mul2(e[q], both(F_C2));
                float s0, s1, a0, a1, b0, b1, g0, g1, q0, q1;
                upk(s[q], s0, s1);
                upk(mul2(ce, fma2(s[q], p, both(0.33333333333333333f))), a0, a1);
                upk(mul2(mul2(ce, p), isig2[q]), b0, b1);
                upk(G[q], g0, g1);
                upk(Q[q], q0, q1);
                const bool l0 = s0 < S_SERIES, l1 = s1 < S_SERIES;
                G[q] = pk(l0 ? a0 : g0, l1 ? a1 : g1);
                Q[q] = pk(l0 ? b0 : q0, l1 ? b1 : q1);
            }
        }
    } else {
#pragma unroll
        for (int q = 0; q < N; q++) {
            float s0, s1;
            upk(s[q], s0, s1);
            if constexpr (K == K_WNKLMNS) {
                float q0, q1;
                upk(add2(s[q], both(1.f)), q0, q1);
                const f32x2 t = pk(frcp(q0), frcp(q1));
                const f32x2 t2u = mul2(mul2(t, t), pk(frsqrt(q0), frsqrt(q1)));
                G[q] = mul2(add2(s[q], both(2.5f)), t2u);
                Q[q] = mul2(mul2(mul2(add2(s[q], both(3.5f)), t), t2u), isig2[q]);
            } else {
                float i0, i1, g0, g1, q0, q1;
                upk(isig2[q], i0, i1);
                near_GQ<K, false>(s0, i0, g0, q0);
                near_GQ<K, false>(s1, i1, g1, q1);
                G[q] = pk(g0, g1);
                Q[q] = pk(q0, q1);
            }
        }
    }
}

// (a + b) - (oh + ol) for two double-floats (hi a / oh, lo b / ol) in FP32: the
// difference of the high parts is made exact by TwoSum (s + e), the rest added
// after, so the result is rounded once, nearly correctly.  The same operations
// on the same inputs give the same bits: a point's offset from an origin
// equals itself wherever it is formed (the self pair has r^2 == 0 exactly).
__device__ __forceinline__ float df_offset(float a, float b, float oh, float ol)
{
    const float s = a - oh;
    const float v = s - a;
    const float e = (a - (s - v)) - (oh + v);
    return s + (e + (b - ol));
}

// ... and `rest`, what its rounding left (two-sum: exact)
__device__ __forceinline__ float df_offset(float a, float b, float oh, float ol, float& rest)
{
    const float s = a - oh, v = s - a;
    const float t = ((a - (s - v)) + (-oh - v)) + (b - ol);
    const float h = s + t, w = h - s;
    rest = (s - (h - w)) + (t - w);
    return h;
}

// the least of the eight (a NaN if one is)
__device__ __forceinline__ float min8_nan(const f32x2 (&v)[4])
{
    float a[8], r;
#pragma unroll
    for (int k = 0; k < 4; k++) upk(v[k], a[2 * k], a[2 * k + 1]);
    asm("{\n\t.reg .f32 t;\n\tmin.NaN.f32 t, %1, %2, %3;\n\tmin.NaN.f32 t, t, %4, %5;\n\t"
        "min.NaN.f32 t, t, %6, %7;\n\tmin.NaN.f32 %0, t, %8;\n\t}"
        : "=f"(r) : "f"(a[0]), "f"(a[1]), "f"(a[2]), "f"(a[3]), "f"(a[4]), "f"(a[5]), "f"(a[6]), "f"(a[7]));
    return r;
}

// s += y, with the rounding error of the addition accumulated in c (Fast2Sum;
// exact when |s| >= |y|, which a running sum of like terms keeps after its
// first additions).  s + c is the compensated sum.
__device__ __forceinline__ void comp_add(float& s, float& c, float y)
{
    const float t = s + y;
    c += (s - t) + y;
    s = t;
}
__device__ __forceinline__ void comp_add2(f32x2& s, f32x2& c, f32x2 y)
{
    const f32x2 t = add2(s, y);
    c = add2(c, add2(sub2(s, t), y));
    s = t;
}

// zeta(rho)/ZNORM as a function of s = rho^2 (FP32).
template <int K>
__device__ __forceinline__ float zhat_f32(float s)
{
    if constexpr (K == K_SING) return s == 0.0f ? 1.0f : 0.0f;
    else if constexpr (K == K_GAUS) { const float rho = sqrtf(s); return expf(-s * rho); }
    else if constexpr (K == K_GAUSERF) return fexp2(s * -0.72134752044448170f);  // e^{-s/2}
    else {
        const float q = s + 1.0f;
        const float t = frcp(q);
        return t * t * t * frsqrt(q);
    }
}

// s above which zeta/zeta(0) < 1e-13 for the Gaussian kernels (contribution
// skipped when every lane of a warp is past it); 0 = never skip.
template <int K>
__host__ __device__ constexpr float zeta_skip_s()
{
    return K == K_GAUSERF ? 60.0f : K == K_GAUS ? 10.0f : 0.0f;
}

}  // namespace vpm
