// uj_pair.cuh -- the UJ pair machinery (FP32-comp and FP64) shared by the all-pairs
// kernels (uj.cu) and the near-field warp-group kernels (leaflist.cu).
#pragma once
#include "internal.h"
#include "vpm_math.cuh"

namespace vpm {

// true for kernels equal to their singular form beyond some rho
template <int K>
__host__ __device__ constexpr bool singular_tail() { return K != K_WNKLMNS; }

// ----------------------------------------------------------- pair: mixed
// Accumulates U += G c, W += G gam, J' += Q c_i dx_j with c = dx x gam.  The
// trace of J' vanishes (c . dx = 0), so J'_33 is not accumulated; the caller
// sets it to -(J'_11 + J'_22).
__device__ __forceinline__ void accum_pair(float dx, float dy, float dz, float G, float Q, const float4& g,
                                           float (&u)[3], float (&jq)[8], float (&w)[3])
{
    const float cx = fmaf(dy, g.z, -dz * g.y);
    const float cy = fmaf(dz, g.x, -dx * g.z);
    const float cz = fmaf(dx, g.y, -dy * g.x);
    u[0] = fmaf(G, cx, u[0]);
    u[1] = fmaf(G, cy, u[1]);
    u[2] = fmaf(G, cz, u[2]);
    w[0] = fmaf(G, g.x, w[0]);
    w[1] = fmaf(G, g.y, w[1]);
    w[2] = fmaf(G, g.z, w[2]);
    const float bx = Q * cx, by = Q * cy, bz = Q * cz;
    jq[0] = fmaf(bx, dx, jq[0]);
    jq[1] = fmaf(by, dx, jq[1]);
    jq[2] = fmaf(bz, dx, jq[2]);
    jq[3] = fmaf(bx, dy, jq[3]);
    jq[4] = fmaf(by, dy, jq[4]);
    jq[5] = fmaf(bz, dy, jq[5]);
    jq[6] = fmaf(bx, dz, jq[6]);
    jq[7] = fmaf(by, dz, jq[7]);
}

// Far form of four sources j0..j0+3 whose pairs with every target of the warp are
// known to be past the kernel's reach and past (2 b)^2: FP32 offsets, no test.
// off[].w is 1/sigma^2 for the kernels without a singular tail (Winckelmans).
template <int K>
__device__ __forceinline__ void pair4_far(const float3& to, const float4* __restrict__ off,
                                          const SrcMixed* __restrict__ tile, int j0, float (&u)[3],
                                          float (&jq)[8], float (&w)[3])
{
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float4 h = off[j0 + q];
        const float dx = to.x - h.x, dy = to.y - h.y, dz = to.z - h.z;
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        float G, Q;
        if constexpr (singular_tail<K>()) {
            const float rs = frsqrt(r2);
            const float rs2 = rs * rs;
            G = rs * rs2;
            Q = G * rs2;
        } else {
            near_GQ<K>(r2 * h.w, h.w, G, Q);
        }
        accum_pair(dx, dy, dz, G, Q, tile[j0 + q].gam, u, jq, w);
    }
}

// Full form of four sources j0..j0+3, per pair, with the displacement from the
// double-float positions (th + tl) - (a + b); r == 0 contributes nothing.
// off[].w as in pair4_far.
template <int K>
__device__ __forceinline__ void pair4_near(const float3& th, const float3& tl, const float4* __restrict__ off,
                                           const SrcMixed* __restrict__ tile, int j0, float (&u)[3],
                                           float (&jq)[8], float (&w)[3])
{
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float4 a = tile[j0 + q].a, b = tile[j0 + q].b;
        const float ex = (th.x - a.x) + (tl.x - b.x);
        const float ey = (th.y - a.y) + (tl.y - b.y);
        const float ez = (th.z - a.z) + (tl.z - b.z);
        const float e2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
        float G, Q;
        if constexpr (singular_tail<K>()) {
            const float isig2 = b.w * b.w;
            near_GQ<K>(e2 * isig2, isig2, G, Q);
            const float isig3 = isig2 * b.w;
            G *= isig3;
            Q *= isig3;
        } else {
            const float hw = off[j0 + q].w;
            near_GQ<K>(e2 * hw, hw, G, Q);
        }
        const bool nz = e2 > 0.0f;
        G = nz ? G : 0.0f;
        Q = nz ? Q : 0.0f;
        accum_pair(ex, ey, ez, G, Q, tile[j0 + q].gam, u, jq, w);
    }
}

// ----------------------------------------------------------- pair: FP64
// The FP64 pair in the accumulated form of the mixed kernels: with c = dx x Gamma,
//     u += G c,   w += G Gamma,   jq[3 i + j] += Q c_j dx_i,
// G = g / r^3 and Q = -aux / (3 r^3) = (G - g' rho' r^-2 / 3) / r^2 (aux, g' = dg/drho and
// rho' = 1/sigma as in src/FLOWVPM_fmm.jl:122-146); the target's U = -u/(4 pi), and
// J = 3 jq/(4 pi) plus the Kronecker terms of src/FLOWVPM_fmm.jl:148-159 from -w/(4 pi)
// (uj_f64_finish).  Algebraically the reference's terms, regrouped so that the strength
// factor -1/(4 pi) and the products shared by the nine J entries are taken once.
// Gaussian-erf pairs past rho = 9 take g = 1, g' = 0 (the reference's cut) from the
// pack's threshold 81 sigma^2 without forming rho.  Pairs with r^2 == 0 are skipped.  Both
// tests are made on the words of r^2 (a compare costs an FP64-pipe slot); r^2 between the
// threshold and the next higher top word takes the near form, which holds there too.
// T: exp_table.
template <int K>
__device__ __forceinline__ void pair_f64_acc(double tx, double ty, double tz, const SrcF64& s, double (&u)[3],
                                             double (&w)[3], double (&jq)[9], const double* T)
{
    const double dx = tx - s.xy.x, dy = ty - s.xy.y, dz = tz - s.z_isig.x;
    const double r2 = dx * dx + dy * dy + dz * dz;
    if ((__double2hiint(r2) | __double2loint(r2)) == 0) return;
    double G, Q;
    if constexpr (K == K_WNKLMNS) {
        // (s + 2.5) q^-2.5 / sigma^3 and (s + 3.5) q^-3.5 / sigma^5, q = s + 1
        const double isig = s.z_isig.y, isig2 = isig * isig;
        const double sq = r2 * isig2;
        const double t = rsqrt(sq + 1.0), t2 = t * t;
        const double f = t2 * t2 * t * (isig2 * isig);
        G = (sq + 2.5) * f;
        Q = (sq + 3.5) * f * (t2 * isig2);
    } else if (K == K_SING || (K == K_GAUSERF && __double2hiint(r2) > __double2hiint(s.gz_sig.y))) {
        const double rinv = rsqrt(r2), rinv2 = rinv * rinv;
        G = rinv * rinv2;
        Q = G * rinv2;
    } else if constexpr (K == K_GAUSERF) {
        const double isig = s.z_isig.y, isig2 = isig * isig;
        const double sq = r2 * isig2;
        const double e = C2 * exp_neg(-0.5 * sq, T);
        if (sq < 2.0) {
            const double p = gerf_S2_f64(sq), f = e * (isig2 * isig);
            G = f * fma(sq, p, 1.0 / 3.0);
            Q = f * p * isig2;
        } else {
            const double rinv = rsqrt(r2), rinv2 = rinv * rinv, rinv3 = rinv * rinv2;
            const double rho = r2 * rinv * isig;
            const double g = fma(-e, gerf_h_f64(rho) * (1.0 / C2), 1.0);
            G = g * rinv3;
            Q = fma(-e * (1.0 / 3.0), rho * sq, g) * (rinv3 * rinv2);
        }
    } else {   // Gaussian: g = 1 - e^{-rho^3}, rho g' = 3 rho^3 e^{-rho^3}
        const double rinv = rsqrt(r2), rinv2 = rinv * rinv, rinv3 = rinv * rinv2;
        const double isig = s.z_isig.y;
        const double rho = r2 * rinv * isig, t = rho * rho * rho;
        const double e = exp_neg(-t, T);
        G = (1.0 - e) * rinv3;
        Q = fma(-t, e, 1.0 - e) * (rinv3 * rinv2);
    }
    const double gx = s.gxy.x, gy = s.gxy.y, gz = s.gz_sig.x;
    const double cx = dy * gz - dz * gy, cy = dz * gx - dx * gz, cz = dx * gy - dy * gx;
    u[0] += G * cx; u[1] += G * cy; u[2] += G * cz;
    w[0] += G * gx; w[1] += G * gy; w[2] += G * gz;
    const double bx = Q * cx, by = Q * cy, bz = Q * cz;
    jq[0] += bx * dx; jq[1] += by * dx; jq[2] += bz * dx;
    jq[3] += bx * dy; jq[4] += by * dy; jq[5] += bz * dy;
    jq[6] += bx * dz; jq[7] += by * dz; jq[8] += bz * dz;
}

// U and J (the layout of pair_f64's acc) from the sums of pair_f64_acc.
__device__ __forceinline__ void uj_f64_finish(const double (&u)[3], const double (&w)[3], const double (&jq)[9],
                                              double (&acc)[12])
{
    constexpr double k = -C4;
#pragma unroll
    for (int m = 0; m < 3; m++) acc[m] = k * u[m];
#pragma unroll
    for (int m = 0; m < 9; m++) acc[3 + m] = (-3.0 * k) * jq[m];
    const double wx = k * w[0], wy = k * w[1], wz = k * w[2];
    acc[4] -= wz;
    acc[5] += wy;
    acc[6] += wz;
    acc[8] -= wx;
    acc[9] -= wy;
    acc[10] += wx;
}

// U and J of one target from the mixed kernels' sums f = (U, W, J'): J = -3 J' (J'_33 =
// -J'_11 - J'_22) plus the Kronecker term of src/FLOWVPM_fmm.jl:148-159 (W = sum aux2 Gamma).
__device__ __forceinline__ void uj_mixed_finish(const double (&f)[14], double (&acc)[12])
{
#pragma unroll
    for (int k = 0; k < 3; k++) acc[k] = f[k];
#pragma unroll
    for (int k = 0; k < 8; k++) acc[3 + k] = -3.0 * f[6 + k];
    acc[11] = 3.0 * (f[6] + f[10]);
    acc[4] -= f[5];
    acc[5] += f[4];
    acc[6] += f[5];
    acc[8] -= f[3];
    acc[9] -= f[4];
    acc[10] += f[3];
}

// One target's sums: added to its rows, or written to its split's partial sums.
__device__ __forceinline__ void write_uj(int64_t t, int32_t idx, const double (&acc)[12], double* U,
                                         int64_t ldU, double* J, int64_t ldJ, double* partial, int64_t nt_pad)
{
    if (partial) {
        double* p = partial + (int64_t)blockIdx.y * 12 * nt_pad + t;
#pragma unroll
        for (int k = 0; k < 12; k++) p[k * nt_pad] = acc[k];
    } else {
        const int64_t i = idx;
#pragma unroll
        for (int k = 0; k < 3; k++) U[i * ldU + k] += acc[k];
#pragma unroll
        for (int k = 0; k < 9; k++) J[i * ldJ + k] += acc[3 + k];
    }
}

}  // namespace vpm
