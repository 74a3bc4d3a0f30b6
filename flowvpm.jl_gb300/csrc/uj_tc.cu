// uj_tc.cu -- the all-pairs U and J sums of one particle set on itself, FP32-comp, with
// the far pairs' sums on the tensor cores.
//
// For a target x and the sources of a compact tile with centre c, with d = x - c and
// y = x_s - c (dx = d - y), the pair terms of the mixed kernel (uj.cu),
//     U += G dx x gam,   W += G gam,   J'_ij += Q (dx x gam)_i dx_j,
// are polynomials in y with coefficients in d, so over a tile
//     W = sum G gam,   U = d x W - sum G (y x gam),
//     J' = v d^T - [d x T_j]_ij + sum Q (y x gam) y^T,
//     v = d x sum Q gam - sum Q (y x gam),   T_j = sum Q gam y_j :
// 26 sums of the two weights G(r), Q(r) times quantities of the source alone.  They are a
// matrix product, weights[targets x sources] * B[sources x 26], which tcgen05.mma does; the
// CUDA cores are left with r^2 and the weights.
//
// Arithmetic.  A weight is split into two f16 numbers, hi + lo, and so is every entry of B; all
// four products are accumulated in FP32 (TMEM), over one tile of 64 sources at a time, and added to
// FP32 mid-level sums (TC_MID tiles) and FP64 ones.  Scales are powers of two: distances are taken
// in units of R = 4..8 times the least distance of the warp's targets from the tile (so that
// G <= 2^9, Q <= 2^15), y in units of the tile's radius, and each column of B so that its largest
// entry is near 2^14: a small component of the strengths or positions keeps its own digits.  hi + lo
// holds 22 to 24 bits, except for Q past 1.5 R, where lo is subnormal: 20 bits at 2 R, the farthest
// pairs.  (Pairs alone at 1.5 R, measured: error of J 2.9e-7 to 3.0e-7 rms, 2.4e-7 to 2.9e-7 in
// uj_mixed_kernel, most of it r^-5 from the approximate square root; R within 6.4..8 of the least
// distance, 22 bits everywhere, gave 2.9e-7 to 3.1e-7.)  Errors against 64 bits stay at or below
// uj_mixed_kernel's (U / J, 2-norm): rings of 100,000 3.6e-8 / 4.1e-8 (4.0e-8 / 6.8e-8 there, in Morton order), random cloud of
// 65,536 1.9e-7 / 2.8e-7 (2.2e-7 / 3.2e-7).
//
// Classes, box to box, for a warp's 32 targets and a tile (tile_class):
//   far   every pair past the kernel's singular reach and past TC_RAD tile radii (little
//         cancellation in the polynomials), distances within a factor of 8 (the f16 range):
//         the singular weights (Winckelmans has no reach: its own weights);
//   mid   within the reach, past s = 2 (Gaussian-erf): the kernel's full form as the weight;
//   near  the rest, pair by pair after the tensor pass as in uj_mixed_kernel.
// At 65,536 random particles 87.6 / 9.2 / 3.2 % of the pairs, at 2^20 94.1 / 5.5 / 0.4 %.
//
// Layout: blocks of 128 targets in curve order, one a thread (4 warps), and a fifth warp that
// loads the tiles (bulk copies, two stages) and issues the MMAs from uniform registers (12 to
// 24 cycles each; 45 from a divergent branch).  The weights of 32 sources at a time go to TMEM
// as the A operand (lane = target, two f16 a column): 64 columns, the sums 64 more, so the 512
// columns hold 4 blocks a SM.  While a step's MMAs run, the weights of the next 16 sources are
// already computed.  B is made once per call (pack_tiles) as the shared-memory image the MMA
// reads.
//
// Bound: issue slots.  A far pair takes 10.5 instructions (packed f32x2 r^2 and weights, one
// MUFU, the f16 splits) plus 4.5 for its share of a tile's set-up, waits and recombination; all
// classes together 19.0 at 262,144, against 40.4 in uj_mixed_kernel.  68 % of the issue slots are
// used (4 warps a scheduler, the TMEM's limit), the tensor pipe 14 %.  Measured, whole calls,
// Gaussian-erf: N = 2^20 1360 -> 758 ms, 262,144 102.8 -> 53.4, 65,536 7.83 -> 4.12, rings of
// 200,000 57.8 -> 41.4, ring of 32,000 2.40 -> 1.62; Winckelmans 50,001 4.61 -> 2.77.  Tried: packed pairs split back to
// scalar FP32 13 % slower, f16 remainders by conversion instead of the mixed-precision
// subtraction 11 %, three blocks a SM 6 %, two A buffers of 16 sources (twice the barriers)
// 16 %.
#include "internal.h"
#include "tc05.cuh"
#include "uj_pair.cuh"
#include "vpm_math.cuh"

#include <cuda_fp16.h>

namespace vpm {

constexpr int TCS = 64;                       // sources per tile
constexpr int TC_GN = 16, TC_QN = 48;         // B columns of the G and Q products (12 and 40 used)
constexpr int TC_BG = TC_GN * 16 * 2;         // bytes of 16 sources' B: G part, then Q part
constexpr int TC_BK = TC_BG + TC_QN * 16 * 2;
constexpr int TC_B = (TCS / 16) * TC_BK;      // 8192
constexpr int TC_POS = TCS * 4;               // bytes of one coordinate of the tile's y
constexpr int TC_REC = TC_B + 4 * TC_POS + 64;      // B, y (x, y, z), sigma^2, header
constexpr int TC_SC = 128;                          // then the scales of B's 26 columns
constexpr int TC_STRIDE = (TC_REC + TC_SC + 127) / 128 * 128;
constexpr int TC_SIZE = (TC_REC + 127) / 128 * 128; // a stage, without the scales
constexpr int TC_THREADS = UJ_THREADS + 32;
constexpr int TC_COLS = 128;                  // TMEM columns of a block: A 64, G sums 16, Q sums 48
constexpr int TC_DG = 64, TC_DQ = 80;
constexpr int WT = 32;
// Tiles between FP64 adds of the tensor pass (1,024 sources, as in uj_mixed_kernel) and of the near pass,
// whose terms are the largest (32 and the 32 tiles' near ones: error of J, rings of 100,000, 7.0e-8
// against 4.1e-8, 6.8e-8 in uj_mixed_kernel in Morton order; UJ of 65,000 random particles 3.92 against 3.98
// ms, of the rings 9.94 against 10.16).
constexpr int TC_MID = 16, TC_MID_NEAR = 4;
// tcgen05.mma truncates: a step's products and the accumulator are aligned to the largest of them and
// cut two bits below FP32's last, and the sum is cut to FP32.  (This arithmetic, simulated, loses what is
// measured, in 1e-7 of the sum: 64 equal sources 2.0 / 1.8, one in 2 1.4 / 1.3, in 4 1.2 / 1.0, in 8 0.95 /
// 0.86, in 16 0.77 / 0.66, one alone 0.5 / 0.4, lognormal strengths 2.3 / 2.4.)  pack_tiles works the
// expected loss of each tile out from its strengths and scales B up by it: every cut at half a unit, at
// nominal weights of 1, projected on the sum.  Without it far velocities that add up coherently were
// low by 0.8e-7 to 2.2e-7 (rings of 100,000, a cloud of strengths of one sign); with it they are within the
// 2e-8 to 3e-8 of the weights' own rounding.
constexpr float TC_UNIT = 0x1p-24f * 1.4427f;   // FP32's unit over the value, on average: 2^-24 / m, m in [1/2, 1)
// a source's products of 22 bits (2^-20.5 of themselves to their last) beside a sum of `top`
__device__ __forceinline__ float cut_loss(float mine, float top)
{
    return fminf(fmaxf(0.5f * (0.25f * TC_UNIT * top - 6.74e-7f * mine), 0.f), mine);
}

// A tile's header, 64 B: centre as a double-float, radius, half extents, the scales.
struct __align__(16) TileHdr {
    float chx, chy, chz, rad;
    float clx, cly, clz, sig2;     // sig2: the tile's largest sigma^2
    float hx, hy, hz, gscale;      // gscale: gam = gscale * (the pack's strength)
    float yscale, ok, sig2lo, p1;  // yscale: y = yscale * (the pack's y); sig2lo: the smallest sigma^2
};
static_assert(sizeof(TileHdr) == 64, "header layout");

static inline int64_t tc_tiles(int64_t n) { return (n + TCS - 1) / TCS; }
static inline size_t align128(size_t b) { return (b + 127) / 128 * 128; }

size_t uj_tc_bytes(int64_t n)
{
    return align128((size_t)tc_tiles(n) * sizeof(TileHdr)) + (size_t)tc_tiles(n) * TC_STRIDE;
}

__device__ __forceinline__ float pow2_at_least(float v)   // power of two >= v (v > 0, normal)
{
    return __uint_as_float((__float_as_uint(v) + 0x7fffffu) & 0x7f800000u);
}

// ------------------------------------------------------------------ packing
// One block of 64 threads per tile, one source each, in the targets' curve order.
template <int K>
__global__ void __launch_bounds__(TCS)
pack_tiles(int64_t n, const double* __restrict__ gs, const double* __restrict__ sgs,
           const TgtPos* __restrict__ order, TileHdr* __restrict__ hdr, char* __restrict__ rec)
{
    __shared__ double red[2][7];
    __shared__ float redf[2][3];
    __shared__ uint32_t redc[2][26];
    __shared__ float steps[4][4], redl[2][2];
    __shared__ __align__(16) char img[TC_B];
    const int k = threadIdx.x, warp = k >> 5, lane = k & 31;
    const int64_t o = (int64_t)blockIdx.x * TCS + k;
    const bool on = o < n;
    const TgtPos p = order[on ? o : n - 1];
    const double x[3] = {p.x, p.y, p.z};
    double g[3] = {0.0, 0.0, 0.0}, sig = 1.0;
    if (on) {
        for (int m = 0; m < 3; m++) g[m] = -C4 * gs[3 * (int64_t)p.idx + m];
        if (K != K_SING) sig = sgs[p.idx];
    }
    // box, largest sigma^2 and largest strength component of the tile
    double b[7] = {x[0], x[1], x[2], -x[0], -x[1], -x[2], fmax(fabs(g[0]), fmax(fabs(g[1]), fabs(g[2])))};
    for (int m = 0; m < 7; m++) {
        for (int s = 16; s > 0; s >>= 1) {
            const double v = __shfl_xor_sync(0xffffffffu, b[m], s);
            b[m] = m < 6 ? fmin(b[m], v) : fmax(b[m], v);
        }
        if (lane == 0) red[warp][m] = b[m];
    }
    __syncthreads();
    double c[3], y[3];
    float half[3];
    for (int m = 0; m < 3; m++) {
        const double lo = fmin(red[0][m], red[1][m]), hi = -fmin(red[0][3 + m], red[1][3 + m]);
        const double mid = 0.5 * (lo + hi);
        const float ch = (float)mid, cl = (float)(mid - (double)ch);
        c[m] = (double)ch + (double)cl;
        half[m] = (float)fmax(hi - c[m], c[m] - lo) * 1.000001f;
        y[m] = x[m] - c[m];
    }
    const float gmax = (float)fmax(red[0][6], red[1][6]);
    float r2 = (float)(y[0] * y[0] + y[1] * y[1] + y[2] * y[2]), s2 = on ? (float)(sig * sig) : 0.f, s2lo = on ? s2 : 3.0e38f;
    const float own_s2 = s2;
    // a NaN position or core size must not hide in a maximum: it clears `ok`
    const bool fine = isfinite(r2) && isfinite(s2) && isfinite(g[0]) && isfinite(g[1]) && isfinite(g[2]);
    for (int s = 16; s > 0; s >>= 1) {
        r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, s));
        s2 = fmaxf(s2, __shfl_xor_sync(0xffffffffu, s2, s));
        s2lo = fminf(s2lo, __shfl_xor_sync(0xffffffffu, s2lo, s));
    }
    if (lane == 0) { redf[warp][0] = r2; redf[warp][1] = s2; redf[warp][2] = s2lo; }
    const bool ok = __syncthreads_and(fine) && gmax < 1e30f && (gmax > 1e-30f || gmax == 0.f);
    // the tile's fourth array: sigma^2 for Winckelmans, 1/sigma for the kernels with a singular tail.  Sources
    // past n take the tile's largest core: they have no strength, but a weight outside the f16 range that
    // tile_class works out from the tile's own cores would be infinite, and NaN times their zeros.  1/sigma
    // stays below 1e6 of the largest core's, where the mid form (r > 1.4 of the largest core) is long the
    // singular one: past rho = 7e12 its rho^3 e^{-rho^2/2} would be infinity times zero.
    const float s2max = fmaxf(redf[0][1], redf[1][1]);
    const float islo = 1.f / sqrtf(s2max);
    const float mys2 = singular_tail<K>() ? on ? fminf((float)(1.0 / sig), 1e6f * islo) : islo : on ? own_s2 : s2max;
    const float rad = sqrtf(fmaxf(redf[0][0], redf[1][0])) * 1.000001f;
    // expected losses, in units of the largest strength: `along` of sums over strengths as they are, `across`
    // of sums whose terms change sign within the tile (strengths times y; or strengths that cancel)
    double along = 0.0, across = 0.0;
    {
        const double in = ok && gmax > 0.f ? 1.0 / (double)gmax : 0.0;
        const float v[3] = {(float)(g[0] * in), (float)(g[1] * in), (float)(g[2] * in)};
        const float a2 = fmaf(v[0], v[0], fmaf(v[1], v[1], v[2] * v[2])), amp = sqrtf(a2);
        float q[5] = {v[0], v[1], v[2], a2, amp};     // of the source's step of 16: sum, sum of squares, largest
        for (int m = 8; m > 0; m >>= 1) {
            for (int j = 0; j < 4; j++) q[j] += __shfl_xor_sync(0xffffffffu, q[j], m);
            q[4] = fmaxf(q[4], __shfl_xor_sync(0xffffffffu, q[4], m));
        }
        if ((k & 15) == 0)
            for (int j = 0; j < 4; j++) steps[k >> 4][j] = q[j];
        __syncthreads();
        float before[4] = {0.f, 0.f, 0.f, 0.f}, whole[4] = {0.f, 0.f, 0.f, 0.f};
        for (int m = 0; m < 4; m++)
            for (int j = 0; j < 4; j++) {
                if (m < (k >> 4)) before[j] += steps[m][j];
                whole[j] += steps[m][j];
            }
        const float top1 = sqrtf(fmaf(before[0], before[0], fmaf(before[1], before[1], before[2] * before[2])));
        const float l1 = cut_loss(amp, fmaxf(top1, q[4])), l2 = cut_loss(amp, fmaxf(sqrtf(before[3]), q[4]));
        // the two cuts of the step's sums (lo and hi products), 3/8 of a unit each, shared by its 16 sources
        const float cut = q[4] > 0.f ? 0.375f * TC_UNIT / 16.f : 0.f, ia = amp > 0.f ? l1 / amp : 0.f;
        float r[2] = {0.f, fmaf(l2, amp, cut * (2.f * before[3] + q[3]))};
        for (int j = 0; j < 3; j++) r[0] = fmaf(whole[j], fmaf(ia, v[j], cut * (2.f * before[j] + q[j])), r[0]);
        for (int m = 16; m > 0; m >>= 1)
            for (int j = 0; j < 2; j++) r[j] += __shfl_xor_sync(0xffffffffu, r[j], m);
        if (lane == 0) { redl[warp][0] = r[0]; redl[warp][1] = r[1]; }
        __syncthreads();
        r[0] = redl[0][0] + redl[1][0];
        r[1] = redl[0][1] + redl[1][1];
        // (weights that vary by a quarter within the tile keep sums from cancelling below that)
        const float s2 = fmaf(whole[0], whole[0], fmaf(whole[1], whole[1], whole[2] * whole[2]));
        if (whole[3] > 0.f) {
            along = (double)((r[0] + r[1] / 16.f) / (s2 + whole[3] / 16.f));
            across = (double)(r[1] / whole[3]);
        }
    }
    const float ys = rad > 1e-30f ? pow2_at_least(rad) : 1.f;
    const float gsc = gmax > 1e-30f ? pow2_at_least(gmax) * (1.f / 64.f) : 1.f;

    // B columns of this source, scaled: G part gam, y x gam; Q part gam, gam y_j, (y x gam) y_j
    const double iy = 1.0 / (double)ys, ig = 1.0 / (double)gsc;
    for (int m = 0; m < 3; m++) { y[m] *= iy; g[m] *= ig; }
    double col[26];
    const double mx[3] = {y[1] * g[2] - y[2] * g[1], y[2] * g[0] - y[0] * g[2], y[0] * g[1] - y[1] * g[0]};
    for (int m = 0; m < 3; m++) { col[m] = g[m]; col[3 + m] = mx[m]; col[6 + m] = g[m]; }
    for (int j = 0; j < 3; j++)
        for (int i = 0; i < 3; i++) {
            col[9 + 3 * j + i] = g[i] * y[j];
            if (3 * j + i < 8) col[18 + 3 * j + i] = mx[i] * y[j];
        }
    for (int m = 0; m < 26; m++) col[m] = fma(col[m], m < 3 || (m >= 6 && m < 9) ? along : across, col[m]);
    // each column to a largest entry of 2^14 in magnitude
    for (int m = 0; m < 26; m++) {
        const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf((float)col[m])));
        if (lane == 0) redc[warp][m] = top;
    }
    for (int w = k; w < TC_B / 16; w += TCS) ((uint4*)img)[w] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    auto scale = [&](int m) {
        const float top = __uint_as_float(max(redc[0][m], redc[1][m]));
        return top > 1e-30f && top < 1e30f ? pow2_at_least(top) * 0x1p-14f : 1.f;
    };
    char* kb = img + (k >> 4) * TC_BK;
    const int kc = (k >> 3) & 1, k8 = k & 7;
    for (int m = 0; m < 26; m++) {
        const bool q = m >= 6;
        const float sc = scale(m), isc = __uint_as_float((254u << 23) - __float_as_uint(sc));   // a power of two
        const __half h = __float2half_rn((float)col[m] * isc);
        const __half l = __float2half_rn((float)(col[m] - (double)(__half2float(h) * sc)) * isc);
        const int base = q ? TC_BG : 0, nh = q ? m - 6 : m, nl = q ? m - 6 + 20 : m + 6;
        *(__half*)(kb + base + ((nh >> 3) * 2 + kc) * 128 + (nh & 7) * 16 + k8 * 2) = h;
        *(__half*)(kb + base + ((nl >> 3) * 2 + kc) * 128 + (nl & 7) * 16 + k8 * 2) = l;
    }
    __syncthreads();
    char* out = rec + (int64_t)blockIdx.x * TC_STRIDE;
    for (int w = k; w < TC_B / 16; w += TCS) ((uint4*)out)[w] = ((const uint4*)img)[w];
    // y, in absolute units (the pair's dx needs no scale of its own); sources past n at the centre
    for (int m = 0; m < 3; m++) ((float*)(out + TC_B + m * TC_POS))[k] = on ? (float)(x[m] - c[m]) : 0.f;
    ((float*)(out + TC_B + 3 * TC_POS))[k] = mys2;
    if (k < 26) ((float*)(out + TC_REC))[k] = scale(k);
    if (k == 0) {
        TileHdr h;
        h.chx = (float)c[0]; h.chy = (float)c[1]; h.chz = (float)c[2]; h.rad = rad;
        h.clx = (float)(c[0] - (double)h.chx); h.cly = (float)(c[1] - (double)h.chy); h.clz = (float)(c[2] - (double)h.chz);
        h.sig2 = s2max;
        h.hx = half[0]; h.hy = half[1]; h.hz = half[2];
        h.gscale = gsc;
        h.yscale = ys; h.ok = ok ? 1.f : 0.f; h.sig2lo = fminf(redf[0][2], redf[1][2]); h.p1 = 0.f;
        hdr[blockIdx.x] = h;
        *(TileHdr*)(out + TC_B + 4 * TC_POS) = h;
    }
}

// ---------------------------------------------------------- packed FP32 pairs
// hi = the two values as f16x2; nlo = minus their remainders as f16x2
__device__ __forceinline__ void split2(f32x2 v, uint32_t& hi, uint32_t& nlo)
{
    float a, b, na, nb;
    upk(v, a, b);
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(b), "f"(a));
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\t"
        "sub.rn.f32.f16 %0, l, %3;\n\tsub.rn.f32.f16 %1, h, %4;\n\t}"
        : "=f"(na), "=f"(nb) : "r"(hi), "f"(a), "f"(b));
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(nlo) : "f"(nb), "f"(na));
}

// Weights of two pairs at squared distance r2 (in units R^2): G = g/r^3, Q = (3g - r g')/(3 r^5).
// s2: sigma^2 in units R^2 (Winckelmans only; r2 then is r^2 + sigma^2).
template <int K>
__device__ __forceinline__ void weights2(f32x2 r2, f32x2 s2, f32x2& G, f32x2& Q)
{
    float a, b;
    upk(r2, a, b);
    const f32x2 t = pk(frsqrt(a), frsqrt(b));
    const f32x2 t2 = mul2(t, t);
    if constexpr (singular_tail<K>()) {
        G = mul2(t2, t);
        Q = mul2(G, t2);
    } else {   // (r^2 + 2.5 s^2) p^-2.5 and (r^2 + 3.5 s^2) p^-3.5 with p = r^2 + s^2
        const f32x2 t3 = mul2(t2, t), t5 = mul2(t3, t2), u = mul2(s2, t5);
        G = fma2(u, pk(1.5f, 1.5f), t3);
        Q = mul2(fma2(u, pk(2.5f, 2.5f), t3), t2);
    }
}

// The Gaussian-erf weights at s = (r/sigma)^2 >= 2 (gerf_G_erfcx's fit; valid at any larger s):
// G = g/r^3, Q = (g - c2 rho^3 e/3)/r^5 with e = e^{-s/2}.  is: 1/sigma in units 1/R.
__device__ __forceinline__ void weights2_erf(f32x2 r2, f32x2 is, f32x2& G, f32x2& Q)
{
    float a, b;
    upk(r2, a, b);
    const f32x2 t = pk(frsqrt(a), frsqrt(b));
    const f32x2 rho = mul2(mul2(r2, t), is), s = mul2(rho, rho);
    float v0, v1;
    upk(fma2(rho, pk(0.5f, 0.5f), pk(1.f, 1.f)), v0, v1);
    const f32x2 x = pk(frcp(v0), frcp(v1));
    upk(mul2(s, pk(-0.72134752044448170f, -0.72134752044448170f)), v0, v1);
    const f32x2 e = pk(fexp2(v0), fexp2(v1));
    const f32x2 w = fma2(x, pk(4.77190564267067f, 4.77190564267067f), pk(-1.795317607111778f, -1.795317607111778f));
    f32x2 p = pk(-5.1560079373370265e-06f, -5.1560079373370265e-06f);
    p = fma2(p, w, pk(5.998428003101994e-06f, 5.998428003101994e-06f));
    p = fma2(p, w, pk(0.00010125038777505872f, 0.00010125038777505872f));
    p = fma2(p, w, pk(-0.00030713426402493693f, -0.00030713426402493693f));
    p = fma2(p, w, pk(-0.0023330098304451836f, -0.0023330098304451836f));
    p = fma2(p, w, pk(0.009623567049071946f, 0.009623567049071946f));
    p = fma2(p, w, pk(0.13016216050000662f, 0.13016216050000662f));
    p = fma2(p, w, pk(0.5926831417002281f, 0.5926831417002281f));
    const f32x2 h = fma2(rho, pk(F_C2, F_C2), mul2(p, x));
    const f32x2 ne = mul2(e, pk(-1.f, -1.f));
    const f32x2 g = fma2(ne, h, pk(1.f, 1.f));
    const f32x2 gq = fma2(mul2(ne, mul2(rho, s)), pk(F_C2 / 3.f, F_C2 / 3.f), g);
    const f32x2 t2 = mul2(t, t), t3 = mul2(t2, t);
    G = mul2(g, t3);
    Q = mul2(gq, mul2(t3, t2));
}

// The weights of 2 N sources (p: their x; y, z and the fourth array follow at TC_POS) for a
// target at d from the tile's centre, in units R, as the A operand's f16 pairs.  MID: the
// kernel's full form instead of the singular one.
template <int K, int N, bool MID = false>
__device__ __forceinline__ void weigh(const ulonglong2* p, float dx, float dy, float dz, float iR,
                                      uint32_t (&gh)[N], uint32_t (&gl)[N], uint32_t (&qh)[N], uint32_t (&ql)[N])
{
    const f32x2 DX = pk(dx, dx), DY = pk(dy, dy), DZ = pk(dz, dz), NR = pk(-iR, -iR);
    f32x2 SC = 0ull;
    if constexpr (!singular_tail<K>()) SC = pk(iR * iR, iR * iR);
    if constexpr (MID) {
        const float R = __uint_as_float((254u << 23) - __float_as_uint(iR));   // iR is a power of two
        SC = pk(R, R);
    }
#pragma unroll
    for (int w = 0; w < N / 2; w++) {
        const ulonglong2 X = p[w], Y = p[w + TC_POS / 16], Z = p[w + 2 * (TC_POS / 16)];
        ulonglong2 S = make_ulonglong2(0ull, 0ull);
        if constexpr (!singular_tail<K>() || MID) S = p[w + 3 * (TC_POS / 16)];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const f32x2 ex = fma2(e ? X.y : X.x, NR, DX), ey = fma2(e ? Y.y : Y.x, NR, DY),
                        ez = fma2(e ? Z.y : Z.x, NR, DZ);
            f32x2 s2 = 0ull, r2;
            if constexpr (!singular_tail<K>()) {
                s2 = mul2(e ? S.y : S.x, SC);
                r2 = fma2(ez, ez, s2);
            } else {
                r2 = mul2(ez, ez);
            }
            r2 = fma2(ex, ex, fma2(ey, ey, r2));
            f32x2 G, Q;
            if constexpr (MID) weights2_erf(r2, mul2(e ? S.y : S.x, SC), G, Q);
            else weights2<K>(r2, s2, G, Q);
            split2(G, gh[2 * w + e], gl[2 * w + e]);
            split2(Q, qh[2 * w + e], ql[2 * w + e]);
        }
    }
}

// 16 sources' weights into A (a: the TMEM address of their first G hi column)
__device__ __forceinline__ void store_a(uint32_t a, const uint32_t (&gh)[8], const uint32_t (&gl)[8],
                                        const uint32_t (&qh)[8], const uint32_t (&ql)[8])
{
    tmem_st8(a, gh);
    tmem_st8(a + 16, gl);
    tmem_st8(a + 32, qh);
    tmem_st8(a + 48, ql);
}

// Box-to-box test of one tile against the warp's targets (centre wc as a double-float, half
// extents wh): TILE_FAR, every pair past the kernel's singular reach; TILE_MID, within it but
// past s = 2 (Gaussian-erf); both past the geometry's limits; else TILE_NEAR.  iR receives 1/R.
enum : int { TILE_NEAR = 0, TILE_MID = 1, TILE_FAR = 2 };
// Least distance of a far or mid tile, in tile radii.  Nearer ones are evaluated pair by pair, at four
// times the cost: 1.5 / 1.0 / 0.75 / 0.5 radii measured 4.30 / 4.06 / 4.00 / 3.92 ms at 65,536 random
// particles, with the same errors but at 0.5 (rings of 30,000, Winckelmans: largest error of J
// 3.7e-7 -> 6.6e-7 of the rms).
constexpr float TC_RAD = 0.75f;
// (A call of its own: it runs once for 32 tiles, and inlined its square roots cost the tile loop up to
// 10 % through the registers and the order of the code around it: Winckelmans 100,000 10.0 -> 9.04 ms.)
template <int K>
__device__ __noinline__ int tile_class(const TileHdr& h, const float3& wch, const float3& wcl, const float3& wh,
                                          float wdiag, float& iR)
{
    const float ax = fmaxf(fabsf((h.chx - wch.x) + (h.clx - wcl.x)) - h.hx - wh.x, 0.f);
    const float ay = fmaxf(fabsf((h.chy - wch.y) + (h.cly - wcl.y)) - h.hy - wh.y, 0.f);
    const float az = fmaxf(fabsf((h.chz - wch.z) + (h.clz - wcl.z)) - h.hz - wh.z, 0.f);
    const float d2 = fmaf(ax, ax, fmaf(ay, ay, az * az));
    const float dmin = sqrtf(d2);
    const float span = 2.f * (sqrtf(fmaf(h.hx, h.hx, fmaf(h.hy, h.hy, h.hz * h.hz))) + wdiag);
    // R: the power of two in (4, 8] dmin.  Winckelmans' weights go by p = r^2 + sigma^2, up to 3.5 p^-2.5:
    // there dmin^2 is the least p times 3.5^-0.4, and the p of the tile stay within 8^2
    float unit = dmin;
    bool range = span < 7.f * dmin;
    if constexpr (!singular_tail<K>()) {
        const float p = d2 + h.sig2lo, far = dmin + span;
        unit = 0.778f * sqrtf(p);
        range = fmaf(far, far, h.sig2) < 64.f * p;
    }
    iR = __uint_as_float((251u << 23) - (__float_as_uint(unit) & 0x7f800000u));
    if (!(h.ok != 0.f && dmin > TC_RAD * h.rad && range && dmin > 1e-9f && unit < 1e9f)) return TILE_NEAR;
    const float sw = h.gscale * iR * iR * iR;      // the sums' unit stays well inside FP32
    if (!(sw > 1e-30f && sw < 1e30f)) return TILE_NEAR;
    if (!singular_tail<K>() || d2 > s_far<K>() * h.sig2) return TILE_FAR;
    return K == K_GAUSERF && d2 > 2.f * h.sig2 ? TILE_MID : TILE_NEAR;
}

struct TcStage { char rec[TC_SIZE]; };

template <int K>
__global__ void __launch_bounds__(TC_THREADS, 4)
uj_tc_kernel(int64_t nt, const TgtPos* __restrict__ tgt, int ntiles_all, const TileHdr* __restrict__ hdr,
             const char* __restrict__ rec, const SrcMixed* __restrict__ src,
             double* U, int64_t ldU, double* J, int64_t ldJ, double* partial, int64_t nt_pad, uint32_t rounds,
             int* __restrict__ gave_up)
{
    __shared__ __align__(128) TcStage stage[2];
    // The scales of a tile's columns, read when its sums are, in the next tile's first half: a slot is
    // filled again three tiles on, after every warp's arrival for that half.
    __shared__ __align__(16) ulonglong2 scales[3][TC_SC / 16];
    __shared__ SrcMixed near_s[UJ_WARPS][WT];
    __shared__ float4 near_o[UJ_WARPS][WT];
    __shared__ double acc64[14][UJ_THREADS];
    __shared__ __align__(8) uint64_t bfull[2], afull, adone, drain;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // this split's tiles: every gridDim.y-th, so that the near ones (a target's neighbours
    // on the curve) spread over the splits
    const int t0 = blockIdx.y, tstep = gridDim.y;
    const int ntiles = (ntiles_all - t0 + tstep - 1) / tstep;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; s++) mbar_init(&bfull[s], 1);
        mbar_init(&afull, UJ_WARPS);
        mbar_init(&adone, 1);
        mbar_init(&drain, 1);
        mbar_init_fence();
        failed = 0;
    }
    if (warp == UJ_WARPS) tmem_alloc(&tmem_slot, TC_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp == UJ_WARPS) {
        // loads and MMAs: the whole warp runs the loop (uniform descriptors), one lane issues
        const bool one = elect_one();
        bool ok = true;
        int loaded = min(ntiles, 2);
        int slot = 0;                       // of the next tile's scales
        auto load = [&](int q) {
            if (one) {
                const char* r = rec + (int64_t)(t0 + q * tstep) * TC_STRIDE;
                mbar_expect_tx(&bfull[q & 1], TC_REC + TC_SC);
                bulk_load(&stage[q & 1], r, TC_REC, &bfull[q & 1]);
                bulk_load(scales[slot], r + TC_REC, TC_SC, &bfull[q & 1]);
            }
            slot = slot == 2 ? 0 : slot + 1;
        };
        for (int q = 0; q < loaded; q++) load(q);
        constexpr uint32_t ig = idesc_f16(128, TC_GN), iq = idesc_f16(128, TC_QN);
        constexpr uint32_t neg = 1u << 13;   // the lo operands are stored negated
        for (int it = 0; ok && it < ntiles; it++) {
            const int s = it & 1;
            ok = mbar_wait(&bfull[s], (uint32_t)(it >> 1) & 1u, rounds);
            const uint32_t b0 = smem_u32(&stage[s]);
            const uint64_t dg0 = smem_desc(b0, 128, 256), dq0 = smem_desc(b0 + TC_BG, 128, 256);
#pragma unroll 1
            for (int h = 0; ok && h < 2; h++) {   // 32 sources: step 2 it + h
                ok = mbar_wait(&afull, (uint32_t)h, rounds);
                tc_fence_after();
                if (ok && one) {
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        const uint64_t dg = dg0 + (2 * h + k) * (TC_BK >> 4), dq = dq0 + (2 * h + k) * (TC_BK >> 4);
                        const bool acc = h + k > 0;
                        mma_f16_ts(tmem + TC_DG, tmem + 16 + 8 * k, dg, ig | neg, acc);
                        mma_f16_ts(tmem + TC_DQ, tmem + 48 + 8 * k, dq, iq | neg, acc);
                        mma_f16_ts(tmem + TC_DG, tmem + 8 * k, dg, ig, true);
                        mma_f16_ts(tmem + TC_DQ, tmem + 32 + 8 * k, dq, iq, true);
                    }
                    mma_commit(&adone);
                }
            }
            if (ok && loaded < ntiles) {
                // the stage is free: every warp has read its y (afull of the last step), and
                // the tile's MMAs are done with its B
                ok = mbar_wait(&adone, 1u, rounds);
                if (ok) load(loaded++);
            }
        }
        if (!ok) {   // a wait that gave up: wait (bounded) for what is in flight
            if (one) { failed = 1; mma_commit(&drain); }
            for (int q = max(0, loaded - 2); q < loaded; q++) mbar_wait(&bfull[q & 1], (uint32_t)(q >> 1) & 1u, WAIT_ROUNDS);
            mbar_wait(&drain, 0, WAIT_ROUNDS);
        }
        __syncwarp();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        tmem_dealloc(tmem, TC_COLS);
        return;
    }

    // ------------------------------------------------------------------- targets
    const int64_t t = (int64_t)blockIdx.x * UJ_THREADS + threadIdx.x;
    const bool valid = t < nt;
    const bool wvalid = (int64_t)blockIdx.x * UJ_THREADS + warp * 32 < nt;
    const TgtPos me = tgt[valid ? t : nt - 1];      // lanes past nt repeat the last target
    const float3 th = make_float3((float)me.x, (float)me.y, (float)me.z);
    const float3 tl = make_float3((float)(me.x - (double)th.x), (float)(me.y - (double)th.y), (float)(me.z - (double)th.z));
    // warp origin: lane 0's target; offsets and their box
    const double ox = __shfl_sync(0xffffffffu, me.x, 0), oy = __shfl_sync(0xffffffffu, me.y, 0),
                 oz = __shfl_sync(0xffffffffu, me.z, 0);
    const float3 to = make_float3((float)(me.x - ox), (float)(me.y - oy), (float)(me.z - oz));
    float3 blo = to, bhi = to;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
        blo.x = fminf(blo.x, __shfl_xor_sync(0xffffffffu, blo.x, m));
        blo.y = fminf(blo.y, __shfl_xor_sync(0xffffffffu, blo.y, m));
        blo.z = fminf(blo.z, __shfl_xor_sync(0xffffffffu, blo.z, m));
        bhi.x = fmaxf(bhi.x, __shfl_xor_sync(0xffffffffu, bhi.x, m));
        bhi.y = fmaxf(bhi.y, __shfl_xor_sync(0xffffffffu, bhi.y, m));
        bhi.z = fmaxf(bhi.z, __shfl_xor_sync(0xffffffffu, bhi.z, m));
    }
    const float3 wh = make_float3(0.500001f * (bhi.x - blo.x), 0.500001f * (bhi.y - blo.y), 0.500001f * (bhi.z - blo.z));
    const float wdiag = sqrtf(fmaf(wh.x, wh.x, fmaf(wh.y, wh.y, wh.z * wh.z)));
    const double wcx = ox + 0.5 * ((double)blo.x + (double)bhi.x), wcy = oy + 0.5 * ((double)blo.y + (double)bhi.y),
                 wcz = oz + 0.5 * ((double)blo.z + (double)bhi.z);
    const float3 wch = make_float3((float)wcx, (float)wcy, (float)wcz);
    const float3 wcl = make_float3((float)(wcx - (double)wch.x), (float)(wcy - (double)wch.y), (float)(wcz - (double)wch.z));
#pragma unroll
    for (int k = 0; k < 14; k++) acc64[k][threadIdx.x] = 0.0;
    float mu[3] = {0.f, 0.f, 0.f}, mw[3] = {0.f, 0.f, 0.f}, mj[8];
#pragma unroll
    for (int k = 0; k < 8; k++) mj[k] = 0.f;
    auto flush = [&]() {
        __syncwarp();   // keeps the FP64 adds a branch of their own (see below)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            acc64[k][threadIdx.x] += (double)mu[k];
            acc64[3 + k][threadIdx.x] += (double)mw[k];
            mu[k] = 0.f;
            mw[k] = 0.f;
        }
#pragma unroll
        for (int k = 0; k < 8; k++) { acc64[6 + k][threadIdx.x] += (double)mj[k]; mj[k] = 0.f; }
        __syncwarp();
    };

    // ------------------------------------------------- tensor pass over the far tiles
    // The mid-level sums go to FP64 after TC_MID tiles (the FP64 adds stand outside the tile loop:
    // as a condition inside it they were issued, predicated off, for every tile and kept the
    // FP64 pipe 42 % busy).
    const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16);
    bool ok = true;
    // the tile's sums, back in absolute units
    auto collect = [&](const ulonglong2* sc, float pdx, float pdy, float pdz, float iR, float hg, float hy) {
        const float kap = hy * iR, su = hg * iR * iR, sw = su * iR;
        {
            float v[16];
            tmem_ld8(ta + TC_DG, v);
            tmem_ld8(ta + TC_DG + 8, v + 8);
            tc_wait_ld(v);
            const ulonglong2 s0 = sc[0], s1 = sc[1];
            float wx, wy, wz, mx, my, mz;
            upk(mul2(add2(pk(v[0], v[1]), pk(v[6], v[7])), s0.x), wx, wy);
            upk(mul2(add2(pk(v[2], v[3]), pk(v[8], v[9])), s0.y), wz, mx);
            upk(mul2(add2(pk(v[4], v[5]), pk(v[10], v[11])), s1.x), my, mz);
            mu[0] = fmaf(su, fmaf(pdy, wz, fmaf(-pdz, wy, -kap * mx)), mu[0]);
            mu[1] = fmaf(su, fmaf(pdz, wx, fmaf(-pdx, wz, -kap * my)), mu[1]);
            mu[2] = fmaf(su, fmaf(pdx, wy, fmaf(-pdy, wx, -kap * mz)), mu[2]);
            mw[0] = fmaf(sw, wx, mw[0]);
            mw[1] = fmaf(sw, wy, mw[1]);
            mw[2] = fmaf(sw, wz, mw[2]);
        }
        {
            float v[40];
#pragma unroll
            for (int k = 0; k < 5; k++) tmem_ld8(ta + TC_DQ + 8 * k, v + 8 * k);
            tc_wait_ld(v);
#pragma unroll
            for (int k = 0; k < 10; k++) {
                const ulonglong2 s2 = sc[(3 + k) >> 1];
                upk(mul2(add2(pk(v[2 * k], v[2 * k + 1]), pk(v[20 + 2 * k], v[21 + 2 * k])), k & 1 ? s2.x : s2.y), v[2 * k], v[2 * k + 1]);
            }
            const float* T = v + 3;          // T[3 j + i] = sum Q gam_i y_j
            const float kx = kap * pdx, ky = kap * pdy, kz = kap * pdz, k2 = kap * kap;
            // v = d x A - kappa sum Q (y x gam), the latter from the antisymmetric part of T
            const float vx = fmaf(pdy, v[2], fmaf(-pdz, v[1], -kap * (T[5] - T[7])));
            const float vy = fmaf(pdz, v[0], fmaf(-pdx, v[2], -kap * (T[6] - T[2])));
            const float vz = fmaf(pdx, v[1], fmaf(-pdy, v[0], -kap * (T[1] - T[3])));
            const float* N = v + 12;
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const float dj = j == 0 ? pdx : j == 1 ? pdy : pdz;
                const float* Tj = T + 3 * j;
                const float c0 = fmaf(ky, Tj[2], -kz * Tj[1]), c1 = fmaf(kz, Tj[0], -kx * Tj[2]);
                mj[3 * j] = fmaf(sw, fmaf(k2, N[3 * j], fmaf(vx, dj, -c0)), mj[3 * j]);
                mj[3 * j + 1] = fmaf(sw, fmaf(k2, N[3 * j + 1], fmaf(vy, dj, -c1)), mj[3 * j + 1]);
                if (j < 2) {
                    const float c2 = fmaf(kx, Tj[1], -ky * Tj[0]);
                    mj[3 * j + 2] = fmaf(sw, fmaf(k2, N[3 * j + 2], fmaf(vz, dj, -c2)), mj[3 * j + 2]);
                }
            }
        }
    };
    bool pend = false;                           // the last tile's sums are still to be read
    float pdx = 0.f, pdy = 0.f, pdz = 0.f, pR = 0.f, pg = 0.f, py = 0.f;   // its d, 1/R and scales
    int slot = 2;                                // where the scales of the tile before are
    for (int base = 0; ok && base < ntiles; base += 32) {
        float iRl = 0.f;
        int cls = 0;
        if (wvalid && base + lane < ntiles) {   // 32 tiles, one a lane
            const TileHdr h = hdr[t0 + (base + lane) * tstep];
            cls = tile_class<K>(h, wch, wcl, wh, wdiag, iRl);
        }
        const unsigned far = __ballot_sync(0xffffffffu, cls == TILE_FAR);
        const unsigned mid = __ballot_sync(0xffffffffu, cls == TILE_MID);
        for (int part = base; ok && part < min(base + 32, ntiles); part += TC_MID) {
#pragma unroll 1
            for (int it = part; it < min(part + TC_MID, ntiles); it++) {
                const bool isfar = (far >> (it & 31)) & 1u;
                if (!isfar && !((mid >> (it & 31)) & 1u)) {
                    // not this warp's: its rows of A keep stale values and its sums are not read
                    ok = mbar_wait(&adone, 1u, rounds);      // the previous tile's second half
                    if (!ok) break;
                    tc_fence_after();
                    if (pend) { collect(scales[slot], pdx, pdy, pdz, pR, pg, py); tc_fence_before(); __syncwarp(); }
                    pend = false;
                    if (lane == 0) mbar_arrive(&afull);
                    ok = mbar_wait(&adone, 0u, rounds);
                    if (!ok) break;
                    if (lane == 0) mbar_arrive(&afull);
                    slot = slot == 2 ? 0 : slot + 1;
                    continue;
                }
                const char* r = stage[it & 1].rec;
                const float iR = __shfl_sync(0xffffffffu, iRl, it & 31);
                ok = mbar_wait(&bfull[it & 1], (uint32_t)(it >> 1) & 1u, rounds);
                if (!ok) break;
                const TileHdr& h = *(const TileHdr*)(r + TC_B + 4 * TC_POS);
                const float dx = ((th.x - h.chx) + (tl.x - h.clx)) * iR, dy = ((th.y - h.chy) + (tl.y - h.cly)) * iR,
                            dz = ((th.z - h.chz) + (tl.z - h.clz)) * iR;
                const float hg = h.gscale, hy = h.yscale;   // the stage is not read after the last arrival
#pragma unroll 1
                for (int hh = 0; hh < 2; hh++) {
                    const ulonglong2* p = (const ulonglong2*)(r + TC_B) + hh * 8;
                    if (isfar) {
                        uint32_t gh[8], gl[8], qh[8], ql[8];
                        weigh<K, 8>(p, dx, dy, dz, iR, gh, gl, qh, ql);   // while the last step's MMAs run
                        ok = mbar_wait(&adone, (uint32_t)(hh ^ 1), rounds);
                        if (!ok) break;
                        tc_fence_after();
                        store_a(ta, gh, gl, qh, ql);
                        if (hh == 0 && pend) collect(scales[slot], pdx, pdy, pdz, pR, pg, py);
                        weigh<K, 8>(p + 4, dx, dy, dz, iR, gh, gl, qh, ql);
                        store_a(ta + 8, gh, gl, qh, ql);
                    } else if constexpr (K == K_GAUSERF) {
                        ok = mbar_wait(&adone, (uint32_t)(hh ^ 1), rounds);
                        if (!ok) break;
                        tc_fence_after();
                        if (hh == 0 && pend) collect(scales[slot], pdx, pdy, pdz, pR, pg, py);
#pragma unroll 1
                        for (int c = 0; c < 4; c++) {
                            uint32_t gh[4], gl[4], qh[4], ql[4];
                            weigh<K, 4, true>(p + 2 * c, dx, dy, dz, iR, gh, gl, qh, ql);
                            tmem_st4(ta + 4 * c, gh);
                            tmem_st4(ta + 16 + 4 * c, gl);
                            tmem_st4(ta + 32 + 4 * c, qh);
                            tmem_st4(ta + 48 + 4 * c, ql);
                        }
                    }
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&afull);
                }
                if (!ok) break;
                pend = true;
                slot = slot == 2 ? 0 : slot + 1;
                pdx = dx; pdy = dy; pdz = dz; pR = iR; pg = hg; py = hy;
            }
            flush();
        }
    }
    if (ok) {
        ok = mbar_wait(&adone, 1u, rounds);
        tc_fence_after();
        if (ok && pend) collect(scales[slot], pdx, pdy, pdz, pR, pg, py);
    }
    if (!ok && lane == 0) failed = 1;

    // --------------------------------------------------- near tiles, pair by pair
    if (wvalid && ok) {
        float b2 = fmaf(to.x, to.x, fmaf(to.y, to.y, to.z * to.z));
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) b2 = fmaxf(b2, __shfl_xor_sync(0xffffffffu, b2, m));
        const float r2n = fmaxf(4.0f * b2, 1.0e-30f);
        const float3 oh = make_float3(__shfl_sync(0xffffffffu, th.x, 0), __shfl_sync(0xffffffffu, th.y, 0),
                                      __shfl_sync(0xffffffffu, th.z, 0));
        const float3 ol = make_float3(__shfl_sync(0xffffffffu, tl.x, 0), __shfl_sync(0xffffffffu, tl.y, 0),
                                      __shfl_sync(0xffffffffu, tl.z, 0));
        int in_mid = 0;
        for (int base = 0; base < ntiles; base += 32) {
            int cls = TILE_FAR;
            if (base + lane < ntiles) {
                const TileHdr h = hdr[t0 + (base + lane) * tstep];
                float iR;
                cls = tile_class<K>(h, wch, wcl, wh, wdiag, iR);
            }
            unsigned near = __ballot_sync(0xffffffffu, cls == TILE_NEAR);
            if (!near) continue;
            // sub-tiles of 32 sources, each loaded to registers while the one before is evaluated
            int sub = 0;
            SrcMixed p = src[(int64_t)(t0 + (base + __ffs(near) - 1) * tstep) * TCS + lane];
#pragma unroll 1
            while (near) {
                __syncwarp();   // every lane is done with the previous sub-tile
                near_s[warp][lane] = p;
                const float px = (p.a.x - oh.x) + (p.b.x - ol.x), py = (p.a.y - oh.y) + (p.b.y - ol.y),
                            pz = (p.a.z - oh.z) + (p.b.z - ol.z);
                near_o[warp][lane] = make_float4(px, py, pz, p.b.w * p.b.w);
                const float ex = fmaxf(fmaxf(blo.x - px, px - bhi.x), 0.0f);
                const float ey = fmaxf(fmaxf(blo.y - py, py - bhi.y), 0.0f);
                const float ez = fmaxf(fmaxf(blo.z - pz, pz - bhi.z), 0.0f);
                const float thr = singular_tail<K>() ? fmaxf(s_far<K>() * p.a.w, r2n) : r2n;
                const unsigned fb = __ballot_sync(0xffffffffu, fmaf(ex, ex, fmaf(ey, ey, ez * ez)) > thr);
                __syncwarp();
                if (sub) near &= near - 1;
                sub ^= 1;
                if (near) p = src[(int64_t)(t0 + (base + __ffs(near) - 1) * tstep) * TCS + sub * WT + lane];
                float u[3] = {0.f, 0.f, 0.f}, w[3] = {0.f, 0.f, 0.f}, jq[8];
#pragma unroll
                for (int k = 0; k < 8; k++) jq[k] = 0.f;
#pragma unroll 1
                for (int j = 0; j < WT; j += 4) {
                    if (((fb >> j) & 0xFu) == 0xFu)
                        pair4_far<K>(to, near_o[warp], near_s[warp], j, u, jq, w);
                    else
                        pair4_near<K>(th, tl, near_o[warp], near_s[warp], j, u, jq, w);
                }
#pragma unroll
                for (int k = 0; k < 3; k++) { mu[k] += u[k]; mw[k] += w[k]; }
#pragma unroll
                for (int k = 0; k < 8; k++) mj[k] += jq[k];
                if (sub == 0 && ++in_mid == TC_MID_NEAR) {
                    in_mid = 0;
                    flush();
                }
            }
        }
    }
    flush();
    tc_fence_before();
    __syncthreads();
    if (failed && threadIdx.x == 0) *(volatile int*)gave_up = 1;     // and the block's sums are NaN
    if (!valid) return;
    double f[14];
#pragma unroll
    for (int k = 0; k < 14; k++) f[k] = failed ? __longlong_as_double(0x7ff8000000000000LL) : acc64[k][threadIdx.x];
    double acc[12];
    uj_mixed_finish(f, acc);
    write_uj(t, me.idx, acc, U, ldU, J, ldJ, partial, nt_pad);
}

int uj_tc_splits(int64_t n, int num_sms)
{
    // two to six waves of resident blocks where there are tiles enough (near tiles make blocks
    // uneven), the least waves x (tiles a block + its fixed cost, about 3 tiles)
    const int64_t blocks = (n + UJ_THREADS - 1) / UJ_THREADS, tiles = tc_tiles(n), slots = 4LL * num_sms;
    int64_t lo = (2 * slots + blocks - 1) / blocks, hi = 6 * slots / blocks;
    if (lo > (tiles + 3) / 4) lo = (tiles + 3) / 4;
    if (hi > tiles) hi = tiles;
    int64_t best = lo, cost = INT64_MAX;
    for (int64_t s = lo; s <= hi; s++) {
        const int64_t c = ((blocks * s + slots - 1) / slots) * ((tiles + s - 1) / s + 3);
        if (c < cost) { cost = c; best = s; }
    }
    return (int)best;
}

template <int K>
static cudaError_t launch_k(const UJArgs& a, const TgtPos* tgt, const SrcMixed* src, const Workspace& w, int nsplit,
                            double* partial, int64_t nt_pad, cudaStream_t st)
{
    void* work = w.tiles;
    const int tiles = (int)tc_tiles(a.ns);
    TileHdr* hdr = (TileHdr*)work;
    char* rec = (char*)work + align128((size_t)tiles * sizeof(TileHdr));
    pack_tiles<K><<<tiles, TCS, 0, st>>>(a.ns, a.gs, a.sgs, tgt, hdr, rec);
    const dim3 grid((unsigned)(nt_pad / UJ_THREADS), (unsigned)nsplit);
    uj_tc_kernel<K><<<grid, TC_THREADS, 0, st>>>(a.nt, tgt, tiles, hdr, rec, src, a.U, a.ldU, a.J, a.ldJ, partial, nt_pad,
                                              (uint32_t)w.wait_rounds, w.gave_up);
    return cudaGetLastError();
}

cudaError_t launch_uj_tc(const UJArgs& a, const TgtPos* tgt, const SrcMixed* src, const Workspace& w,
                         int nsplit, double* partial, int64_t nt_pad, cudaStream_t st, int64_t* launches)
{
    *launches += 2;
    switch (a.kernel) {
    case K_SING: return launch_k<K_SING>(a, tgt, src, w, nsplit, partial, nt_pad, st);
    case K_GAUS: return launch_k<K_GAUS>(a, tgt, src, w, nsplit, partial, nt_pad, st);
    case K_GAUSERF: return launch_k<K_GAUSERF>(a, tgt, src, w, nsplit, partial, nt_pad, st);
    default: return launch_k<K_WNKLMNS>(a, tgt, src, w, nsplit, partial, nt_pad, st);
    }
}

}  // namespace vpm
