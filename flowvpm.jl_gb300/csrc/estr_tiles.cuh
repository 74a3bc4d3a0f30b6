// estr_tiles.cuh -- per-tile boxes of a source pack and the walk over the tiles within
// reach of a warp's targets, shared by the mixed Estr (estr.cu), its adjoint
// (estr_adjoint.cu) and the filter differences (dynamic.cu).  Their Gaussian terms fall
// below FP32 resolution past a reach (zeta_skip_s, dyn_skip_s), so whole 32-source tiles
// out of a warp's reach need not be loaded.
#pragma once
#include "dyn_math.cuh"
#include "internal.h"
#include "vpm_math.cuh"

namespace vpm {

constexpr int EST_TILE = 32;   // particles per tile (one per lane of a warp)

// The rounding of two FP32 offsets of size |o| changes a weight by dlog(zeta)/ds 2 sqrt(s) |o|/sigma
// 2^-24 or so, with |o| up to the box's extent E plus the distance.  Within E = 4 sigma that is at most
// 4 ulp of zeta(0) at any distance; in wider boxes sources nearer than 3 sigma to the box take
// both parts of the offsets (farther ones are below 3 ulp of zeta(0) up to E = 100 sigma, since zeta
// itself falls off).  A random cloud of 1,600 has E = 40 sigma, and its sums are a few close pairs: their
// SFS was 2e-6 of its norm off.  Rings of 60,000 and more stay on the offsets (E = 0.9 to 2.7 sigma for
// nine warps in ten).
constexpr float ESTR_WIDE = 16.0f;       // (E/sigma)^2
constexpr float ESTR_CLOSE = 9.0f;       // (distance from the box/sigma)^2

// A tile of sources for the mixed Estr kernels (estr.cu, leaflist.cu), in the form their inner loop
// reads: coordinates (x, y, z high parts, xl, yl, zl low
// parts; both turned into offsets in place by estr.cu) and w = 1/sigma^2 as arrays, so that one 16-byte broadcast read serves four sources and
// f32x2 instructions take two of them; and the payload g, v = ZNORM (Gamma, J^T Gamma)/sigma^3 as
// (gx gy)(gz vx)(vy vz), three f32x2 a source, 24 bytes instead of two float4.
struct __align__(128) EstrTile {
    float x[EST_TILE], y[EST_TILE], z[EST_TILE], w[EST_TILE], xl[EST_TILE], yl[EST_TILE], zl[EST_TILE];
    float2 gv[3 * EST_TILE];
};
static_assert(sizeof(EstrTile) == 1664, "whole 16-byte chunks, no padding");

// r^2 and s = r^2/sigma^2 of the tile's sources j .. j + 7 for a target at th + tl, from both
// parts of the positions: the rounding is of the displacement's own size.
__device__ __forceinline__ void estr_r2s8(const EstrTile& T, int j, const float3& th, const float3& tl, f32x2 (&r2)[4],
                                          f32x2 (&s)[4])
{
    const f32x2 HX = pk(-th.x, -th.x), HY = pk(-th.y, -th.y), HZ = pk(-th.z, -th.z);
    const f32x2 LX = pk(-tl.x, -tl.x), LY = pk(-tl.y, -tl.y), LZ = pk(-tl.z, -tl.z);
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const int i = j + 4 * c;
        const ulonglong2 X = *(const ulonglong2*)&T.x[i], Y = *(const ulonglong2*)&T.y[i],
                         Z = *(const ulonglong2*)&T.z[i], W = *(const ulonglong2*)&T.w[i],
                         XL = *(const ulonglong2*)&T.xl[i], YL = *(const ulonglong2*)&T.yl[i],
                         ZL = *(const ulonglong2*)&T.zl[i];
        f32x2 dx = add2(add2(X.x, HX), add2(XL.x, LX)), dy = add2(add2(Y.x, HY), add2(YL.x, LY)),
              dz = add2(add2(Z.x, HZ), add2(ZL.x, LZ));
        r2[2 * c] = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        s[2 * c] = mul2(r2[2 * c], W.x);
        dx = add2(add2(X.y, HX), add2(XL.y, LX)); dy = add2(add2(Y.y, HY), add2(YL.y, LY));
        dz = add2(add2(Z.y, HZ), add2(ZL.y, LZ));
        r2[2 * c + 1] = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        s[2 * c + 1] = mul2(r2[2 * c + 1], W.y);
    }
}

// ... from the high parts (offsets) alone
__device__ __forceinline__ void estr_r2s8(const EstrTile& T, int j, const float3& to, f32x2 (&r2)[4], f32x2 (&s)[4])
{
    const f32x2 TX = pk(-to.x, -to.x), TY = pk(-to.y, -to.y), TZ = pk(-to.z, -to.z);
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const int i = j + 4 * c;
        const ulonglong2 X = *(const ulonglong2*)&T.x[i], Y = *(const ulonglong2*)&T.y[i],
                         Z = *(const ulonglong2*)&T.z[i], W = *(const ulonglong2*)&T.w[i];
        f32x2 dx = add2(X.x, TX), dy = add2(Y.x, TY), dz = add2(Z.x, TZ);
        r2[2 * c] = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        s[2 * c] = mul2(r2[2 * c], W.x);
        dx = add2(X.y, TX); dy = add2(Y.y, TY); dz = add2(Z.y, TZ);
        r2[2 * c + 1] = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        s[2 * c + 1] = mul2(r2[2 * c + 1], W.y);
    }
}

// Payload sums of 8 sources: f[0..2] += z (gx gy)(gz vx)(vy vz) for the weights of r2/s pairs
// (s = r2/sigma^2).  MASKED: sources whose target mask (`mask`) lacks `bit` add nothing.
// ZERO: sources at r2 = 0 may be among them, which add nothing.
template <int K, bool ZETA, bool DZ, bool MASKED, bool ZERO>
__device__ __forceinline__ void estr_add8(const f32x2 (&r2)[4], const f32x2 (&s)[4], const float2* gv, unsigned bit,
                                          const uint4* mask, float3 fd, f32x2 (&f)[3])
{
    const ulonglong2* p = (const ulonglong2*)gv;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        float s0, s1;
        upk(s[q], s0, s1);
        float z0 = zhat_f32<K>(s0), z1 = zhat_f32<K>(s1);
        if constexpr (DZ) { z0 *= zeta_ratio_m1<K>(s0, fd); z1 *= zeta_ratio_m1<K>(s1, fd); }
        if constexpr (MASKED) {
            const uint4 m = mask[q >> 1];
            z0 = (q & 1 ? m.z : m.x) & bit ? z0 : 0.0f;
            z1 = (q & 1 ? m.w : m.y) & bit ? z1 : 0.0f;
        }
        if constexpr (ZERO) {
            float a, b;
            upk(r2[q], a, b);
            z0 = a == 0.0f ? 0.0f : z0;
            z1 = b == 0.0f ? 0.0f : z1;
        }
        const ulonglong2 a = p[3 * q], b = p[3 * q + 1], c = p[3 * q + 2];
        const f32x2 Z0 = pk(z0, z0), Z1 = pk(z1, z1);
        f[0] = fma2(Z0, a.x, f[0]);
        f[1] = fma2(Z0, a.y, f[1]);
        if constexpr (!ZETA) f[2] = fma2(Z0, b.x, f[2]);
        f[0] = fma2(Z1, b.y, f[0]);
        f[1] = fma2(Z1, c.x, f[1]);
        if constexpr (!ZETA) f[2] = fma2(Z1, c.y, f[2]);
    }
}

// The compensated sums sm + cm, added to FP64.  A branch of its own (the warp barriers): as a
// predicated block in the tile loop its FP64 instructions took their turn in the FP64 pipe for every
// tile (24 % busy).
__device__ __forceinline__ void estr_flush(f32x2 (&sm)[3], f32x2 (&cm)[3], double (&zg)[3], double (&zv)[3])
{
    __syncwarp();
    float a[6], c[6];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        upk(sm[k], a[2 * k], a[2 * k + 1]);
        upk(cm[k], c[2 * k], c[2 * k + 1]);
        sm[k] = cm[k] = 0ull;
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        zg[k] += (double)a[k] + (double)c[k];
        zv[k] += (double)a[3 + k] + (double)c[3 + k];
    }
    __syncwarp();
}

// The box of every 32-source tile of a pack of ns_pad sources (ns real ones): for tile i,
// box[2 i] = (min x, min y, min z, min 1/sigma^2) and box[2 i + 1] = (max x, max y, max z, 0)
// over its real sources, in FP32 (the high parts); a tile of padding has an empty box.
// Called by whole warps, one tile per warp (ns_pad is a multiple of 32).
__device__ __forceinline__ void estr_tile_box(int64_t o, int64_t ns, float xh, float yh, float zh, float isig2,
                                              float4* __restrict__ box)
{
    const bool real = o < ns;
    float lo[4] = {real ? xh : 3.0e38f, real ? yh : 3.0e38f, real ? zh : 3.0e38f, real ? isig2 : 3.0e38f};
    float hi[3] = {real ? xh : -3.0e38f, real ? yh : -3.0e38f, real ? zh : -3.0e38f};
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
#pragma unroll
        for (int k = 0; k < 4; k++) lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], m));
#pragma unroll
        for (int k = 0; k < 3; k++) hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], m));
    }
    if ((o & (EST_TILE - 1)) == 0) {
        box[2 * (o / EST_TILE)] = make_float4(lo[0], lo[1], lo[2], lo[3]);
        box[2 * (o / EST_TILE) + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
    }
}

// The tiles of a warp's share (every step-th of ntiles from `first`: a target's tiles in reach
// are its neighbours on the curve, so contiguous shares would leave them all to one split) that
// can be within reach of its targets, in order: lane l tests tile 32 c + l of chunk c against the targets' FP32 box (lo, hi) with the
// tile's box from the pack (estr_tile_box), a ballot gives the chunk's tiles in reach, and
// next() pops them.  A tile is out of reach when its box is farther than zeta_skip_s
// sigma^2 from the target box at the tile's largest sigma (every pair then has
// zeta/zeta(0) < 1e-13); the FP32 boxes shift that bound by a few ulp of the
// coordinates, where the weights are already far below the FP32 resolution of the sums.
// With wfix > 0 the test takes 1/sigma^2 = wfix instead of the tile's (the adjoint's second
// pass, whose tiles hold targets and whose sigma is the lanes' sources').  next_s takes the
// reach skip_s explicitly (the filter differences' dyn_skip_s); skip_s <= 0 or >= 1e37 (a
// kernel without a reach) takes every tile.  All 32 lanes call it, with the same values.
struct TileWalk {
    int n, c, first, step;
    unsigned mask;
    __device__ __forceinline__ void init(int ntiles, int first_ = 0, int step_ = 1)
    {
        n = (ntiles - first_ + step_ - 1) / step_;
        first = first_;
        step = step_;
        c = -1;
        mask = 0u;
    }
    template <int K>
    __device__ __forceinline__ int next(const float4* __restrict__ box, const float4 lo, const float4 hi, int lane,
                                        float wfix = 0.0f)
    {
        return next_s(box, lo, hi, lane, zeta_skip_s<K>(), wfix);
    }
    __device__ __forceinline__ int next_s(const float4* __restrict__ box, const float4 lo, const float4 hi, int lane,
                                          float skip_s, float wfix = 0.0f)
    {
        while (mask == 0u) {
            if ((c + 1) * 32 >= n) return -1;
            ++c;
            const int i = first + (c * 32 + lane) * step;
            bool in = c * 32 + lane < n;
            if (skip_s > 0.0f && skip_s < 1.0e37f && in) {
                const float4 bl = box[2 * i], bh = box[2 * i + 1];
                const float ex = fmaxf(fmaxf(lo.x - bh.x, bl.x - hi.x), 0.0f);
                const float ey = fmaxf(fmaxf(lo.y - bh.y, bl.y - hi.y), 0.0f);
                const float ez = fmaxf(fmaxf(lo.z - bh.z, bl.z - hi.z), 0.0f);
                in = !(fmaf(ex, ex, fmaf(ey, ey, ez * ez)) * (wfix > 0.0f ? wfix : bl.w) > skip_s);
            }
            mask = __ballot_sync(0xffffffffu, in);
        }
        const int b = __ffs(mask) - 1;
        mask &= mask - 1u;
        return first + (c * 32 + b) * step;
    }
};

}  // namespace vpm
