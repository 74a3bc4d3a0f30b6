// estr.cu -- SFS vortex-stretching pass Estr (src/FLOWVPM_subfilterscale_models.jl:16-92).
//
// The reference adds, for every non-static target t and non-static source s,
//     SFS_t += zeta(r/sigma_s)/sigma_s^3 * (J_t - J_s)^T Gamma_s      (transposed)
// This is evaluated in the exactly equivalent factored form
//     SFS_t += J_t^T Zg_t - Zv_t,   Zg_t = sum_s z_ts Gamma_s,  Zv_t = sum_s z_ts v_s,
// with z_ts = zeta(r/sigma_s)/sigma_s^3 and v_s = J_s^T Gamma_s (J_s Gamma_s for
// the classic scheme), so a source carries 10 numbers instead of 16 and a pair
// costs about 25 flop.  The self pair, which the reference includes but which
// contributes exactly zero there, is excluded by index (in the factored form
// its two terms would only cancel to rounding).  Static sources are packed with
// zero strength; static targets are left untouched.  Targets run in curve
// order (order.cu) like the UJ kernels.  The FP64 kernel takes
// zeta from r^2 with a table exponential or one rsqrt; the mixed kernel uses FP32 pair math on per-warp FP32 offsets
// (see uj.cu) and FP64 accumulation of FP32 blocks, and skips every pair at
// r = 0 (the self pair, and coincident particles, whose J are equal so that
// their reference term is zero; in the factored form their two terms would
// only cancel to FP32 rounding, at the largest weight zeta(0)).
#include "dyn_math.cuh"
#include "estr_tiles.cuh"
#include "internal.h"
#include "vpm_math.cuh"

#include <type_traits>

namespace vpm {

static inline int64_t round_up(int64_t a, int64_t b) { return (a + b - 1) / b * b; }

// Sources summed in plain FP32 before a compensated add.  J_t^T Zg - Zv is a
// difference of two sums far larger than itself (by |J| / |J_t - J_s| and by
// the cancellation of neighbours on either side of a target), so their FP32
// rounding is what limits the mixed Estr; sums of 8 added with compensation
// bring it from ~1e-5 to ~2e-6 of max |SFS| on a smooth field.
constexpr int ESTR_SUB = 8;

static_assert(UJ_BLOCK % ESTR_SUB == 0, "whole sub-blocks");

constexpr int EWT = EST_TILE;   // sources per tile of the mixed kernel's streams (one per lane)

size_t estr_src_pack_bytes(int64_t ns, int precision)
{
    const int64_t n = round_up(ns, UJ_TILE);
    // FP32-comp: the tiles, then two float4 a tile (estr_tile_box)
    return precision ? (size_t)(n / EWT) * (sizeof(EstrTile) + 2 * sizeof(float4))
                     : (size_t)n * sizeof(SrcEstrF64);
}

// v = J^T Gamma (transposed) or J Gamma (classic); J column-major 3x3.
__device__ __forceinline__ void stretch_vec(const double* J, double gx, double gy, double gz,
                                            bool transposed, double& vx, double& vy, double& vz)
{
    if (transposed) {
        vx = J[0] * gx + J[1] * gy + J[2] * gz;
        vy = J[3] * gx + J[4] * gy + J[5] * gz;
        vz = J[6] * gx + J[7] * gy + J[8] * gz;
    } else {
        vx = J[0] * gx + J[3] * gy + J[6] * gz;
        vy = J[1] * gx + J[4] * gy + J[7] * gz;
        vz = J[2] * gx + J[5] * gy + J[8] * gz;
    }
}

template <int K>
__global__ void pack_estr_mixed(int64_t ns, int64_t ns_pad, const double* __restrict__ xs,
                                const double* __restrict__ gs, const double* __restrict__ sgs,
                                const double* __restrict__ Js, int64_t ldJs,
                                const uint8_t* __restrict__ static_s, bool transposed,
                                const TgtPos* __restrict__ order, EstrTile* __restrict__ out,
                                float4* __restrict__ box)
{
    // with `order` (sources = targets) the pack follows the targets' curve order
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= ns_pad) return;   // whole warps: ns_pad is a multiple of 32
    float x[3] = {1.0e6f, 1.0e6f, 1.0e6f}, xl[3] = {0.f, 0.f, 0.f}, w = 1.f, g[3] = {0.f, 0.f, 0.f}, v[3] = {0.f, 0.f, 0.f};
    if (o < ns) {   // past ns: far away, no strength
        const int64_t i = order ? (int64_t)order[o].idx : o;
        const double isig = 1.0 / sgs[i];
        const double isig2 = isig * isig;
        w = (float)isig2;
        const bool off = static_s && static_s[i];
        const double k = off ? 0.0 : zeta_norm(K) * isig2 * isig;
        const double gx = gs[3 * i], gy = gs[3 * i + 1], gz = gs[3 * i + 2];
        double vv[3] = {0.0, 0.0, 0.0};   // the zeta field (Js null) needs no v
        if (Js) stretch_vec(Js + i * ldJs, gx, gy, gz, transposed, vv[0], vv[1], vv[2]);
#pragma unroll
        for (int m = 0; m < 3; m++) {
            const double c = xs[3 * i + m];
            x[m] = (float)c;
            xl[m] = (float)(c - (double)x[m]);
            g[m] = (float)(k * gs[3 * i + m]);
            v[m] = (float)(k * vv[m]);
        }
    }
    EstrTile& T = out[o / EWT];
    const int l = (int)(o % EWT);
    T.x[l] = x[0]; T.y[l] = x[1]; T.z[l] = x[2]; T.w[l] = w;
    T.xl[l] = xl[0]; T.yl[l] = xl[1]; T.zl[l] = xl[2];
    T.gv[3 * l] = make_float2(g[0], g[1]);
    T.gv[3 * l + 1] = make_float2(g[2], v[0]);
    T.gv[3 * l + 2] = make_float2(v[1], v[2]);
    estr_tile_box(o, ns, x[0], x[1], x[2], w, box);
}

template <int K>
__global__ void pack_estr_f64(int64_t ns, int64_t ns_pad, const double* __restrict__ xs,
                              const double* __restrict__ gs, const double* __restrict__ sgs,
                              const double* __restrict__ Js, int64_t ldJs,
                              const uint8_t* __restrict__ static_s, bool transposed,
                              SrcEstrF64* __restrict__ out)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= ns_pad) return;
    SrcEstrF64 p;
    if (i < ns) {
        const bool off = static_s && static_s[i];
        const double isig = 1.0 / sgs[i], k = off ? 0.0 : zeta_norm(K) * isig * isig * isig;
        const double gx = off ? 0.0 : k * gs[3 * i], gy = off ? 0.0 : k * gs[3 * i + 1],
                     gz = off ? 0.0 : k * gs[3 * i + 2];
        double vx = 0.0, vy = 0.0, vz = 0.0;
        if (Js) stretch_vec(Js + i * ldJs, gx, gy, gz, transposed, vx, vy, vz);
        p.xy = make_double2(xs[3 * i], xs[3 * i + 1]);
        p.z_isig = make_double2(xs[3 * i + 2], isig * isig);
        p.gxy = make_double2(gx, gy);
        p.gz_vx = make_double2(gz, vx);
        p.vyz = make_double2(vy, vz);
    } else {
        p.xy = make_double2(0.0, 0.0);
        p.z_isig = make_double2(0.0, 1.0);
        p.gxy = p.gz_vx = p.vyz = make_double2(0.0, 0.0);
    }
    out[i] = p;
}

// SFS contribution J_t^T Zg - Zv  (or J_t Zg - Zv), FP64.
__device__ __forceinline__ void estr_combine(const double* Jt, const double (&zg)[3], const double (&zv)[3],
                                             bool transposed, double (&out)[3])
{
    double sx, sy, sz;
    stretch_vec(Jt, zg[0], zg[1], zg[2], transposed, sx, sy, sz);
    out[0] = sx - zv[0];
    out[1] = sy - zv[1];
    out[2] = sz - zv[2];
}

__device__ __forceinline__ void write_estr(int64_t t, int64_t idx, const double (&o)[3], double* SFS, int64_t ldS,
                                           double* partial, int64_t nt_pad)
{
    if (partial) {
        double* p = partial + (int64_t)blockIdx.y * 3 * nt_pad + t;
        p[0] = o[0]; p[nt_pad] = o[1]; p[2 * nt_pad] = o[2];
    } else {
        SFS[idx * ldS] += o[0]; SFS[idx * ldS + 1] += o[1]; SFS[idx * ldS + 2] += o[2];
    }
}

__global__ void estr_reduce(int64_t nt, int nsplit, const double* __restrict__ partial, int64_t nt_pad,
                            const TgtPos* __restrict__ tgt, const uint8_t* __restrict__ static_t,
                            double* SFS, int64_t ldS)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const int64_t i = tgt[t].idx;
    if (static_t && static_t[i]) return;
    const double* p = partial + blockIdx.y * nt_pad + t;
    double s = 0.0;
#pragma unroll 8
    for (int sp = 0; sp < nsplit; sp++) s += p[(int64_t)sp * 3 * nt_pad];
    SFS[i * ldS + blockIdx.y] += s;
}

// With ZETA the kernels evaluate zeta_direct instead (src/FLOWVPM_viscous.jl:467-488):
// W_t += sum_s zeta(r/sigma_s)/sigma_s^3 Gamma_s over every source and target, the
// self pair included, written to the SFS output.
template <int K, bool ZETA>
__global__ void __launch_bounds__(UJ_THREADS)
estr_f64_kernel(int64_t nt, const TgtPos* __restrict__ tgt, const double* __restrict__ Jt, int64_t ldJt,
                const uint8_t* __restrict__ static_t, int64_t ns_pad, const SrcEstrF64* __restrict__ src,
                bool self, bool transposed, double* SFS, int64_t ldS, double* partial, int64_t nt_pad)
{
    __shared__ SrcEstrF64 tile[UJ_TILE];
    __shared__ double T[64];
    exp_table(T);
    const int64_t t = (int64_t)blockIdx.x * UJ_THREADS + threadIdx.x;
    double tx = 1.0e3, ty = 1.0e3, tz = 1.0e3;
    int64_t idx = -1;
    if (t < nt) {
        const TgtPos p = tgt[t];
        tx = p.x; ty = p.y; tz = p.z; idx = p.idx;
    }
    const bool valid = t < nt && (ZETA || !(static_t && static_t[idx]));
    const int64_t self_q = (self && !ZETA) ? split_position(idx, blockIdx.y, gridDim.y) : -1;
    double zg[3] = {0.0, 0.0, 0.0}, zv[3] = {0.0, 0.0, 0.0};
    const int64_t nq = split_count(ns_pad, blockIdx.y, gridDim.y);
    for (int64_t base = 0; base < nq; base += UJ_TILE) {
        __syncthreads();
        if (base + threadIdx.x < nq) tile[threadIdx.x] = src[split_source(base + threadIdx.x, blockIdx.y, gridDim.y)];
        __syncthreads();
        const int m = (int)min((int64_t)UJ_TILE, nq - base);
#pragma unroll 2
        for (int j = 0; j < m; j++) {
            const SrcEstrF64& p = tile[j];
            if (base + j == self_q) continue;
            const double dx = p.xy.x - tx, dy = p.xy.y - ty, dz = p.z_isig.x - tz;
            const double z = zhat_f64<K>((dx * dx + dy * dy + dz * dz) * p.z_isig.y, T);
            zg[0] += z * p.gxy.x; zg[1] += z * p.gxy.y; zg[2] += z * p.gz_vx.x;
            if constexpr (!ZETA) { zv[0] += z * p.gz_vx.y; zv[1] += z * p.vyz.x; zv[2] += z * p.vyz.y; }
        }
    }
    if (!valid) return;
    double o[3];
    if constexpr (ZETA) { o[0] = zg[0]; o[1] = zg[1]; o[2] = zg[2]; }
    else estr_combine(Jt + idx * ldJt, zg, zv, transposed, o);
    write_estr(t, idx, o, SFS, ldS, partial, nt_pad);
}

// 16-byte asynchronous global->shared copy (LDGSTS), L2-cached.
__device__ __forceinline__ void ecp_async16(void* smem, const void* gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void ecp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void ecp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

constexpr int ESTR_FLUSH_TILES = 24;     // evaluated warp tiles between FP64 adds (768 sources)

// The mixed Estr.  Each warp streams the sources on its own, 32 per tile,
// double-buffered with cp.async (no block-wide barrier); the loading lane
// converts its source to an FP32 offset from the warp's first target with
// FP32 double-float arithmetic (df_offset: rounded once), and each target's
// own offset is formed by the same operations, so that the self pair and
// coincident particles have
// r^2 == 0 exactly (they are skipped: their terms would only cancel to FP32
// rounding, at the largest weight).  Where the targets' box is wide against a source's
// core and the source close to it, the displacement takes in what the offsets' rounding left
// and is rounded to its own size: ESTR_WIDE, ESTR_CLOSE.  For the Gaussian kernels the terms past
// zeta_skip_s (zeta/zeta(0) < 1e-13: below the FP32 resolution of the sums) are
// skipped at three levels: a tile whose pack box is out of reach of the warp's
// targets is not loaded (TileWalk); of a loaded tile, the 8-source sub-blocks whose
// sources are all out of reach of the warp's target box, before their distances are
// formed, or of every target, after.  Sums: 8-source FP32 partials added with
// compensation (comp_add2), FP64 every ESTR_FLUSH_TILES evaluated tiles.
// Bound: shared-memory reads (74 % of the rate) and the FMA pipe (61 % busy).  With two sources to an f32x2
// instruction and 16-byte reads of four sources' coordinates a pair takes 18 issue slots; one
// source at a time from 64-byte records took 24 and 80 % of the shared-memory rate (every lane
// reads every source, and the records' copies and conversions met bank conflicts).  Rings of
// 200,000: 3.77 -> 3.15 ms; jet of 100,000, Winckelmans (no reach): 9.70 -> 8.69 ms (2.98 and
// 8.49 before the choice for coarse offsets).
// With DZ (the weight difference of the dynamic procedure's test filter,
// dynamic.cu) each weight zeta~(r, sigma_s) is replaced by
// zeta~(r, alpha sigma_s) - zeta~(r, sigma_s) = zeta~(r, sigma_s) (ratio - 1),
// ratio - 1 from zeta_ratio_m1 with the factors fd = (alpha^-3 - 1, alpha^-3, alpha^-2 - 1).
template <int K, bool ZETA, bool DZ = false>
__global__ void __launch_bounds__(UJ_THREADS)
estr_mixed_kernel(int64_t nt, const TgtPos* __restrict__ tgt, const double* __restrict__ Jt, int64_t ldJt,
                  const uint8_t* __restrict__ static_t, int64_t ns_pad, const EstrTile* __restrict__ src,
                  const float4* __restrict__ box, bool self, bool transposed, double* SFS,
                  int64_t ldS, double* partial, int64_t nt_pad, float3 fd = make_float3(0.f, 0.f, 0.f))
{
    __shared__ EstrTile stage[UJ_WARPS][2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t = (int64_t)blockIdx.x * UJ_THREADS + threadIdx.x;
    double tx = 0.0, ty = 0.0, tz = 0.0;
    int64_t idx = -1;
    if (t < nt) {
        const TgtPos p = tgt[t];
        tx = p.x; ty = p.y; tz = p.z; idx = p.idx;
    }
    const bool valid = t < nt && (ZETA || !(static_t && static_t[idx]));
    // warp origin: lane 0's target as a double-float
    const double ox = __shfl_sync(0xffffffffu, tx, 0), oy = __shfl_sync(0xffffffffu, ty, 0),
                 oz = __shfl_sync(0xffffffffu, tz, 0);
    const float3 oh = make_float3((float)ox, (float)oy, (float)oz);
    const float3 ol = make_float3((float)(ox - (double)oh.x), (float)(oy - (double)oh.y), (float)(oz - (double)oh.z));
    // the target's offset by the same FP32 double-float operations as the sources' (below);
    // padding lanes sit at the origin
    float3 to = make_float3(0.f, 0.f, 0.f), tr = to;      // and what its rounding left
    if (t < nt) {
        const float3 th = make_float3((float)tx, (float)ty, (float)tz);
        const float3 tl = make_float3((float)(tx - (double)th.x), (float)(ty - (double)th.y),
                                      (float)(tz - (double)th.z));
        to = make_float3(df_offset(th.x, tl.x, oh.x, ol.x, tr.x), df_offset(th.y, tl.y, oh.y, ol.y, tr.y),
                         df_offset(th.z, tl.z, oh.z, ol.z, tr.z));
    }
    // the warp's target boxes: offsets (for the per-source test of a tile) and FP32
    // positions of its targets (for the tile boxes of the pack); [0], [1] = offsets low,
    // high; [2], [3] = positions low, high (empty without a target)
    __shared__ float4 wbox[UJ_WARPS][4];
    float ext;
    {
        float v[12] = {to.x, to.y, to.z, -to.x, -to.y, -to.z};
        const bool real = t < nt;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float h = (float)(k == 0 ? tx : k == 1 ? ty : tz);
            v[6 + k] = real ? h : 3.0e38f;
            v[9 + k] = real ? -h : 3.0e38f;
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1)
#pragma unroll
            for (int k = 0; k < 12; k++) v[k] = fminf(v[k], __shfl_xor_sync(0xffffffffu, v[k], m));
        ext = fmaxf(fmaxf(-v[3] - v[0], -v[4] - v[1]), -v[5] - v[2]);
        if (lane == 0) {
            wbox[warp][0] = make_float4(v[0], v[1], v[2], 0.f);
            wbox[warp][1] = make_float4(-v[3], -v[4], -v[5], 0.f);
            wbox[warp][2] = make_float4(v[6], v[7], v[8], 0.f);
            wbox[warp][3] = make_float4(-v[9], -v[10], -v[11], 0.f);
        }
        __syncwarp();
    }
    double zg[3] = {0.0, 0.0, 0.0}, zv[3] = {0.0, 0.0, 0.0};
    f32x2 sm[3] = {0ull, 0ull, 0ull}, cm[3] = {0ull, 0ull, 0ull};   // compensated sums (gx gy)(gz vx)(vy vz)
    const float ext2 = ext * ext;
    auto load = [&](int tile, int b) {   // 104 chunks of 16 bytes
        const float4* g = (const float4*)&src[tile];
        float4* d = (float4*)&stage[warp][b];
#pragma unroll
        for (int q = 0; q < 3; q++) ecp_async16(d + 32 * q + lane, g + 32 * q + lane);
        if (lane < 8) ecp_async16(d + 96 + lane, g + 96 + lane);
        ecp_commit();
    };
    // the split's tiles within reach of the warp's targets, 32 tiles per ballot
    TileWalk walk;
    walk.init((int)(ns_pad / EWT), blockIdx.y, gridDim.y);
    int cur = walk.next<K>(box, wbox[warp][2], wbox[warp][3], lane);
    if (cur >= 0) load(cur, 0);
    int in_flush = 0, buf = 0;
    while (cur >= 0) {
        const int nxt = walk.next<K>(box, wbox[warp][2], wbox[warp][3], lane);
        if (nxt >= 0) {
            load(nxt, buf ^ 1);
            ecp_wait<1>();
        } else {
            ecp_wait<0>();
        }
        __syncwarp();
        EstrTile& T = stage[warp][buf];
        // the tile's sources out of reach of the whole target box, those inside it, the only ones that
        // can be at r = 0 from a target, and those whose offsets are too coarse
        unsigned beyond, inside, coarse;
        {   // this lane's source: FP32 offset
            const float hx = T.x[lane], hy = T.y[lane], hz = T.z[lane], w = T.w[lane];
            const float lx = T.xl[lane], ly = T.yl[lane], lz = T.zl[lane];
            const float px = df_offset(hx, lx, oh.x, ol.x), py = df_offset(hy, ly, oh.y, ol.y),
                        pz = df_offset(hz, lz, oh.z, ol.z);
            T.x[lane] = px; T.y[lane] = py; T.z[lane] = pz;
            const float4 lo = wbox[warp][0], hi = wbox[warp][1];
            const float ex = fmaxf(fmaxf(lo.x - px, px - hi.x), 0.0f);
            const float ey = fmaxf(fmaxf(lo.y - py, py - hi.y), 0.0f);
            const float ez = fmaxf(fmaxf(lo.z - pz, pz - hi.z), 0.0f);
            const float d2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez)), ds = d2 * w;
            beyond = __ballot_sync(0xffffffffu, zeta_skip_s<K>() > 0.0f && ds > zeta_skip_s<K>());
            inside = __ballot_sync(0xffffffffu, !(d2 > 0.0f));
            coarse = __ballot_sync(0xffffffffu, ext2 * w > ESTR_WIDE && ds < ESTR_CLOSE);
            if (__builtin_expect(coarse != 0u, 0)) {
                float rx, ry, rz;
                df_offset(hx, lx, oh.x, ol.x, rx);
                df_offset(hy, ly, oh.y, ol.y, ry);
                df_offset(hz, lz, oh.z, ol.z, rz);
                T.xl[lane] = rx; T.yl[lane] = ry; T.zl[lane] = rz;
            }
        }
        __syncwarp();
        if (beyond != 0xffffffffu) {
            // (two loops cost dense fields, which take the second, 5 %; the choice inside one loop cost them 15,
            // a call for the first 5, and a pass of its own after the others 18)
            auto sources = [&](auto two_parts) {
#pragma unroll 1
                for (int sub = 0; sub < EWT; sub += ESTR_SUB) {
                    if (((beyond >> sub) & 0xffu) == 0xffu) continue;
                    f32x2 r2[4], s[4];
                    if (decltype(two_parts)::value && ((coarse >> sub) & 0xffu)) estr_r2s8(T, sub, to, tr, r2, s);
                    else estr_r2s8(T, sub, to, r2, s);
                    if (zeta_skip_s<K>() > 0.0f && __all_sync(0xffffffffu, min8_nan(s) > zeta_skip_s<K>())) continue;
                    f32x2 f[3] = {0ull, 0ull, 0ull};
                    if (!ZETA && ((inside >> sub) & 0xffu))
                        estr_add8<K, ZETA, DZ, false, !ZETA>(r2, s, &T.gv[3 * sub], 0u, nullptr, fd, f);
                    else
                        estr_add8<K, ZETA, DZ, false, false>(r2, s, &T.gv[3 * sub], 0u, nullptr, fd, f);
#pragma unroll
                    for (int k = 0; k < (ZETA ? 2 : 3); k++) comp_add2(sm[k], cm[k], f[k]);
                }
            };
            if (__builtin_expect(coarse != 0u, 0)) sources(std::true_type());
            else sources(std::false_type());
            // skipped tiles add nothing, so only the tiles taken count towards a flush
            if (++in_flush == ESTR_FLUSH_TILES) {
                in_flush = 0;
                estr_flush(sm, cm, zg, zv);
            }
        }
        __syncwarp();   // every lane is done with `buf` before it is refilled
        cur = nxt;
        buf ^= 1;
    }
    estr_flush(sm, cm, zg, zv);
    if (!valid) return;
    double o[3];
    if constexpr (ZETA) { o[0] = zg[0]; o[1] = zg[1]; o[2] = zg[2]; }
    else estr_combine(Jt + idx * ldJt, zg, zv, transposed, o);
    write_estr(t, idx, o, SFS, ldS, partial, nt_pad);
}

template <int K>
static cudaError_t launch_estr_k(const EstrArgs& a, const Workspace& w, int num_sms, cudaStream_t st,
                                 int64_t* launches)
{
    const int64_t ns_pad = round_up(a.ns, UJ_TILE);
    const int64_t nt_pad = round_up(a.nt, UJ_THREADS);
    const int nsplit = uj_num_splits(a.nt, a.ns, num_sms, a.precision, REACH_SPLITS);
    double* partial = nsplit > 1 ? w.partial : nullptr;
    const dim3 grid((unsigned)(nt_pad / UJ_THREADS), (unsigned)nsplit);
    const int pb = 256;
    const unsigned pgrid = (unsigned)((ns_pad + pb - 1) / pb);
    const TgtPos* tgt = nullptr;
    if (a.ordered) {
        tgt = ordered_targets(a.nt, w.order);
    } else {
        cudaError_t e = order_targets(a.nt, a.xt, w.order, w.order_bytes, st, launches, &tgt);
        if (e != cudaSuccess) return e;
    }
    const uint8_t* static_s = a.zeta ? nullptr : a.static_s;
    const uint8_t* static_t = a.zeta ? nullptr : a.static_t;
    if (a.dz_alpha > 0.0 && a.precision == 0) return cudaErrorInvalidValue;   // FP32-comp only
    if (a.precision == 0) {
        SrcEstrF64* src = (SrcEstrF64*)w.src_pack;
        pack_estr_f64<K><<<pgrid, pb, 0, st>>>(a.ns, ns_pad, a.xs, a.gs, a.sgs, a.zeta ? nullptr : a.Js, a.ldJs,
                                                static_s, a.transposed, src);
        if (a.zeta)
            estr_f64_kernel<K, true><<<grid, UJ_THREADS, 0, st>>>(a.nt, tgt, a.Jt, a.ldJt, static_t, ns_pad, src,
                                                                  a.self, a.transposed, a.SFS, a.ldS, partial,
                                                                  nt_pad);
        else
            estr_f64_kernel<K, false><<<grid, UJ_THREADS, 0, st>>>(a.nt, tgt, a.Jt, a.ldJt, static_t, ns_pad, src,
                                                                   a.self, a.transposed, a.SFS, a.ldS, partial,
                                                                   nt_pad);
    } else {
        EstrTile* src = (EstrTile*)w.src_pack;
        float4* box = (float4*)(src + ns_pad / EWT);   // the tile boxes follow the tiles
        pack_estr_mixed<K><<<pgrid, pb, 0, st>>>(a.ns, ns_pad, a.xs, a.gs, a.sgs, a.zeta ? nullptr : a.Js, a.ldJs,
                                                  static_s, a.transposed, a.self ? tgt : nullptr, src, box);
        if (a.zeta)
            estr_mixed_kernel<K, true><<<grid, UJ_THREADS, 0, st>>>(a.nt, tgt, a.Jt, a.ldJt, static_t, ns_pad, src,
                                                                    box, a.self, a.transposed, a.SFS,
                                                                    a.ldS, partial, nt_pad);
        else if (a.dz_alpha > 0.0) {
            const double al = a.dz_alpha;
            const float3 fd = make_float3((float)(1.0 / (al * al * al) - 1.0), (float)(1.0 / (al * al * al)),
                                          (float)(1.0 / (al * al) - 1.0));
            estr_mixed_kernel<K, false, true><<<grid, UJ_THREADS, 0, st>>>(a.nt, tgt, a.Jt, a.ldJt, static_t, ns_pad,
                                                                           src, box, a.self, a.transposed,
                                                                           a.SFS, a.ldS, partial, nt_pad, fd);
        } else
            estr_mixed_kernel<K, false><<<grid, UJ_THREADS, 0, st>>>(a.nt, tgt, a.Jt, a.ldJt, static_t, ns_pad, src,
                                                                     box, a.self, a.transposed, a.SFS,
                                                                     a.ldS, partial, nt_pad);
    }
    *launches += 2;
    if (partial) {
        estr_reduce<<<dim3((unsigned)((a.nt + 127) / 128), 3), 128, 0, st>>>(a.nt, nsplit, partial, nt_pad, tgt,
                                                                   static_t, a.SFS, a.ldS);
        *launches += 1;
    }
    return cudaGetLastError();
}

cudaError_t launch_estr(const EstrArgs& a, const Workspace& w, int num_sms, cudaStream_t st,
                        int64_t* launches)
{
    if (a.nt <= 0 || a.ns <= 0) return cudaSuccess;
    switch (a.kernel) {
    case K_SING: return launch_estr_k<K_SING>(a, w, num_sms, st, launches);
    case K_GAUS: return launch_estr_k<K_GAUS>(a, w, num_sms, st, launches);
    case K_GAUSERF: return launch_estr_k<K_GAUSERF>(a, w, num_sms, st, launches);
    case K_WNKLMNS: return launch_estr_k<K_WNKLMNS>(a, w, num_sms, st, launches);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace vpm
