// leaflist.cu -- near-field P2P over octree leaf pairs: the direct leg of
// UJ_fmm (FastMultipole's direct_list, src/FLOWVPM_UJ.jl:90-100) and the Estr
// pass over the same list (Estr_fmm!, src/FLOWVPM_subfilterscale_models.jl:94-188).
//
// Particles are processed in the tree's Morton order (nearfield.cu), so every
// leaf is a contiguous range.  Leaves are small (leaf_size is a maximum; a
// uniform cloud at leaf_size 64 averages ~11 particles a leaf), so work is not
// cut per leaf: one warp takes 32 consecutive Morton positions -- a few
// neighbouring leaves -- and walks the union of their source lists as
// particle intervals, each with the mask of the warp's leaves that need it.
// Sources are staged 32 at a time in the warp's shared memory, the tiles
// running on across interval boundaries so that they are full, each source
// carrying its interval's mask; a lane whose leaf is not in a source's mask
// computes that pair with zero weight.  Pair math is
// that of the all-pairs kernels (two sources to an f32x2 instruction for FP32-comp, uj_pair.cuh for
// FP64); Estr uses the factored form of estr.cu with the self
// pair excluded by position.
#include "dyn_math.cuh"
#include "estr_tiles.cuh"
#include "internal.h"
#include "uj_pair.cuh"
#include "vpm_math.cuh"

namespace vpm {

constexpr int NF_WARPS = 4;                  // warp groups per block
constexpr int NF_THREADS = 32 * NF_WARPS;
constexpr int NF_BLK_TILES = 2;              // 32-source tiles summed in FP32 per block
constexpr int NF_ESTR_FLUSH = 24;            // nf_estr: tiles of compensated FP32 sums between FP64 adds
// Resident blocks per SM the UJ kernel is compiled for; a fifth hides the Gaussian kernel's divergent
// branches (jet of 200,000: 4.05 -> 3.85 ms) and gains nothing elsewhere.
constexpr int nf_min_blocks(int kernel) { return kernel == K_GAUS ? 5 : 4; }
constexpr int NF_MID_BLKS = 4;               // blocks summed in FP32 before the FP64 add

__global__ void tgt_from_perm(int64_t n, const double* __restrict__ x, const int32_t* __restrict__ perm,
                              TgtPos* __restrict__ out)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t j = perm[i];
    TgtPos t;
    t.x = x[3 * j]; t.y = x[3 * j + 1]; t.z = x[3 * j + 2];
    t.idx = (int32_t)j; t.pad = 0;
    out[i] = t;
}

template <int K>
__global__ void leaf_pack_mixed(int64_t n, const double* __restrict__ x, const double* __restrict__ gs,
                                const double* __restrict__ sgs, const int32_t* __restrict__ perm,
                                SrcMixed* __restrict__ out)
{
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= n) return;
    const int64_t i = perm[o];
    const double px = x[3 * i], py = x[3 * i + 1], pz = x[3 * i + 2];
    const float xh = (float)px, yh = (float)py, zh = (float)pz;
    const double sig = (K == K_SING) ? 1.0 : sgs[i];
    const double k = singular_tail<K>() ? -C4 : -C4 / (sig * sig * sig);
    SrcMixed p;
    p.a = make_float4(xh, yh, zh, (float)(sig * sig));
    p.b = make_float4((float)(px - (double)xh), (float)(py - (double)yh), (float)(pz - (double)zh), (float)(1.0 / sig));
    p.gam = make_float4((float)(k * gs[3 * i]), (float)(k * gs[3 * i + 1]), (float)(k * gs[3 * i + 2]), 0.f);
    out[o] = p;
}

template <int K>
__global__ void leaf_pack_f64(int64_t n, const double* __restrict__ x, const double* __restrict__ gs,
                              const double* __restrict__ sgs, const int32_t* __restrict__ perm,
                              SrcF64* __restrict__ out)
{
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= n) return;
    const int64_t i = perm[o];
    const double sig = (K == K_SING) ? 1.0 : sgs[i];
    SrcF64 p;
    p.xy = make_double2(x[3 * i], x[3 * i + 1]);
    p.z_isig = make_double2(x[3 * i + 2], 1.0 / sig);
    p.gxy = make_double2(gs[3 * i], gs[3 * i + 1]);
    // .y: for Gaussian-erf the r^2 past which g = 1, g' = 0 (pair_f64_acc), else sigma
    p.gz_sig = make_double2(gs[3 * i + 2], K == K_GAUSERF ? 81.0 * sig * sig : sig);
    out[o] = p;
}

// Estr source payloads in Morton order (v = J^T Gamma or J Gamma, zero for static sources;
// Js = NULL: v = 0, the zeta sum's payload).
template <int K>
__global__ void leaf_pack_estr(int64_t n, const double* __restrict__ x, const double* __restrict__ gs,
                               const double* __restrict__ sgs, const double* __restrict__ Js,
                               const uint8_t* __restrict__ static_s, bool transposed,
                               const int32_t* __restrict__ perm, int precision, void* __restrict__ out)
{
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= n) return;
    const int64_t i = perm[o];
    const bool off = static_s && static_s[i];
    const double gx = gs[3 * i], gy = gs[3 * i + 1], gz = gs[3 * i + 2];
    double vx = 0.0, vy = 0.0, vz = 0.0;
    if (Js) {
        const double* J = Js + 9 * i;
        if (transposed) {
            vx = J[0] * gx + J[1] * gy + J[2] * gz; vy = J[3] * gx + J[4] * gy + J[5] * gz; vz = J[6] * gx + J[7] * gy + J[8] * gz;
        } else {
            vx = J[0] * gx + J[3] * gy + J[6] * gz; vy = J[1] * gx + J[4] * gy + J[7] * gz; vz = J[2] * gx + J[5] * gy + J[8] * gz;
        }
    }
    const double isig = 1.0 / sgs[i];
    if (precision) {   // the position as a double-float, so that the kernel's staging is plain loads
        const double k = off ? 0.0 : zeta_norm(K) * isig * isig * isig;
        const double px = x[3 * i], py = x[3 * i + 1], pz = x[3 * i + 2];
        const float xh = (float)px, yh = (float)py, zh = (float)pz;
        SrcEstrDF p;
        p.a = make_float4(xh, yh, zh, (float)(isig * isig));
        p.b = make_float4((float)(px - (double)xh), (float)(py - (double)yh), (float)(pz - (double)zh), 0.f);
        p.g = make_float4((float)(k * gx), (float)(k * gy), (float)(k * gz), 0.f);
        p.v = make_float4((float)(k * vx), (float)(k * vy), (float)(k * vz), 0.f);
        ((SrcEstrDF*)out)[o] = p;
    } else {
        const double m = off ? 0.0 : 1.0;
        SrcEstrF64 p;
        p.xy = make_double2(x[3 * i], x[3 * i + 1]);
        p.z_isig = make_double2(x[3 * i + 2], isig);
        p.gxy = make_double2(m * gx, m * gy);
        p.gz_vx = make_double2(m * gz, m * vx);
        p.vyz = make_double2(m * vy, m * vz);
        ((SrcEstrF64*)out)[o] = p;
    }
}

// Warp-group geometry shared by the kernels: this lane's target (FP64
// position, caller index) and its bit in the interval masks (its leaf relative
// to the group's first leaf; 0 for the padding lanes of the last group).
struct GroupTarget {
    double tx, ty, tz;
    int32_t idx;
    unsigned bit;
    bool valid;
};

__device__ __forceinline__ GroupTarget group_target(int64_t n, int64_t p0, int lane, const TgtPos* __restrict__ tgt,
                                                    const int32_t* __restrict__ leaf_of)
{
    GroupTarget g;
    const int64_t t = p0 + lane;
    g.valid = t < n;
    const TgtPos p = tgt[g.valid ? t : p0];
    g.tx = p.x; g.ty = p.y; g.tz = p.z; g.idx = p.idx;
    g.bit = g.valid ? 1u << (leaf_of[t] - leaf_of[p0]) : 0u;
    return g;
}

// A launch of few groups (20,000 particles: 157 blocks) gives each group to gridDim.y warps, part
// p taking every gridDim.y-th tile of its walk from the p-th; their sums go to `partial` and
// leaf_reduce adds them, in part order, to the outputs.
struct PartTurn {
    int turn, parts;
    __device__ __forceinline__ PartTurn() : turn(blockIdx.y), parts(gridDim.y) {}
    __device__ __forceinline__ bool mine()      // whether the walk's next tile is this part's
    {
        if (turn == 0) { turn = parts - 1; return true; }
        turn--;
        return false;
    }
};

__global__ void leaf_reduce(int64_t n, int parts, int na, int nb, const double* __restrict__ partial, int64_t n_pad,
                            const TgtPos* __restrict__ tgt, const uint8_t* __restrict__ skip, double* __restrict__ A,
                            double* __restrict__ B)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int64_t i = tgt[t].idx;
    if (skip && skip[i]) return;                 // static targets of Estr
    const int k = blockIdx.y, nk = na + nb;
    const double* p = partial + k * n_pad + t;
    double s = 0.0;
#pragma unroll 4
    for (int q = 0; q < parts; q++) s += p[(int64_t)q * nk * n_pad];
    if (k < na) A[na * i + k] += s;
    else B[nb * i + (k - na)] += s;
}

// Walks a group's intervals 32 sources at a time, across interval boundaries,
// so that tiles are full.  Lane i keeps interval wbase + i of a 32-interval
// window in registers; the walk itself is warp-uniform.
struct IntervalWalk {
    const int4* ivs;
    int e, e1, off, wbase;
    int4 win;

    __device__ __forceinline__ void init(const int4* v, int e0, int e_end, int lane)
    {
        ivs = v; e = e0; e1 = e_end; off = 0; wbase = e0;
        win = (e0 + lane < e_end) ? ivs[e0 + lane] : make_int4(0, 0, 0, 0);
    }
    // Next tile: this lane's source position (-1 for none) and target mask; returns the tile's size.
    __device__ __forceinline__ int next(int lane, int& my_p, unsigned& my_mask)
    {
        int filled = 0;
        my_p = -1;
        my_mask = 0u;
        while (filled < 32 && e < e1) {
            if (e - wbase >= 32) {
                wbase = e;
                win = (wbase + lane < e1) ? ivs[wbase + lane] : make_int4(0, 0, 0, 0);
            }
            const int k = e - wbase;
            const int p0 = __shfl_sync(0xffffffffu, win.x, k);
            const int p1 = __shfl_sync(0xffffffffu, win.y, k);
            const unsigned m = (unsigned)__shfl_sync(0xffffffffu, win.z, k);
            const int take = min(p1 - p0 - off, 32 - filled);
            if (lane >= filled && lane < filled + take) {
                my_p = p0 + off + (lane - filled);
                my_mask = m;
            }
            filled += take;
            off += take;
            if (off == p1 - p0) { e++; off = 0; }
        }
        return filled;
    }
};

// ------------------------------------------------------------- UJ, FP32-comp
// Sources of nf_uj_mixed: the double-float position with 1/sigma^2 in a.w, and
// gam = -Gamma/(4 pi sigma^3) for every kernel (the near form's sigma^-3 taken once).
template <int K>
__global__ void leaf_pack_lane(int64_t n, const double* __restrict__ x, const double* __restrict__ gs,
                               const double* __restrict__ sgs, const int32_t* __restrict__ perm,
                               SrcMixed* __restrict__ out)
{
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= n) return;
    const int64_t i = perm[o];
    const double px = x[3 * i], py = x[3 * i + 1], pz = x[3 * i + 2];
    const float xh = (float)px, yh = (float)py, zh = (float)pz;
    const double sig = (K == K_SING) ? 1.0 : sgs[i];
    const double k = -C4 / (sig * sig * sig);
    SrcMixed p;
    p.a = make_float4(xh, yh, zh, (float)(1.0 / (sig * sig)));
    p.b = make_float4((float)(px - (double)xh), (float)(py - (double)yh), (float)(pz - (double)zh), 0.f);
    p.gam = make_float4((float)(k * gs[3 * i]), (float)(k * gs[3 * i + 1]), (float)(k * gs[3 * i + 2]), 0.f);
    out[o] = p;
}

// A tile of nf_uj_mixed: minus the positions (nx, ny, nz + their low parts), w = 1/sigma^2, the
// strength and its negative (f32x2 instructions have no subtraction), as arrays, so that a 16-byte
// broadcast read serves four sources and an f32x2 instruction takes two.
struct __align__(16) UjTile {
    float nx[32], ny[32], nz[32], w[32], nxl[32], nyl[32], nzl[32];
    float g[3][32], ng[3][32];
    unsigned mask[32];
};

// Box of a warp's targets, by its lane 0 to box[0..1]: their FP32 high parts, widened by 2^-21 of
// the coordinates, more than what the low parts of targets and sources can add to a distance.
__device__ __forceinline__ void target_box(const float3& th, int lane, float4* box)
{
    float3 lo = th, hi = th;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
        lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, m)); hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, m));
        lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, m)); hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, m));
        lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, m)); hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, m));
    }
    if (lane == 0) {
        const float d = 4.76837158203125e-07f * fmaxf(fmaxf(fmaxf(fabsf(lo.x), fabsf(hi.x)), fmaxf(fabsf(lo.y), fabsf(hi.y))),
                                                      fmaxf(fabsf(lo.z), fabsf(hi.z)));
        box[0] = make_float4(lo.x - d, lo.y - d, lo.z - d, 0.f);
        box[1] = make_float4(hi.x + d, hi.y + d, hi.z + d, 0.f);
    }
    __syncwarp();
}

// Squared distance of a source (high parts) from that box; 0 (or NaN) inside.
__device__ __forceinline__ float box_d2(const float4* box, float x, float y, float z)
{
    const float4 lo = box[0], hi = box[1];
    const float ex = fmaxf(fmaxf(lo.x - x, x - hi.x), 0.0f);
    const float ey = fmaxf(fmaxf(lo.y - y, y - hi.y), 0.0f);
    const float ez = fmaxf(fmaxf(lo.z - z, z - hi.z), 0.0f);
    return fmaf(ex, ex, fmaf(ey, ey, ez * ez));
}

// The two halves of an f32x2 sum.
__device__ __forceinline__ float halves(f32x2 v)
{
    float a, b;
    upk(v, a, b);
    return a + b;
}

// Sums of four sources at a time, two to an instruction.  Masks and r = 0 are looked at only in
// groups of four where a source does not act on all of the group's targets or lies inside their
// box, the series form of Gaussian-erf (s < 2) only where one is that near to the box.
// Bound: the FMA pipe; f32x2 instructions with three distinct operands take about 2.4 of its cycles
// (62 % busy at 2), and the issue slots fell from 82 % to 56 %.  Kernel at jet 2^20 10.0 -> 9.3 ms
// against one source at a time with masks, r = 0 and form looked at in every pair; errors 0.65
// times as large, each half being a sum of its own.  Tried: offsets from the group's first target
// for sources far enough away (3 operations instead of 9 for a displacement): 4 % slower, few are.
template <int K>
__global__ void __launch_bounds__(NF_THREADS, nf_min_blocks(K))
nf_uj_mixed(int64_t n, int64_t ngroups, const TgtPos* __restrict__ tgt, const int32_t* __restrict__ leaf_of,
            const int32_t* __restrict__ grp_row, const int4* __restrict__ ivs, const SrcMixed* __restrict__ src,
            double* U, double* J, double* __restrict__ partial, int64_t n_pad)
{
    __shared__ UjTile tiles_s[NF_WARPS];
    __shared__ float4 box[NF_WARPS][2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t grp = (int64_t)blockIdx.x * NF_WARPS + warp;
    if (grp >= ngroups) return;
    const int64_t p0 = 32 * grp;
    const GroupTarget me = group_target(n, p0, lane, tgt, leaf_of);
    const float3 th = make_float3((float)me.tx, (float)me.ty, (float)me.tz);
    const float3 tl = make_float3((float)(me.tx - (double)th.x), (float)(me.ty - (double)th.y),
                                  (float)(me.tz - (double)th.z));
    target_box(th, lane, box[warp]);
    const unsigned all = __reduce_or_sync(0xffffffffu, me.bit);
    const f32x2 HX = pk(th.x, th.x), HY = pk(th.y, th.y), HZ = pk(th.z, th.z);
    const f32x2 LX = pk(tl.x, tl.x), LY = pk(tl.y, tl.y), LZ = pk(tl.z, tl.z);

    // sums of this lane ([0..2] U, [3..5] W, [6..13] J'): FP32 over NF_BLK_TILES tiles in registers,
    // FP32 over NF_MID_BLKS of those and FP64 in shared memory
    __shared__ double acc64[14][NF_THREADS];
    __shared__ float mid[14][NF_THREADS];
#pragma unroll
    for (int k = 0; k < 14; k++) { acc64[k][threadIdx.x] = 0.0; mid[k][threadIdx.x] = 0.f; }
    f32x2 a[14];
#pragma unroll
    for (int k = 0; k < 14; k++) a[k] = 0ull;
    int tiles = 0, blks = 0;
    PartTurn part;
    IntervalWalk walk;
    walk.init(ivs, grp_row[grp], grp_row[grp + 1], lane);
    UjTile& T = tiles_s[warp];
    for (;;) {
        int sp;
        unsigned smask;
        const int cnt = walk.next(lane, sp, smask);
        if (cnt == 0) break;
        if (!part.mine()) continue;
        SrcMixed sj;
        if (sp >= 0) {
            sj = src[sp];
        } else {   // padding: far away, no strength, no target
            sj.a = make_float4(1.0e6f, 1.0e6f, 1.0e6f, 1.f);
            sj.b = sj.gam = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();
        T.nx[lane] = -sj.a.x; T.ny[lane] = -sj.a.y; T.nz[lane] = -sj.a.z; T.w[lane] = sj.a.w;
        T.nxl[lane] = -sj.b.x; T.nyl[lane] = -sj.b.y; T.nzl[lane] = -sj.b.z;
        T.g[0][lane] = sj.gam.x; T.g[1][lane] = sj.gam.y; T.g[2][lane] = sj.gam.z;
        T.ng[0][lane] = -sj.gam.x; T.ng[1][lane] = -sj.gam.y; T.ng[2][lane] = -sj.gam.z;
        T.mask[lane] = smask;
        const float d2 = box_d2(box[warp], sj.a.x, sj.a.y, sj.a.z);
        const unsigned care = __ballot_sync(0xffffffffu, !(d2 > 0.0f) || (smask & all) != all);
        const unsigned close = __ballot_sync(0xffffffffu, !(d2 * sj.a.w > 2.01f));   // 2, and room for roundings
        __syncwarp();
#pragma unroll 1
        for (int j = 0; j < cnt; j += 4) {   // cnt <= 32: j + 3 stays in the tile
            const bool series = ((close >> j) & 0xfu) != 0u;
            f32x2 dx[2], dy[2], dz[2], r2[2], G[2], Q[2];
            {
                const ulonglong2 X = *(const ulonglong2*)&T.nx[j], Y = *(const ulonglong2*)&T.ny[j],
                                 Z = *(const ulonglong2*)&T.nz[j], XL = *(const ulonglong2*)&T.nxl[j],
                                 YL = *(const ulonglong2*)&T.nyl[j], ZL = *(const ulonglong2*)&T.nzl[j],
                                 W = *(const ulonglong2*)&T.w[j];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    dx[q] = add2(add2(HX, q ? X.y : X.x), add2(LX, q ? XL.y : XL.x));
                    dy[q] = add2(add2(HY, q ? Y.y : Y.x), add2(LY, q ? YL.y : YL.x));
                    dz[q] = add2(add2(HZ, q ? Z.y : Z.x), add2(LZ, q ? ZL.y : ZL.x));
                    r2[q] = fma2(dx[q], dx[q], fma2(dy[q], dy[q], mul2(dz[q], dz[q])));
                }
                const f32x2 w[2] = {W.x, W.y}, s[2] = {mul2(r2[0], W.x), mul2(r2[1], W.y)};
                near_GQ2<K, 2>(s, w, series, G, Q);
            }
            if ((care >> j) & 0xfu) {
                const uint4 m = *(const uint4*)&T.mask[j];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    float r0, r1, g0, g1, q0, q1;
                    upk(r2[q], r0, r1);
                    upk(G[q], g0, g1);
                    upk(Q[q], q0, q1);
                    const bool on0 = r0 > 0.0f && ((q ? m.z : m.x) & me.bit), on1 = r1 > 0.0f && ((q ? m.w : m.y) & me.bit);
                    G[q] = pk(on0 ? g0 : 0.f, on1 ? g1 : 0.f);
                    Q[q] = pk(on0 ? q0 : 0.f, on1 ? q1 : 0.f);
                }
            }
            const ulonglong2 GX = *(const ulonglong2*)&T.g[0][j], GY = *(const ulonglong2*)&T.g[1][j],
                             GZ = *(const ulonglong2*)&T.g[2][j], NX = *(const ulonglong2*)&T.ng[0][j],
                             NY = *(const ulonglong2*)&T.ng[1][j], NZ = *(const ulonglong2*)&T.ng[2][j];
#pragma unroll
            for (int q = 0; q < 2; q++) {   // accum_pair
                const f32x2 gx = q ? GX.y : GX.x, gy = q ? GY.y : GY.x, gz = q ? GZ.y : GZ.x;
                const f32x2 cx = fma2(dy[q], gz, mul2(dz[q], q ? NY.y : NY.x));
                const f32x2 cy = fma2(dz[q], gx, mul2(dx[q], q ? NZ.y : NZ.x));
                const f32x2 cz = fma2(dx[q], gy, mul2(dy[q], q ? NX.y : NX.x));
                a[0] = fma2(G[q], cx, a[0]);
                a[1] = fma2(G[q], cy, a[1]);
                a[2] = fma2(G[q], cz, a[2]);
                a[3] = fma2(G[q], gx, a[3]);
                a[4] = fma2(G[q], gy, a[4]);
                a[5] = fma2(G[q], gz, a[5]);
                const f32x2 bx = mul2(Q[q], cx), by = mul2(Q[q], cy), bz = mul2(Q[q], cz);
                a[6] = fma2(bx, dx[q], a[6]);
                a[7] = fma2(by, dx[q], a[7]);
                a[8] = fma2(bz, dx[q], a[8]);
                a[9] = fma2(bx, dy[q], a[9]);
                a[10] = fma2(by, dy[q], a[10]);
                a[11] = fma2(bz, dy[q], a[11]);
                a[12] = fma2(bx, dz[q], a[12]);
                a[13] = fma2(by, dz[q], a[13]);
            }
        }
        if (++tiles == NF_BLK_TILES) {
            tiles = 0;
            __syncwarp();   // these flushes are branches of their own, not predicated
            const bool up = ++blks == NF_MID_BLKS;
#pragma unroll
            for (int k = 0; k < 14; k++) {
                mid[k][threadIdx.x] += halves(a[k]);
                a[k] = 0ull;
            }
            if (up) {
                blks = 0;
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 14; k++) {
                    acc64[k][threadIdx.x] += (double)mid[k][threadIdx.x];
                    mid[k][threadIdx.x] = 0.f;
                }
                __syncwarp();
            }
        }
    }
    double f[14], acc[12];
#pragma unroll
    for (int k = 0; k < 14; k++) f[k] = acc64[k][threadIdx.x] + ((double)mid[k][threadIdx.x] + (double)halves(a[k]));
    if (!me.valid) return;
    uj_mixed_finish(f, acc);
    write_uj(p0 + lane, me.idx, acc, U, 3, J, 9, partial, n_pad);
}

// ------------------------------------------- dynamic procedure, FP32-comp
// dJ_t += the test-filter difference of every near pair's J term,
// j(dx, Gamma_s, alpha sigma_s) - j(dx, Gamma_s, sigma_s), evaluated as a
// difference (dynamic.cu) over the group's intervals, four pairs at a time
// without branches (masked pairs and pairs at r = 0 add zero); M as in
// filter_diff.  No far vote: near-list pairs are almost all within reach.
template <int K, int M>
__global__ void __launch_bounds__(NF_THREADS)
nf_filter_diff(int64_t n, int64_t ngroups, const TgtPos* __restrict__ tgt, const int32_t* __restrict__ leaf_of,
               const int32_t* __restrict__ grp_row, const int4* __restrict__ ivs, const SrcMixed* __restrict__ src,
               float hm, int panels, double* dJ, double* __restrict__ partial, int64_t n_pad)
{
    __shared__ SrcMixed tile[NF_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t grp = (int64_t)blockIdx.x * NF_WARPS + warp;
    if (grp >= ngroups) return;
    const int64_t p0 = 32 * grp;
    const GroupTarget me = group_target(n, p0, lane, tgt, leaf_of);
    const float3 th = make_float3((float)me.tx, (float)me.ty, (float)me.tz);
    const float3 tl = make_float3((float)(me.tx - (double)th.x), (float)(me.ty - (double)th.y),
                                  (float)(me.tz - (double)th.z));
    double acc[9];
    float f[9];
#pragma unroll
    for (int k = 0; k < 9; k++) { acc[k] = 0.0; f[k] = 0.f; }
    int tiles = 0;
    PartTurn part;
    IntervalWalk walk;
    walk.init(ivs, grp_row[grp], grp_row[grp + 1], lane);
    for (;;) {
        int sp;
        unsigned smask;
        const int cnt = walk.next(lane, sp, smask);
        if (cnt == 0) break;
        if (!part.mine()) continue;
        SrcMixed sj;
        if (sp >= 0) {
            sj = src[sp];
        } else {   // padding: far away, no strength, no target
            sj.a = make_float4(1.0e6f, 1.0e6f, 1.0e6f, 1.f);
            sj.b = make_float4(0.f, 0.f, 0.f, 1.f);
            sj.gam = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        sj.gam.w = __uint_as_float(smask);
        __syncwarp();
        tile[warp][lane] = sj;
        __syncwarp();
        for (int j0 = 0; j0 < cnt; j0 += 4) {   // cnt <= 32: j0 + 3 stays in the tile
            float ex[4], ey[4], ez[4], r2[4];
            bool on[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const SrcMixed& s = tile[warp][j0 + q];
                ex[q] = (th.x - s.a.x) + (tl.x - s.b.x);
                ey[q] = (th.y - s.a.y) + (tl.y - s.b.y);
                ez[q] = (th.z - s.a.z) + (tl.z - s.b.z);
                r2[q] = fmaf(ex[q], ex[q], fmaf(ey[q], ey[q], ez[q] * ez[q]));
                on[q] = (__float_as_uint(s.gam.w) & me.bit) != 0u && r2[q] > 0.0f;
                r2[q] = on[q] ? r2[q] : 1.0f;
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                filter_diff_pair<K, M>(ex[q], ey[q], ez[q], r2[q], tile[warp][j0 + q].b.w, tile[warp][j0 + q].gam, hm,
                                       panels, on[q], f);
        }
        if (++tiles == NF_BLK_TILES) {
            tiles = 0;
#pragma unroll
            for (int k = 0; k < 9; k++) { acc[k] += (double)f[k]; f[k] = 0.f; }
        }
    }
    if (!me.valid) return;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const double v = acc[k] + (double)f[k];
        if (partial) partial[((int64_t)blockIdx.y * 9 + k) * n_pad + 32 * grp + lane] = v;
        else dJ[9 * (int64_t)me.idx + k] += v;
    }
}

// --------------------------------------------------------------------- UJ, FP64
// pair_f64_acc (uj_pair.cuh) over the group's intervals, for the targets of each source's mask.
template <int K>
__global__ void __launch_bounds__(NF_THREADS)
nf_uj_f64(int64_t n, int64_t ngroups, const TgtPos* __restrict__ tgt, const int32_t* __restrict__ leaf_of,
          const int32_t* __restrict__ grp_row, const int4* __restrict__ ivs, const SrcF64* __restrict__ src,
          double* U, double* J, double* __restrict__ partial, int64_t n_pad)
{
    __shared__ SrcF64 tile[NF_WARPS][32];
    __shared__ unsigned tmask[NF_WARPS][32];
    __shared__ double T[64];
    exp_table(T);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t grp = (int64_t)blockIdx.x * NF_WARPS + warp;
    if (grp >= ngroups) return;
    const GroupTarget me = group_target(n, 32 * grp, lane, tgt, leaf_of);
    double u[3] = {0.0, 0.0, 0.0}, w[3] = {0.0, 0.0, 0.0}, jq[9];
#pragma unroll
    for (int k = 0; k < 9; k++) jq[k] = 0.0;
    PartTurn part;
    IntervalWalk walk;
    walk.init(ivs, grp_row[grp], grp_row[grp + 1], lane);
    for (;;) {
        int sp;
        unsigned smask;
        const int cnt = walk.next(lane, sp, smask);
        if (cnt == 0) break;
        if (!part.mine()) continue;
        __syncwarp();
        if (sp >= 0) tile[warp][lane] = src[sp];
        tmask[warp][lane] = smask;
        __syncwarp();
        for (int j = 0; j < cnt; j++)
            if (tmask[warp][j] & me.bit) pair_f64_acc<K>(me.tx, me.ty, me.tz, tile[warp][j], u, w, jq, T);
    }
    if (!me.valid) return;
    double acc[12];
    uj_f64_finish(u, w, jq, acc);
    write_uj(32 * grp + lane, me.idx, acc, U, 3, J, 9, partial, n_pad);
}

// ------------------------------------------------------------------------- Estr
// SFS_t += J_t^T sum_s z_s g_s - sum_s z_s v_s  (z = zeta(r/sigma_s), g and v
// pre-scaled by ZNORM / sigma_s^3 in the pack), over the group's intervals,
// skipping the self pair (mixed: every pair at r = 0, as in estr.cu), for
// non-static targets.  With DZ (mixed only) each weight is the dynamic
// procedure's weight difference zeta~(r, alpha sigma_s) - zeta~(r, sigma_s),
// fd as in estr.cu.  With ZETA the kernel is zeta_fmm's near-field sum
// (src/FLOWVPM_viscous.jl:523-556): SFS_t += sum_s z_s g_s over every target,
// the self pair and static particles included (payload packed with Js = NULL).
template <int K, bool MIXED, bool DZ = false, bool ZETA = false>
__global__ void __launch_bounds__(NF_THREADS)
nf_estr(int64_t n, int64_t ngroups, const TgtPos* __restrict__ tgt, const int32_t* __restrict__ leaf_of,
        const int32_t* __restrict__ grp_row, const int4* __restrict__ ivs, const void* __restrict__ srcv,
        const double* __restrict__ Jt, const uint8_t* __restrict__ static_t, bool transposed, double* SFS,
        double* __restrict__ partial, int64_t n_pad, float3 fd = make_float3(0.f, 0.f, 0.f))
{
    static_assert(MIXED || !DZ, "weight differences are FP32-comp only");
    static_assert(!(DZ && ZETA), "one mode at a time");
    // mixed: the sources as in the all-pairs kernel (estr.cu), two to an f32x2 instruction, without a
    // look at the masks where the group's targets all take all eight sources (jet of 2^20 with the
    // list build and UJ: 22.05 -> 21.34 ms);  FP64: the packed source
    __shared__ EstrTile mtile[MIXED ? NF_WARPS : 1];
    __shared__ SrcEstrF64 dtile[MIXED ? 1 : NF_WARPS][32];
    __shared__ int spos[NF_WARPS][32];                          // source position, -1 for padding
    __shared__ __align__(16) unsigned tmask[NF_WARPS][32];
    __shared__ double T[64];
    if constexpr (!MIXED) {
        exp_table(T);
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t grp = (int64_t)blockIdx.x * NF_WARPS + warp;
    if (grp >= ngroups) return;
    const int64_t p0 = 32 * grp;
    const GroupTarget me = group_target(n, p0, lane, tgt, leaf_of);
    const bool live = me.valid && (ZETA || !(static_t && static_t[me.idx]));
    const unsigned bit = live ? me.bit : 0u;
    const int tpos = (int)(p0 + lane);
    const float3 th = make_float3((float)me.tx, (float)me.ty, (float)me.tz);
    const float3 tl = make_float3((float)(me.tx - (double)th.x), (float)(me.ty - (double)th.y),
                                  (float)(me.tz - (double)th.z));
    double zg[3] = {0.0, 0.0, 0.0}, zv[3] = {0.0, 0.0, 0.0};
    // mixed: compensated FP32 sums of 8-source partial sums (comp_add), FP64 every NF_ESTR_FLUSH tiles
    // (as the all-pairs mixed Estr; the FP64 pipe runs at 1/64 of the FP32 rate)
    f32x2 sm[3] = {0ull, 0ull, 0ull}, cm[3] = {0ull, 0ull, 0ull};
    const unsigned all = __reduce_or_sync(0xffffffffu, bit);   // the group's live leaves
    // box of the group's targets (high parts): sources out of its reach are skipped as in the
    // all-pairs kernel, and only those inside it can be at r = 0 from a target
    __shared__ float4 gbox[MIXED ? NF_WARPS : 1][2];
    if constexpr (MIXED) target_box(th, lane, gbox[warp]);
    int tiles = 0;
    PartTurn part;
    IntervalWalk walk;
    walk.init(ivs, grp_row[grp], grp_row[grp + 1], lane);
    for (;;) {
        int sp;
        unsigned smask;
        const int cnt = walk.next(lane, sp, smask);
        if (cnt == 0) break;
        if (!part.mine()) continue;
        __syncwarp();
        unsigned beyond = 0u, inside = 0u;
        if constexpr (MIXED) {
            EstrTile& q = mtile[warp];
            SrcEstrDF p;
            if (sp >= 0) {
                p = ((const SrcEstrDF*)srcv)[sp];
            } else {   // padding: far away, no payload, mask 0
                p.a = make_float4(1.0e6f, 1.0e6f, 1.0e6f, 1.f);
                p.b = p.g = p.v = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            q.x[lane] = p.a.x; q.y[lane] = p.a.y; q.z[lane] = p.a.z; q.w[lane] = p.a.w;
            q.xl[lane] = p.b.x; q.yl[lane] = p.b.y; q.zl[lane] = p.b.z;
            q.gv[3 * lane] = make_float2(p.g.x, p.g.y);
            q.gv[3 * lane + 1] = make_float2(p.g.z, p.v.x);
            q.gv[3 * lane + 2] = make_float2(p.v.y, p.v.z);
            tmask[warp][lane] = smask;
            const float d2 = box_d2(gbox[warp], p.a.x, p.a.y, p.a.z);
            beyond = __ballot_sync(0xffffffffu, zeta_skip_s<K>() > 0.0f && d2 * p.a.w > zeta_skip_s<K>());
            inside = __ballot_sync(0xffffffffu, !(d2 > 0.0f));
        } else {
            if (sp >= 0) dtile[warp][lane] = ((const SrcEstrF64*)srcv)[sp];
        }
        if constexpr (!MIXED) {
            spos[warp][lane] = sp;
            tmask[warp][lane] = smask;
        }
        __syncwarp();
        if constexpr (MIXED) {
            const EstrTile& q = mtile[warp];
            const unsigned whole = __ballot_sync(0xffffffffu, (smask & all) == all);   // sources of every target
            for (int j0 = 0; j0 < cnt; j0 += 8) {   // cnt <= 32: j0 + 7 stays in the tile (padding has mask 0)
                if (((beyond >> j0) & 0xffu) == 0xffu) continue;
                f32x2 r2[4], s[4], f[3] = {0ull, 0ull, 0ull};
                estr_r2s8(q, j0, th, tl, r2, s);
                if (zeta_skip_s<K>() > 0.0f && __all_sync(0xffffffffu, min8_nan(s) > zeta_skip_s<K>())) continue;
                if (((whole >> j0) & 0xffu) == 0xffu && (ZETA || !((inside >> j0) & 0xffu))) {
                    estr_add8<K, ZETA, DZ, false, false>(r2, s, &q.gv[3 * j0], 0u, nullptr, fd, f);
                } else {
                    const uint4* m = (const uint4*)&tmask[warp][j0];
                    const uint4 on[2] = {m[0], m[1]};
                    estr_add8<K, ZETA, DZ, true, !ZETA>(r2, s, &q.gv[3 * j0], bit, on, fd, f);
                }
#pragma unroll
                for (int k = 0; k < (ZETA ? 2 : 3); k++) comp_add2(sm[k], cm[k], f[k]);
            }
            if (++tiles == NF_ESTR_FLUSH) {
                tiles = 0;
                estr_flush(sm, cm, zg, zv);
            }
        } else {
            for (int j = 0; j < cnt; j++) {
                if (!(tmask[warp][j] & bit) || (!ZETA && spos[warp][j] == tpos)) continue;
                const SrcEstrF64& p = dtile[warp][j];
                const double dx = p.xy.x - me.tx, dy = p.xy.y - me.ty, dz = p.z_isig.x - me.tz;
                const double isig = p.z_isig.y;
                const double isig2 = isig * isig;
                const double z = zhat_f64<K>((dx * dx + dy * dy + dz * dz) * isig2, T) * (zeta_norm(K) * isig * isig2);
                zg[0] += z * p.gxy.x; zg[1] += z * p.gxy.y; zg[2] += z * p.gz_vx.x;
                zv[0] += z * p.gz_vx.y; zv[1] += z * p.vyz.x; zv[2] += z * p.vyz.y;
            }
        }
    }
    if constexpr (MIXED) estr_flush(sm, cm, zg, zv);
    if (!live) return;      // a static target's partial sums are not read
    double o[3] = {0.0, 0.0, 0.0};
    if constexpr (ZETA) {
#pragma unroll
        for (int k = 0; k < 3; k++) o[k] = zg[k];
    } else {
        const double* Jp = Jt + 9 * (int64_t)me.idx;
        const int sr = transposed ? 3 : 1, sc = transposed ? 1 : 3;
#pragma unroll
        for (int k = 0; k < 3; k++) o[k] = Jp[sr * k] * zg[0] + Jp[sr * k + sc] * zg[1] + Jp[sr * k + 2 * sc] * zg[2] - zv[k];
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (partial) partial[((int64_t)blockIdx.y * 3 + k) * n_pad + p0 + lane] = o[k];
        else SFS[3 * (int64_t)me.idx + k] += o[k];
    }
}

// ---------------------------------------------------------------------- launcher
static inline size_t al256(size_t b) { return (b + 255) / 256 * 256; }

// Warps a group: enough for 16 blocks a SM, at most 8 (each walks the whole list to find its
// tiles).  With one warp a group a few blocks of uneven groups left most of the chip idle: near-field
// UJ and Estr calls of a 20,000-particle jet 1.94 -> 1.70 ms, 100,000 6.34 -> 5.52, 2^20 unchanged
// (one warp a group there).
static int near_parts(int64_t n, int num_sms)
{
    const int64_t blocks = (n + NF_THREADS - 1) / NF_THREADS;
    const int64_t p = (16LL * num_sms + blocks - 1) / blocks;
    return (int)(p < 1 ? 1 : p > 8 ? 8 : p);
}

// The launch's buffers: targets, packed sources, and the parts' partial sums (12 a target at most).
struct LeafWork {
    TgtPos* tgt;
    void* src;
    double* partial;     // null with one part a group
    int64_t n_pad;
    dim3 grid;           // groups x parts
    unsigned gt;         // blocks of 256 threads over the targets
};

size_t leaf_work_bytes(int64_t n, int num_sms)
{
    const size_t src = sizeof(SrcEstrDF) > sizeof(SrcEstrF64) ? sizeof(SrcEstrDF) : sizeof(SrcEstrF64);
    const int parts = near_parts(n, num_sms);
    const int64_t n_pad = (n + 31) / 32 * 32;
    return al256(n * sizeof(TgtPos)) + al256(n * src) + (parts > 1 ? (size_t)parts * 12 * n_pad * sizeof(double) : 0);
}

static LeafWork leaf_work(const LeafArgs& a, const NearLists& L, void* work)
{
    const size_t src = sizeof(SrcEstrDF) > sizeof(SrcEstrF64) ? sizeof(SrcEstrDF) : sizeof(SrcEstrF64);
    const int parts = near_parts(a.n, a.num_sms);
    LeafWork w;
    w.tgt = (TgtPos*)work;
    w.src = (char*)work + al256(a.n * sizeof(TgtPos));
    w.partial = parts > 1 ? (double*)((char*)w.src + al256(a.n * src)) : nullptr;
    w.n_pad = (a.n + 31) / 32 * 32;
    w.grid = dim3((unsigned)((L.ngroups + NF_WARPS - 1) / NF_WARPS), (unsigned)parts);
    w.gt = (unsigned)((a.n + 255) / 256);
    return w;
}

static void reduce_parts(const LeafArgs& a, const LeafWork& w, int na, double* A, int nb, double* B, cudaStream_t st,
                         int64_t* launches, const uint8_t* skip = nullptr)
{
    if (!w.partial) return;
    leaf_reduce<<<dim3((unsigned)((a.n + 127) / 128), (unsigned)(na + nb)), 128, 0, st>>>(
        a.n, (int)w.grid.y, na, nb, w.partial, w.n_pad, w.tgt, skip, A, B);
    *launches += 1;
}

template <int K>
static cudaError_t launch_leaf_k(const LeafArgs& a, const NearLists& L, void* work, cudaStream_t st,
                                 int64_t* launches)
{
    const int64_t n = a.n;
    const LeafWork w = leaf_work(a, L, work);
    tgt_from_perm<<<w.gt, 256, 0, st>>>(n, a.x, L.perm, w.tgt);
    *launches += 1;
    if (a.uj) {
        if (a.precision) {
            leaf_pack_lane<K><<<w.gt, 256, 0, st>>>(n, a.x, a.gam, a.sig, L.perm, (SrcMixed*)w.src);
            nf_uj_mixed<K><<<w.grid, NF_THREADS, 0, st>>>(n, L.ngroups, w.tgt, L.leaf_of, L.grp_row, L.ivs,
                                                          (const SrcMixed*)w.src, a.U, a.J, w.partial, w.n_pad);
        } else {
            leaf_pack_f64<K><<<w.gt, 256, 0, st>>>(n, a.x, a.gam, a.sig, L.perm, (SrcF64*)w.src);
            nf_uj_f64<K><<<w.grid, NF_THREADS, 0, st>>>(n, L.ngroups, w.tgt, L.leaf_of, L.grp_row, L.ivs,
                                                        (const SrcF64*)w.src, a.U, a.J, w.partial, w.n_pad);
        }
        *launches += 2;
        reduce_parts(a, w, 3, a.U, 9, a.J, st, launches);
    }
    if (a.sfs) {
        leaf_pack_estr<K><<<w.gt, 256, 0, st>>>(n, a.x, a.gam, a.sig, a.J, a.static_flags, a.transposed, L.perm,
                                                 a.precision, w.src);
        if (a.precision)
            nf_estr<K, true><<<w.grid, NF_THREADS, 0, st>>>(n, L.ngroups, w.tgt, L.leaf_of, L.grp_row, L.ivs, w.src,
                                                            a.J, a.static_flags, a.transposed, a.SFS, w.partial,
                                                            w.n_pad);
        else
            nf_estr<K, false><<<w.grid, NF_THREADS, 0, st>>>(n, L.ngroups, w.tgt, L.leaf_of, L.grp_row, L.ivs, w.src,
                                                             a.J, a.static_flags, a.transposed, a.SFS, w.partial,
                                                             w.n_pad);
        *launches += 2;
        reduce_parts(a, w, 3, a.SFS, 0, nullptr, st, launches, a.static_flags);
    }
    return cudaGetLastError();
}

// The dynamic procedure's differences over the near lists, FP32-comp:
// dJ = the filter difference of J; dSFS = the weight-difference Estr at J plus
// the Estr of dJ at alpha sigma (sig_a); a.J is J, a.sfs and a.U unused.
template <int K>
static cudaError_t launch_leaf_dyn_k(const LeafArgs& a, const NearLists& L, double alpha, const double* sig_a,
                                     double* dJ, double* dSFS, void* work, cudaStream_t st, int64_t* launches)
{
    const int64_t n = a.n;
    const LeafWork w = leaf_work(a, L, work);
    const double ha = 1.0 / alpha - 1.0;
    tgt_from_perm<<<w.gt, 256, 0, st>>>(n, a.x, L.perm, w.tgt);
    *launches += 1;
    if constexpr (K != K_SING) {   // g = 1 has no sigma dependence: dJ = 0
        leaf_pack_mixed<K><<<w.gt, 256, 0, st>>>(n, a.x, a.gam, a.sig, L.perm, (SrcMixed*)w.src);
        const int m = filter_panels(ha);
        if (m == 1)
            nf_filter_diff<K, 1><<<w.grid, NF_THREADS, 0, st>>>(n, L.ngroups, w.tgt, L.leaf_of, L.grp_row, L.ivs,
                                                                (const SrcMixed*)w.src, (float)ha, 1, dJ, w.partial,
                                                                w.n_pad);
        else
            nf_filter_diff<K, 0><<<w.grid, NF_THREADS, 0, st>>>(n, L.ngroups, w.tgt, L.leaf_of, L.grp_row, L.ivs,
                                                                (const SrcMixed*)w.src, (float)(ha / m), m, dJ,
                                                                w.partial, w.n_pad);
        *launches += 2;
        reduce_parts(a, w, 9, dJ, 0, nullptr, st, launches);
    }
    const float3 fd = make_float3((float)(1.0 / (alpha * alpha * alpha) - 1.0), (float)(1.0 / (alpha * alpha * alpha)),
                                  (float)(1.0 / (alpha * alpha) - 1.0));
    leaf_pack_estr<K><<<w.gt, 256, 0, st>>>(n, a.x, a.gam, a.sig, a.J, a.static_flags, a.transposed, L.perm, 1, w.src);
    nf_estr<K, true, true><<<w.grid, NF_THREADS, 0, st>>>(n, L.ngroups, w.tgt, L.leaf_of, L.grp_row, L.ivs, w.src, a.J,
                                                          a.static_flags, a.transposed, dSFS, w.partial, w.n_pad, fd);
    reduce_parts(a, w, 3, dSFS, 0, nullptr, st, launches, a.static_flags);
    leaf_pack_estr<K><<<w.gt, 256, 0, st>>>(n, a.x, a.gam, sig_a, dJ, a.static_flags, a.transposed, L.perm, 1, w.src);
    nf_estr<K, true><<<w.grid, NF_THREADS, 0, st>>>(n, L.ngroups, w.tgt, L.leaf_of, L.grp_row, L.ivs, w.src, dJ,
                                                    a.static_flags, a.transposed, dSFS, w.partial, w.n_pad);
    reduce_parts(a, w, 3, dSFS, 0, nullptr, st, launches, a.static_flags);
    *launches += 4;
    return cudaGetLastError();
}

cudaError_t launch_leaf_dynamic(const LeafArgs& a, const NearLists& L, double alpha, const double* sig_a, double* dJ,
                                double* dSFS, void* work, cudaStream_t st, int64_t* launches)
{
    if (a.n <= 0) return cudaSuccess;
    if (!a.precision) return cudaErrorInvalidValue;   // FP32-comp only
    switch (a.kernel) {
    case K_SING: return launch_leaf_dyn_k<K_SING>(a, L, alpha, sig_a, dJ, dSFS, work, st, launches);
    case K_GAUS: return launch_leaf_dyn_k<K_GAUS>(a, L, alpha, sig_a, dJ, dSFS, work, st, launches);
    case K_GAUSERF: return launch_leaf_dyn_k<K_GAUSERF>(a, L, alpha, sig_a, dJ, dSFS, work, st, launches);
    case K_WNKLMNS: return launch_leaf_dyn_k<K_WNKLMNS>(a, L, alpha, sig_a, dJ, dSFS, work, st, launches);
    default: return cudaErrorInvalidValue;
    }
}

// zeta_fmm's near-field sum: W += sum over the near lists of zeta(r/sigma_s)/sigma_s^3 Gamma_s
// (a.x, a.gam, a.sig; every particle a target, the self pair included).
template <int K>
static cudaError_t launch_leaf_zeta_k(const LeafArgs& a, const NearLists& L, double* W, void* work, cudaStream_t st,
                                      int64_t* launches)
{
    const int64_t n = a.n;
    const LeafWork w = leaf_work(a, L, work);
    tgt_from_perm<<<w.gt, 256, 0, st>>>(n, a.x, L.perm, w.tgt);
    leaf_pack_estr<K><<<w.gt, 256, 0, st>>>(n, a.x, a.gam, a.sig, nullptr, nullptr, true, L.perm, a.precision, w.src);
    if (a.precision)
        nf_estr<K, true, false, true><<<w.grid, NF_THREADS, 0, st>>>(n, L.ngroups, w.tgt, L.leaf_of, L.grp_row, L.ivs,
                                                                     w.src, nullptr, nullptr, true, W, w.partial,
                                                                     w.n_pad);
    else
        nf_estr<K, false, false, true><<<w.grid, NF_THREADS, 0, st>>>(n, L.ngroups, w.tgt, L.leaf_of, L.grp_row, L.ivs,
                                                                      w.src, nullptr, nullptr, true, W, w.partial,
                                                                      w.n_pad);
    *launches += 3;
    reduce_parts(a, w, 3, W, 0, nullptr, st, launches);
    return cudaGetLastError();
}

cudaError_t launch_leaf_zeta(const LeafArgs& a, const NearLists& L, double* W, void* work, cudaStream_t st,
                             int64_t* launches)
{
    if (a.n <= 0) return cudaSuccess;
    switch (a.kernel) {
    case K_SING: return launch_leaf_zeta_k<K_SING>(a, L, W, work, st, launches);
    case K_GAUS: return launch_leaf_zeta_k<K_GAUS>(a, L, W, work, st, launches);
    case K_GAUSERF: return launch_leaf_zeta_k<K_GAUSERF>(a, L, W, work, st, launches);
    case K_WNKLMNS: return launch_leaf_zeta_k<K_WNKLMNS>(a, L, W, work, st, launches);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_leaflist(const LeafArgs& a, const NearLists& L, void* work, cudaStream_t st, int64_t* launches)
{
    if (a.n <= 0) return cudaSuccess;
    switch (a.kernel) {
    case K_SING: return launch_leaf_k<K_SING>(a, L, work, st, launches);
    case K_GAUS: return launch_leaf_k<K_GAUS>(a, L, work, st, launches);
    case K_GAUSERF: return launch_leaf_k<K_GAUSERF>(a, L, work, st, launches);
    case K_WNKLMNS: return launch_leaf_k<K_WNKLMNS>(a, L, work, st, launches);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace vpm
