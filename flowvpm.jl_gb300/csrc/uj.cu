// uj.cu -- all-pairs U and J kernels (the P2P pair loop of
// src/FLOWVPM_fmm.jl:102-168, over all sources as UJ_direct does,
// src/FLOWVPM_UJ.jl:35).
//
// Layout: one target per thread, UJ_THREADS targets per block, targets in
// curve order (order.cu) so each warp holds 32 neighbouring targets.  Sources
// are packed once per call (in the same curve order when they are the
// targets).  The FP64 kernel streams them through shared memory in block-wide
// tiles of UJ_TILE; in the mixed kernel every warp streams them on its own in
// tiles of 32, double-buffered with cp.async, so warps never wait for one
// another.  gridDim.y splits the sources when there are too few target blocks
// to fill the GPU; each split then writes FP64 partial sums to scratch and
// uj_reduce adds them, in split order, to the outputs.
//
// Mixed (FP32-comp) kernel.  Positions are double-floats (hi + lo in FP32).
//  * Far pairs: each warp takes its first target as origin and, once per tile,
//    converts every source to an FP32 offset from it; dx = o_t - o_s then costs
//    3 FP32 subtractions with an error of a few ulp of |dx| + the warp's extent
//    b.  A source is "far" for a lane when r^2 > max(s_far sigma^2, (2b)^2):
//    the kernel is then in its singular form (G = r^-3, Q = r^-5, no sigma) and
//    the offset error is below 1.5 ulp of |dx|.
//  * When any lane of the warp has a near pair among 4 sources (one vote), the
//    warp evaluates those 4 pairs with dx = (x_t,hi - x_s,hi) + (x_t,lo - x_s,lo)
//    and the full regular form of the kernel (vpm_math.cuh).
// Sums run in FP32 over blocks of UJ_BLOCK sources, then in an FP32 mid-level
// sum over MID_BLOCKS of those, then in FP64.  In tiles with near sources the
// FP32 blocks are of 8: a target's largest terms stand in one or two tiles of the
// curve and often add with one sign (ring of 1,000, J: error 1.7e-7 with blocks of
// 64, 0.8e-7 so, for 2 % of the time; 1.6e-7 in the caller's order).
#include "internal.h"
#include "uj_pair.cuh"
#include "vpm_math.cuh"

namespace vpm {

static_assert(UJ_TILE == UJ_THREADS, "one source loaded per thread per tile");
static_assert(UJ_TILE % UJ_BLOCK == 0, "FP32 blocks must tile the shared tile");
static_assert(UJ_BLOCK % 4 == 0, "far/near votes cover groups of 4 sources");
static_assert(UJ_TILE % 32 == 0, "per-warp conversion covers the tile in whole passes");

static inline int64_t round_up(int64_t a, int64_t b) { return (a + b - 1) / b * b; }

size_t uj_src_pack_bytes(int64_t ns, int precision)
{
    const int64_t n = round_up(ns, UJ_TILE);
    return (size_t)n * (precision ? sizeof(SrcMixed) : sizeof(SrcF64));
}

int uj_num_splits(int64_t nt, int64_t ns, int num_sms, int precision, int per_sm)
{
    // per_sm blocks per SM (about four waves at the default), from shares of at least one unit
    // (FP64) or two warp tiles.  With shares of at least 512 sources 1,400 particles made 22
    // blocks for 152 SMs (UJ 2.39 ms, Estr 1.27 ms in FP64); with 12 blocks a SM the uneven
    // blocks left SMs idle at the end: FP64 gradient of 5,600 particles 21.1 ms, 20.4 at 24 and
    // 20.3 at 36; Estr of the 200,000-particle rings 4.20, 3.78 and 3.77 ms; filter differences
    // of 100,000 8.9 ms unsplit, 6.8, 6.1 and 5.7 (whole calls).
    const int64_t tblocks = (nt + UJ_THREADS - 1) / UJ_THREADS;
    const int64_t units = precision ? (ns + 63) / 64 : (ns + F64_UNIT - 1) / F64_UNIT;
    const int64_t want = (int64_t)per_sm * num_sms;
    int64_t nsplit = (want + tblocks - 1) / tblocks;
    if (nsplit > units) nsplit = units;
    if (nsplit < 1) nsplit = 1;
    return (int)nsplit;
}

// The tile kernels (uj_tc.cu) take a set on itself from 10,240 particles.  Below, most tiles of
// 64 are near ones (4,099 random particles: 73 % of the pairs) and the tile pack is pure cost.
// With uj_mixed_kernel / with tiles, us: random 8,192 306 / 299, 10,240 382 / 390, 12,000 454 / 435,
// 14,000 542 / 495; rings of 8,192 300 / 304, of 10,240 372 / 387, of 12,000 439 / 431; Winckelmans
// 8,192 288 / 287, 10,240 373 / 364; jet of 10,240 408 / 429, of 12,000 477 / 472.
bool uj_takes_tiles(const UJArgs& a) { return a.self && a.precision == 1 && a.ns >= 10240; }

size_t uj_partial_bytes(int64_t nt, int nsplit, int components)
{
    return nsplit > 1 ? (size_t)nsplit * components * (size_t)round_up(nt, UJ_THREADS) * sizeof(double) : 0;
}


// ------------------------------------------------------------------ packing
// When `order` is given (sources = targets), source i of the pack is particle
// order[i].idx, i.e. the sources follow the targets' curve order: a warp's
// near sources then sit in few 4-source groups, so fewer groups take the near
// path.  The order of a sum's terms does not otherwise matter.
template <int K>
__global__ void pack_src_mixed(int64_t ns, int64_t ns_pad, const double* __restrict__ xs,
                               const double* __restrict__ gs, const double* __restrict__ sgs,
                               const TgtPos* __restrict__ order, SrcMixed* __restrict__ out)
{
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= ns_pad) return;
    SrcMixed p;
    if (o < ns) {
        const int64_t i = order ? (int64_t)order[o].idx : o;
        const double x = xs[3 * i], y = xs[3 * i + 1], z = xs[3 * i + 2];
        const float xh = (float)x, yh = (float)y, zh = (float)z;
        const double sig = (K == K_SING) ? 1.0 : sgs[i];
        const double k = singular_tail<K>() ? -C4 : -C4 / (sig * sig * sig);
        p.a = make_float4(xh, yh, zh, (float)(sig * sig));
        p.b = make_float4((float)(x - (double)xh), (float)(y - (double)yh), (float)(z - (double)zh),
                          (float)(1.0 / sig));
        p.gam = make_float4((float)(k * gs[3 * i]), (float)(k * gs[3 * i + 1]), (float)(k * gs[3 * i + 2]), 0.f);
    } else {  // padding: no strength, at the origin, unit core
        p.a = make_float4(0.f, 0.f, 0.f, 1.f);
        p.b = make_float4(0.f, 0.f, 0.f, 1.f);
        p.gam = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    out[o] = p;
}

template <int K>
__global__ void pack_src_f64(int64_t ns, int64_t ns_pad, const double* __restrict__ xs,
                             const double* __restrict__ gs, const double* __restrict__ sgs,
                             SrcF64* __restrict__ out)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= ns_pad) return;
    SrcF64 p;
    if (i < ns) {
        const double sig = (K == K_SING) ? 1.0 : sgs[i];
        p.xy = make_double2(xs[3 * i], xs[3 * i + 1]);
        p.z_isig = make_double2(xs[3 * i + 2], 1.0 / sig);
        p.gxy = make_double2(gs[3 * i], gs[3 * i + 1]);
        // .y: for Gaussian-erf the r^2 past which g = 1, g' = 0 (rho > 9), else sigma
        p.gz_sig = make_double2(gs[3 * i + 2], K == K_GAUSERF ? 81.0 * sig * sig : sig);
    } else {
        p.xy = make_double2(0.0, 0.0);
        p.z_isig = make_double2(0.0, 1.0);
        p.gxy = make_double2(0.0, 0.0);
        p.gz_sig = make_double2(0.0, 1.0);
    }
    out[i] = p;
}

// --------------------------------------------------------------- epilogue
// One thread per target and component (coalesced along the targets): with one thread a target
// the 12 sums ran one after the other (30 us for 7 splits of 4,099 targets).
__global__ void uj_reduce(int64_t nt, int nsplit, const double* __restrict__ partial, int64_t nt_pad,
                          const TgtPos* __restrict__ tgt, double* U, int64_t ldU, double* J, int64_t ldJ)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const int64_t i = tgt[t].idx;
    const int k = blockIdx.y;
    const double* p = partial + k * nt_pad + t;
    double s = 0.0;
#pragma unroll 8
    for (int sp = 0; sp < nsplit; sp++) s += p[(int64_t)sp * 12 * nt_pad];
    if (k < 3) U[i * ldU + k] += s;
    else J[i * ldJ + (k - 3)] += s;
}

__global__ void sum_splits_kernel(double* __restrict__ p, int nsplit, int nk, int64_t nt, int64_t nt_pad)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nt) return;
    double* q = p + blockIdx.y * nt_pad + t;
    double s = 0.0;
#pragma unroll 8
    for (int sp = 0; sp < nsplit; sp++) s += q[(int64_t)sp * nk * nt_pad];
    q[0] = s;
}

void sum_splits(double* p, int nsplit, int nk, int64_t nt, int64_t nt_pad, cudaStream_t st, int64_t* launches)
{
    if (nsplit < 2) return;
    sum_splits_kernel<<<dim3((unsigned)((nt + 127) / 128), (unsigned)nk), 128, 0, st>>>(p, nsplit, nk, nt, nt_pad);
    *launches += 1;
}

// ------------------------------------------------------------ main kernels
template <int K>
__global__ void __launch_bounds__(UJ_THREADS)
uj_f64_kernel(int64_t nt, const TgtPos* __restrict__ tgt, int64_t ns_pad, const SrcF64* __restrict__ src,
              double* U, int64_t ldU, double* J, int64_t ldJ, double* partial, int64_t nt_pad)
{
    __shared__ SrcF64 tile[UJ_TILE];
    __shared__ double T[64];
    exp_table(T);
    const int64_t t = (int64_t)blockIdx.x * UJ_THREADS + threadIdx.x;
    const bool valid = t < nt;
    double tx = 1.0e3, ty = 1.0e3, tz = 1.0e3;
    int32_t idx = 0;
    if (valid) {
        const TgtPos p = tgt[t];
        tx = p.x; ty = p.y; tz = p.z; idx = p.idx;
    }
    double acc[12];
    double u[3] = {0.0, 0.0, 0.0}, w[3] = {0.0, 0.0, 0.0}, jq[9];
#pragma unroll
    for (int k = 0; k < 9; k++) jq[k] = 0.0;
    const int64_t nq = split_count(ns_pad, blockIdx.y, gridDim.y);
    for (int64_t base = 0; base < nq; base += UJ_TILE) {
        __syncthreads();
        if (base + threadIdx.x < nq) tile[threadIdx.x] = src[split_source(base + threadIdx.x, blockIdx.y, gridDim.y)];
        __syncthreads();
        const int m = (int)min((int64_t)UJ_TILE, nq - base);
#pragma unroll 2
        for (int j = 0; j < m; j++) pair_f64_acc<K>(tx, ty, tz, tile[j], u, w, jq, T);
    }
    uj_f64_finish(u, w, jq, acc);
    if (valid) write_uj(t, idx, acc, U, ldU, J, ldJ, partial, nt_pad);
}

// 16-byte asynchronous global->shared copy (LDGSTS), L2-cached.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }


constexpr int WT = 32;                      // sources per warp tile (one per lane)
constexpr int BLOCK_TILES = UJ_BLOCK / WT;  // warp tiles per FP32 block
// FP32 blocks per FP32 mid-level sum: 16 x 64 sources between FP64 adds (4 measured 1.2 %
// slower -- the FP64 pipe runs at 1/64 rate -- with the same U, J error against the oracle)
constexpr int MID_BLOCKS = 16;
// Resident blocks per SM the register budget targets, per kernel: at N = 2^20 with the
// per-tile far flags, Gaussian-erf ran 1360 ms a launch at 5 (96 registers), 1400 at 6
// (80) and 1408 at 7 (72, a few spills); Winckelmans, whose far form is its full form,
// 1522 at 5 and 1503 at 6.
template <int K>
__host__ __device__ constexpr int uj_min_blocks()
{
    return K == K_WNKLMNS ? 6 : 5;
}
constexpr int UJ_UNROLL = 2;                // 4-source groups unrolled per iteration of a tile

// Each warp streams the sources on its own: 32 per tile, double-buffered with
// cp.async, so warps never wait for each other (no block-wide barrier).
template <int K>
__global__ void __launch_bounds__(UJ_THREADS, uj_min_blocks<K>())
uj_mixed_kernel(int64_t nt, const TgtPos* __restrict__ tgt, int64_t ns_pad,
                const SrcMixed* __restrict__ src, double* U, int64_t ldU,
                double* J, int64_t ldJ, double* partial, int64_t nt_pad)
{
    __shared__ SrcMixed stage[UJ_WARPS][2][WT];
    __shared__ float4 offs[UJ_WARPS][2][WT];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t = (int64_t)blockIdx.x * UJ_THREADS + threadIdx.x;
    const bool valid = t < nt;
    double tx = 3.0e4, ty = 3.0e4, tz = 3.0e4;
    int32_t idx = 0;
    if (valid) {
        const TgtPos p = tgt[t];
        tx = p.x; ty = p.y; tz = p.z; idx = p.idx;
    }
    const float3 th = make_float3((float)tx, (float)ty, (float)tz);
    const float3 tl = make_float3((float)(tx - (double)th.x), (float)(ty - (double)th.y), (float)(tz - (double)th.z));
    // warp origin: lane 0's target (valid whenever any lane of the warp is)
    const double ox = __shfl_sync(0xffffffffu, tx, 0);
    const double oy = __shfl_sync(0xffffffffu, ty, 0);
    const double oz = __shfl_sync(0xffffffffu, tz, 0);
    const float3 oh = make_float3(__shfl_sync(0xffffffffu, th.x, 0), __shfl_sync(0xffffffffu, th.y, 0),
                                  __shfl_sync(0xffffffffu, th.z, 0));
    const float3 ol = make_float3(__shfl_sync(0xffffffffu, tl.x, 0), __shfl_sync(0xffffffffu, tl.y, 0),
                                  __shfl_sync(0xffffffffu, tl.z, 0));
    const float3 to = valid ? make_float3((float)(tx - ox), (float)(ty - oy), (float)(tz - oz))
                            : make_float3(3.0e4f, 3.0e4f, 3.0e4f);
    // (2 b)^2 with b the largest |offset| of the warp's valid targets
    float b2 = valid ? fmaf(to.x, to.x, fmaf(to.y, to.y, to.z * to.z)) : 0.0f;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) b2 = fmaxf(b2, __shfl_xor_sync(0xffffffffu, b2, m));
    const float r2n = fmaxf(4.0f * b2, 1.0e-30f);
    const float sfar = s_far<K>();
    // the box of the warp's valid targets (offsets; empty when it has none), read by the
    // loading lanes
    __shared__ float4 wbox[UJ_WARPS][2];
    {
        float lo[3] = {valid ? to.x : 3.0e38f, valid ? to.y : 3.0e38f, valid ? to.z : 3.0e38f};
        float hi[3] = {valid ? to.x : -3.0e38f, valid ? to.y : -3.0e38f, valid ? to.z : -3.0e38f};
#pragma unroll
        for (int m = 16; m > 0; m >>= 1)
#pragma unroll
            for (int k = 0; k < 3; k++) {
                lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], m));
                hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], m));
            }
        if (lane == 0) {
            wbox[warp][0] = make_float4(lo[0], lo[1], lo[2], 0.f);
            wbox[warp][1] = make_float4(hi[0], hi[1], hi[2], 0.f);
        }
        __syncwarp();
    }

    // FP64 sums of this thread: [0..2] U, [3..5] W, [6..13] J' (touched once per mid-level flush)
    __shared__ double acc64[14][UJ_THREADS];
#pragma unroll
    for (int k = 0; k < 14; k++) acc64[k][threadIdx.x] = 0.0;
#define ACC_DU(k) acc64[k][threadIdx.x]
#define ACC_DW(k) acc64[3 + (k)][threadIdx.x]
#define ACC_DJ(k) acc64[6 + (k)][threadIdx.x]
    float mu[3] = {0.f, 0.f, 0.f}, mw[3] = {0.f, 0.f, 0.f}, mj[8];
    float u[3] = {0.f, 0.f, 0.f}, w[3] = {0.f, 0.f, 0.f}, jq[8];
#pragma unroll
    for (int k = 0; k < 8; k++) { mj[k] = 0.f; jq[k] = 0.f; }

    // the split's warp tiles: every gridDim.y-th (a target's near tiles are neighbours)
    const int ntiles = (int)((ns_pad / WT - blockIdx.y + gridDim.y - 1) / gridDim.y);
    const int64_t step = (int64_t)gridDim.y * WT;
    const SrcMixed* wsrc = src + (int64_t)blockIdx.y * WT + lane;
    if (ntiles > 0) {
        SrcMixed* d = &stage[warp][0][lane];
        cp_async16(&d->a, &wsrc->a);
        cp_async16(&d->b, &wsrc->b);
        cp_async16(&d->gam, &wsrc->gam);
        cp_async_commit();
    }
    int in_block = 0, in_mid = 0;
    for (int it = 0; it < ntiles; it++) {
        const int buf = it & 1;
        if (it + 1 < ntiles) {
            const SrcMixed* g = wsrc + (it + 1) * step;
            SrcMixed* d = &stage[warp][buf ^ 1][lane];
            cp_async16(&d->a, &g->a);
            cp_async16(&d->b, &g->b);
            cp_async16(&d->gam, &g->gam);
            cp_async_commit();
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncwarp();
        bool far_src;
        {   // this lane's source: FP32 offset from the warp origin, and whether every pair
            // with the warp's targets is past max(reach, (2 b)^2)
            const float4 a = stage[warp][buf][lane].a, b = stage[warp][buf][lane].b;
            const float px = (a.x - oh.x) + (b.x - ol.x), py = (a.y - oh.y) + (b.y - ol.y),
                        pz = (a.z - oh.z) + (b.z - ol.z);
            offs[warp][buf][lane] = make_float4(px, py, pz, b.w * b.w);
            const float4 lo = wbox[warp][0], hi = wbox[warp][1];
            const float ex = fmaxf(fmaxf(lo.x - px, px - hi.x), 0.0f);
            const float ey = fmaxf(fmaxf(lo.y - py, py - hi.y), 0.0f);
            const float ez = fmaxf(fmaxf(lo.z - pz, pz - hi.z), 0.0f);
            const float thr = singular_tail<K>() ? fmaxf(sfar * a.w, r2n) : r2n;
            far_src = fmaf(ex, ex, fmaf(ey, ey, ez * ez)) > thr;
        }
        const unsigned farbits = __ballot_sync(0xffffffffu, far_src);
        __syncwarp();
        if (farbits == 0xffffffffu) {
#pragma unroll (UJ_UNROLL)
            for (int j = 0; j < WT; j += 4) pair4_far<K>(to, offs[warp][buf], stage[warp][buf], j, u, jq, w);
        } else {
#pragma unroll 1
            for (int j = 0; j < WT; j += 4) {
                if (((farbits >> j) & 0xFu) == 0xFu)
                    pair4_far<K>(to, offs[warp][buf], stage[warp][buf], j, u, jq, w);
                else
                    pair4_near<K>(th, tl, offs[warp][buf], stage[warp][buf], j, u, jq, w);
                if (j & 4) {   // 8 sources at a time where near ones are (see the head of the file)
#pragma unroll
                    for (int k = 0; k < 3; k++) { mu[k] += u[k]; mw[k] += w[k]; u[k] = 0.f; w[k] = 0.f; }
#pragma unroll
                    for (int k = 0; k < 8; k++) { mj[k] += jq[k]; jq[k] = 0.f; }
                }
            }
        }
        if (++in_block == BLOCK_TILES) {
#pragma unroll
            for (int k = 0; k < 3; k++) { mu[k] += u[k]; mw[k] += w[k]; u[k] = 0.f; w[k] = 0.f; }
#pragma unroll
            for (int k = 0; k < 8; k++) { mj[k] += jq[k]; jq[k] = 0.f; }
            in_block = 0;
            if (++in_mid == MID_BLOCKS) {
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    ACC_DU(k) += (double)mu[k]; ACC_DW(k) += (double)mw[k]; mu[k] = 0.f; mw[k] = 0.f;
                }
#pragma unroll
                for (int k = 0; k < 8; k++) { ACC_DJ(k) += (double)mj[k]; mj[k] = 0.f; }
                in_mid = 0;
            }
        }
        __syncwarp();   // every lane is done with `buf` before it is refilled
    }
    // remaining partial block and mid-level sums
    double fU[3], fW[3], fJ[8];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        fU[k] = ACC_DU(k) + ((double)mu[k] + (double)u[k]);
        fW[k] = ACC_DW(k) + ((double)mw[k] + (double)w[k]);
    }
#pragma unroll
    for (int k = 0; k < 8; k++) fJ[k] = ACC_DJ(k) + ((double)mj[k] + (double)jq[k]);
#undef ACC_DU
#undef ACC_DW
#undef ACC_DJ
    if (!valid) return;
    const double f[14] = {fU[0], fU[1], fU[2], fW[0], fW[1], fW[2], fJ[0], fJ[1], fJ[2], fJ[3], fJ[4], fJ[5], fJ[6], fJ[7]};
    double acc[12];
    uj_mixed_finish(f, acc);
    write_uj(t, idx, acc, U, ldU, J, ldJ, partial, nt_pad);
}
// --------------------------------------------------------------- launcher
template <int K>
static cudaError_t launch_uj_k(const UJArgs& a, const Workspace& w, int num_sms, cudaStream_t st,
                               int64_t* launches)
{
    const int64_t ns_pad = round_up(a.ns, UJ_TILE);
    const int64_t nt_pad = round_up(a.nt, UJ_THREADS);
    const bool tc = uj_takes_tiles(a) && w.tiles && w.gave_up;
    int nsplit = tc ? uj_tc_splits(a.nt, num_sms) : uj_num_splits(a.nt, a.ns, num_sms, a.precision);
    while (!tc && nsplit > 1 && uj_partial_bytes(a.nt, nsplit) > w.partial_bytes) nsplit--;   // a caller's fixed scratch
    double* partial = nsplit > 1 ? w.partial : nullptr;
    const dim3 grid((unsigned)(nt_pad / UJ_THREADS), (unsigned)nsplit);
    const int pb = 256;
    const TgtPos* tgt = nullptr;
    cudaError_t e = order_targets(a.nt, a.xt, w.order, w.order_bytes, st, launches, &tgt);
    if (e != cudaSuccess) return e;
    if (a.precision == 0) {
        SrcF64* src = (SrcF64*)w.src_pack;
        pack_src_f64<K><<<(unsigned)((ns_pad + pb - 1) / pb), pb, 0, st>>>(a.ns, ns_pad, a.xs, a.gs, a.sgs, src);
        uj_f64_kernel<K><<<grid, UJ_THREADS, 0, st>>>(a.nt, tgt, ns_pad, src, a.U, a.ldU,
                                                       a.J, a.ldJ, partial, nt_pad);
    } else {
        SrcMixed* src = (SrcMixed*)w.src_pack;
        pack_src_mixed<K><<<(unsigned)((ns_pad + pb - 1) / pb), pb, 0, st>>>(a.ns, ns_pad, a.xs, a.gs, a.sgs,
                                                                             a.self ? tgt : nullptr, src);
        if (tc) {
            e = launch_uj_tc(a, tgt, src, w, nsplit, partial, nt_pad, st, launches);
            if (e != cudaSuccess) return e;
        } else
        uj_mixed_kernel<K><<<grid, UJ_THREADS, 0, st>>>(a.nt, tgt, ns_pad, src, a.U, a.ldU,
                                                         a.J, a.ldJ, partial, nt_pad);
    }
    *launches += 2;
    if (partial) {
        uj_reduce<<<dim3((unsigned)((a.nt + 127) / 128), 12), 128, 0, st>>>(a.nt, nsplit, partial, nt_pad, tgt, a.U,
                                                                 a.ldU, a.J, a.ldJ);
        *launches += 1;
    }
    return cudaGetLastError();
}

cudaError_t launch_uj(const UJArgs& a, const Workspace& w, int num_sms, cudaStream_t st, int64_t* launches)
{
    if (a.nt <= 0 || a.ns <= 0) return cudaSuccess;
    switch (a.kernel) {
    case K_SING: return launch_uj_k<K_SING>(a, w, num_sms, st, launches);
    case K_GAUS: return launch_uj_k<K_GAUS>(a, w, num_sms, st, launches);
    case K_GAUSERF: return launch_uj_k<K_GAUSERF>(a, w, num_sms, st, launches);
    case K_WNKLMNS: return launch_uj_k<K_WNKLMNS>(a, w, num_sms, st, launches);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace vpm
