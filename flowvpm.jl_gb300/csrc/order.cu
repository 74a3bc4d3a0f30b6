// order.cu -- space-filling-curve (Hilbert) ordering of the targets of a UJ / Estr call.
//
// The pair kernels give each warp 32 consecutive targets of this order, and the tile kernels
// 32 or 64 consecutive sources, so that each sits in a small box: far-field and reach tests
// are then the same for a whole warp or tile, and the FP32 offsets of the mixed kernels, taken
// from a per-warp FP64 origin, stay small.  The order is internal: results are written back to
// each target's original index.
//
// Hilbert's curve, in the cube of the largest extent: consecutive cells are neighbours, where
// Morton's order jumps, so runs of 32 or 64 particles are more compact (65,536-particle random
// cloud: median radius of 64-particle tiles 0.093 against 0.101, and the pairs in tiles closer
// than two radii 10.8 % against 20.8 % of all).  On flat sets the cube matters more than the
// curve: with each axis scaled to its own extent the cells of a 32,000-particle ring were 11
// times as wide as high (tile radius 0.161 against 0.074).
//
// Steps: per-block bounding boxes (bbox_partial), curve keys (hilbert_keys), CUB radix sort and a
// gather of the sorted positions into TgtPos records; up to RANK_MAX particles order_rank counts
// places instead.  Keys have 21 bits an axis at every size: the cube is as wide as the farthest
// particle makes it, and with 10 bits one particle 1,000 extents away left all others in the
// caller's order, every tile of 64 near every other (FP32-comp UJ of 60,000 3.4 -> 10.8 ms; 4.7
// with 21, for the few wide tiles and warps that hold the particle).  order_rank compares their
// top 32 bits at first, four to a 16-byte read, and all 63 where particles share those.
#include "internal.h"

#include <cub/device/device_radix_sort.cuh>

namespace vpm {

constexpr int BB_BLOCKS = 256;
constexpr int BB_THREADS = 256;

constexpr int KEY_BITS = 21;   // an axis

// Spread the low 21 bits of v so that bit i moves to bit 3i.
__device__ __forceinline__ uint64_t spread3(uint64_t v)
{
    v &= 0x1fffffULL;
    v = (v | (v << 32)) & 0x1f00000000ffffULL;
    v = (v | (v << 16)) & 0x1f0000ff0000ffULL;
    v = (v | (v << 8)) & 0x100f00f00f00f00fULL;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ULL;
    v = (v | (v << 2)) & 0x1249249249249249ULL;
    return v;
}

// Index along Hilbert's curve of the cell q of a 2^KEY_BITS cube (J. Skilling, "Programming the
// Hilbert curve", AIP Conf. Proc. 707, 2004: axes to transpose, then the bits interleaved).
__device__ __forceinline__ uint64_t hilbert_index(uint32_t (&q)[3])
{
    for (uint32_t m = 1u << (KEY_BITS - 1); m > 1; m >>= 1) {
        const uint32_t p = m - 1;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            if (q[i] & m) {
                q[0] ^= p;
            } else {
                const uint32_t t = (q[0] ^ q[i]) & p;
                q[0] ^= t;
                q[i] ^= t;
            }
        }
    }
    q[1] ^= q[0];
    q[2] ^= q[1];
    uint32_t t = 0;
    for (uint32_t m = 1u << (KEY_BITS - 1); m > 1; m >>= 1)
        if (q[2] & m) t ^= m - 1;
#pragma unroll
    for (int i = 0; i < 3; i++) q[i] ^= t;
    return spread3(q[0]) << 2 | spread3(q[1]) << 1 | spread3(q[2]);
}

__global__ void __launch_bounds__(BB_THREADS)
bbox_partial(int64_t n, const double* __restrict__ x, double* __restrict__ part)
{
    __shared__ double red[6][BB_THREADS];
    double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t i = blockIdx.x * (int64_t)BB_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * BB_THREADS) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double v = x[3 * i + k];
            mn[k] = fmin(mn[k], v);
            mx[k] = fmax(mx[k], v);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) { red[k][threadIdx.x] = mn[k]; red[3 + k][threadIdx.x] = mx[k]; }
    __syncthreads();
    for (int off = BB_THREADS / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                red[k][threadIdx.x] = fmin(red[k][threadIdx.x], red[k][threadIdx.x + off]);
                red[3 + k][threadIdx.x] = fmax(red[3 + k][threadIdx.x], red[3 + k][threadIdx.x + off]);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x < 6) part[blockIdx.x * 6 + threadIdx.x] = red[threadIdx.x][0];
}

__device__ __forceinline__ TgtPos target_of(const double* __restrict__ x, int64_t i)
{
    TgtPos t;
    t.x = x[3 * i]; t.y = x[3 * i + 1]; t.z = x[3 * i + 2];
    t.idx = (int32_t)i; t.pad = 0;
    return t;
}

// aux receives the key's top 32 bits (RANK) or the index
template <bool RANK>
__global__ void __launch_bounds__(BB_THREADS)
hilbert_keys(int64_t n, const double* __restrict__ x, const double* __restrict__ part, uint64_t* __restrict__ keys,
             uint32_t* __restrict__ aux)
{
    // The box from the 256 partial ones, a warp a side, and the scale, once a block: the FP64 pipe
    // (16 cycles a warp instruction) is what this kernel waits for, and with every thread at all of
    // it 5,600 particles took 11.2 us and 100,000 took 28.
    __shared__ double box[6], scale;
    static_assert(BB_BLOCKS == 256 && BB_THREADS >= 192, "six warps, eight boxes a lane");
    constexpr uint32_t TOP = (1u << KEY_BITS) - 1u;
    if (threadIdx.x < 192) {
        const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
        double v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = part[(lane + 32 * j) * 6 + k];
#pragma unroll
        for (int j = 1; j < 8; j++) v[0] = k < 3 ? fmin(v[0], v[j]) : fmax(v[0], v[j]);
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) {
            const double o = __shfl_xor_sync(0xffffffffu, v[0], m);
            v[0] = k < 3 ? fmin(v[0], o) : fmax(v[0], o);
        }
        if (lane == 0) box[k] = v[0];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double ext = fmax(fmax(fmax(box[3] - box[0], box[4] - box[1]), box[5] - box[2]), 0.0);
        scale = ext > 0.0 ? (double)TOP / ext : 0.0;
    }
    __syncthreads();
    const int64_t i = blockIdx.x * (int64_t)BB_THREADS + threadIdx.x;
    if (i >= n) return;
    uint32_t q[3];
#pragma unroll
    for (int k = 0; k < 3; k++)   // the conversion takes values below 0 to 0, the minimum the rest (NaN too) to the top
        q[k] = min(__double2uint_rz((x[3 * i + k] - box[k]) * scale), TOP);
    const uint64_t key = hilbert_index(q);
    keys[i] = key;
    aux[i] = RANK ? (uint32_t)(key >> (3 * KEY_BITS - 32)) : (uint32_t)i;
}

__global__ void gather_targets(int64_t n, const double* __restrict__ x, const uint32_t* __restrict__ perm,
                               TgtPos* __restrict__ out)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n) return;
    out[t] = target_of(x, perm ? (int64_t)perm[t] : t);
}

static inline size_t align256(size_t b) { return (b + 255) / 256 * 256; }

// Up to RANK_MAX particles: each one's place is the number of keys before it, counted (lane =
// particle, the block's warps share the keys), and its record goes there: one launch for the sort's
// nine and the gather, but n^2 compares.  UJ calls with the sort / with ranks, us: 4,099 293 / 197,
// 16,000 618 / 557, 20,000 754 / 710, 24,000 949 / 921, 28,000 1118 / 1125, 32,000 1370 / 1412.  A sort
// of everything in one block took 20 us more at 6,100 than the ranks, and as long at 1,400.
constexpr int64_t RANK_MAX = 27648;
constexpr int RANK_THREADS = 1024;
__global__ void __launch_bounds__(RANK_THREADS)
order_rank(int n, const double* __restrict__ x, const uint32_t* __restrict__ hi, const uint64_t* __restrict__ keys,
           TgtPos* __restrict__ out)
{
    __shared__ int part[RANK_THREADS / 32][32];
    constexpr int W = RANK_THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i0 = blockIdx.x * 32, i = i0 + lane, ic = min(i, n - 1);
    const uint32_t top = hi[ic];
    const uint64_t key = keys[ic];
    TgtPos t;
    if (warp == 0) t = target_of(x, ic);
    // The keys before the block's own 32 and those after them, by their top bits or, where a lane's own
    // are among these, in full; then the 32 (quads own .. own + 7).  Equal keys keep the caller's order.
    const uint4* h4 = (const uint4*)hi;
    const ulonglong2* k2 = (const ulonglong2*)keys;
    const int own = i0 / 4, quads = n / 4;
    int c = 0;
    bool tie = false;
    auto tops = [&](int q) {
        const uint4 k = h4[q];
        c += (k.x < top) + (k.y < top) + (k.z < top) + (k.w < top);
        tie = tie || k.x == top || k.y == top || k.z == top || k.w == top;
    };
#pragma unroll 4
    for (int q = warp; q < own; q += W) tops(q);
#pragma unroll 4
    for (int q = own + 8 + warp; q < quads; q += W) tops(q);
    if (__any_sync(0xffffffffu, tie)) {
        c = 0;
#pragma unroll 4
        for (int q = warp; q < own; q += W) {
            const ulonglong2 a = k2[2 * q], b = k2[2 * q + 1];
            c += (a.x <= key) + (a.y <= key) + (b.x <= key) + (b.y <= key);
        }
#pragma unroll 4
        for (int q = own + 8 + warp; q < quads; q += W) {
            const ulonglong2 a = k2[2 * q], b = k2[2 * q + 1];
            c += (a.x < key) + (a.y < key) + (b.x < key) + (b.y < key);
        }
    }
    auto before = [&](uint64_t k, int j) { return k < key || (k == key && j < i); };
    if (warp < 8 && own + warp < quads) {
        const int j = 4 * (own + warp);
        const ulonglong2 a = k2[j / 2], b = k2[j / 2 + 1];
        c += before(a.x, j) + before(a.y, j + 1) + before(b.x, j + 2) + before(b.y, j + 3);
    }
    if (warp == 0)
        for (int j = n / 4 * 4; j < n; j++) c += before(keys[j], j);
    part[warp][lane] = c;
    __syncthreads();
    if (warp != 0 || i >= n) return;
    c = 0;
#pragma unroll
    for (int w = 0; w < RANK_THREADS / 32; w++) c += part[w][lane];
    out[c] = t;
}

static cudaError_t sort_keys(void* tmp, size_t& bytes, uint64_t* k0, uint64_t* k1, uint32_t* i0, uint32_t* i1,
                             int64_t n, cudaStream_t st)
{
    return cub::DeviceRadixSort::SortPairs(tmp, bytes, k0, k1, i0, i1, (int)n, 0, 3 * KEY_BITS, st);
}

static size_t sort_tmp(int64_t nt)
{
    size_t tmp = 0;
    sort_keys(nullptr, tmp, nullptr, nullptr, nullptr, nullptr, nt, nullptr);
    return tmp;
}

size_t order_bytes(int64_t nt)
{
    return align256(BB_BLOCKS * 6 * sizeof(double)) + 2 * align256(nt * sizeof(uint64_t)) +
           2 * align256(nt * sizeof(int32_t)) + align256(sort_tmp(nt)) + align256(nt * sizeof(TgtPos));
}

const TgtPos* ordered_targets(int64_t nt, void* scratch)
{
    return (const TgtPos*)((char*)scratch + order_bytes(nt) - align256(nt * sizeof(TgtPos)));
}

cudaError_t order_targets(int64_t nt, const double* xt, void* scratch, size_t scratch_bytes, cudaStream_t st,
                          int64_t* launches, const TgtPos** out)
{
    char* p = (char*)scratch;
    double* part = (double*)p;            p += align256(BB_BLOCKS * 6 * sizeof(double));
    uint64_t* k0 = (uint64_t*)p;          p += align256(nt * sizeof(uint64_t));
    uint64_t* k1 = (uint64_t*)p;          p += align256(nt * sizeof(uint64_t));
    uint32_t* i0 = (uint32_t*)p;          p += align256(nt * sizeof(int32_t));
    uint32_t* i1 = (uint32_t*)p;          p += align256(nt * sizeof(int32_t));
    size_t tmp = sort_tmp(nt);
    void* tmpp = p;                       p += align256(tmp);
    TgtPos* tp = (TgtPos*)p;              p += align256(nt * sizeof(TgtPos));
    if ((size_t)(p - (char*)scratch) > scratch_bytes) return cudaErrorInvalidValue;
    const unsigned nb = (unsigned)((nt + BB_THREADS - 1) / BB_THREADS);
    const uint32_t* perm = nullptr;
    if (nt > 1) {
        bbox_partial<<<BB_BLOCKS, BB_THREADS, 0, st>>>(nt, xt, part);
        *launches += 2;
        if (nt <= RANK_MAX) {
            hilbert_keys<true><<<nb, BB_THREADS, 0, st>>>(nt, xt, part, k0, i0);
            order_rank<<<(unsigned)((nt + 31) / 32), RANK_THREADS, 0, st>>>((int)nt, xt, i0, k0, tp);
            *launches += 1;
            *out = tp;
            return cudaGetLastError();
        }
        hilbert_keys<false><<<nb, BB_THREADS, 0, st>>>(nt, xt, part, k0, i0);
        cudaError_t e = sort_keys(tmpp, tmp, k0, k1, i0, i1, nt, st);
        if (e != cudaSuccess) return e;
        *launches += 1;  // CUB's onesweep passes are counted as one library call
        perm = i1;
    }
    gather_targets<<<nb, BB_THREADS, 0, st>>>(nt, xt, perm, tp);
    *launches += 1;
    *out = tp;
    return cudaGetLastError();
}

}  // namespace vpm
