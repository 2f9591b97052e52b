// Learned output-size predictor (no counterpart in the reference): per-block
// statistics of a volume, exact per-block triangle counts, and a small MLP
// (34 -> 64 -> 64 -> 1, ReLU, float32) with hand-written forward, backward
// and Adam kernels.
//
// Blocks are 16^3 cells (17^3 points, clipped at the grid's far faces),
// numbered (bz * nby + by) * nbx + bx.  A block's statistics (34 floats):
// min, max and a 32-bin histogram of its point values over [min, max]
// (fractions of its points).  They do not depend on the isovalue, so they are
// computed once per resident volume; the network's 34 inputs for an
// isovalue are (min - iso) / (max - min), (max - iso) / (max - min) and the
// 32 fractions.  A block has triangles only when min < iso <= max (some
// corner below, some at or above); the network is trained on and applied to
// those blocks; the package trains its output on triangles / 256.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "../../include/miniiso.h"
#include "iso_device.cuh"
#include "iso_kernels.h"

namespace iso {

constexpr int kBlock = ISO_BLOCK;  // cells per block edge
constexpr int kIn = ISO_MLP_IN, kHid = ISO_MLP_HIDDEN;
// parameter layout: W1 [kIn][kHid], b1 [kHid], W2 [kHid][kHid], b2 [kHid], W3 [kHid], b3
constexpr int kOffB1 = kIn * kHid, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid, kOffW3 = kOffB2 + kHid,
              kOffB3 = kOffW3 + kHid, kParams = kOffB3 + 1;
static_assert(kParams == ISO_MLP_PARAMS, "parameter count");

struct BlockDims {
    int nbx, nby, nbz;
};

inline BlockDims block_dims(const Grid& g)
{
    auto nb = [](int n) { return n < 2 ? 0 : (n - 1 + kBlock - 1) / kBlock; };
    return {nb(g.nx), nb(g.ny), nb(g.nz)};
}

// ---- per-block statistics: one CTA per block ------------------------------
// Thread t takes the points (t & 15, t >> 4 and t >> 4 | 8, z) of the block's 17
// planes and five or so of the points past its 16th column and row: 39 values,
// loaded once, all at the same time, and kept in registers from the minimum and
// maximum to the histogram, which has a copy for every fourth lane.  What bounds
// it: a block's chain from its first load to its last store, and 20 instructions a
// point.  320^3 (8,000 blocks): 36 us against 42 with 256 threads of 20 values, whose
// fixed work was 40% of the instructions, and 238 with each point's place divided
// out of its number and the block read twice.  64 threads of 77 values spill (48 us).
constexpr int kStatThreads = 128, kStatRows = 256 / kStatThreads, kStatWarps = kStatThreads / 32;
constexpr int kStatVals = kStatRows * (kBlock + 3) + 1, kHistCopies = 4;

__global__ void __launch_bounds__(kStatThreads, 1024 / kStatThreads) k_block_stats(const float* __restrict__ vol, Grid g, BlockDims bd,
                                                        float* __restrict__ stats)
{
    __shared__ float s_min[kStatWarps], s_max[kStatWarps];
    __shared__ unsigned s_hist[32 * kHistCopies];
    const int b = blockIdx.x;
    const int bx = b % bd.nbx, by = (b / bd.nbx) % bd.nby, bz = b / (bd.nbx * bd.nby);
    const int x0 = bx * kBlock, y0 = by * kBlock, z0 = bz * kBlock;
    const int ex = min(kBlock, g.nx - 1 - x0) + 1, ey = min(kBlock, g.ny - 1 - y0) + 1,
              ez = min(kBlock, g.nz - 1 - z0) + 1;  // points per edge
    const int npts = ex * ey * ez;
    const int t = threadIdx.x, u = t & 15, v = t >> 4;
    const long long plane = (long long)g.nx * g.ny;
    const float* base = vol + (long long)z0 * plane + (long long)y0 * g.nx + x0;
    float val[kStatVals];
    unsigned long long have = 0ull;  // bit q: val[q] is a point of a block that is cut off
    const bool full = ex == kBlock + 1 && ey == kBlock + 1 && ez == kBlock + 1;
    // the last of them: (16, t, 16) and (t, 16, 16) for t < 16, (16, 16, t) for t <= 16
    const int wx = t < 16 ? kBlock : (t < 32 ? t - 16 : kBlock), wy = t < 16 ? t : kBlock, wz = t < 32 ? kBlock : t - 32;
    const bool wmine = t < 32 + kBlock + 1;
    const float* rest = base + wz * plane + (long long)wy * g.nx + wx;
    if (full) {
#pragma unroll
        for (int h = 0; h < kStatRows; ++h) {
            const int vv = v + kStatThreads / 16 * h;
            const float* core = base + (long long)vv * g.nx + u;
#pragma unroll
            for (int z = 0; z <= kBlock; ++z) val[(kBlock + 3) * h + z] = __ldg(core + z * plane);
            val[(kBlock + 3) * h + kBlock + 1] = __ldg(base + vv * plane + (long long)u * g.nx + kBlock);  // (16, u, vv)
            val[(kBlock + 3) * h + kBlock + 2] = __ldg(base + vv * plane + (long long)kBlock * g.nx + u);  // (u, 16, vv)
        }
        val[kStatVals - 1] = wmine ? __ldg(rest) : val[0];
    } else {  // a block cut off at the grid's far faces; a value it does not have stands for its first point
        auto take = [&](int q, const float* p, bool ok) {
            val[q] = __ldg(ok ? p : base);
            have |= (ok ? 1ull : 0ull) << q;
        };
#pragma unroll
        for (int h = 0; h < kStatRows; ++h) {
            const int vv = v + kStatThreads / 16 * h;
            const float* core = base + (long long)vv * g.nx + u;
#pragma unroll
            for (int z = 0; z <= kBlock; ++z) take((kBlock + 3) * h + z, core + z * plane, u < ex && vv < ey && z < ez);
            take((kBlock + 3) * h + kBlock + 1, base + vv * plane + (long long)u * g.nx + kBlock,
                 kBlock < ex && u < ey && vv < ez);
            take((kBlock + 3) * h + kBlock + 2, base + vv * plane + (long long)kBlock * g.nx + u,
                 u < ex && kBlock < ey && vv < ez);
        }
        take(kStatVals - 1, rest, wmine && wx < ex && wy < ey && wz < ez);
    }
    float lo = 3.402823466e38f, hi = -3.402823466e38f;
#pragma unroll
    for (int q = 0; q < kStatVals; ++q) {  // every val is one of the block's points
        lo = fminf(lo, val[q]);
        hi = fmaxf(hi, val[q]);
    }
    for (int d = 16; d > 0; d >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d));
    }
    const int warp = t >> 5, lane = t & 31;
    if (lane == 0) {
        s_min[warp] = lo;
        s_max[warp] = hi;
    }
#pragma unroll
    for (int q = 0; q < 32 * kHistCopies; q += kStatThreads) s_hist[q + t] = 0u;
    __syncthreads();
    lo = s_min[0];
    hi = s_max[0];
    for (int w = 1; w < kStatWarps; ++w) {
        lo = fminf(lo, s_min[w]);
        hi = fmaxf(hi, s_max[w]);
    }
    const float range = hi - lo;
    const float scale = range > 0.f ? 32.f / range : 0.f;
    unsigned* hist = s_hist + (t & (kHistCopies - 1));
    auto count = [&](int q) { atomicAdd(hist + kHistCopies * min(31, max(0, (int)((val[q] - lo) * scale))), 1u); };
    if (full) {
#pragma unroll
        for (int q = 0; q < kStatVals - 1; ++q) count(q);
        if (wmine) count(kStatVals - 1);
    } else {
#pragma unroll
        for (int q = 0; q < kStatVals; ++q)
            if ((have >> q) & 1ull) count(q);
    }
    __syncthreads();
    float* o = stats + (size_t)b * kIn;
    if (t == 0) {
        o[0] = lo;
        o[1] = hi;
    }
    constexpr int kPer = kStatThreads / 32, kEach = kHistCopies / kPer;  // threads to a bin, copies to a thread
    unsigned n = 0u;
#pragma unroll
    for (int q = 0; q < kEach; ++q) n += s_hist[kEach * t + q];
#pragma unroll
    for (int d = kPer / 2; d > 0; d >>= 1) n += __shfl_xor_sync(0xffffffffu, n, d);
    if (t % kPer == 0) o[2 + t / kPer] = (float)n / (float)npts;
}

// ---- exact triangles per block from the count pass's bit rows -------------
// One thread per (cell row (j, k), word w): the triangles of the word's 32
// cells (tris_of_word, the count pass's formula) split into its two
// 16-cell halves, each half one block's.
__global__ void k_block_tris(const uint32_t* __restrict__ bits, Grid g, BlockDims bd, int* __restrict__ counts)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long rows = (long long)(g.ny - 1) * (g.nz - 1);
    if (t >= rows * g.W) return;
    const int w = (int)(t % g.W);
    const long long cr = t / g.W;
    const int j = (int)(cr % (g.ny - 1)), k = (int)(cr / (g.ny - 1));
    auto word = [&](int jj, int kk, int ww) -> uint32_t {
        return ww < g.W ? __ldg(&bits[((long long)kk * g.ny + jj) * g.W + ww]) : 0u;
    };
    const uint32_t a = word(j, k, w), b = word(j + 1, k, w), c = word(j, k + 1, w), d = word(j + 1, k + 1, w);
    const uint32_t ash = (a >> 1) | (word(j, k, w + 1) << 31), bsh = (b >> 1) | (word(j + 1, k, w + 1) << 31);
    const uint32_t csh = (c >> 1) | (word(j, k + 1, w + 1) << 31), dsh = (d >> 1) | (word(j + 1, k + 1, w + 1) << 31);
    const uint32_t cells = validmask(w, g.nx - 1);
    const int by = j / kBlock, bz = k / kBlock;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const uint32_t m = cells & (half ? 0xffff0000u : 0x0000ffffu);
        if (!m) continue;
        const uint32_t n = tris_of_word(a, ash, bsh, b, c, csh, dsh, d, m);
        if (n) atomicAdd(&counts[((long long)bz * bd.nby + by) * bd.nbx + 2 * w + half], (int)n);
    }
}

// ---- the network -----------------------------------------------------------
// A CTA of 256 threads takes tiles of 64 samples.  Everything that is summed over
// is the slow index in shared memory (x, h1, d2, d1 by input or unit, 64 samples
// side by side; the weights by input, 64 units side by side), so that a thread
// makes a 4 x 4 part of a product from two 16-byte loads per term; a warp's lanes
// cover 32 samples by 16 units.  The weight gradients are sums over the samples: a
// thread makes those of 4 (of the first layer 3) units by 4 of the next layer from
// 16-byte loads of four samples, two samples per instruction, in registers over
// all tiles of the CTA; eight CTAs of a cluster then add theirs up through
// distributed shared memory, so that a gradient gets one global addition per
// cluster instead of one per CTA (1.7 million on 6,465 addresses for 16,384
// samples).  Sums are fused multiply-adds.
// What bounds it, for 16,384 samples (256 tiles; 34 us, 38 with 512 threads of 4 x
// 2, 106 with a row of 16 units per thread and every CTA's own additions): the
// bytes that shared memory returns to registers (a broadcast counts like any other
// load; 0.5 floats per multiply-add, 0.75 with 4 x 2), then the latency of the
// weights' way in, five barriers a tile and the cluster's end.
constexpr int kTile = 64, kRow = kTile + 4;  // samples of a tile; of a row in shared memory (16-byte aligned)
constexpr int kMlpCluster = 8;
constexpr int kUnitRow = kHid + 4;
constexpr int kMlpThreads = 256;

struct __align__(16) MlpSmem {
    float w1[kIn * kHid], w2[kHid * kHid], b1[kHid], b2[kHid], w3[kHid], b3[4];
    float x[kIn * kRow], h1[kHid * kRow];
    float yp[4 * kTile];                    // the outputs' parts, by group of 16 units
};

struct __align__(16) MlpGradSmem {
    MlpSmem f;
    float w2t[kHid * kUnitRow];             // w2 by unit of the second layer, rows four floats apart in the banks
    float d2[kHid * kRow], d1[kHid * kRow];
    float dy[kTile], w3p[2 * kHid];         // the two sample halves' parts of dW3
};
static_assert(sizeof(float) * kParams <= sizeof(float) * 2 * kHid * kRow, "a CTA's gradients fit over d2 and d1");

// The parameters into shared memory, w2t (if any) the second layer's weights by its unit. Unrolled, so that a thread's
// loads are on their way together.
__device__ __forceinline__ void load_params(MlpSmem& s, const float* __restrict__ p, float* w2t = nullptr)
{
    const int t = threadIdx.x;
    static_assert(kHid * kHid % kMlpThreads == 0, "");
#pragma unroll
    for (int q = 0; q < kHid * kHid; q += kMlpThreads) {
        const int i = q + t;
        const float w = __ldg(p + kOffW2 + i);
        s.w2[i] = w;
        if (w2t) w2t[(i % kHid) * kUnitRow + i / kHid] = w;
    }
#pragma unroll
    for (int q = 0; q < kIn * kHid; q += kMlpThreads)
        if (q + t < kIn * kHid) s.w1[q + t] = __ldg(p + q + t);
    if (t < kHid) {
        s.b1[t] = __ldg(p + kOffB1 + t);
        s.b2[t] = __ldg(p + kOffB2 + t);
        s.w3[t] = __ldg(p + kOffW3 + t);
    }
    if (t == 0) s.b3[0] = __ldg(p + kOffB3);
}

// A thread's 4 x 4 part of a tile: warp w the samples 32 (w & 1) on and units 16 (w >> 1) on, lane l of them 4 (l >> 2)
// and 4 (l & 3) on.
__device__ __forceinline__ int part_row() { return 32 * ((threadIdx.x >> 5) & 1) + 4 * ((threadIdx.x & 31) >> 2); }
__device__ __forceinline__ int part_col() { return 16 * (threadIdx.x >> 6) + 4 * (threadIdx.x & 3); }

// Output of the tile's sample r, after forward_tile.
__device__ __forceinline__ float tile_y(const MlpSmem& s, int r)
{
    float y = s.b3[0];
#pragma unroll
    for (int q = 0; q < 4; ++q) y += s.yp[q * kTile + r];
    return y;
}

// Input c of a block's statistics st for the isovalue iso.
__device__ __forceinline__ float mlp_input(const float* __restrict__ st, float iso, int c)
{
    if (c >= 2) return st[c];
    const float range = st[1] - st[0];
    return range > 0.f ? (st[c] - iso) / range : 0.f;
}

// Inputs of the tile's samples from their block statistics.
__device__ __forceinline__ void load_tile(MlpSmem& s, const float* __restrict__ stats, const float* __restrict__ iso,
                                          long long base, long long n)
{
#pragma unroll
    for (int i0 = 0; i0 < kTile * kIn; i0 += kMlpThreads) {
        const int i = i0 + threadIdx.x, r = i / kIn, c = i % kIn;
        if (kTile * kIn % kMlpThreads != 0 && i >= kTile * kIn) break;
        const long long q = base + r;
        s.x[c * kRow + r] = q < n ? mlp_input(stats + q * kIn, iso[q], c) : 0.f;
    }
}

// out[b][a] = the product's value for sample r0 + a and unit c0 + b: bias + sum over K of in[k][sample] w[k][unit].
template <int K, int WROW = kHid>
__device__ __forceinline__ void mlp_product(const float* in, const float* w, const float* bias, int r0, int c0,
                                            float (&out)[4][4])
{
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int a = 0; a < 4; ++a) out[b][a] = bias ? bias[c0 + b] : 0.f;
#pragma unroll 8
    for (int k = 0; k < K; ++k) {
        const float4 xv = *reinterpret_cast<const float4*>(in + k * kRow + r0);
        const float4 wv = *reinterpret_cast<const float4*>(w + k * WROW + c0);
        const float xs[4] = {xv.x, xv.y, xv.z, xv.w}, ws[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int a = 0; a < 4; ++a) out[b][a] = __fmaf_rn(xs[a], ws[b], out[b][a]);
    }
}

// Two fused multiply-adds at once, and the sum of a pair.
__device__ __forceinline__ void fma_pair(unsigned long long& acc, unsigned long long a, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pair_sum(unsigned long long v)
{
    return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

__device__ __forceinline__ void store_units(float* o, int r0, int c0, const float (&v)[4][4])
{
#pragma unroll
    for (int b = 0; b < 4; ++b)
        *reinterpret_cast<float4*>(o + (c0 + b) * kRow + r0) = make_float4(v[b][0], v[b][1], v[b][2], v[b][3]);
}

// h1 (in shared memory), h2 (the thread's 4 x 4 part) and the parts of the outputs of the tile.
__device__ __forceinline__ void forward_tile(MlpSmem& s, float (&h2)[4][4])
{
    const int r0 = part_row(), c0 = part_col();
    float h1[4][4];
    mlp_product<kIn>(s.x, s.w1, s.b1, r0, c0, h1);
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int a = 0; a < 4; ++a) h1[b][a] = fmaxf(h1[b][a], 0.f);
    store_units(s.h1, r0, c0, h1);
    __syncthreads();
    mlp_product<kHid>(s.h1, s.w2, s.b2, r0, c0, h2);
    float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            h2[b][a] = fmaxf(h2[b][a], 0.f);
            part[a] = __fmaf_rn(h2[b][a], s.w3[c0 + b], part[a]);
        }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int d = 1; d < 4; d <<= 1) part[a] += __shfl_xor_sync(0xffffffffu, part[a], d);
    }
    if ((threadIdx.x & 3) == 0)
        *reinterpret_cast<float4*>(s.yp + (c0 / 16) * kTile + r0) = make_float4(part[0], part[1], part[2], part[3]);
    __syncthreads();
}

__global__ void __launch_bounds__(kMlpThreads) k_mlp_forward(const float* __restrict__ params, const float* __restrict__ stats,
                                                     const float* __restrict__ iso, long long n, float* __restrict__ y)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    MlpSmem& s = *reinterpret_cast<MlpSmem*>(s_raw);
    load_params(s, params);
    for (long long base = (long long)blockIdx.x * kTile; base < n; base += (long long)gridDim.x * kTile) {
        load_tile(s, stats, iso, base, n);
        __syncthreads();
        float h2[4][4];
        forward_tile(s, h2);
        if (threadIdx.x < kTile && base + threadIdx.x < n) y[base + threadIdx.x] = tile_y(s, threadIdx.x);
    }
}

// Prediction for many (block statistics, isovalue) sets in one launch: the
// samples are the sets' blocks one after another; a block counts when
// min < iso <= max, and max(y, 0) of those is added to its set's total.  A tile's
// samples of one set are summed before the global addition.
constexpr int kMaxSets = 128;
struct PredictSets {
    int n;
    long long start[kMaxSets + 1];  // first sample of each set; start[n] = all samples
    const float* stats[kMaxSets];
    float iso[kMaxSets];
};

__global__ void __launch_bounds__(kMlpThreads) k_mlp_predict(const float* __restrict__ params, PredictSets sets,
                                                     float* __restrict__ totals)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    MlpSmem& s = *reinterpret_cast<MlpSmem*>(s_raw);
    __shared__ int s_set[kTile];
    load_params(s, params);
    const long long n = sets.start[sets.n];
    for (long long base = (long long)blockIdx.x * kTile; base < n; base += (long long)gridDim.x * kTile) {
        if (threadIdx.x < kTile) {  // the set of sample base + t (-1: past the end or an inactive block)
            const long long q = base + threadIdx.x;
            int set = -1;
            if (q < n) {
                int lo = 0, hi = sets.n - 1;  // last set with start <= q
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (sets.start[mid] <= q) lo = mid;
                    else hi = mid - 1;
                }
                const float* st = sets.stats[lo] + (q - sets.start[lo]) * kIn;
                if (st[0] < sets.iso[lo] && st[1] >= sets.iso[lo]) set = lo;
            }
            s_set[threadIdx.x] = set;
        }
        if (!__syncthreads_or(threadIdx.x < kTile && s_set[threadIdx.x] >= 0)) continue;  // no active block
#pragma unroll
        for (int i0 = 0; i0 < kTile * kIn; i0 += kMlpThreads) {
            const int i = i0 + threadIdx.x, r = i / kIn, c = i % kIn;
            if (kTile * kIn % kMlpThreads != 0 && i >= kTile * kIn) break;
            const int set = s_set[r];
            s.x[c * kRow + r] =
                set >= 0 ? mlp_input(sets.stats[set] + (base + r - sets.start[set]) * kIn, sets.iso[set], c) : 0.f;
        }
        __syncthreads();
        float h2[4][4];
        forward_tile(s, h2);
        if (threadIdx.x < 32) {  // the sets of a tile are neighbours
            const int lane = threadIdx.x, a = s_set[lane], b = s_set[lane + 32];
            const float ya = a >= 0 ? fmaxf(tile_y(s, lane), 0.f) : 0.f, yb = b >= 0 ? fmaxf(tile_y(s, lane + 32), 0.f) : 0.f;
            const int none = sets.n;
            int q = __reduce_min_sync(0xffffffffu, min(a >= 0 ? a : none, b >= 0 ? b : none));
            while (q < none) {
                float v = (a == q ? ya : 0.f) + (b == q ? yb : 0.f);
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
                if (lane == 0) atomicAdd(&totals[q], v);
                q = __reduce_min_sync(0xffffffffu, min(a > q ? a : none, b > q ? b : none));
            }
        }
        __syncthreads();
    }
}

// Gradient of the mean squared error (1/n) sum (y - target)^2 with respect
// to every parameter, added into grads (zeroed by the caller); the loss
// into *loss.
__global__ void __cluster_dims__(kMlpCluster, 1, 1) __launch_bounds__(kMlpThreads, 2)
    k_mlp_gradient(const float* __restrict__ params, const float* __restrict__ stats, const float* __restrict__ iso,
                   const float* __restrict__ target, long long n, float* __restrict__ grads, float* __restrict__ loss)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    MlpGradSmem& s = *reinterpret_cast<MlpGradSmem*>(s_raw);
    const int t = threadIdx.x, r0 = part_row(), c0 = part_col();
    // weight gradients: units i = gi + 16 a of one layer by l = gl + 32 b of the next
    const int gi = 4 * ((t >> 5) & 3) + ((t & 31) >> 3), gl = 8 * (t >> 7) + (t & 7);
    load_params(s.f, params, s.w2t);
    unsigned long long gw2[4][4] = {}, gw1[3][4] = {};  // two sums each, of the even and of the odd samples
    float gw3[4] = {};
    float gb1 = 0.f, gb2 = 0.f, gb3 = 0.f, lsum = 0.f;
    const float inv_n = 1.f / (float)n;
    for (long long base = (long long)blockIdx.x * kTile; base < n; base += (long long)gridDim.x * kTile) {
        load_tile(s.f, stats, iso, base, n);
        __syncthreads();
        float h2[4][4];
        forward_tile(s.f, h2);
        if (t < kTile) {
            const long long q = base + t;
            float dy = 0.f;
            if (q < n) {
                const float e = tile_y(s.f, t) - target[q];
                lsum = __fmaf_rn(e, e, lsum);
                dy = 2.f * e * inv_n;
            }
            s.dy[t] = dy;
            gb3 += dy;
        }
        __syncthreads();
        // d2 = dy * w3 where h2 > 0; dW3 += h2 dy
        float d[4][4];
        {
            const float4 dv = *reinterpret_cast<const float4*>(s.dy + r0);
            const float dys[4] = {dv.x, dv.y, dv.z, dv.w};
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    d[b][a] = h2[b][a] > 0.f ? dys[a] * s.f.w3[c0 + b] : 0.f;
                    gw3[b] = __fmaf_rn(h2[b][a], dys[a], gw3[b]);
                }
        }
        store_units(s.d2, r0, c0, d);
        __syncthreads();
        // d1[sample][i] = sum_u d2[sample][u] w2[i][u] where h1 > 0
        mlp_product<kHid, kUnitRow>(s.d2, s.w2t, nullptr, r0, c0, d);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float4 hv = *reinterpret_cast<const float4*>(s.f.h1 + (c0 + b) * kRow + r0);
            d[b][0] = hv.x > 0.f ? d[b][0] : 0.f;
            d[b][1] = hv.y > 0.f ? d[b][1] : 0.f;
            d[b][2] = hv.z > 0.f ? d[b][2] : 0.f;
            d[b][3] = hv.w > 0.f ? d[b][3] : 0.f;
        }
        store_units(s.d1, r0, c0, d);
        __syncthreads();
        // the tile's weight gradients, four samples at a time
#pragma unroll 1
        for (int r = 0; r < kTile; r += 4) {
            ulonglong2 hv[4], dv[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) hv[a] = *reinterpret_cast<const ulonglong2*>(s.f.h1 + (gi + 16 * a) * kRow + r);
#pragma unroll
            for (int b = 0; b < 4; ++b) dv[b] = *reinterpret_cast<const ulonglong2*>(s.d2 + (gl + 16 * b) * kRow + r);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    fma_pair(gw2[a][b], hv[a].x, dv[b].x);
                    fma_pair(gw2[a][b], hv[a].y, dv[b].y);
                }
#pragma unroll
            for (int a = 0; a < 3; ++a)
                hv[a] = gi + 16 * a < kIn ? *reinterpret_cast<const ulonglong2*>(s.f.x + (gi + 16 * a) * kRow + r)
                                          : make_ulonglong2(0ull, 0ull);
#pragma unroll
            for (int b = 0; b < 4; ++b) dv[b] = *reinterpret_cast<const ulonglong2*>(s.d1 + (gl + 16 * b) * kRow + r);
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    fma_pair(gw1[a][b], hv[a].x, dv[b].x);
                    fma_pair(gw1[a][b], hv[a].y, dv[b].y);
                }
        }
        if (t < 2 * kHid) {  // db1, db2: one unit's samples per thread
            const float* row = t < kHid ? s.d1 + t * kRow : s.d2 + (t - kHid) * kRow;
            float sum = 0.f;
            for (int r = 0; r < kTile; r += 4) {
                const float4 v = *reinterpret_cast<const float4*>(row + r);
                sum += (v.x + v.y) + (v.z + v.w);
            }
            if (t < kHid) gb1 += sum;
            else gb2 += sum;
        }
        __syncthreads();  // the next tile overwrites x, h1, d2, d1
    }
    // the CTA's gradients, in the parameters' layout, over d2 and d1
    float* own = s.d2;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) own[kOffW2 + (gi + 16 * a) * kHid + gl + 16 * b] = pair_sum(gw2[a][b]);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (gi + 16 * a < kIn) own[(gi + 16 * a) * kHid + gl + 16 * b] = pair_sum(gw1[a][b]);
    if (t < kHid) own[kOffB1 + t] = gb1;
    else if (t < 2 * kHid) own[kOffB2 + t - kHid] = gb2;
#pragma unroll
    for (int b = 0; b < 4; ++b) {  // dW3: a warp's samples, then the halves
#pragma unroll
        for (int d = 4; d < 32; d <<= 1) gw3[b] += __shfl_xor_sync(0xffffffffu, gw3[b], d);
        if ((t & 31) < 4) s.w3p[((t >> 5) & 1) * kHid + c0 + b] = gw3[b];
    }
    if (t < kTile) {  // db3 and the loss: two warps
        for (int d = 16; d > 0; d >>= 1) {
            gb3 += __shfl_xor_sync(0xffffffffu, gb3, d);
            lsum += __shfl_xor_sync(0xffffffffu, lsum, d);
        }
        if ((t & 31) == 0) {
            s.dy[t >> 5] = gb3;
            s.dy[2 + (t >> 5)] = lsum;
        }
    }
    __syncthreads();
    if (t < kHid) own[kOffW3 + t] = s.w3p[t] + s.w3p[kHid + t];
    if (t == kHid) {
        own[kOffB3] = s.dy[0] + s.dy[1];
        atomicAdd(loss, (s.dy[2] + s.dy[3]) * inv_n);
    }
    // every CTA of the cluster adds up its eighth of the parameters
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    uint32_t rank;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    constexpr int kShare = (kParams + kMlpCluster - 1) / kMlpCluster;
    for (int i = t; i < kShare; i += kMlpThreads) {
        const int q = (int)rank * kShare + i;
        if (q < kParams) {
            float sum = 0.f;
#pragma unroll
            for (uint32_t c = 0; c < kMlpCluster; ++c) {
                uint32_t at;
                float v;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(own + q)), "r"(c));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
                sum += v;
            }
            if (sum != 0.f) atomicAdd(&grads[q], sum);
        }
    }
    // no CTA ends while another reads its shared memory
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// Adam (Kingma & Ba 2015) with bias correction; step counts from 1.
__global__ void k_mlp_adam(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                           const float* __restrict__ g, float lr, float c1, float c2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kParams) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

size_t mlp_smem() { return sizeof(MlpSmem); }

int mlp_blocks(long long n, int nsm, int per_sm)
{
    const long long tiles = (n + kTile - 1) / kTile;
    return (int)std::min<long long>(tiles, (long long)nsm * per_sm);
}

int device_sms()
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm > 0 ? nsm : 1;
}

void launch_block_tris(const Grid& g, const uint32_t* bits, int* counts, cudaStream_t s)
{
    const BlockDims bd = block_dims(g);
    const long long threads = (long long)(g.ny - 1) * (g.nz - 1) * g.W;
    if (threads <= 0) return;
    k_block_tris<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(bits, g, bd, counts);
}

long long block_count(const Grid& g)
{
    const BlockDims bd = block_dims(g);
    return (long long)bd.nbx * bd.nby * bd.nbz;
}

}  // namespace iso

namespace {
using iso::Grid;

iso_status launch_status(cudaError_t e) { return e == cudaSuccess ? ISO_OK : ISO_ERR_CUDA; }

bool grid_of(const iso_grid* gr, Grid& g)
{
    if (!gr) return false;
    for (int a = 0; a < 3; ++a)
        if (gr->dims[a] < 1 || gr->dims[a] > (1ll << 30)) return false;
    g = Grid{};
    g.nx = (int)gr->dims[0];
    g.ny = (int)gr->dims[1];
    g.nz = (int)gr->dims[2];
    g.W = (g.nx + 31) / 32;
    g.kd = g.kr = 0;
    g.ke = g.nz;
    g.R = (long long)g.ny * g.nz;
    return true;
}
}  // namespace

extern "C" {

int64_t iso_block_count(const iso_grid* grid)
{
    Grid g;
    if (!grid_of(grid, g)) return -1;
    return iso::block_count(g);
}

iso_status iso_block_stats(const float* volume, const iso_grid* grid, float* stats, void* stream)
{
    Grid g;
    if (!grid_of(grid, g)) return ISO_ERR_INVALID_ARG;
    const long long nb = iso::block_count(g);
    if (nb == 0) return ISO_OK;
    if (!volume || !stats) return ISO_ERR_INVALID_ARG;
    iso::k_block_stats<<<(unsigned)nb, iso::kStatThreads, 0, static_cast<cudaStream_t>(stream)>>>(volume, g, iso::block_dims(g),
                                                                                   stats);
    return launch_status(cudaGetLastError());
}

iso_status iso_mlp_forward(const float* params, const float* stats, const float* isovals, int64_t n, float* y,
                           void* stream)
{
    if (n < 0 || (n > 0 && (!params || !stats || !isovals || !y))) return ISO_ERR_INVALID_ARG;
    if (n == 0) return ISO_OK;
    const size_t smem = iso::mlp_smem();
    cudaFuncSetAttribute(iso::k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    iso::k_mlp_forward<<<iso::mlp_blocks(n, iso::device_sms(), 4), iso::kMlpThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        params, stats, isovals, n, y);
    return launch_status(cudaGetLastError());
}

iso_status iso_mlp_predict(const float* params, int64_t n_sets, const iso_block_set* sets, float* totals,
                           void* stream)
{
    if (n_sets < 0 || (n_sets > 0 && (!params || !sets || !totals))) return ISO_ERR_INVALID_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (n_sets == 0) return ISO_OK;
    if (cudaMemsetAsync(totals, 0, sizeof(float) * (size_t)n_sets, s) != cudaSuccess) return ISO_ERR_CUDA;
    const size_t smem = iso::mlp_smem();
    cudaFuncSetAttribute(iso::k_mlp_predict, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int nsm = iso::device_sms();
    for (int64_t s0 = 0; s0 < n_sets; s0 += iso::kMaxSets) {  // kMaxSets sets per launch
        iso::PredictSets ps{};
        ps.n = (int)std::min<int64_t>(iso::kMaxSets, n_sets - s0);
        long long at = 0;
        for (int q = 0; q < ps.n; ++q) {
            const iso_block_set& b = sets[s0 + q];
            if (b.n_blocks < 0 || (b.n_blocks > 0 && !b.stats)) return ISO_ERR_INVALID_ARG;
            ps.start[q] = at;
            ps.stats[q] = b.stats;
            ps.iso[q] = b.isoval;
            at += b.n_blocks;
        }
        ps.start[ps.n] = at;
        if (at == 0) continue;
        iso::k_mlp_predict<<<iso::mlp_blocks(at, nsm, 4), iso::kMlpThreads, smem, s>>>(params, ps, totals + s0);
        if (cudaGetLastError() != cudaSuccess) return ISO_ERR_CUDA;
    }
    return ISO_OK;
}

iso_status iso_mlp_gradient(const float* params, const float* stats, const float* isovals, const float* target,
                            int64_t n, float* grads, float* loss, void* stream)
{
    if (n <= 0 || !params || !stats || !isovals || !target || !grads || !loss) return ISO_ERR_INVALID_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(grads, 0, sizeof(float) * ISO_MLP_PARAMS, s) != cudaSuccess ||
        cudaMemsetAsync(loss, 0, sizeof(float), s) != cudaSuccess)
        return ISO_ERR_CUDA;
    const size_t smem = sizeof(iso::MlpGradSmem);
    cudaFuncSetAttribute(iso::k_mlp_gradient, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    // whole clusters; a CTA without a tile adds zeros
    const int blocks = (iso::mlp_blocks(n, iso::device_sms(), 2) + iso::kMlpCluster - 1) / iso::kMlpCluster *
                       iso::kMlpCluster;
    iso::k_mlp_gradient<<<blocks, iso::kMlpThreads, smem, s>>>(params, stats, isovals, target, n, grads, loss);
    return launch_status(cudaGetLastError());
}

iso_status iso_mlp_adam(float* params, float* m, float* v, const float* grads, int64_t step, float lr, void* stream)
{
    if (!params || !m || !v || !grads || step < 1) return ISO_ERR_INVALID_ARG;
    const double c1 = 1.0 - std::pow(0.9, (double)step), c2 = 1.0 - std::pow(0.999, (double)step);
    iso::k_mlp_adam<<<(ISO_MLP_PARAMS + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        params, m, v, grads, lr, (float)c1, (float)c2);
    return launch_status(cudaGetLastError());
}

}  // extern "C"
