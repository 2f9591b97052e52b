// Passes 1-3 of Flying Edges (flyingEdges/serial/FlyingEdgesAlgorithm.cpp:23-269)
// on sm_103a, with pass 1 (x-edge classification, trims) fused into pass 2
// (cube cases, per-row counts):
//
//   k_count_rows   (rows up to 1024 points, the volume at a 16-byte boundary;
//                  count_rows.cuh) a warp owns 1 to 64 neighbouring grid rows
//                  and a run of KC planes and marches along z, a bulk copy of
//                  its rows of plane k+2 in flight while plane k is counted.
//   k_count_warps  (up to 2048 points, any boundary) a CTA owns a block of 8
//                  grid rows, a warp per row.
//                  Either way each row's words of plane k+1 are classified
//                  straight from the volume into bit-per-point words -- the
//                  reference's edgeCases bytes are never materialised -- and
//                  counted for grid row (j,k): its cut x, y and z edges (the
//                  vertices it owns), the trims xl/xr, the triangles of cell
//                  row (j,k) and, for Marching Cubes, the vertices cell row
//                  (j,k) owns, all 32 cells of a word at once.  Writes the bit
//                  words for pass 4.  No warp waits for another.
//   k_count_wide   rows longer than 2048 points, walked in chunks.
//   k_scan_*       exclusive scans of the per-row counts in (k, j) order, the
//                  reference's row order: the first vertex / triangle / MC
//                  vertex of every row (gridEdge xstart and triCounter after
//                  pass 3) and the totals.
#include "batch_kernels.cuh"
#include "count_rows.cuh"
#include "iso_kernels.h"
#include <algorithm>

namespace iso {


// Raw values of one row held by a warp: lane l holds float4 l + 32u.
template <int U>
struct RowVals {
    float4 v[U];
};

template <int U>
__device__ __forceinline__ void load_row_vec4(const float* __restrict__ row, int nq, int lane, bool ok, RowVals<U>& r)
{
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int q = lane + 32 * u;
        r.v[u] = (ok && q < nq) ? __ldg(reinterpret_cast<const float4*>(row) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// Bit words "value >= iso" of a row: word w ends up in lane w % 32, slot w / 32.
template <int U, int NW>
__device__ __forceinline__ void words_vec4(const RowVals<U>& r, int nq, int lane, float iso, uint32_t (&out)[NW])
{
#pragma unroll
    for (int q = 0; q < NW; ++q) out[q] = 0u;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int f = lane + 32 * u;
        const float4 v = r.v[u];
        const uint32_t nib = f < nq ? ((uint32_t)(v.x >= iso) | ((uint32_t)(v.y >= iso) << 1) |
                                       ((uint32_t)(v.z >= iso) << 2) | ((uint32_t)(v.w >= iso) << 3))
                                    : 0u;
        uint32_t word = nib << (4 * (lane & 7));
        word |= __shfl_xor_sync(0xffffffffu, word, 1);
        word |= __shfl_xor_sync(0xffffffffu, word, 2);
        word |= __shfl_xor_sync(0xffffffffu, word, 4);
        // lanes 8g..8g+7 now hold word 4u+g; lane L wants word L + 32q
        const uint32_t x = __shfl_sync(0xffffffffu, word, 8 * (lane & 3));
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            if (u == (lane >> 2) + 8 * q) out[q] = x;
        }
    }
}

template <int NW>
__device__ __forceinline__ void words_scalar(const float* __restrict__ row, int nx, int W, bool ok, int lane, float iso,
                                             uint32_t (&out)[NW])
{
#pragma unroll
    for (int q = 0; q < NW; ++q) out[q] = 0u;
    for (int w = 0; w < W; ++w) {
        const int i = 32 * w + lane;
        const float v = (ok && i < nx) ? __ldg(row + i) : 0.f;
        const uint32_t m = __ballot_sync(0xffffffffu, ok && i < nx && v >= iso);
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            if (w == lane + 32 * q) out[q] = m;
        }
    }
}

// Next word (the source of bit i+1) of the lane's slot q.
template <int NW>
__device__ __forceinline__ uint32_t next_word(const uint32_t (&w)[NW], int q, int lane)
{
    const uint32_t dn = __shfl_down_sync(0xffffffffu, w[q], 1);
    const uint32_t wrap = __shfl_sync(0xffffffffu, w[q + 1 < NW ? q + 1 : q], 0);
    if (lane < 31) return dn;
    return q + 1 < NW ? wrap : 0u;
}

// Warp totals of row r; lane 0 stores them.
template <bool MC>
__device__ __forceinline__ void finish_row(RowCounts& rc, int lane, long long r, const Grid& g,
                                           uint4* __restrict__ rowcnt, uint2* __restrict__ trims,
                                           uint32_t* __restrict__ mccnt)
{
    rc.xc = __reduce_add_sync(0xffffffffu, rc.xc);
    rc.yc = __reduce_add_sync(0xffffffffu, rc.yc);
    rc.zc = __reduce_add_sync(0xffffffffu, rc.zc);
    rc.tc = __reduce_add_sync(0xffffffffu, rc.tc);
    if (MC) rc.mc = __reduce_add_sync(0xffffffffu, rc.mc);
    if (trims) {
        rc.first = __reduce_min_sync(0xffffffffu, rc.first);
        rc.last = __reduce_max_sync(0xffffffffu, rc.last);
    }
    if (lane == 0) {
        rowcnt[r] = make_uint4(rc.xc, rc.yc, rc.zc, rc.tc);
        if (trims) trims[r] = make_uint2(rc.first == 0xffffffffu ? (uint32_t)g.nx : rc.first, rc.last);
        if (MC) mccnt[r] = rc.mc;
    }
}

template <bool MC, bool VEC4, int U, int NW>
__global__ void __launch_bounds__(kThreads) k_count_warps(const float* __restrict__ vol, Grid g, float iso, int KC,
                                                          int nyb, const CaseTables* __restrict__ cases,
                                                          uint4* __restrict__ rowcnt, uint2* __restrict__ trims,
                                                          uint32_t* __restrict__ mccnt, uint32_t* __restrict__ bits_out)
{
    (void)cases;  // the counts need no case table (tris_of_word, mc_verts_of_word)
    const int jb = blockIdx.x % nyb, kc = blockIdx.x / nyb;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = jb * kCountRows + warp;
    if (j >= g.ny) return;
    const int kb = g.kr + kc * KC, ke = min(kb + KC, g.ke);
    const bool hasY = j < g.ny - 1;
    const int jy = hasY ? j + 1 : j;  // row B (a valid address even when B does not exist)
    const int nq = g.nx >> 2;
    auto rowptr = [&](int k, int jj) { return vol + ((long long)(k - g.kd) * g.ny + jj) * g.nx; };

    // words of rows A = (j,k), B = (j+1,k); Cw, Dw = the same rows at plane k+1
    uint32_t A[NW], B[NW], Cw[NW], Dw[NW];
    RowVals<U> pc, pd;  // raw values of plane k+1 (VEC4), loaded one step ahead
    if (VEC4) {
        RowVals<U> ra, rbv;
        load_row_vec4<U>(rowptr(kb, j), nq, lane, true, ra);
        load_row_vec4<U>(rowptr(kb, jy), nq, lane, hasY, rbv);
        if (kb + 1 < g.nz) {
            load_row_vec4<U>(rowptr(kb + 1, j), nq, lane, true, pc);
            load_row_vec4<U>(rowptr(kb + 1, jy), nq, lane, hasY, pd);
        }
        words_vec4<U, NW>(ra, nq, lane, iso, A);
        words_vec4<U, NW>(rbv, nq, lane, iso, B);
    } else {
        words_scalar<NW>(rowptr(kb, j), g.nx, g.W, true, lane, iso, A);
        words_scalar<NW>(rowptr(kb, jy), g.nx, g.W, hasY, lane, iso, B);
    }
    for (int k = kb; k < ke; ++k) {
        const bool hasZ = k + 1 < g.nz;
        if (VEC4) {
            words_vec4<U, NW>(pc, nq, lane, iso, Cw);
            words_vec4<U, NW>(pd, nq, lane, iso, Dw);
            if (k + 2 < g.nz && k + 1 < ke) {  // plane k+2 for the next step
                load_row_vec4<U>(rowptr(k + 2, j), nq, lane, true, pc);
                load_row_vec4<U>(rowptr(k + 2, jy), nq, lane, hasY, pd);
            }
        } else if (hasZ) {
            words_scalar<NW>(rowptr(k + 1, j), g.nx, g.W, true, lane, iso, Cw);
            words_scalar<NW>(rowptr(k + 1, jy), g.nx, g.W, hasY, lane, iso, Dw);
        }
        if (!hasZ) {
#pragma unroll
            for (int q = 0; q < NW; ++q) Cw[q] = Dw[q] = 0u;
        }
        RowCounts rc;
        const long long r = (long long)(k - g.kr) * g.ny + j;
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            const int w = lane + 32 * q;
            RowWords rw;
            rw.a = A[q];
            rw.b = B[q];
            rw.c = Cw[q];
            rw.d = Dw[q];
            rw.ash = (rw.a >> 1) | (next_word<NW>(A, q, lane) << 31);
            rw.bsh = (rw.b >> 1) | (next_word<NW>(B, q, lane) << 31);
            rw.csh = (rw.c >> 1) | (next_word<NW>(Cw, q, lane) << 31);
            rw.dsh = (rw.d >> 1) | (next_word<NW>(Dw, q, lane) << 31);
            count_word<MC>(rw, w, g, j, k, hasY, hasZ, trims != nullptr, rc);
            if (w < g.W) bits_out[r * g.W + w] = rw.a;
        }
        finish_row<MC>(rc, lane, r, g, rowcnt, trims, mccnt);
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            A[q] = Cw[q];
            B[q] = Dw[q];
        }
    }
}

// Rows of up to 32 words, the volume at a 16-byte boundary (count_rows.cuh).  Against the kernel it replaced (lanes
// per row a power of two, every row classified twice), us: 768^3 302 / 453, 667 x 228 x 724 94 / 152, 301 x 217 x 190
// 18.6 / 32, 64^3 10 / 21; 512^3 104 / 103, both at the HBM rate (the kernel by itself 88 us, 6.1 TB/s; in a sequence
// of extractions the mesh written before drains at the same time).
template <bool MC, int S, bool ALIGNED>
__global__ void __launch_bounds__(kCountThreads) k_count_rows(const float* __restrict__ vol, Grid g, float below,
                                                              int KC, int ngroups, unsigned nitems, int stage_bytes,
                                                              uint4* __restrict__ rowcnt,
                                                              uint2* __restrict__ trims, uint32_t* __restrict__ mccnt,
                                                              uint32_t* __restrict__ bits_out,
                                                              unsigned long long* __restrict__ status)
{
    extern __shared__ __align__(128) unsigned char s_raw[];
    __shared__ uint64_t s_bar[kCountWarps];
    next_may_start();
    const int warp = threadIdx.x >> 5;
    const unsigned item = blockIdx.x * kCountWarps + warp;
    if (item >= nitems) return;
    const FloatSamples<ALIGNED> smp(below);
    count_rows_item<FloatSamples<ALIGNED>, MC, S>(vol, g, smp, KC, ngroups, item,
                                                  s_raw + (size_t)warp * stage_bytes,
                                                  s_bar + warp, rowcnt, trims, mccnt, bits_out, status);
}

// The Flying Edges counts of a list of requests (batch_kernels.cuh), one launch: block x is block x - first[q] of
// request list[q].
template <bool ALIGNED>
__global__ void __launch_bounds__(kCountThreads) k_count_rows_batch(const BatchReq* __restrict__ reqs,
                                                                    const int* __restrict__ list,
                                                                    const unsigned* __restrict__ first, int m,
                                                                    int stage_bytes)
{
    extern __shared__ __align__(128) unsigned char s_raw[];
    __shared__ uint64_t s_bar[kCountWarps];
    const int warp = threadIdx.x >> 5;
    const int q = batch_find(first, m, blockIdx.x);
    const BatchReq* d = reqs + __ldg(&list[q]);
    const Grid g = d->g;
    const unsigned item = (blockIdx.x - __ldg(&first[q])) * kCountWarps + warp;
    const FloatSamples<ALIGNED> smp(d->below);
    count_rows_item<FloatSamples<ALIGNED>, false, kBatchCountRows>(
        d->vol, g, smp, d->count_KC, d->count_groups, item, s_raw + (size_t)warp * stage_bytes,
        s_bar + warp, d->rowcnt, nullptr, nullptr, d->bits, d->totals + 3);
}

// Word c*32 + lane of a row and, uniform over the warp, word c*32 + 32 (the
// source of lane 31's bit 32): 33 coalesced 128-byte loads.
__device__ __forceinline__ void chunk_words(const float* __restrict__ row, bool ok, int c, int nx, int lane, float iso,
                                            uint32_t& word, uint32_t& next)
{
    word = 0u;
    for (int t = 0; t <= 32; ++t) {
        const long long i = 32ll * (32 * c + t) + lane;
        const bool in = ok && i < nx;
        const uint32_t m = __ballot_sync(0xffffffffu, in && __ldg(row + i) >= iso);
        if (t == lane) word = m;
        next = m;
    }
}

// Rows longer than 64 words (nx > 2048): the same counts as k_count_warps,
// the row walked in chunks of 32 words, the four rows of a step re-read from
// the volume for every plane (twice the reads of the narrow kernel).
template <bool MC>
__global__ void __launch_bounds__(kThreads) k_count_wide(const float* __restrict__ vol, Grid g, float iso, int KC,
                                                         int nyb, const CaseTables* __restrict__ cases,
                                                         uint4* __restrict__ rowcnt, uint2* __restrict__ trims,
                                                         uint32_t* __restrict__ mccnt, uint32_t* __restrict__ bits_out)
{
    (void)cases;  // the counts need no case table (tris_of_word, mc_verts_of_word)
    const int jb = blockIdx.x % nyb, kc = blockIdx.x / nyb;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = jb * kCountRows + warp;
    if (j >= g.ny) return;
    const int kb = g.kr + kc * KC, ke = min(kb + KC, g.ke);
    const bool hasY = j < g.ny - 1;
    const int jy = hasY ? j + 1 : j;
    const int nchunks = (g.W + 31) / 32;
    auto rowptr = [&](int k, int jj) { return vol + ((long long)(k - g.kd) * g.ny + jj) * g.nx; };
    for (int k = kb; k < ke; ++k) {
        const bool hasZ = k + 1 < g.nz;
        const int kz = hasZ ? k + 1 : k;
        RowCounts rc;
        const long long r = (long long)(k - g.kr) * g.ny + j;
        for (int c = 0; c < nchunks; ++c) {
            RowWords rw;
            uint32_t na, nb, nc, nd;
            chunk_words(rowptr(k, j), true, c, g.nx, lane, iso, rw.a, na);
            chunk_words(rowptr(k, jy), hasY, c, g.nx, lane, iso, rw.b, nb);
            chunk_words(rowptr(kz, j), hasZ, c, g.nx, lane, iso, rw.c, nc);
            chunk_words(rowptr(kz, jy), hasY && hasZ, c, g.nx, lane, iso, rw.d, nd);
            const uint32_t da = __shfl_down_sync(0xffffffffu, rw.a, 1), db = __shfl_down_sync(0xffffffffu, rw.b, 1);
            const uint32_t dc = __shfl_down_sync(0xffffffffu, rw.c, 1), dd = __shfl_down_sync(0xffffffffu, rw.d, 1);
            rw.ash = (rw.a >> 1) | ((lane < 31 ? da : na) << 31);
            rw.bsh = (rw.b >> 1) | ((lane < 31 ? db : nb) << 31);
            rw.csh = (rw.c >> 1) | ((lane < 31 ? dc : nc) << 31);
            rw.dsh = (rw.d >> 1) | ((lane < 31 ? dd : nd) << 31);
            const int w = 32 * c + lane;
            count_word<MC>(rw, w, g, j, k, hasY, hasZ, trims != nullptr, rc);
            if (w < g.W) bits_out[r * g.W + w] = rw.a;
        }
        finish_row<MC>(rc, lane, r, g, rowcnt, trims, mccnt);
    }
}

// ---------------------------------------------------------------------------
// Exclusive scans of the per-row counts (vertices = x+y+z cuts, triangles,
// MC vertices) over the R = ny*nz rows, in two launches over segments of
// kSeg rows (256 threads x 4):
//   k_scan_partial  one CTA per segment: segment totals
//   k_scan_final    one CTA per segment: offset of the segment + scan inside
//                   it -> starts[n][R]; grand totals.
// ---------------------------------------------------------------------------
constexpr int kScanPer = 4;  // 4 rather than 8 rows per thread: twice the CTAs, 15.2 -> 12.9 us at 512^3
constexpr int kSeg = kThreads * kScanPer;

// Scan modes: the components scanned per row.
//   kScanFE   0: vertices (x+y+z cuts)  1: triangles
//   kScanMC   0: vertices  1: triangles  2: MC vertices
//   kScanDup  0: x cuts  1: triangles  2: y cuts  3: z cuts (the blocks of the
//             global-edge-index order; totals[4], totals[5] = all x, all y cuts)
template <int SM>
struct ScanComps {
    static constexpr int n = SM == kScanDup ? 4 : (SM == kScanMC ? 3 : 2);
};

template <int SM>
__device__ __forceinline__ void load_counts(const uint4* rowcnt, const uint32_t* mccnt,
                                            long long R, long long b, uint32_t (&v)[4][kScanPer],
                                            unsigned long long (&s)[4])
{
    s[0] = s[1] = s[2] = s[3] = 0;
#pragma unroll
    for (int q = 0; q < kScanPer; ++q) {
        const bool ok = b + q < R;
        const uint4 c = ok ? load_written(rowcnt + b + q) : make_uint4(0, 0, 0, 0);
        if (SM == kScanDup) {
            v[0][q] = c.x;
            v[2][q] = c.y;
            v[3][q] = c.z;
        } else {
            v[0][q] = c.x + c.y + c.z;
            v[2][q] = (SM == kScanMC && ok) ? load_written(mccnt + b + q) : 0u;
            v[3][q] = 0u;
        }
        v[1][q] = c.w;
#pragma unroll
        for (int a = 0; a < 4; ++a) s[a] += v[a][q];
    }
}

// Segment blk of the scan: its totals into part[a * nseg + blk].
template <int SM>
__device__ __forceinline__ void scan_partial_block(const uint4* rowcnt,
                                                   const uint32_t* mccnt, long long R,
                                                   unsigned long long* __restrict__ part, int nseg, int blk)
{
    constexpr int NC = ScanComps<SM>::n;
    __shared__ unsigned long long s_w[NC][kThreads / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t v[4][kScanPer];
    unsigned long long s[4];
    load_counts<SM>(rowcnt, mccnt, R, (long long)blk * kSeg + (long long)t * kScanPer, v, s);
#pragma unroll
    for (int a = 0; a < NC; ++a) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) s[a] += __shfl_xor_sync(0xffffffffu, s[a], d);
        if (lane == 0) s_w[a][warp] = s[a];
    }
    __syncthreads();
    if (t < NC) {
        unsigned long long tot = 0;
        for (int w = 0; w < kThreads / 32; ++w) tot += s_w[t][w];
        part[t * nseg + blk] = tot;
    }
}

template <int SM>
__global__ void __launch_bounds__(kThreads) k_scan_partial(const uint4* rowcnt,
                                                           const uint32_t* mccnt, long long R,
                                                           unsigned long long* __restrict__ part, int nseg)
{
    wait_for_previous();
    next_may_start();
    scan_partial_block<SM>(rowcnt, mccnt, R, part, nseg, (int)blockIdx.x);
}

// The totals' other duties, by one thread of the scan: the work counter of pass 4 starts at zero, and the counts go
// to the host (launch_scan).
__device__ __forceinline__ void scan_publish(unsigned long long* __restrict__ totals, unsigned long long v,
                                             unsigned long long t, unsigned long long m,
                                             unsigned long long* __restrict__ publish,
                                             unsigned long long* __restrict__ kept)
{
    totals[7] = 0;
    if (publish) {
        publish[0] = v;
        publish[1] = t;
        publish[2] = m;
        publish[3] = totals[3] = *kept;  // pass 4 looks at totals[3]
        *kept = 0;
    }
}

// 32 bytes at a 32-byte boundary. A thread's rows lie next to each other; in smaller stores a warp wrote every sector
// several times: 768^3 13.5 us before, 9.3 now, 64 uneven volumes 74 / 60.
__device__ __forceinline__ void store_sector(unsigned long long* p, unsigned long long a, unsigned long long b,
                                             unsigned long long c, unsigned long long d)
{
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}

// Segment blk: the starts of its rows from the segments' totals; segment 0 also writes the totals.
template <int SM>
__device__ __forceinline__ void scan_final_block(const uint4* rowcnt,
                                                 const uint32_t* mccnt, long long R,
                                                 const unsigned long long* part, int nseg,
                                                 unsigned long long* __restrict__ starts, uint4* __restrict__ row4,
                                                 unsigned long long* __restrict__ totals,
                                                 unsigned long long* __restrict__ publish,
                                                 unsigned long long* __restrict__ kept, int blk)
{
    constexpr int NC = ScanComps<SM>::n;
    __shared__ unsigned long long s_w[NC][kThreads / 32];
    __shared__ unsigned long long s_base[NC], s_tot[NC];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (warp < NC) {  // warp a: the segments before this one and all of them, for component a
        unsigned long long b = 0, tot = 0;
        for (int q = lane; q < nseg; q += 32) {
            const unsigned long long x = load_written(part + warp * nseg + q);
            if (q < blk) b += x;
            tot += x;
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            b += __shfl_xor_sync(0xffffffffu, b, d);
            tot += __shfl_xor_sync(0xffffffffu, tot, d);
        }
        if (lane == 0) {
            s_base[warp] = b;
            s_tot[warp] = tot;
        }
    }
    const long long b = (long long)blk * kSeg + (long long)t * kScanPer;
    uint32_t v[4][kScanPer];
    unsigned long long s[4], inc[4];
    load_counts<SM>(rowcnt, mccnt, R, b, v, s);
#pragma unroll
    for (int a = 0; a < NC; ++a) {
        inc[a] = s[a];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, inc[a], d);
            if (lane >= d) inc[a] += y;
        }
        if (lane == 31) s_w[a][warp] = inc[a];
    }
    __syncthreads();
    if (blk == 0 && t == 0) {
        const unsigned long long e2 = NC > 2 ? s_tot[NC > 2 ? 2 : 0] : 0ull, e3 = NC > 3 ? s_tot[NC > 3 ? 3 : 0] : 0ull;
        const unsigned long long V = SM == kScanDup ? s_tot[0] + e2 + e3 : s_tot[0], m = SM == kScanDup ? 0ull : e2;
        totals[0] = V;
        totals[1] = s_tot[1];
        totals[2] = m;
        if (SM == kScanDup) {
            totals[4] = s_tot[0];
            totals[5] = e2;
        }
        scan_publish(totals, V, s_tot[1], m, publish, kept);
    }
#pragma unroll
    for (int a = 0; a < NC; ++a) {
        unsigned long long run = s_base[a] + inc[a] - s[a];
        for (int w = 0; w < warp; ++w) run += s_w[a][w];
        unsigned long long first[kScanPer];
#pragma unroll
        for (int q = 0; q < kScanPer; ++q) {
            first[q] = run;
            run += v[a][q];
        }
        if (b + kScanPer <= R && (reinterpret_cast<uintptr_t>(starts + a * R + b) & 31) == 0) {
            store_sector(starts + a * R + b, first[0], first[1], first[2], first[3]);
        } else {
#pragma unroll
            for (int q = 0; q < kScanPer; ++q)
                if (b + q < R) starts[a * R + b + q] = first[q];
        }
        if (SM != kScanDup && a == 0) {  // the row's vertices are its x, its y, then its z cuts
            unsigned long long r4[2 * kScanPer];
#pragma unroll
            for (int q = 0; q < kScanPer; ++q) {
                const uint2 c = b + q < R ? __ldg(reinterpret_cast<const uint2*>(rowcnt + b + q)) : make_uint2(0u, 0u);
                const uint32_t f = (uint32_t)first[q];
                r4[2 * q] = (unsigned long long)(f + c.x) << 32 | f;
                r4[2 * q + 1] = f + c.x + c.y;
            }
            if (b + kScanPer <= R) {
#pragma unroll
                for (int q = 0; q < kScanPer; q += 2)
                    store_sector(reinterpret_cast<unsigned long long*>(row4 + b + q), r4[2 * q], r4[2 * q + 1],
                                 r4[2 * q + 2], r4[2 * q + 3]);
            } else {
#pragma unroll
                for (int q = 0; q < kScanPer; ++q)
                    if (b + q < R)
                        *reinterpret_cast<ulonglong2*>(row4 + b + q) = make_ulonglong2(r4[2 * q], r4[2 * q + 1]);
            }
        }
    }
}

template <int SM>
__global__ void __launch_bounds__(kThreads) k_scan_final(const uint4* rowcnt,
                                                         const uint32_t* mccnt, long long R,
                                                         const unsigned long long* part, int nseg,
                                                         unsigned long long* __restrict__ starts,
                                                         uint4* __restrict__ row4,
                                                         unsigned long long* __restrict__ totals,
                                                         unsigned long long* __restrict__ publish,
                                                         unsigned long long* __restrict__ kept)
{
    wait_for_previous();
    next_may_start();
    scan_final_block<SM>(rowcnt, mccnt, R, part, nseg, starts, row4, totals, publish, kept, (int)blockIdx.x);
}

// The whole scan of a small grid in one CTA: one launch less than the two above where launches are most of the time.
// A warp takes a run of 128 consecutive rows, a lane every 32nd of them, read once.  Events around the pass, us: 64^3
// (4,096 rows) 9.0 against 11.4 with the two.  The limit is where a thread's four rows end.  With sixteen, up to 16,384
// rows, the call (rows of 64 points) takes longer at every size, us: 3,000 rows 44-48 (with four 40), 5,120 rows 46-49
// (the two kernels 43), 8,000 rows 48-52 (45), 12,000 rows 53-56 (47), 16,384 rows 58-59 (49).
constexpr int kScanSmallPer = 4;
constexpr long long kScanSmall = 1024ll * kScanSmallPer;

template <int SM>
__global__ void __launch_bounds__(1024) k_scan_small(const uint4* rowcnt,
                                                     const uint32_t* mccnt, int R,
                                                     unsigned long long* __restrict__ starts, uint4* __restrict__ row4,
                                                     unsigned long long* __restrict__ totals,
                                                     unsigned long long* __restrict__ publish,
                                                     unsigned long long* __restrict__ kept)
{
    constexpr int NC = ScanComps<SM>::n, PER = kScanSmallPer;
    __shared__ uint32_t s_w[NC][32];
    wait_for_previous();
    next_may_start();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int r0 = warp * PER * 32 + lane;
    uint32_t v[NC][PER], cx[PER], cxy[PER], sum[NC];  // 32 bits hold the counts of so many rows (scan_launch)
#pragma unroll
    for (int a = 0; a < NC; ++a) sum[a] = 0u;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int r = r0 + 32 * q;
        const uint4 c = r < R ? load_written(rowcnt + r) : make_uint4(0u, 0u, 0u, 0u);
        cx[q] = c.x;
        cxy[q] = c.x + c.y;
        v[0][q] = SM == kScanDup ? c.x : c.x + c.y + c.z;
        v[1][q] = c.w;
        if (NC > 2) v[NC > 2 ? 2 : 0][q] = SM == kScanDup ? c.y : (r < R ? load_written(mccnt + r) : 0u);
        if (NC > 3) v[NC > 3 ? 3 : 0][q] = c.z;
#pragma unroll
        for (int a = 0; a < NC; ++a) sum[a] += v[a][q];
    }
#pragma unroll
    for (int a = 0; a < NC; ++a) {
        const uint32_t w = __reduce_add_sync(0xffffffffu, sum[a]);
        if (lane == 0) s_w[a][warp] = w;
    }
    __syncthreads();
    if (warp < NC) {  // warp a: the warps' sums before each; the last lane's end with the totals
        const uint32_t x = s_w[warp][lane];
        uint32_t inc = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += y;
        }
        s_w[warp][lane] = inc - x;
    }
    __syncthreads();
    uint32_t run[NC];
#pragma unroll
    for (int a = 0; a < NC; ++a) run[a] = s_w[a][warp];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int r = r0 + 32 * q;
#pragma unroll
        for (int a = 0; a < NC; ++a) {
            uint32_t inc = v[a][q];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += y;
            }
            const uint32_t first = run[a] + inc - v[a][q];
            if (r < R) {
                starts[(long long)a * R + r] = first;
                if (SM != kScanDup && a == 0) row4[r] = make_uint4(first, first + cx[q], first + cxy[q], 0u);
            }
            run[a] += __shfl_sync(0xffffffffu, inc, 31);
        }
    }
    if (t == 1023) {
        const unsigned long long e2 = NC > 2 ? run[NC > 2 ? 2 : 0] : 0u, e3 = NC > 3 ? run[NC > 3 ? 3 : 0] : 0u;
        const unsigned long long V = SM == kScanDup ? run[0] + e2 + e3 : run[0], m = SM == kScanDup ? 0ull : e2;
        totals[0] = V;
        totals[1] = run[1];
        totals[2] = m;
        if (SM == kScanDup) {
            totals[4] = run[0];
            totals[5] = e2;
        }
        scan_publish(totals, V, run[1], m, publish, kept);
    }
}

// The Flying Edges scans of a list of requests, one launch per phase: block x is segment
// x - first[q] of request list[q].
__global__ void __launch_bounds__(kThreads) k_scan_partial_batch(const BatchReq* __restrict__ reqs,
                                                                 const int* __restrict__ list,
                                                                 const unsigned* __restrict__ first, int m)
{
    const int q = batch_find(first, m, blockIdx.x);
    const BatchReq* d = reqs + __ldg(&list[q]);
    const int blk = (int)(blockIdx.x - __ldg(&first[q]));
    if (blk >= d->nseg) return;  // past the request's segments (the launch holds exactly first[m] blocks)
    scan_partial_block<kScanFE>(d->rowcnt, nullptr, d->g.R, d->part, d->nseg, blk);
}

__global__ void __launch_bounds__(kThreads) k_scan_final_batch(const BatchReq* __restrict__ reqs,
                                                               const int* __restrict__ list,
                                                               const unsigned* __restrict__ first, int m)
{
    const int q = batch_find(first, m, blockIdx.x);
    const BatchReq* d = reqs + __ldg(&list[q]);
    const int blk = (int)(blockIdx.x - __ldg(&first[q]));
    if (blk >= d->nseg) return;
    scan_final_block<kScanFE>(d->rowcnt, nullptr, d->g.R, d->part, d->nseg, d->starts, d->row4,
                              d->totals, nullptr, nullptr, blk);
}

// vfirst[q] = the vertices of requests list[0 .. q-1] whose meshes hold their counts (one CTA of 1024 threads,
// each summing a run of consecutive requests).
__global__ void __launch_bounds__(1024) k_batch_vfirst(const BatchReq* __restrict__ reqs, const int* __restrict__ list,
                                                       int m, unsigned long long* __restrict__ vfirst)
{
    __shared__ unsigned long long s_w[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int per = (m + 1023) / 1024, q0 = t * per, q1 = min(m, q0 + per);
    auto verts = [&](int q) -> unsigned long long {
        const BatchReq* d = reqs + __ldg(&list[q]);
        return mesh_holds(d->totals, d->capV, d->capT) ? d->totals[0] : 0ull;
    };
    unsigned long long mine = 0;
    for (int q = q0; q < q1; ++q) mine += verts(q);
    unsigned long long inc = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += y;
    }
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    unsigned long long run = inc - mine;
    for (int w = 0; w < warp; ++w) run += s_w[w];
    for (int q = q0; q < q1; ++q) {
        vfirst[q] = run;
        run += verts(q);
    }
    if (t == 1023) vfirst[m] = run;
}

// Block-wide exclusive sums of two values per thread (one CTA of 1024 threads): returns this thread's offsets.
__device__ __forceinline__ void block_excl2(unsigned long long a, unsigned long long b, unsigned long long& ea,
                                            unsigned long long& eb, unsigned long long* s_a, unsigned long long* s_b)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long ia = a, ib = b;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long ya = __shfl_up_sync(0xffffffffu, ia, d), yb = __shfl_up_sync(0xffffffffu, ib, d);
        if (lane >= d) {
            ia += ya;
            ib += yb;
        }
    }
    if (lane == 31) {
        s_a[warp] = ia;
        s_b[warp] = ib;
    }
    __syncthreads();
    ea = ia - a;
    eb = ib - b;
    for (int w = 0; w < warp; ++w) {
        ea += s_a[w];
        eb += s_b[w];
    }
    __syncthreads();  // s_a / s_b free for the next call
}

// The packed placement (launch_place_batch): one CTA of 1024 threads, each over a run of consecutive requests.
// Request list[q] goes to vertex offset vat and triangle offset tat, the sums of the counts before it; it is
// placed when both ranges end within the capacities and, for 32-bit indices, its vertices number below 2^32.
// vfirst sums the vertices of the placed requests only.
__global__ void __launch_bounds__(1024) k_batch_place(BatchReq* __restrict__ reqs, const int* __restrict__ list, int m,
                                                      PackedOut o, unsigned long long* __restrict__ vfirst)
{
    __shared__ unsigned long long s_a[32], s_b[32];
    const int t = threadIdx.x;
    const int per = (m + 1023) / 1024, q0 = t * per, q1 = min(m, q0 + per);
    unsigned long long sv = 0, st = 0;
    for (int q = q0; q < q1; ++q) {
        const unsigned long long* tot = reqs[__ldg(&list[q])].totals;
        sv += tot[0];
        st += tot[1];
    }
    unsigned long long vat, tat;
    block_excl2(sv, st, vat, tat, s_a, s_b);
    unsigned long long placed = 0;  // vertices of this thread's placed requests
    for (int q = q0; q < q1; ++q) {
        BatchReq* d = reqs + __ldg(&list[q]);
        const unsigned long long V = d->totals[0], T = d->totals[1];
        const bool ok = vat + V <= (unsigned long long)o.cap_points && tat + T <= (unsigned long long)o.cap_tris &&
                        (o.index_bytes == 8 || V <= 0xffffffffull) && d->totals[3] == 0ull;
        d->points = o.points + 3 * vat;
        d->normals = o.normals + 3 * vat;
        d->tris = static_cast<char*>(o.tris) + 3 * tat * (unsigned long long)o.index_bytes;
        d->capV = ok ? (long long)V : -1;
        d->capT = ok ? (long long)T : -1;
        d->totals[4] = vat;
        d->totals[5] = tat;
        placed += ok ? V : 0ull;
        vat += V;
        tat += T;
    }
    unsigned long long at, unused;
    block_excl2(placed, 0ull, at, unused, s_a, s_b);
    for (int q = q0; q < q1; ++q) {
        const BatchReq* d = reqs + __ldg(&list[q]);
        vfirst[q] = at;
        at += d->capV >= 0 ? d->totals[0] : 0ull;
    }
    if (t == 1023) vfirst[m] = at;
}

// gridEdge records {xl, xr, xstart, ystart, zstart} and triCounter for
// inspection (counts before the scan, offsets after it).
__global__ void k_grid_edges(Grid g, RowStarts rs, const uint4* __restrict__ rowcnt, const uint2* __restrict__ trims,
                             int scanned, unsigned long long* __restrict__ ge,
                             unsigned long long* __restrict__ tri_counter)
{
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= g.R) return;
    const uint4 c = rowcnt[r];
    const uint2 tr = trims[r];
    unsigned long long* o = ge + 5 * r;
    o[0] = tr.x;
    o[1] = tr.y;
    if (scanned) {
        const unsigned long long b = rs.get(r, 0);
        o[2] = b; o[3] = b + c.x; o[4] = b + c.x + c.y;
    } else {
        o[2] = c.x; o[3] = c.y; o[4] = c.z;
    }
    const int j = (int)(r % g.ny), k = (int)(r / g.ny);
    if (j < g.ny - 1 && k < g.nz - 1) tri_counter[(long long)k * (g.ny - 1) + j] = scanned ? rs.get(r, 1) : c.w;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
int lanes_per_row(int W)
{
    int G = 1;
    while (G < W && G < 32) G <<= 1;
    return G;
}

CountPlan count_plan(const Grid& g, int nsm)
{
    CountPlan p;
    p.J = kCountRows;
    p.nyb = (g.ny + p.J - 1) / p.J;
    // ~8 CTAs per SM in total, at least 8 planes per column
    const int nzw = g.ke - g.kr;  // planes of the window
    const long long target = (long long)nsm * 8;
    int nkc = (int)((target + p.nyb - 1) / p.nyb);
    if (nkc < 1) nkc = 1;
    p.KC = (nzw + nkc - 1) / nkc;
    if (p.KC < 8) p.KC = 8;
    if (p.KC > nzw) p.KC = nzw;
    if (p.KC < 1) p.KC = 1;
    p.nkc = (nzw + p.KC - 1) / p.KC;
    p.nseg = (int)((g.R + kSeg - 1) / kSeg);
    p.nsm = nsm;
    return p;
}

CountRows count_rows_plan(const Grid& g, int nsm, int sample_bytes, bool aligned, bool trims)
{
    CountRows r;
    const int nzw = g.ke - g.kr;  // planes of the window
    auto resident = [&](int S) {  // warps of one wave with S rows per lane
        r.S = S;
        r.stage = count_stage_bytes(g.nx, g.W, S, sample_bytes, aligned);
        r.groups = (g.ny + (32 / g.W) * S - 1) / ((32 / g.W) * S);
        const long long per_sm = (227ll * 1024) / (kCountWarps * (long long)r.stage + 1024);
        return (long long)nsm * kCountWarps * std::max(1ll, std::min(8ll, per_sm));
    };
    // Rows of 17-32 words, one per warp at a time: four per lane where that leaves every warp of a wave at least 8
    // planes (768^3: 302 us against 312 with two and 395 with one).  Else two, which is the best or within 1% of it
    // from 256^3 (20.2 us, with four 21.8) to 512^3 (103.5, with four 105), and one where a wave's half has less
    // than a plane each (64^3: 10.0 us against 11.9 with two).
    long long warps = resident(trims ? 1 : (g.W > 16 ? 4 : 2));
    if (r.S == 4 && (long long)r.groups * nzw < 8 * warps) warps = resident(2);
    if (r.S == 2 && 2ll * r.groups * nzw < warps) warps = resident(1);
    const long long cols = std::max(1ll, warps / r.groups);  // one wave
    r.KC = (int)std::max(1ll, (nzw + cols - 1) / cols);
    r.items = (unsigned)((long long)r.groups * ((nzw + r.KC - 1) / r.KC));
    return r;
}

template <bool MC>
static void count_launch(const CountPlan& p, const float* vol, const Grid& g, float iso, const CaseTables* cases,
                         FeBuffers& b, unsigned long long* status, cudaStream_t s)
{
    const unsigned blocks = (unsigned)(p.nyb * p.nkc);
    const bool base16 = (reinterpret_cast<uintptr_t>(vol) & 15) == 0;
    const bool vec4 = g.W <= 64 && (g.nx % 4 == 0) && base16;
    uint2* trims = p.trims ? b.trims : nullptr;  // the kernels skip the trims when null
    if (base16 && g.W <= 32) {
        const bool aligned = g.nx % 4 == 0;
        const CountRows r = count_rows_plan(g, p.nsm, 4, aligned, p.trims);
        const size_t smem = (size_t)kCountWarps * r.stage;
        const unsigned nb = (r.items + kCountWarps - 1) / kCountWarps;
        auto kern = r.S == 4 ? (aligned ? k_count_rows<MC, 4, true> : k_count_rows<MC, 4, false>)
                  : r.S == 2 ? (aligned ? k_count_rows<MC, 2, true> : k_count_rows<MC, 2, false>)
                             : (aligned ? k_count_rows<MC, 1, true> : k_count_rows<MC, 1, false>);
        allow_smem(kern, smem);
        kern<<<nb, kCountThreads, smem, s>>>(vol, g, count_below(iso), r.KC, r.groups, r.items, r.stage, b.rowcnt,
                                             trims, b.mccnt, b.bits, status);
        return;
    }
    if (g.W > 64) {
        k_count_wide<MC><<<blocks, kThreads, 0, s>>>(vol, g, iso, p.KC, p.nyb, cases, b.rowcnt, trims, b.mccnt,
                                                     b.bits);
        return;
    }
#define ISO_COUNT(VEC, UU, NWW)                                                                                \
    k_count_warps<MC, VEC, UU, NWW><<<blocks, kThreads, 0, s>>>(vol, g, iso, p.KC, p.nyb, cases, b.rowcnt,     \
                                                                trims, b.mccnt, b.bits)
    if (vec4) {  // rows of 33-64 words; the shorter ones ran above
        ISO_COUNT(true, 16, 2);
    } else if (g.W <= 32) {
        ISO_COUNT(false, 1, 1);
    } else {
        ISO_COUNT(false, 1, 2);
    }
#undef ISO_COUNT
}

void launch_count(const float* vol, const Grid& g, float iso, const CaseTables* cases, bool mc,
                  const CountPlan& p, FeBuffers& b, cudaStream_t s, bool zero_status)
{
    unsigned long long* status = count_status(b, zero_status, s);
    if (mc) count_launch<true>(p, vol, g, iso, cases, b, status, s);
    else count_launch<false>(p, vol, g, iso, cases, b, status, s);
}

BatchCount batch_count(const Grid& g, int planes)
{
    BatchCount c;
    const int G = (32 / g.W) * kBatchCountRows;
    c.aligned = g.nx % 4 == 0;
    c.stage = count_stage_bytes(g.nx, g.W, kBatchCountRows, 4, c.aligned);
    c.groups = (g.ny + G - 1) / G;
    c.KC = std::min(planes, g.nz);
    c.blocks = ((long long)c.groups * ((g.nz + c.KC - 1) / c.KC) + kCountWarps - 1) / kCountWarps;
    return c;
}

void launch_count_batch(bool aligned, const BatchReq* reqs, const int* list, const unsigned* first, int m,
                        unsigned blocks, int stage, cudaStream_t s)
{
    const size_t smem = (size_t)kCountWarps * stage;
    auto kern = aligned ? k_count_rows_batch<true> : k_count_rows_batch<false>;
    allow_smem(kern, smem);
    kern<<<blocks, kCountThreads, smem, s>>>(reqs, list, first, m, stage);
}

void launch_scan_batch(const BatchReq* reqs, const int* list, const unsigned* first, int m, unsigned blocks,
                       cudaStream_t s)
{
    k_scan_partial_batch<<<blocks, kThreads, 0, s>>>(reqs, list, first, m);
    k_scan_final_batch<<<blocks, kThreads, 0, s>>>(reqs, list, first, m);
}

void launch_vfirst_batch(const BatchReq* reqs, const int* list, int m, unsigned long long* vfirst, cudaStream_t s)
{
    k_batch_vfirst<<<1, 1024, 0, s>>>(reqs, list, m, vfirst);
}

void launch_place_batch(BatchReq* reqs, const int* list, int m, const PackedOut& out, unsigned long long* vfirst,
                        cudaStream_t s)
{
    k_batch_place<<<1, 1024, 0, s>>>(reqs, list, m, out, vfirst);
}

template <int SM>
static void scan_launch(const Grid& g, const CountPlan& p, FeBuffers& b, cudaStream_t s, unsigned long long* publish)
{
    if (g.R <= kScanSmall && g.nx <= (1 << 15)) {  // their triangles stay below 2^32
        launch_after(k_scan_small<SM>, 1, 1024, 0, s, b.rowcnt, b.mccnt, (int)g.R, b.starts, b.row4, b.totals, publish,
                     b.kept);
        return;
    }
    launch_after(k_scan_partial<SM>, p.nseg, kThreads, 0, s, b.rowcnt, b.mccnt, g.R, b.part, p.nseg);
    launch_after(k_scan_final<SM>, p.nseg, kThreads, 0, s, b.rowcnt, b.mccnt, g.R, b.part, p.nseg, b.starts, b.row4,
                 b.totals, publish, b.kept);
}

void launch_scan(const Grid& g, const CountPlan& p, int mode, FeBuffers& b, cudaStream_t s,
                 unsigned long long* publish)
{
    if (mode == kScanMC) scan_launch<kScanMC>(g, p, b, s, publish);
    else if (mode == kScanDup) scan_launch<kScanDup>(g, p, b, s, publish);
    else scan_launch<kScanFE>(g, p, b, s, publish);
}

RowStarts row_starts(const Grid& g, const CountPlan& p, const FeBuffers& b)
{
    (void)p;
    RowStarts rs;
    rs.starts = b.starts;
    rs.R = g.R;
    rs.ny = g.ny;
    rs.kr = g.kr;
    rs.add[0] = rs.add[1] = rs.add[2] = rs.add[3] = 0;
    return rs;
}

// Where a slab begins and ends in its window's counts, for the host, written by
// one warp straight into mapped pinned host memory (no copy engine: the read-back
// does not queue behind bulk copies of other streams): out[a] the start of row
// rlo and out[3 + a] that of row rhi, for a = vertices, triangles, MC vertices.
__global__ void k_slab_readback(const unsigned long long* __restrict__ starts, int comps, long long R, long long rlo,
                                long long rhi, int has_lo, int has_hi, unsigned long long* out)
{
    const int a = threadIdx.x;
    if (a < 3) {
        if (has_lo) out[a] = a < comps ? starts[a * R + rlo] : 0ull;
        if (has_hi) out[3 + a] = a < comps ? starts[a * R + rhi] : 0ull;
    }
}

void launch_slab_readback(const FeBuffers& b, const Grid& g, int comps, long long rlo, long long rhi, bool has_lo,
                          bool has_hi, unsigned long long* out, cudaStream_t s)
{
    k_slab_readback<<<1, 32, 0, s>>>(b.starts, comps, g.R, rlo, rhi, has_lo ? 1 : 0, has_hi ? 1 : 0, out);
}

void launch_grid_edges(const Grid& g, const CountPlan& p, const FeBuffers& b, int scanned, unsigned long long* ge,
                       unsigned long long* tri_counter, cudaStream_t s)
{
    const long long blocks = (g.R + 255) / 256;
    k_grid_edges<<<(unsigned)blocks, 256, 0, s>>>(g, row_starts(g, p, b), b.rowcnt, b.trims, scanned, ge,
                                                  tri_counter);
}

ISO_WAIT_STATS_ACCESSOR(iso_dbg_count_waits)

}  // namespace iso
