// The count pass over rows of up to 32 words (1024 points), shared by the
// float32 kernels (count_kernels.cu) and the 8- and 16-bit ones
// (count_narrow.cu): bit words, cut edges, triangles and Marching Cubes
// vertices of every grid row.
//
// A row's W words go to W neighbouring lanes, 32 / W rows side by side in a
// warp, so 91% of the lanes hold a word on average over the widths up to 16, 84%
// up to 32 (powers of two of lanes per row left a 5-word row 3 of 8 lanes idle;
// rows of 17 to 31 words leave 32 - W idle either way).  A lane holds S
// consecutive rows of its place plus the row after them: a warp's rows are
// jw .. jw + G - 1, G = (32 / W) * S, and they read rows jw .. jw + G of every
// plane, which lie next to each other in memory, so one bulk copy per plane
// and warp brings them in.  Everything that belongs to one row of one plane
// (its word, the word shifted by one point, its corners and the face between
// it and the next row) is computed once and kept in registers for the next row
// and the next plane; with S = 4 a row's word is built 1.25 times, not twice.
//
// What bounds it: the volume's bytes on large grids (one read, 4 bytes a
// point).  The sample compare is a subtraction on the FMA pipe, two samples
// per instruction, and one funnel shift that collects the sign (the ALU pipe's
// whole share of a sample).
#pragma once
#include <cmath>
#include <cstring>
#include <limits>

#include "count_words.cuh"

namespace iso {

constexpr int kCountWarps = 4;             // warps per CTA, each on its own
constexpr int kCountThreads = 32 * kCountWarps;
constexpr int kCountPad = 192;             // bytes past a buffer that a row's last word may read

// value >= iso as the sign bit of (the float below iso) - value: exact, because
// a difference of floats is zero only for equal ones, and clear for a NaN on
// either side.  Minus infinity has no float below it: there the bit is "no
// NaN", the one case that is compared sample by sample (FloatSamples::word).
constexpr uint32_t kAllButNaN = 0xffffffffu;  // a NaN that no other isovalue is passed as
inline float count_below(float iso)
{
    if (std::isnan(iso)) return std::numeric_limits<float>::quiet_NaN();
    float below = std::nextafterf(iso, -std::numeric_limits<float>::infinity());
    if (std::isinf(iso) && iso < 0.f) std::memcpy(&below, &kAllButNaN, sizeof below);
    return below;
}

__device__ __forceinline__ uint32_t push_sign(uint32_t acc, uint32_t v) { return __funnelshift_l(v, acc, 1); }

// Bits "value >= iso" of four floats, the first in the lowest bit, pushed above acc's.
__device__ __forceinline__ uint32_t push4(uint32_t acc, ulonglong2 v, unsigned long long below2)
{
    unsigned long long a, b;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(a) : "l"(below2), "l"(v.x));
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(b) : "l"(below2), "l"(v.y));
    acc = push_sign(acc, (uint32_t)(b >> 32));
    acc = push_sign(acc, (uint32_t)b);
    acc = push_sign(acc, (uint32_t)(a >> 32));
    return push_sign(acc, (uint32_t)a);
}

// Float32 rows.  A word is eight float4; lane l starts at float4 rot of its
// word, so that the eight lanes of a quarter warp read different bank groups,
// and rotates the word into place at the end.
template <bool ALIGNED>
struct FloatSamples {
    typedef float T;
    static constexpr bool kAligned = ALIGNED;
    unsigned long long below2;
    // places of the lane's eight float4 in reading order, and its rotation
    struct Lane {
        int off[8];
        int rot;
    };
    __device__ __forceinline__ FloatSamples(float below)
    {
        const uint32_t b = __float_as_uint(below);
        below2 = (unsigned long long)b << 32 | b;
    }
    // first: float index of the lane's first row in the buffer
    __device__ __forceinline__ Lane lane(int lane, int first) const
    {
        Lane x;
        x.rot = (lane - (first >> 2)) & 7;
#pragma unroll
        for (int u = 0; u < 8; ++u) x.off[u] = ((u + x.rot) & 7) * 16;
        return x;
    }
    // Word at float index `at` of the buffer (row start + 32 * word); bits past the row are garbage.  Every lane
    // of the warp calls it.  last: the lane's word is the row's last, nv its points inside the row.
    __device__ __forceinline__ uint32_t word(const unsigned char* buf, int at, const Lane& x, bool last, int nv) const
    {
        const unsigned char* p = buf + 16 * (at >> 2);
        uint32_t w = 0u;
        if ((uint32_t)below2 != kAllButNaN) {
#pragma unroll
            for (int u = 7; u >= 0; --u) w = push4(w, *reinterpret_cast<const ulonglong2*>(p + x.off[u]), below2);
            w = __funnelshift_l(w, w, 4 * x.rot);
        } else {
#pragma unroll 1
            for (int q = 31; q >= 0; --q) {
                const float v = reinterpret_cast<const float*>(p)[q];
                w = 2u * w + (v == v ? 1u : 0u);
            }
        }
        if (ALIGNED) return w;
        // the row starts at & 3 floats into its first float4: the points shifted out come from the first float4 of
        // the next lane's word, or from one more load
        const int sh = at & 3;
        uint32_t hi = __shfl_down_sync(0xffffffffu, w, 1);
        if (last && nv + sh > 32) {
            const float4 v = *reinterpret_cast<const float4*>(p + 128);
            const float below = __uint_as_float((uint32_t)below2);
            const bool all = (uint32_t)below2 == kAllButNaN;
            hi = (uint32_t)(all ? v.x == v.x : v.x > below) | (uint32_t)(all ? v.y == v.y : v.y > below) << 1 |
                 (uint32_t)(all ? v.z == v.z : v.z > below) << 2;  // at most three points were shifted out
        }
        return __funnelshift_r(w, hi, sh);
    }
};

// The values a lane keeps per row of a plane.
struct PlaneRow {
    uint32_t w, sh;  // the word, and the word shifted down by one point (within the row's cells)
    uint32_t pv;     // set corners of the row's cells
};

// v summed over the lanes of a row, in its first lane.
__device__ __forceinline__ uint32_t row_total(uint32_t v, int lw, int W)
{
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        if (d >= W) break;
        const uint32_t t = __shfl_down_sync(0xffffffffu, v, d);
        if (lw + d < W) v += t;
    }
    return v;
}

// Bytes of one plane's rows in a warp's buffer.
__host__ __device__ inline int count_stage_bytes(int nx, int W, int S, int sample_bytes, bool aligned)
{
    const int rows = (32 / W) * S + 1;
    return ((rows * nx + (aligned ? 0 : 16 / sample_bytes - 1)) * sample_bytes + kCountPad + 15) & ~15;
}

// Item `item` of a grid: row group item % ngroups, planes [kc * KC, ...) of
// column item / ngroups; one warp, its buffer at buf and the buffer's barrier at
// bar.  A plane's copy is issued as soon as the words of the plane before it are
// built and runs while those are counted; a second buffer per warp was no faster
// (512^3: 100 us with two rows per lane and two buffers, 100 us with four and one;
// 768^3: 415 against 302 us, for the warps that the buffers take).
template <class Samples, bool MC, int S>
__device__ __forceinline__ void count_rows_item(const typename Samples::T* __restrict__ vol, const Grid& g,
                                                const Samples& smp, int KC, int ngroups, unsigned item,
                                                unsigned char* buf, uint64_t* bar,
                                                uint4* __restrict__ rowcnt, uint2* __restrict__ trims,
                                                uint32_t* __restrict__ mccnt, uint32_t* __restrict__ bits_out,
                                                unsigned long long* __restrict__ status)
{
    typedef typename Samples::T T;
    constexpr bool ALIGNED = Samples::kAligned;
    constexpr int PER = 16 / (int)sizeof(T);  // samples of 16 bytes
    const int lane = threadIdx.x & 31;
    const int W = g.W, rpw = 32 / W, G = rpw * S;
    const int grp = (int)(item % (unsigned)ngroups), kc = (int)(item / (unsigned)ngroups);
    const int kb = g.kr + kc * KC, ke = min(kb + KC, g.ke);
    if (kb >= ke) return;  // past the grid's last plane column: nothing to copy
    const int hl = lane / W, lw = lane - hl * W;
    const int h = min(hl, rpw - 1);  // lanes past the last row repeat its addresses and hold no row
    const int jw = grp * G, j0 = jw + h * S;
    const int nrow = hl < rpw ? max(0, min(S + 1, g.ny - j0)) : 0;  // rows of the lane inside the grid
    const int nrows = min(G + 1, g.ny - jw);
    const uint32_t evalid = validmask(lw, g.nx - 1), pvalid = validmask(lw, g.nx);
    const int first = h * S * g.nx + 32 * lw;  // the lane's word of its first row
    const typename Samples::Lane place = smp.lane(lane, h * S * g.nx);
    const bool last = lw == W - 1;
    const int nv = g.nx - 32 * lw;
    const int plast = min(g.ke, g.nz - 1);  // the last plane the pass reads

    if (lane == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    __syncwarp();

    auto plane_start = [&](int p) { return ((long long)(p - g.kd) * g.ny + jw) * g.nx; };
    // Rows that are not a multiple of 16 bytes: the copy runs from the 16-byte boundary at or below their first
    // point to the one at or above their last, except past the end of the pass' last plane, where the last points
    // come by plain loads.  points [s0, e) -> copied [a0, e1)
    auto extent = [&](long long s0, long long& a0, long long& e1) {
        a0 = s0 & ~(long long)(PER - 1);
        const long long e = s0 + (long long)nrows * g.nx;
        e1 = (e + PER - 1) & ~(long long)(PER - 1);
        if (e1 > (long long)(plast - g.kd + 1) * g.ny * g.nx) e1 = e & ~(long long)(PER - 1);
        return e;
    };
    auto issue = [&](int p) {  // lane 0; the buffer's readers were joined by a __syncwarp
        const long long s0 = plane_start(p);
        fence_proxy_async();
        if (ALIGNED) {
            const unsigned bytes = (unsigned)(nrows * g.nx * (int)sizeof(T));
            mbar_arrive_expect_tx(bar, bytes);
            bulk_copy_g2s(buf, vol + s0, bytes, bar);
        } else {
            long long a0, e1;
            extent(s0, a0, e1);
            const unsigned bytes = (unsigned)((e1 - a0) * (int)sizeof(T));
            mbar_arrive_expect_tx(bar, bytes);
            if (bytes) bulk_copy_g2s(buf, vol + a0, bytes, bar);
        }
    };
    // the rows of plane p, the n-th of the item
    auto take = [&](int p, int n, PlaneRow (&r)[S + 1]) -> bool {
        const bool done = mbar_wait(bar, (unsigned)n & 1u);
        if (!__all_sync(0xffffffffu, done)) return false;
        int at = first;
        if (!ALIGNED) {
            const long long s0 = plane_start(p);
            long long a0, e1;
            const long long e = extent(s0, a0, e1);
            at += (int)(s0 - a0);
            // the last points of the pass' last plane. No copy into these bytes follows: the planes after it, which there
            // are only where a plane has fewer than PER points, end in the same 16 bytes and copy nothing.
            if (e1 < e) {
                if (lane < (int)(e - e1)) reinterpret_cast<T*>(buf)[(int)(e1 - a0) + lane] = __ldg(vol + e1 + lane);
                __syncwarp();
            }
        }
#pragma unroll
        for (int s = 0; s <= S; ++s) {
            const uint32_t w = smp.word(buf, at + s * g.nx, place, last, nv) & (s < nrow ? pvalid : 0u);
            const uint32_t nx = __shfl_down_sync(0xffffffffu, w, 1);
            r[s].w = w;
            r[s].sh = __funnelshift_r(w, nx, 1) & evalid;
            r[s].pv = __popc(w & evalid) + __popc(r[s].sh);
        }
        __syncwarp();  // every lane has read the buffer before it is refilled
        return true;
    };

    PlaneRow A[S + 1], C[S + 1];
    uint32_t zA[S], zC[S];  // set faces of the plane between a row and the next
    int n = 0;              // planes taken after the first
    if (lane == 0) issue(kb);
    bool ok = take(kb, 0, A);
    if (ok && kb + 1 < g.nz && lane == 0) issue(kb + 1);
#pragma unroll
    for (int s = 0; s < S; ++s) zA[s] = __popc(A[s].w & A[s].sh & A[s + 1].w & A[s + 1].sh);
    for (int k = kb; ok && k < ke; ++k) {
        const bool hasZ = k + 1 < g.nz;
        if (hasZ) {
            ++n;
            if (!(ok = take(k + 1, n, C))) break;
            if (k + 2 < g.nz && k + 2 <= ke && lane == 0) issue(k + 2);
        } else {
#pragma unroll
            for (int s = 0; s <= S; ++s) C[s].w = C[s].sh = C[s].pv = 0u;
        }
        uint32_t xy[S], zt[S], mc[S], y0 = __popc(A[0].w & A[0].sh & C[0].w & C[0].sh);
        uint32_t tfirst = 0xffffffffu, tlast = 0u;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const uint32_t a = A[s].w, b = A[s + 1].w, c = C[s].w, d = C[s + 1].w;
            const uint32_t as = A[s].sh, bs = A[s + 1].sh, cs = C[s].sh, ds = C[s + 1].sh;
            const bool hasY = s + 1 < nrow;
            const uint32_t xm = (a ^ as) & evalid, ym = hasY ? a ^ b : 0u, zm = hasZ ? a ^ c : 0u;
            xy[s] = __popc(xm) | (__popc(ym) << 16);
            // the triangles of the word's cells (tris_of_word): corners - 2 faces - 4 rings + 4 full cells, the
            // corners and the faces between rows and planes taken from the rows' own counts
            const uint32_t y1 = __popc(b & bs & d & ds);
            const uint32_t e1 = a & b, e2 = c & d, xlo = e1 & e2 & evalid, xhi = as & bs & cs & ds;
            zC[s] = __popc(c & cs & d & ds);
            const uint32_t faces = zA[s] + zC[s] + y0 + y1 + __popc(xlo) + __popc(xhi);
            y0 = y1;
            // body diagonals 0-6 1-7 2-4 3-5 (corners a as bs b c cs ds d): one unset, the other three set
            const uint32_t p0 = a & ds, p1 = as & d, p2 = bs & c, p3 = b & cs;
            const uint32_t o0 = a | ds, o1 = as | d, o2 = bs | c, o3 = b | cs;
            const uint32_t p01 = p0 & p1, p23 = p2 & p3;
            const uint32_t ring = (p23 & ((p0 & ~o1) | (p1 & ~o0))) | (p01 & ((p2 & ~o3) | (p3 & ~o2)));
            const uint32_t nt = A[s].pv + A[s + 1].pv + C[s].pv + C[s + 1].pv - 2u * faces +
                                4u * (__popc(p01 & p23) - __popc(ring));
            zt[s] = __popc(zm) | ((hasY && hasZ ? nt : 0u) << 16);
            if (MC)
                mc[s] = hasY && hasZ ? mc_verts_of_word(a, as, bs, b, c, cs, ds, d, evalid, j0 + s == 0, k == 0, lw == 0)
                                     : 0u;
            if (S == 1) {  // trim candidates: isCutEdge (FlyingEdgesAlgorithm.cpp:515-554)
                const uint32_t marked = xm | ((ym | zm) & evalid);
                if (marked) {
                    tfirst = (uint32_t)(32 * lw + __ffs(marked) - 1);
                    tlast = (uint32_t)(32 * lw + 32 - __clz(marked));
                }
            }
        }
        const long long r0 = (long long)(k - g.kr) * g.ny + j0;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            xy[s] = row_total(xy[s], lw, W);
            zt[s] = row_total(zt[s], lw, W);
            if (MC) mc[s] = row_total(mc[s], lw, W);
            if (s < nrow) {
                bits_out[(r0 + s) * W + lw] = A[s].w;
                if (lw == 0) {
                    rowcnt[r0 + s] = make_uint4(xy[s] & 0xffffu, xy[s] >> 16, zt[s] & 0xffffu, zt[s] >> 16);
                    if (MC) mccnt[r0 + s] = mc[s];
                }
            }
        }
        if (S == 1 && trims) {  // the pass-by-pass interface alone asks for them
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t f = __shfl_down_sync(0xffffffffu, tfirst, d), x = __shfl_down_sync(0xffffffffu, tlast, d);
                if (lw + d < W) {
                    tfirst = min(tfirst, f);
                    tlast = max(tlast, x);
                }
            }
            if (nrow > 0 && lw == 0) trims[r0] = make_uint2(tfirst == 0xffffffffu ? (uint32_t)g.nx : tfirst, tlast);
        }
#pragma unroll
        for (int s = 0; s <= S; ++s) A[s] = C[s];
#pragma unroll
        for (int s = 0; s < S; ++s) zA[s] = zC[s];
    }
    if (!ok) {  // a copy did not complete in time: report it, and let the copy land before the CTA ends
        if (lane == 0) atomicOr(status, kStatusTimeout);
        mbar_wait(bar, (unsigned)n & 1u);
    }
}

}  // namespace iso
