// Passes 1+2 of Flying Edges / the Marching Cubes counts over 8- and 16-bit
// samples read as they are: the typed-volume path of iso_extract_device_typed
// without a float32 copy of the volume (flyingEdges/util/ConvertBuffer.h:
// 45-72 converts every sample to float before extracting).
//
// The reference classifies a sample s by (float)s >= iso.  For 8- and 16-bit
// integers the conversion is exact, and for an integer s and a real iso,
// s >= iso exactly when s >= ceil(iso); so the kernel compares the integer
// sample with thr = ceil(iso) (clamped to the int range; a NaN isovalue, for
// which every comparison is false, gives INT_MAX).  The rows, words and counts
// are those of count_rows.cuh, so the scan and the generate pass that follow
// are unchanged; the vertex pass reads the same narrow samples (k_vertices with
// a sample type, vertices.cuh).
#include <climits>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "../../include/miniiso.h"
#include "count_rows.cuh"
#include "iso_kernels.h"

namespace iso {

// Two or four samples of a 32-bit word compared at once.  With a sample's top
// bit set and the threshold's cleared, their difference keeps its top bit
// exactly when the low bits alone are at or above the threshold's, and borrows
// from no neighbour; the top bits then decide by themselves or leave it to
// that.  Signed samples are the unsigned ones with the top bit the other way
// round.  1.35 (8 bits) and 2.6 (16 bits) instructions a sample, where a
// compare, a select and a shift per sample took 4 to 5.
template <typename S, bool ALIGNED>
struct IntSamples {
    typedef S T;
    static constexpr bool kAligned = ALIGNED;
    static constexpr int B = 8 * (int)sizeof(S);
    static constexpr int PER = 16 / (int)sizeof(S);  // samples of a 16-byte chunk
    static constexpr int NV = 2 * (int)sizeof(S);    // chunks of a word
    static constexpr uint32_t kOne = B == 8 ? 0x01010101u : 0x00010001u, kTop = kOne << (B - 1);
    uint32_t low, high;  // the threshold's low bits; all ones where its top bit is clear
    uint32_t on;         // the top bits, none when no sample reaches the threshold
    struct Lane {
        int off[NV];
        int rot;
    };
    __device__ __forceinline__ IntSamples(int thr)
    {
        const int least = std::is_signed<S>::value ? -(1 << (B - 1)) : 0;
        const uint32_t t = thr <= least ? 0u : (uint32_t)thr - (uint32_t)least;  // as of unsigned samples
        on = (thr > least && t >> B) ? 0u : kTop;
        low = (t & ((1u << (B - 1)) - 1u)) * kOne;
        high = (t >> (B - 1)) & 1u ? 0u : 0xffffffffu;
    }
    // Neighbouring lanes start at different chunks of their words, so that a quarter warp reads different banks.
    __device__ __forceinline__ Lane lane(int lane, int first) const
    {
        Lane x;
        x.rot = (lane / (8 / NV) - first / PER) & (NV - 1);
#pragma unroll
        for (int u = 0; u < NV; ++u) x.off[u] = ((u + x.rot) & (NV - 1)) * 16;
        return x;
    }
    // the top bit of every sample of w: sample >= threshold
    __device__ __forceinline__ uint32_t ge(uint32_t w) const
    {
        const uint32_t d = (w | kTop) - low;
        const uint32_t u = std::is_signed<S>::value ? ~w : w;
        return ((u & d) | ((u | d) & high)) & on;
    }
    // Bits of two chunks, the first sample in the lowest (8-bit samples: 32 bits; 16-bit: 16).
    __device__ __forceinline__ uint32_t bits2(uint4 a, uint4 b) const
    {
        if constexpr (B == 8) {
            // two words to a nibble pair per byte, whose bits 3 and 7 a multiplication brings next to the other
            // bytes' in the top byte (no two of its terms meet)
            constexpr uint32_t gather = 1u << 21 | 1u << 14 | 1u << 7 | 1u;
            const uint32_t p0 = (ge(a.x) >> 4 | ge(a.y)) * gather, p1 = (ge(a.z) >> 4 | ge(a.w)) * gather;
            const uint32_t p2 = (ge(b.x) >> 4 | ge(b.y)) * gather, p3 = (ge(b.z) >> 4 | ge(b.w)) * gather;
            return __byte_perm(__byte_perm(p0, p1, 0x0073), __byte_perm(p2, p3, 0x0073), 0x5410);
        } else {
            // every second bit of both halves: odd samples above, even ones below
            uint32_t r = ge(a.x);
            r = r >> 2 | ge(a.y);
            r = r >> 2 | ge(a.z);
            r = r >> 2 | ge(a.w);
            r = r >> 2 | ge(b.x);
            r = r >> 2 | ge(b.y);
            r = r >> 2 | ge(b.z);
            r = r >> 2 | ge(b.w);
            return r;
        }
    }
    // Word at sample index `at` of the buffer (row start + 32 * word); bits past the row are garbage.  Every lane of
    // the warp calls it.  last: the lane's word is the row's last, nv its points inside the row.
    __device__ __forceinline__ uint32_t word(const unsigned char* buf, int at, const Lane& x, bool last, int nv) const
    {
        const unsigned char* p = buf + 16 * (at / PER);
        uint32_t w;
        const uint32_t a = bits2(*reinterpret_cast<const uint4*>(p + x.off[0]),
                                 *reinterpret_cast<const uint4*>(p + x.off[1]));
        if constexpr (B == 8) {
            w = a;
        } else {
            const uint32_t b = bits2(*reinterpret_cast<const uint4*>(p + x.off[2]),
                                     *reinterpret_cast<const uint4*>(p + x.off[3]));
            w = __byte_perm(a, b, 0x7632) | __byte_perm(a, b, 0x5410) >> 1;
        }
        w = __funnelshift_l(w, w, PER * x.rot);
        if (ALIGNED) return w;
        // the row starts at % PER samples into its first chunk: the points shifted out come from the next lane's
        // word, or from one more chunk
        const int sh = at & (PER - 1);
        uint32_t hi = __shfl_down_sync(0xffffffffu, w, 1);
        if (last && nv + sh > 32) {
            const uint32_t c = bits2(*reinterpret_cast<const uint4*>(p + 16 * NV), make_uint4(0u, 0u, 0u, 0u));
            // 16-bit samples: the chunk's bits went eight places further down, past the zeros' ones
            hi = B == 8 ? c : (c >> 16 & 0xaau) | (c >> 1 & 0x55u);
        }
        return __funnelshift_r(w, hi, sh);
    }
};

// R rows per lane by count_rows_plan's rule, which suits these samples too (times of any R above one and of half to
// four times its planes per item lie within 5%).  The ALU pipe bounds it: 512 x 512 x 320 int16 52 us (66 with a
// compare per sample and rows at powers of two of lanes; its bytes take 26), int8 39 (65).  Rows of 17-32 words and
// rows that are not a multiple of 16 bytes come here too instead of through a float32 copy of the volume: extraction
// of 667 x 328 x 324 int16 254 us against 464, 301 x 417 x 290 uint8 141 against 246.
template <bool MC, typename S, int R, bool ALIGNED>
__global__ void __launch_bounds__(kCountThreads) k_count_narrow(const S* __restrict__ vol, Grid g, int thr, int KC,
                                                                int ngroups, unsigned nitems, int stage_bytes,
                                                                uint4* __restrict__ rowcnt,
                                                                uint32_t* __restrict__ mccnt,
                                                                uint32_t* __restrict__ bits_out,
                                                                unsigned long long* __restrict__ status)
{
    extern __shared__ __align__(128) unsigned char s_raw[];
    __shared__ uint64_t s_bar[kCountWarps];
    next_may_start();
    const int warp = threadIdx.x >> 5;
    const unsigned item = blockIdx.x * kCountWarps + warp;
    if (item >= nitems) return;
    const IntSamples<S, ALIGNED> smp(thr);
    count_rows_item<IntSamples<S, ALIGNED>, MC, R>(vol, g, smp, KC, ngroups, item, s_raw + (size_t)warp * stage_bytes,
                                                   s_bar + warp, rowcnt, nullptr, mccnt, bits_out, status);
}

int narrow_threshold(float iso)
{
    if (std::isnan(iso)) return INT_MAX;  // (float)s >= NaN is false for every sample
    const double c = std::ceil((double)iso);
    if (c >= (double)INT_MAX) return INT_MAX;  // above every 8- and 16-bit sample
    if (c <= (double)INT_MIN) return INT_MIN;
    return (int)c;
}

bool narrow_fits(const Grid& g, const void* vol, int dtype)
{
    const size_t sb = dtype_bytes(dtype);
    return (sb == 1 || sb == 2) && g.kd == 0 && g.kr == 0 && g.ke == g.nz && g.W <= 32 &&
           (reinterpret_cast<uintptr_t>(vol) & 15) == 0;
}

template <bool MC, typename S>
static void narrow_launch(const CountPlan& p, const S* vol, const Grid& g, int thr, FeBuffers& b,
                          unsigned long long* status, cudaStream_t s)
{
    const bool aligned = g.nx * (int)sizeof(S) % 16 == 0;
    const CountRows r = count_rows_plan(g, p.nsm, (int)sizeof(S), aligned, false);
    const size_t smem = (size_t)kCountWarps * r.stage;
    const unsigned nb = (r.items + kCountWarps - 1) / kCountWarps;
    auto kern = r.S == 4 ? (aligned ? k_count_narrow<MC, S, 4, true> : k_count_narrow<MC, S, 4, false>)
              : r.S == 2 ? (aligned ? k_count_narrow<MC, S, 2, true> : k_count_narrow<MC, S, 2, false>)
                         : (aligned ? k_count_narrow<MC, S, 1, true> : k_count_narrow<MC, S, 1, false>);
    allow_smem(kern, smem);
    kern<<<nb, kCountThreads, smem, s>>>(vol, g, thr, r.KC, r.groups, r.items, r.stage, b.rowcnt, b.mccnt, b.bits,
                                         status);
}

void launch_count_narrow(const void* vol, int dtype, const Grid& g, float iso, bool mc, const CountPlan& p, FeBuffers& b,
                         cudaStream_t s, bool zero_status)
{
    unsigned long long* status = count_status(b, zero_status, s);
    const int thr = narrow_threshold(iso);
#define ISO_TYPE(T)                                                                   \
    {                                                                                 \
        if (mc) narrow_launch<true, T>(p, static_cast<const T*>(vol), g, thr, b, status, s);  \
        else narrow_launch<false, T>(p, static_cast<const T*>(vol), g, thr, b, status, s);    \
    }
    switch (dtype) {
        case ISO_INT8: ISO_TYPE(int8_t) break;
        case ISO_UINT8: ISO_TYPE(uint8_t) break;
        case ISO_INT16: ISO_TYPE(int16_t) break;
        default: ISO_TYPE(uint16_t) break;
    }
#undef ISO_TYPE
}

}  // namespace iso
