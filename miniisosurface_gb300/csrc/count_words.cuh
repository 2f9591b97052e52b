// Counting helpers of the count kernels (count_kernels.cu): a row's counts word
// by word (cut x, y, z edges, trims, triangles and Marching Cubes vertices of
// its cells).
#pragma once
#include "iso_device.cuh"

namespace iso {

constexpr int kCountRows = 8;  // warps per CTA of the count kernels

// Counts of one grid row, accumulated word by word in each lane.
struct RowCounts {
    uint32_t xc = 0, yc = 0, zc = 0, tc = 0, mc = 0, first = 0xffffffffu, last = 0;
};

// Counts of word w of grid row (j,k): cut x / y / z edges the row owns, the
// trim candidates, the triangles (and MC vertices) of its cells.
// trims: whether the row trims are wanted (only the pass-by-pass interface
// reads them; an extraction skips them).
template <bool MC>
__device__ __forceinline__ void count_word(const RowWords& rw, int w, const Grid& g, int j, int k, bool hasY,
                                           bool hasZ, bool trims, RowCounts& rc)
{
    const uint32_t evalid = validmask(w, g.nx - 1);  // x-edges / cells: i <= nx-2
    const uint32_t pvalid = validmask(w, g.nx);      // points: i <= nx-1
    const uint32_t xm = (rw.a ^ rw.ash) & evalid;
    const uint32_t ym = hasY ? ((rw.a ^ rw.b) & pvalid) : 0u;
    const uint32_t zm = hasZ ? ((rw.a ^ rw.c) & pvalid) : 0u;
    rc.xc += __popc(xm);
    rc.yc += __popc(ym);
    rc.zc += __popc(zm);
    // isCutEdge (FlyingEdgesAlgorithm.cpp:515-554): edge i is marked when
    // it is cut or the y / z edge at its left point is.
    const uint32_t marked = trims ? (xm | ((ym | zm) & evalid)) : 0u;
    if (marked) {
        rc.first = min(rc.first, (uint32_t)(32 * w + __ffs(marked) - 1));
        rc.last = max(rc.last, (uint32_t)(32 * w + 32 - __clz(marked)));
    }
    if (hasY && hasZ) {  // all 32 cells at once (tris_of_word, mc_verts_of_word)
        rc.tc += tris_of_word(rw.a, rw.ash, rw.bsh, rw.b, rw.c, rw.csh, rw.dsh, rw.d, evalid);
        if (MC) rc.mc += mc_verts_of_word(rw.a, rw.ash, rw.bsh, rw.b, rw.c, rw.csh, rw.dsh, rw.d, evalid, j == 0, k == 0,
                                          w == 0);
    }
}

}  // namespace iso
