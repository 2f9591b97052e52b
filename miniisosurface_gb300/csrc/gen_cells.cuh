// Pass 4 (FlyingEdgesAlgorithm.cpp:271-500; Marching Cubes: marchingCubes/
// serial/main.cpp:96-185) for rows of up to 32 words (nx <= 1024), included by
// gen_warps_fe.cu and gen_warps_mc.cu: triangles, and a record per vertex that
// k_vertices (vertices.cuh) turns into its position and normal.
//
// A warp takes work items -- a group of G neighbouring grid rows and a run of
// KC planes -- from a counter and marches along z on its own.  A row's W words
// go to W neighbouring lanes, rpw rows side by side (32 / W of them; fewer on
// grids with too few rows for the GPU), and a lane holds kGenSlots rows (slot
// s: row jw + s * rpw + lane / W), the last row, or one in a slot more, the row
// after the group: the fixed work of a step is shared by up to 64 words, and their active cells and
// triangles fill batches of 32 lanes (one row pair at a time left a third of the
// lanes idle).
//
// Every cut mask belongs to one grid row of one plane (z: to one row between
// two planes) and is computed once, when its plane is entered, not once per
// cell row that touches it: the warp keeps {mask, id of its first cut edge} of
// x, y and z of every word and row in shared memory, the planes' two copies
// side by side, and a triangle corner is one 8-byte load and a popc:
//   tab[idx][axis][plane & 1]   48 bytes per word, idx = w * (2 * rpw + 1) + row,
//                               odd so that neighbouring words fall on different banks
//   pair[idx][plane & 1]        {word, next word} of the row
// With that order the word above in y is 48 bytes on at any width, so a corner
// is the same byte for every grid (axis * 16 + row * 48 + plane * 8, bit 0 the
// edge at point i + 1), and the other plane is bit 3 of the address.
//
// What bounds it: instruction issue (77% of the slots on the 512^3 volume, with 115 M warp instructions; the kernels
// it replaced, which recomputed eight masks and four scans per row and step, took 161 M).  Events around the pass, us,
// Flying Edges, before / now: 512^3 167 / 124, 768^3 (with the vertices, which were in the same kernel) 1252 / 715,
// 667 x 228 x 724 the same 363 / 208, 150 x 700 x 600 110 / 68, 301 x 217 x 190 36 / 27, 128^3 22 / 16.5, 64^3 17 / 12.
// Three rows per lane and one more instead of two and one: 145 us at 512^3 (fewer warps fit).  Vertex runs made dense like the cells
// instead of a loop over each word's bits: 32 M instructions instead of 21 M.
// Marching Cubes: a cell away from the first column, row and plane owns at most three vertices, read ready from a
// table instead of walking the case's edges one by one, and a chunk's vertices are written together: 512^3 187 us
// before, 145 now (667 x 228 x 724 blobs 82 / 72, 64^3 13.9 / 11.9).
#pragma once
#include "batch_kernels.cuh"
#include "gen_warps.cuh"
#include "vertices.cuh"

namespace iso {

constexpr int kGenSlots = 2;       // rows per lane
constexpr int kGenExtra = 2;       // rows side by side up to which a kernel for them gives the row after the group a slot
// Cells whose triangles are listed together: a step of the 512^3 volume has 85, so that most take one list and the
// triangles' batches are full but for its last (64 cells: 126.3 us, 96: 123.7, 128: 123.8; 301 x 217 x 190 28.3 / 26.8 /
// 26.8, 64^3 12.8 / 12.0 / 12.0). Marching Cubes: 64, so that their vertices fit their list (kGenOwned).
__host__ __device__ inline constexpr int gen_chunk(int mode) { return mode == kGenFE ? 96 : 64; }
constexpr int kGenMaxWarps = 16;   // warps per CTA, two CTAs per SM
// ... of the batch kernel, which holds what others take from their parameters in registers: with 16 it spilled 29 of
// them (64 uneven volumes, whole call 2030 us; 14: 1960, 12: 1970, 10: 2013)
constexpr int kGenBatchWarps = 14;

// Rows held by a warp: the group's and the one after it, which takes a slot of its own (extra) or is the last of the
// slots' rows.
__host__ __device__ inline constexpr bool gen_extra_slot(int RPW) { return RPW > 0 && RPW <= kGenExtra; }
__host__ __device__ inline constexpr int gen_group_rows(int rpw, bool extra) { return kGenSlots * rpw - (extra ? 0 : 1); }
// Entries of a word in the warp's tables: odd, so that neighbouring words fall on different banks.
__host__ __device__ inline int gen_word_entries(int rpw) { return kGenSlots * rpw + 1; }

// Per-warp scratch: tab, pair, cell[chunk], the triangle list (u16), and for the Marching Cubes modes the
// cells' places and the owned vertices' list.
__host__ __device__ inline bool gen_owns(int mode) { return mode == kGenMC || mode == kGenMCT; }
__host__ __device__ inline int gen_cells_scratch(int W, int rpw, int mode)
{
    const int list = mode == kGenMC ? 0 : 5 * gen_chunk(mode) * 2;
    const int own = gen_owns(mode) ? 4 * gen_chunk(mode) + 2 * kGenOwned : 0;
    // + 48: the last row of a slot looks one entry past its word's rows
    return (64 * W * gen_word_entries(rpw) + 48 + 4 * gen_chunk(mode) + list + own + 15) & ~15;
}

// The kernel's per-case tables in shared memory (CaseTables holds them ready).
template <int MODE>
struct GenCellTables {
    static constexpr bool OWNS = MODE == kGenMC || MODE == kGenMCT;
    static constexpr bool TRIS = MODE != kGenMC;
    uint32_t corner[TRIS ? 256 * 5 : 1];
    uint32_t nth[256];
    uint64_t order[OWNS ? 256 : 1];
    uint32_t own[OWNS ? 256 : 1];
    uint16_t cut[OWNS ? 256 : 1];
    uint8_t nt[256];
};

template <int MODE>
__device__ __forceinline__ void stage_gen_tables(const CaseTables* __restrict__ cases, GenCellTables<MODE>& t)
{
    if (t.TRIS)
        for (int c = threadIdx.x; c < 256 * 5; c += blockDim.x) t.corner[c] = cases->corner[c];
    for (int c = threadIdx.x; c < 256; c += blockDim.x) {
        t.nth[c] = cases->nth[c];
        t.nt[c] = cases->nt2[c];
        if (t.OWNS) {
            t.order[c] = cases->order2[c];
            t.cut[c] = cases->cut2[c];
            t.own[c] = cases->own2[c];
        }
    }
}

// Place of set bit n (from 0) of m, n < popc(m): two halvings, then a byte's places from a table.
__device__ __forceinline__ int nth_bit(uint32_t m, int n, const uint32_t* nth)
{
    int at = 0;
    int c = __popc(m & 0xffffu);
    if (n >= c) {
        n -= c;
        m >>= 16;
        at = 16;
    }
    c = __popc(m & 0xffu);
    if (n >= c) {
        n -= c;
        m >>= 8;
        at += 8;
    }
    return at + (int)((nth[m & 0xffu] >> (4 * n)) & 7u);
}

// Inclusive sum over the warp's lanes.
__device__ __forceinline__ uint32_t lane_incl_sum(uint32_t v)
{
#define ISO_STEP(D)                                      \
    asm volatile(                                        \
        "{\n\t.reg .pred p;\n\t.reg .b32 t;\n\t"           \
        "shfl.sync.up.b32 t|p, %0, " #D                  \
        ", 0, 0xffffffff;\n\t@p add.u32 %0, %0, t;\n\t}" \
        : "+r"(v))
    ISO_STEP(1);
    ISO_STEP(2);
    ISO_STEP(4);
    ISO_STEP(8);
    ISO_STEP(16);
#undef ISO_STEP
    return v;
}

// Runs of planes of the items: `nbig` columns of `big` planes first, then columns of KC: the long ones for the
// work that entering an item's first plane costs, the short ones so that the warps finish together.
struct GenCols {
    int nbig, big, KC;
};

// A lane's place in the groups of rows of W words, rpw side by side.
struct GenLane {
    int h, lw, idx0;   // its row of a slot, its word, its entry of slot 0 (slot s: + s * rpw)
    int rows;          // slot s holds a row of the warp when s * rpw < rows
    uint32_t evalid;   // x-edges / cells of its word: i <= nx-2
};

__device__ __forceinline__ GenLane gen_lane(const Grid& g, int rpw, bool extra)
{
    GenLane l;
    const int lane = threadIdx.x & 31;
    l.h = lane / g.W;
    l.lw = lane - l.h * g.W;
    l.idx0 = l.lw * gen_word_entries(rpw) + l.h;
    l.rows = l.h < rpw ? gen_group_rows(rpw, extra) + 1 - l.h : 0;
    l.evalid = validmask(l.lw, g.nx - 1);
    return l;
}

// Where an item's records and triangles go: kernel parameters, or the request's copy in shared memory, read anew at
// each use because the batch kernel has no registers left for it.
template <typename IndexT>
struct GenOut {
    float* p;
    IndexT* t;
    __device__ __forceinline__ float* points() const { return p; }
    __device__ __forceinline__ IndexT* tris() const { return t; }
};
template <typename IndexT>
struct GenOutShared {
    const volatile unsigned long long* s;
    __device__ __forceinline__ float* points() const { return reinterpret_cast<float*>(s[0]); }
    __device__ __forceinline__ IndexT* tris() const { return reinterpret_cast<IndexT*>(s[1]); }
};

// Work item `item` of an extraction, run by one warp with its scratch at s_raw + ws.
template <typename IndexT, int MODE, int RPW, typename Out>
__device__ __forceinline__ void gen_cells_item(uint32_t item, unsigned char* s_raw, uint32_t ws,
                                               const GenCellTables<MODE>& tabs, const uint32_t* __restrict__ bits,
                                               const Grid& g, const GenLane& ln, int rpw_, const GenCols& cols, int ngroups,
                                               int kbeg, int kend, int kemit, unsigned long long vbase,
                                               unsigned long long tbase, const uint4* row4,
                                               const RowStarts& rs, const Out& out, uint32_t* __restrict__ fe2mc, int reverse)
{
    constexpr bool OWNS = GenCellTables<MODE>::OWNS, TRIS = GenCellTables<MODE>::TRIS;
    constexpr bool WIDE = MODE == kGenFE && sizeof(IndexT) == 8;  // ids past 32 bits; the map's ids are 32-bit
    constexpr int kChunk = gen_chunk(MODE);
    constexpr int S = kGenSlots, NS = S + (gen_extra_slot(RPW) ? 1 : 0);
    static_assert(S == 2, "the active cells' counts of a lane's slots share a word");
    const int rpw = RPW > 0 ? RPW : rpw_;
    const int lane = threadIdx.x & 31;
    const int W = g.W, RW = rpw * W, E = gen_word_entries(rpw), G = gen_group_rows(rpw, gen_extra_slot(RPW));
    const int h = ln.h, lw = ln.lw, idx0 = ln.idx0;
    unsigned char* tab = s_raw + ws;
    unsigned char* pair = tab + 48 * W * E;
    uint32_t* cell = reinterpret_cast<uint32_t*>(pair + 16 * W * E + 48);
    uint16_t* list = reinterpret_cast<uint16_t*>(cell + kChunk);
    uint32_t* place = reinterpret_cast<uint32_t*>(list + (TRIS ? 5 * kChunk : 0));
    uint16_t* vlist = reinterpret_cast<uint16_t*>(place + kChunk);

    const int col = (int)(item / (uint32_t)ngroups);
    const int jw = G * (int)(item - (uint32_t)col * (uint32_t)ngroups);
    const int from = col < cols.nbig ? col * cols.big : cols.nbig * cols.big + (col - cols.nbig) * cols.KC;
    const int len = min(col < cols.nbig ? cols.big : cols.KC, kend - kbeg - from);
    const int kb = reverse ? kend - from - len : kbeg + from, ke = kb + len, plast = min(ke, g.nz - 1);
    const int nrow = min(ln.rows, g.ny - jw - h);           // slot s holds a row of the grid when s * rpw < nrow
    const int ncell = min(ln.rows - 1, g.ny - 1 - jw - h);  // ... a cell row of the group when s * rpw < ncell
    const uint32_t add0 = (uint32_t)rs.add[0];
    const long long rp0 = (long long)(kb - g.kr) * g.ny + jw;
    const uint32_t* bp = bits + rp0 * W + lane;                // the plane's words
    const uint4* qp = row4 + rp0 + h;                          // the plane's row starts
    const unsigned long long* sp = rs.starts + rp0;            // first vertex of row jw, R on: first triangle

    uint32_t w[NS], wp[NS], zb[NS];  // this plane's words; of the plane before: words, id of the first z cut
    uint4 q[NS];                     // this plane's first x, y and z cut of the row
    uint32_t pand[S], por[S];        // corners all set / any set between a row and the next, of the plane before
    unsigned long long xwp = 0ull, tnext = 0ull, mnext = 0ull;  // of the plane before, row jw: first vertex (WIDE),
                                                                // first triangle, first owned MC vertex
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        wp[s] = zb[s] = 0u;
        w[s] = s * rpw < nrow ? __ldg(bp + s * RW) : 0u;
        q[s] = s * rpw < nrow ? load_written(qp + s * rpw) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int s = 0; s < S; ++s) pand[s] = por[s] = 0u;
    for (int p = kb; p <= plast; ++p) {
        const uint32_t par = (uint32_t)(p & 1) * 8u, kpar = par ^ 8u;  // this plane's copy, the plane before's
        const bool cells = p > kb;
        unsigned long long tcur = tnext, mcur = mnext, xw = 0ull;
        if (TRIS) tnext = load_written(sp + rs.R) + rs.add[1];
        if (OWNS) mnext = load_written(sp + 2 * rs.R) + rs.add[2];
        if (WIDE) xw = load_written(sp) + rs.add[0];
        uint32_t act[S];
        {
            uint32_t wn[NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                wn[s] = __shfl_down_sync(0xffffffffu, w[s], 1);
                if (s * rpw < ln.rows) *reinterpret_cast<uint2*>(pair + 16 * (idx0 + s * rpw) + par) = make_uint2(w[s], wn[s]);
            }
            __syncwarp();
            uint32_t x[NS], y[NS], z[NS], any = 0u;
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const uint32_t sh = __funnelshift_r(w[s], wn[s], 1);
                x[s] = (w[s] ^ sh) & ln.evalid;
                z[s] = cells ? w[s] ^ wp[s] : 0u;
                y[s] = 0u;
                if (s < S) {
                    const uint2 b = *reinterpret_cast<const uint2*>(pair + 16 * (idx0 + s * rpw + 1) + par);
                    const uint32_t bsh = __funnelshift_r(b.x, b.y, 1);
                    const bool row = s * rpw < ncell;
                    y[s] = row ? w[s] ^ b.x : 0u;
                    const uint32_t a4 = w[s] & sh & b.x & bsh, o4 = w[s] | sh | b.x | bsh;
                    act[s] = row ? (por[s] | o4) & ~(pand[s] & a4) & ln.evalid : 0u;
                    pand[s] = a4;
                    por[s] = o4;
                }
                any |= x[s] | y[s] | z[s];
            }
            if (__any_sync(0xffffffffu, any != 0u)) {  // else no cell of either side asks for this plane's masks
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    // exclusive prefixes over the row's words: x, y and z cuts in 11 + 11 + 10 bits (z wraps at the
                    // top), from the warp's sums and those before the row
                    const uint32_t own = __popc(x[s]) + (__popc(y[s]) << 11) + (__popc(z[s]) << 22);
                    uint32_t e = lane_incl_sum(own) - own;
                    e -= __shfl_sync(0xffffffffu, e, h * W);
                    const uint32_t xf = q[s].x + (e & 0x7ffu) + add0, yf = q[s].y + ((e >> 11) & 0x7ffu) + add0;
                    const uint32_t zf = zb[s] + (e >> 22);
                    if (s * rpw < ln.rows) {
                        unsigned char* t = tab + 48 * (idx0 + s * rpw);
                        *reinterpret_cast<uint2*>(t + par) = make_uint2(x[s], xf);
                        if (s < S) *reinterpret_cast<uint2*>(t + 16 + par) = make_uint2(y[s], yf);
                        *reinterpret_cast<uint2*>(t + 32 + kpar) = make_uint2(z[s], zf);
                    }
                    if (MODE == kGenFE && s < S && s * rpw < ln.rows - 1) {  // vertex records of the word's cut edges
                        const uint32_t j = (uint32_t)(jw + s * rpw + h);
                        auto records = [&](uint32_t mk, uint32_t first, unsigned long long row0, uint32_t axis, uint32_t k) {
                            const unsigned long long at = WIDE ? row0 - vbase + (uint32_t)(first - (uint32_t)row0)
                                                               : (unsigned long long)(uint32_t)(first - (uint32_t)vbase);
                            float* o = out.points() + 3 * at;
                            while (mk != 0u) {
                                put_vertex_record(o, 0ull, (uint32_t)(32 * lw + __ffs(mk) - 1), axis, j, k);
                                mk &= mk - 1u;
                                o += 3;
                            }
                        };
                        if (p < ke) {
                            records(x[s], xf, xw, 0u, (uint32_t)p);
                            records(y[s], yf, xw, 1u, (uint32_t)p);
                        }
                        records(z[s], zf, xwp, 2u, (uint32_t)(p - 1));
                    }
                }
            }
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                wp[s] = w[s];
                zb[s] = q[s].z + add0;
            }
            bp += (long long)g.ny * W;
            qp += g.ny;
            sp += g.ny;
            if (p < plast) {  // the next plane's words and row starts, in flight while this plane's cells run
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    w[s] = s * rpw < nrow ? __ldg(bp + s * RW) : 0u;
                    q[s] = s * rpw < nrow ? load_written(qp + s * rpw) : make_uint4(0u, 0u, 0u, 0u);
                }
            }
        }
        __syncwarp();

        if (cells) {
            const int k = p - 1;
            const uint32_t na = __popc(act[0]) | (__popc(act[1]) << 16);
            const uint32_t inc = lane_incl_sum(na);
            const uint32_t tot = __shfl_sync(0xffffffffu, inc, 31);
            const uint32_t tot0 = tot & 0xffffu, ctot = tot0 + (tot >> 16);
            // the owned vertices of a chunk fit their list: a cell owns at most 12 on the first plane and row, else 5
            const uint32_t chunk = OWNS && (k == 0 || jw == 0) ? 32u : (uint32_t)kChunk;
            static_assert(!OWNS || (kGenOwned >= 12 * 32 && kGenOwned >= 5 * kChunk), "owned vertices of a chunk");
            for (uint32_t c0 = 0; c0 < ctot; c0 += chunk) {
                uint32_t ntri = 0, nown = 0;
#pragma unroll 1
                for (uint32_t cb = 0; cb < chunk && c0 + cb < ctot; cb += 32) {
                    // lane L takes active cell c0 + cb + L (slot 0's come first): the first lane whose inclusive
                    // count passes it, by a shuffle binary search, then the bit
                    const uint32_t target = c0 + cb + (uint32_t)lane;
                    const bool live = target < ctot;
                    const bool up = target >= tot0;
                    const uint32_t sel = up ? 0x4432u : 0x4410u, tt = up ? target - tot0 : target;
                    int src = 0;
#pragma unroll
                    for (int step = 16; step > 0; step >>= 1) {
                        const uint32_t before = __byte_perm(__shfl_sync(0xffffffffu, inc, src + step - 1), 0u, sel);
                        if (before <= tt) src += step;
                    }
                    const uint32_t a0 = __shfl_sync(0xffffffffu, act[0], src), a1 = __shfl_sync(0xffffffffu, act[1], src);
                    const uint32_t a = up ? a1 : a0;
                    const uint32_t first = __byte_perm(__shfl_sync(0xffffffffu, inc - na, src), 0u, sel);
                    const uint32_t id = (uint32_t)(__shfl_sync(0xffffffffu, idx0, src) + (up ? rpw : 0));
                    const int slw = OWNS ? __shfl_sync(0xffffffffu, lw, src) : 0;
                    uint32_t cs = 0u, nt = 0u, row = 0u;
                    int b = 0;
                    if (live) {
                        b = nth_bit(a, (int)(tt - first), tabs.nth);
                        const unsigned char* q = pair + 16u * id;
                        const uint2 wa = *reinterpret_cast<const uint2*>(q + kpar);
                        const uint2 wb = *reinterpret_cast<const uint2*>(q + 16 + kpar);
                        const uint2 wc = *reinterpret_cast<const uint2*>(q + par);
                        const uint2 wd = *reinterpret_cast<const uint2*>(q + 16 + par);
                        // the cube case, corners in the order i, i + 1 of rows A, B, C, D (CaseTables)
                        cs = (__funnelshift_r(wa.x, wa.y, b) & 3u) | ((__funnelshift_r(wb.x, wb.y, b) & 3u) << 2) |
                             ((__funnelshift_r(wc.x, wc.y, b) & 3u) << 4) | ((__funnelshift_r(wd.x, wd.y, b) & 3u) << 6);
                        cell[cb + lane] = (48u * id) | ((uint32_t)b << 13) | ((5u * cs) << 18);
                        if (TRIS) nt = tabs.nt[cs];
                        if (OWNS) {
                            row = id - (uint32_t)(slw * E);
                            place[cb + lane] = (uint32_t)(32 * slw + b) | (row << 10);
                        }
                    }
                    if (TRIS && (MODE != kGenMCT || k >= kemit)) {  // rows below kemit belong to the slab below
                        const uint32_t it = lane_incl_sum(nt);
                        uint16_t* l = list + ntri + it - nt;
                        const uint32_t me = cb + (uint32_t)lane;
#pragma unroll
                        for (uint32_t q = 0; q < 5; ++q)
                            if (q < nt) l[q] = (uint16_t)(me | (q << 7));
                        ntri += __shfl_sync(0xffffffffu, it, 31);
                    }
                    if (OWNS) {
                        // the MC vertices the batch's cells own, listed in cell order, then order of first appearance in
                        // the cell's triangle list (marchingCubes/serial/main.cpp:139-177): at most three ready in a
                        // table, but for the cells of the first column, row and plane
                        const uint32_t me = cb + (uint32_t)lane, ready = live ? tabs.own[cs] : 0u;
                        uint32_t own = 0u, no = ready & 3u;
                        const bool edge = live && (slw + b == 0 || (jw == 0 && row == 0u) || k == 0);
                        if (edge) {
                            own = mc_owned_edges(slw + b == 0, jw == 0 && row == 0u, k == 0) & tabs.cut[cs];
                            no = __popc(own);
                        }
                        const uint32_t io = lane_incl_sum(no);
                        uint16_t* o = vlist + nown + io - no;
                        if (edge) {
                            const uint64_t ord = tabs.order[cs];
                            for (int q = 0; q < iso_case_ntris(ord); ++q) {
                                const int ed = iso_case_edge(ord, q);
                                if ((own >> ed) & 1u) *o++ = (uint16_t)(me | ((uint32_t)ed << 7));
                            }
                        } else {
                            if (no > 0u) o[0] = (uint16_t)(me | ((ready >> 1) & 0x780u));
                            if (no > 1u) o[1] = (uint16_t)(me | ((ready >> 5) & 0x780u));
                            if (no > 2u) o[2] = (uint16_t)(me | ((ready >> 9) & 0x780u));
                        }
                        nown += __shfl_sync(0xffffffffu, io, 31);
                    }
                }
                __syncwarp();
                if (OWNS) {
                    for (uint32_t v = (uint32_t)lane; v < nown; v += 32) {
                        const uint32_t vr = vlist[v];
                        const uint32_t cr = cell[vr & 127u], pl = place[vr & 127u];
                        const int e12 = (int)(vr >> 7);
                        const unsigned long long mid = mcur + v;
                        int dx, dy, dz, axis;
                        cube_edge_geometry(e12, dx, dy, dz, axis);
                        if (k >= kemit)  // cell rows below kemit belong to the slab below: map only
                            put_mc_record(out.points(), mid - vbase, (pl & 1023u) + (uint32_t)dx, (uint32_t)axis,
                                          (uint32_t)(dx | (dy << 1) | (dz << 2)), (uint32_t)(jw + dy) + (pl >> 10),
                                          (uint32_t)(k + dz));
                        // the edge's Flying Edges id: its axis, row and plane in tab, dx bits further along x
                        const uint2 pm = *reinterpret_cast<const uint2*>(
                            tab + (((cr & 0x1fffu) + 16u * (uint32_t)axis + 48u * (uint32_t)dy + 8u * (uint32_t)dz) ^ kpar));
                        const uint32_t sft = 32u - ((cr >> 13) & 31u) - (uint32_t)dx;
                        fe2mc[pm.y + __popc(__funnelshift_lc(0u, pm.x, sft))] = (uint32_t)mid;
                    }
                    mcur += nown;
                }
                if (TRIS) {
                    IndexT* o = out.tris() + 3 * (tcur + (uint32_t)lane - tbase);
                    for (uint32_t t = (uint32_t)lane; t < ntri; t += 32, o += 96) {
                        const uint32_t c = list[t];
                        const uint32_t rec = cell[c & 127u];
                        const uint32_t corners = tabs.corner[(rec >> 18) + (c >> 7)];
                        const uint32_t at = ws + (rec & 0x1fffu), sft = 32u - ((rec >> 13) & 31u);
                        uint32_t vid[3];
#pragma unroll
                        for (int q = 0; q < 3; ++q) {
                            const uint32_t v = at + ((corners >> (8 * q)) & 0xffu);
                            const uint2 pm = *reinterpret_cast<const uint2*>(s_raw + ((v ^ kpar) & ~7u));
                            // popc of the mask's bits below the edge's (the funnel shift clamps at 32)
                            vid[q] = pm.y + __popc(__funnelshift_lc(0u, pm.x, sft - (v & 1u)));
                        }
#pragma unroll
                        for (int q = 0; q < 3; ++q) {
                            if (MODE == kGenTri) o[q] = (IndexT)__ldg(fe2mc + vid[q]);
                            else if (WIDE) o[q] = (IndexT)(xwp + (uint32_t)(vid[q] - (uint32_t)xwp));
                            else o[q] = (IndexT)vid[q];
                        }
                    }
                    tcur += ntri;
                }
                __syncwarp();  // the next chunk overwrites the lists
            }
        }
        __syncwarp();  // the next plane overwrites the copies of the plane before
        xwp = xw;
    }
}

// The warp's next work item.  (Taken one item ahead, to overlap the counter's trip to memory, a warp at a long
// item kept a short one waiting: 512^3 140 us against 132, 256^3 40 against 34.)
__device__ __forceinline__ uint32_t gen_take(unsigned int* work)
{
    uint32_t item = 0u;
    if ((threadIdx.x & 31) == 0) item = atomicAdd(work, 1u);
    return __shfl_sync(0xffffffffu, item, 0);
}

// One wave of CTAs; every warp takes work items from the counter `work` until none is left.
template <typename IndexT, int MODE, int RPW>
__global__ void __launch_bounds__(32 * kGenMaxWarps, 2) k_gen_cells(
    const uint32_t* __restrict__ bits, Grid g, int rpw, GenCols cols, int ngroups, uint32_t nitems, int kbeg, int kend, int kemit,
    unsigned long long vbase, unsigned long long tbase, int ws_bytes, const CaseTables* __restrict__ cases,
    const uint4* row4, RowStarts rs, const unsigned long long* totals,
    unsigned int* __restrict__ work, long long capV, long long capT, float* __restrict__ points,
    IndexT* __restrict__ tris, uint32_t* __restrict__ fe2mc, int reverse)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ GenCellTables<MODE> tabs;
    stage_gen_tables<MODE>(cases, tabs);
    wait_for_previous();
    next_may_start();
    __syncthreads();  // the only CTA barrier: from here on every warp runs alone
    // Caller grows buffers.  Past this check every record slot and triangle index written below lies
    // under the totals, because the count pass derives the counts and starts from the same bit words
    // with the same masks; the writes are not checked one by one.
    if (!mesh_holds(totals, capV, capT)) return;
    const uint32_t ws = (threadIdx.x >> 5) * (uint32_t)ws_bytes;
    const GenLane ln = gen_lane(g, RPW > 0 ? RPW : rpw, gen_extra_slot(RPW));
    for (uint32_t item; (item = gen_take(work)) < nitems;) {
        gen_cells_item<IndexT, MODE, RPW>(item, s_raw, ws, tabs, bits, g, ln, rpw, cols, ngroups, kbeg, kend, kemit,
                                          vbase, tbase, row4, rs, GenOut<IndexT>{points, tris}, fe2mc, reverse);
    }
}

// The Flying Edges generate items of a list of requests (batch_kernels.cuh), one launch: item x is item
// x - first[q] of request list[q]; the items of a request whose mesh cannot hold its counts are skipped.
template <typename IndexT>
__global__ void __launch_bounds__(32 * kGenBatchWarps, 2) k_gen_cells_batch(
    const BatchReq* __restrict__ reqs, const int* __restrict__ list, const unsigned* __restrict__ first, int m,
    const CaseTables* __restrict__ cases, unsigned int* __restrict__ work, int ws_bytes, int reverse)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ GenCellTables<kGenFE> tabs;
    __shared__ unsigned long long s_out[kGenBatchWarps][2];
    stage_gen_tables<kGenFE>(cases, tabs);
    __syncthreads();
    const uint32_t ws = (threadIdx.x >> 5) * (uint32_t)ws_bytes;
    const uint32_t nitems = __ldg(&first[m]);
    for (uint32_t item; (item = gen_take(work)) < nitems;) {
        const int q = batch_find(first, m, item);
        const BatchReq* d = reqs + __ldg(&list[q]);
        if (!mesh_holds(d->totals, d->capV, d->capT)) continue;
        if (item - __ldg(&first[q]) >= (uint32_t)d->gen_ngroups * (uint32_t)d->gen_nkc) continue;  // past its items
        const Grid g = d->g;
        unsigned long long* out = s_out[threadIdx.x >> 5];
        __syncwarp();  // the item before has written its last triangle
        if ((threadIdx.x & 31) == 0) {
            out[0] = reinterpret_cast<unsigned long long>(d->points);
            out[1] = reinterpret_cast<unsigned long long>(d->tris);
        }
        __syncwarp();
        RowStarts rs;
        rs.starts = d->starts;
        rs.R = g.R;
        rs.ny = g.ny;
        rs.kr = g.kr;
        rs.add[0] = rs.add[1] = rs.add[2] = rs.add[3] = 0;
        gen_cells_item<IndexT, kGenFE, 0>(item - __ldg(&first[q]), s_raw, ws, tabs, d->bits, g, gen_lane(g, 32 / g.W, false),
                                       32 / g.W, GenCols{0, 1, d->gen_KC}, d->gen_ngroups, g.kr, g.ke, g.kr, 0ull, 0ull, d->row4, rs,
                                       GenOutShared<IndexT>{out}, nullptr, reverse);
    }
}

// Warps per CTA with ws_bytes of scratch each beside `fixed` bytes of tables: two CTAs share an SM's 227 KB.
inline int gen_cells_warps(int ws_bytes, size_t fixed)
{
    const long long room = 227ll * 1024 / 2 - 1024 - (long long)fixed;
    return (int)std::max(1ll, std::min<long long>(kGenMaxWarps, room / ws_bytes));
}

// Rows of up to 32 words (gen_plan's fits) in MODE over the plan's planes [kbeg, kend).  again: not the first such
// launch since the scan, which leaves the work counter at zero.
template <typename IndexT, int MODE>
void launch_gen_cells(const Grid& g, const CaseTables* cases, const FeBuffers& b, const CountPlan& cp,
                      const GenPlan& p, long long capV, long long capT, float* points, IndexT* tris, int reverse,
                      cudaStream_t s, bool again = false)
{
    const int nzw = p.kend - p.kbeg;
    if (nzw <= 0) return;
    // Rows side by side: all that fit, halved on grids whose (row group, plane) steps would not fill three quarters
    // of a wave (128^3: 18.2 us with two against 19.7 with eight; 256^3, filled: 34 with four, 39 with two). The row
    // after the group in a slot of its own (three slots of work for a group of twice rpw rows, against two for one row
    // less) only where one or two rows are all that fit: 512^3 126 us against 131, but 256^3 33.7 against 31.3 without
    // it, 150 x 700 x 600 75.5 / 70, 128^3 17.5 / 16.6.
    int rpw = 32 / g.W, per_cta, rows;
    bool extra = gen_extra_slot(rpw);
    long long ngroups, wave;
    for (;; rpw /= 2, extra = false) {
        per_cta = gen_cells_warps(gen_cells_scratch(g.W, rpw, MODE), sizeof(GenCellTables<MODE>));
        wave = 2ll * p.nsm * per_cta;
        rows = gen_group_rows(rpw, extra);
        ngroups = (g.ny + rows - 1) / rows;
        if (rpw <= 3 || 4 * ngroups * nzw >= 3 * wave) break;
    }
    const int ws_bytes = gen_cells_scratch(g.W, rpw, MODE);
    // Columns: three quarters of the planes in runs of 2/7 of a warp's share of the steps, the rest in runs a quarter
    // of that (512^3: 126 us in runs of 4 and 1, 132 all in 2, 142 all in 1; 768^3: 434 in 12 and 3, 445 all in 7).
    GenCols cols;
    cols.big = (int)std::max(1ll, std::min(12ll, 2 * ngroups * nzw / (7 * wave)));
    cols.KC = std::max(1, cols.big / 4);
    while (ngroups * ((nzw + cols.KC - 1) / cols.KC + 1) >= (1ll << 31)) cols.KC *= 2;  // item numbers stay below 2^31
    cols.big = std::max(cols.big, cols.KC);
    cols.nbig = (int)(3ll * nzw / 4 / cols.big);
    const int nkc = cols.nbig + (nzw - cols.nbig * cols.big + cols.KC - 1) / cols.KC;
    const long long nitems = ngroups * nkc;
    // a grid of fewer items than a wave has warps: small CTAs, so that every SM gets some
    const int warps = nitems >= wave ? per_cta : (int)std::min<long long>(per_cta, 4);
    const long long blocks = std::min((nitems + warps - 1) / warps, wave / warps);
    RowStarts rs = row_starts(g, cp, b);
    for (int a = 0; a < 3; ++a) rs.add[a] = p.add[a];
    unsigned int* work = reinterpret_cast<unsigned int*>(b.totals + 7);
    if (again) cudaMemsetAsync(work, 0, sizeof(unsigned int), s);
    const size_t smem = (size_t)warps * ws_bytes;
    auto kern = !extra ? k_gen_cells<IndexT, MODE, 0> : (rpw == 1 ? k_gen_cells<IndexT, MODE, 1> : k_gen_cells<IndexT, MODE, 2>);
    allow_smem(kern, smem);
    launch_after(kern, (unsigned)blocks, 32u * warps, smem, s, b.bits, g, rpw, cols, (int)ngroups, (uint32_t)nitems,
                 p.kbeg, p.kend, p.kemit, p.vbase, p.tbase, ws_bytes, cases, b.row4, rs, b.totals, work, capV, capT,
                 points, tris, b.fe2mc, reverse);
}

}  // namespace iso
