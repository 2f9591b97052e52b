// Helpers of pass 4 (gen_cells.cuh, vertices.cuh), and the generate kernel of
// the duplicate-free Marching Cubes order (included by gen_warps_mc.cu): one
// grid row per warp, rows of up to 32 words.
//
// One wave of CTAs of 8 warps; every warp takes (grid row j, run of KC planes)
// work items from a counter and marches along z on its own (the only CTA
// barrier stages the case tables).  The count pass's bit rows say where the
// surface is.
//
// Per step a warp handles grid row (j, k) with one 32-bit word of the bit
// mask per lane (the bit words and row starts of the next step load while
// this one runs): the 8 cut masks of the cell row, their popc prefixes (warp
// scans) and with them, per word, the place of each mask's first cut edge in the
// order, in shared memory (mb, db), with the row words (rwt); then the active
// cells of the cell row, 32 at a time: each cell lane finds its cell by a
// shuffle binary search over the lanes' counts and computes its cube case, the
// cells' triangles are written one per lane, and the vertices the cells own, one
// per lane: their record (put_mc_record), which k_vertices (vertices.cuh) turns
// into the vertex afterwards.
#pragma once
#include <cmath>
#include <type_traits>

#include "iso_device.cuh"
#include "iso_kernels.h"

namespace iso {

constexpr int kGenRows = 8;       // grid rows per CTA, one per warp
constexpr int kGenCtasPerSm = 3;  // resident CTAs per SM the kernel is built for
constexpr int kGenCells = 32;  // cells per batch
constexpr int kGenOwned = 12 * kGenCells;  // MC vertices owned by a batch, at most
enum GenMode { kGenFE = 0, kGenMC = 1, kGenTri = 2, kGenMCT = 3 };  // gen_cells.cuh

// Per-warp scratch in shared memory:
//   mb[8][W]   {cut mask, -} per mask (xA xB xC xD yA yC zA zB) and word
//   rwt[W][8]  the word's row words (a ash bsh b c csh dsh d: corners 0..7)
//   cell[32]   the batch's active cells: i | cube case << 16
//   list[...]  the batch's triangles, cell | triangle << 5 (u8), then its owned
//              vertices, cell | cube edge << 5 (u16)
//   db[8][W]   the global-edge-index order id of each mask's first cut edge
__host__ __device__ inline size_t gen_warp_scratch_bytes(int W)
{
    return ((size_t)8 * W * 8 + (size_t)8 * W * 4 + kGenCells * 4 + (size_t)kGenOwned * 2 + (size_t)8 * W * 8 + 15) &
           ~(size_t)15;
}

// Divisors of the gradient: the reference divides by the spacing (one-sided
// differences at the faces) or by twice the spacing.  When every spacing is
// a power of two, dividing equals multiplying by the exact reciprocal: both
// round the same real number.
struct GradScale {
    float sp[3], inv1[3], inv2[3];
    int exact;
};

inline GradScale make_grad_scale(const Grid& g)
{
    GradScale s;
    s.exact = 1;
    for (int a = 0; a < 3; ++a) {
        const float sp = g.sp[a];
        int e = 0;
        const float m = std::frexp(sp, &e);  // sp = m * 2^e, m in [0.5, 1)
        const bool pow2 = sp > 0.f && m == 0.5f && e >= -124 && e <= 126;
        if (!pow2) s.exact = 0;
        s.sp[a] = sp;
        s.inv1[a] = pow2 ? std::ldexp(1.0f, 1 - e) : 0.f;  // 1 / sp
        s.inv2[a] = pow2 ? std::ldexp(1.0f, -e) : 0.f;     // 1 / (2 sp)
    }
    return s;
}

// grad_component() of iso_device.cuh along axis a (negated central
// difference, one-sided at the faces).
__device__ __forceinline__ float grad_axis(float prev, float here, float next, int p, int n, int a,
                                           const GradScale& gs)
{
    const bool lo = p == 0, hi = p == n - 1;
    const float num = lo ? fsub(here, next) : (hi ? fsub(prev, here) : fsub(prev, next));
    const bool one = lo || hi;
    if (gs.exact) {
        const float r1 = a == 0 ? gs.inv1[0] : (a == 1 ? gs.inv1[1] : gs.inv1[2]);
        const float r2 = a == 0 ? gs.inv2[0] : (a == 1 ? gs.inv2[1] : gs.inv2[2]);
        return fmul(num, one ? r1 : r2);
    }
    const float sp = a == 0 ? gs.sp[0] : (a == 1 ? gs.sp[1] : gs.sp[2]);
    return fdiv(num, one ? sp : fmul(2.0f, sp));
}

// Gradient components at one point from its six neighbours (grad_component
// of iso_device.cuh per axis).
__device__ __forceinline__ float3 grad3(float xm, float xp, float ym, float yp, float zm, float zp, float here, int i,
                                        int j, int kk, const Grid& g, const GradScale& gs)
{
    return make_float3(grad_axis(xm, here, xp, i, g.nx, 0, gs), grad_axis(ym, here, yp, j, g.ny, 1, gs),
                       grad_axis(zm, here, zp, kk, g.nz, 2, gs));
}

__device__ __forceinline__ void store_vertex(float* __restrict__ points, float* __restrict__ normals,
                                             unsigned long long id, const float3& p, const float3& n)
{
    points[3 * id + 0] = p.x;
    points[3 * id + 1] = p.y;
    points[3 * id + 2] = p.z;
    normals[3 * id + 0] = n.x;
    normals[3 * id + 1] = n.y;
    normals[3 * id + 2] = n.z;
}

// Marching Cubes vertex record in the first 8 bytes of the vertex's points
// slot: the edge's lower point (i, j, k), its axis and the offset d (bit 0 x,
// 1 y, 2 z) of that point from the owner cell, whose cube places the vertex:
// word 0 = i | axis << 10 | d << 12 | (j & 0x1ffff) << 15, word 1 = j >> 17 |
// k << 10 (i < 1024, j < 2^27, k < 2^22).
__device__ __forceinline__ void put_mc_record(float* points, unsigned long long idx, uint32_t i, uint32_t axis,
                                              uint32_t d, uint32_t j, uint32_t k)
{
    uint32_t* r = reinterpret_cast<uint32_t*>(points) + 3 * idx;
    r[0] = i | (axis << 10) | (d << 12) | ((j & 0x1ffffu) << 15);
    r[1] = (j >> 17) | (k << 10);
}

// Inclusive warp scan.
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane)
{
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += t;
    }
    return v;
}

// Id in the global-edge-index order (x block, y block, z block) of cube edge
// e of the cell at bit `bit` of word w: util::duplicateRemover's order
// (marchingCubes/util/DuplicateRemover.h:38-103).
//   e : 0  1  2  3  4  5  6  7  8  9  10 11
//   mask xA yA xB yA xC yC xD yC zA zA zB zB    (index 0..7 below)
//   +1  .  1  .  .  .  1  .  .  .  1  .  1      (edge at point i+1)
__device__ __forceinline__ unsigned long long dup_edge_id(const uint2* mb, const unsigned long long* db, int W, int e,
                                                          int w, int bit)
{
    const int sel = (int)((0x776653524140ull >> (4 * e)) & 7u);
    const int off = (0xA22 >> e) & 1;
    return db[sel * W + w] + __popc(mb[sel * W + w].x & lowmask(bit + off));
}

template <typename IndexT>
__global__ void __launch_bounds__(kThreads, kGenCtasPerSm) k_gen_warps(
    const uint32_t* __restrict__ bits, Grid g, int KC, int nkc, int ws_bytes, const CaseTables* __restrict__ cases,
    RowStarts rs, const unsigned long long* __restrict__ totals, unsigned int* __restrict__ work, long long capV,
    long long capT, float* __restrict__ points, IndexT* __restrict__ tris, int reverse)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ uint64_t s_tris[256];
    __shared__ uint64_t s_order[256];
    __shared__ uint16_t s_cut[256];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int W = g.W;
    unsigned char* ws = s_raw + (size_t)warp * ws_bytes;
    uint2* mb = reinterpret_cast<uint2*>(ws);
    uint32_t* rwt = reinterpret_cast<uint32_t*>(ws + (size_t)8 * W * 8);
    uint32_t* cell = rwt + 8 * W;
    unsigned char* list = reinterpret_cast<unsigned char*>(cell + kGenCells);
    unsigned long long* db = reinterpret_cast<unsigned long long*>(list + (size_t)kGenOwned * 2);
    for (int c = tid; c < 256; c += kThreads) {
        s_order[c] = cases->order[c];
        s_cut[c] = cases->cut[c];
        s_tris[c] = cases->tris[c];
    }
    __syncthreads();  // the only CTA barrier: from here on every warp runs alone
    if (!mesh_holds(totals, capV, capT)) return;  // caller grows buffers
    const unsigned long long dupY = totals[4];              // all x cuts
    const unsigned long long dupZ = totals[4] + totals[5];  // all x and y cuts

    // work items: grid row j and a run of KC planes, taken from the counter `work`
    // (one wave of CTAs; no warp waits for another, no CTA stays for its slowest warp)
    const uint32_t nitems = (uint32_t)g.ny * (uint32_t)nkc;
    for (;;) {
        uint32_t item = 0u;
        if (lane == 0) item = atomicAdd(work, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= nitems) break;
        const int col = (int)(item / (uint32_t)g.ny);
        const int kc = reverse ? nkc - 1 - col : col;
        const int kb = kc * KC, ke = min(kb + KC, g.nz);
        const int j = (int)(item % (uint32_t)g.ny);
        const bool hasY = j < g.ny - 1;
        const bool in = lane < W, in1 = lane + 1 < W;
        const uint32_t evalid = validmask(lane, g.nx - 1);  // x-edges / cells: i <= nx-2
        const uint32_t pvalid = validmask(lane, g.nx);      // points: i <= nx-1

        // Bit words of rows (j, p) and (j+1, p).
        auto load_words = [&](int p, uint32_t& wa, uint32_t& wb) {
            const bool okp = p < g.nz;
            const long long r = (long long)p * g.ny + j;
            wa = (in && okp) ? __ldg(&bits[r * W + lane]) : 0u;
            wb = (in && okp && hasY) ? __ldg(&bits[(r + 1) * W + lane]) : 0u;
        };
        // Row starts of step p, one per lane: lanes 0..3 the first x cut of rows A = (j,p), B = (j+1,p), C = (j,p+1),
        // D = (j+1,p+1), lane 4 the first triangle of cell row A, lanes 5, 6 the first y cut of rows A, C, lanes 7, 8
        // the first z cut of rows A, B (each block's own numbering).
        auto load_starts = [&](int p) -> unsigned long long {
            const long long rA = (long long)p * g.ny + j;
            const bool hasZp = p + 1 < g.nz;
            int dk = 0, dj = 0, comp = 0;  // row offset dk * ny + dj, component, exists
            bool ok = true;
            if (lane < 4) {
                dk = (lane >> 1) & 1;
                dj = lane & 1;
                ok = (dj == 0 || hasY) && (dk == 0 || hasZp);
            } else if (lane == 4) {
                comp = 1;
            } else if (lane <= 6) {
                comp = 2;
                dk = lane - 5;
                ok = dk == 0 || hasZp;
            } else if (lane <= 8) {
                comp = 3;
                dj = lane - 7;
                ok = dj == 0 || hasY;
            } else {
                ok = false;
            }
            return ok ? rs.get(rA + (long long)dk * g.ny + dj, comp) : 0ull;
        };

        uint32_t wA = 0, wB = 0, wC = 0, wD = 0;
        load_words(kb, wA, wB);
        load_words(kb + 1, wC, wD);
        unsigned long long st = load_starts(kb);

        for (int k = kb; k < ke; ++k) {
            const bool hasZ = k + 1 < g.nz;
            // the next step's words and starts, in flight while this step runs
            uint32_t nC = 0, nD = 0;
            unsigned long long nst = 0;
            if (k + 1 < ke) {
                load_words(k + 2, nC, nD);
                nst = load_starts(k + 1);
            }
            const bool cellrow = hasY && hasZ;
            RowWords rw;
            rw.a = wA;
            rw.b = wB;
            rw.c = hasZ ? wC : 0u;
            rw.d = cellrow ? wD : 0u;
            const uint32_t an = __shfl_down_sync(0xffffffffu, rw.a, 1);
            const uint32_t bn = __shfl_down_sync(0xffffffffu, rw.b, 1);
            const uint32_t cn = __shfl_down_sync(0xffffffffu, rw.c, 1);
            const uint32_t dn = __shfl_down_sync(0xffffffffu, rw.d, 1);
            rw.ash = (rw.a >> 1) | ((in1 ? an : 0u) << 31);
            rw.bsh = (rw.b >> 1) | ((in1 ? bn : 0u) << 31);
            rw.csh = (rw.c >> 1) | ((in1 ? cn : 0u) << 31);
            rw.dsh = (rw.d >> 1) | ((in1 ? dn : 0u) << 31);
            const CutMasks m = cut_masks(rw, evalid, pvalid, hasY, hasZ);
            // popc prefixes, two 16-bit counts per scan
            const uint32_t p0 = __popc(m.xA) | (__popc(m.xB) << 16);
            const uint32_t p1 = __popc(m.xC) | (__popc(m.xD) << 16);
            const uint32_t p2 = __popc(m.yA) | (__popc(m.yC) << 16);
            const uint32_t p3 = __popc(m.zA) | (__popc(m.zB) << 16);
            const uint32_t e0 = warp_incl_scan(p0, lane) - p0, e1 = warp_incl_scan(p1, lane) - p1;
            const uint32_t e2 = warp_incl_scan(p2, lane) - p2, e3 = warp_incl_scan(p3, lane) - p3;
            const unsigned long long ts = __shfl_sync(0xffffffffu, st, 4);
            unsigned long long dxB[8];  // block starts of the 8 masks' rows (x A B C D, y A C, z A B)
#pragma unroll
            for (int q = 0; q < 8; ++q) dxB[q] = __shfl_sync(0xffffffffu, st, q < 4 ? q : q + 1);
            if (in) {
                const uint32_t mk[8] = {m.xA, m.xB, m.xC, m.xD, m.yA, m.yC, m.zA, m.zB};
#pragma unroll
                for (int q = 0; q < 8; ++q) mb[q * W + lane] = make_uint2(mk[q], 0u);
                // ids in the global-edge-index order: x block, y block, z block
                db[0 * W + lane] = dxB[0] + (e0 & 0xffffu);
                db[1 * W + lane] = dxB[1] + (e0 >> 16);
                db[2 * W + lane] = dxB[2] + (e1 & 0xffffu);
                db[3 * W + lane] = dxB[3] + (e1 >> 16);
                db[4 * W + lane] = dupY + dxB[4] + (e2 & 0xffffu);
                db[5 * W + lane] = dupY + dxB[5] + (e2 >> 16);
                db[6 * W + lane] = dupZ + dxB[6] + (e3 & 0xffffu);
                db[7 * W + lane] = dupZ + dxB[7] + (e3 >> 16);
                if (cellrow) {  // corner order of the cube case: bit v = corner v
                    uint4* t = reinterpret_cast<uint4*>(rwt + 8 * lane);
                    t[0] = make_uint4(rw.a, rw.ash, rw.bsh, rw.b);
                    t[1] = make_uint4(rw.c, rw.csh, rw.dsh, rw.d);
                }
            }
            __syncwarp();
            if (cellrow) {
                // ---- active cells of cell row (j, k), 32 at a time
                const uint32_t act = in ? active_cells(rw, evalid) : 0u;
                const uint32_t na = __popc(act);
                const uint32_t ia = warp_incl_scan(na, lane);
                const uint32_t tot = __shfl_sync(0xffffffffu, ia, 31);
                unsigned long long tcur = ts;  // next triangle
                for (uint32_t c0 = 0; c0 < tot; c0 += kGenCells) {
                    // lane L takes active cell c0 + L: the first lane whose inclusive count passes it (a
                    // shuffle binary search over the lanes), then the bit by __fns -- no per-lane loop,
                    // which diverges where the active cells cluster along the surface
                    const uint32_t target = c0 + (uint32_t)lane;
                    int src = 0;
#pragma unroll
                    for (int step = 16; step > 0; step >>= 1) {
                        const uint32_t before = __shfl_sync(0xffffffffu, ia, (src + step - 1) & 31);
                        if (before <= target) src += step;
                    }
                    const uint32_t srcact = __shfl_sync(0xffffffffu, act, src);
                    const uint32_t srcexc = __shfl_sync(0xffffffffu, ia - na, src);
                    const uint32_t nc = min(tot - c0, (uint32_t)kGenCells);
                    const bool live = (uint32_t)lane < nc;
                    uint32_t rec = 0u;
                    if (live) {  // the cell's cube case from its word's row words
                        const uint32_t ci = (uint32_t)(32 * src + (int)__fns(srcact, 0, (int)(target - srcexc) + 1));
                        const uint4* t = reinterpret_cast<const uint4*>(rwt + 8 * (ci >> 5));
                        const uint4 lo4 = t[0], hi4 = t[1];
                        const int b = (int)(ci & 31u);
                        const uint32_t cs = ((lo4.x >> b) & 1u) | (((lo4.y >> b) & 1u) << 1) |
                                            (((lo4.z >> b) & 1u) << 2) | (((lo4.w >> b) & 1u) << 3) |
                                            (((hi4.x >> b) & 1u) << 4) |
                                            (((hi4.y >> b) & 1u) << 5) | (((hi4.z >> b) & 1u) << 6) |
                                            (((hi4.w >> b) & 1u) << 7);
                        rec = ci | (cs << 16);
                        cell[lane] = rec;
                    }
                    const int cs = (int)(rec >> 16);
                    {
                        const uint32_t nt = live ? (uint32_t)iso_case_ntris(s_tris[cs]) : 0u;
                        const uint32_t it = warp_incl_scan(nt, lane);
                        const uint32_t ntb = __shfl_sync(0xffffffffu, it, 31);
                        for (uint32_t q = 0; q < nt; ++q) list[it - nt + q] = (unsigned char)(lane | (q << 5));
                        __syncwarp();
                        for (uint32_t tb = 0; tb < ntb; tb += 32) {
                            const uint32_t t = tb + lane;
                            if (t < ntb) {
                                const uint32_t tr = list[t];
                                const uint32_t cr = cell[tr & 31u];
                                const int q = (int)(tr >> 5);
                                const int ci = (int)(cr & 0xffffu);
                                const uint64_t tl = s_tris[cr >> 16];
                                IndexT* o = tris + 3 * (tcur + t);
#pragma unroll
                                for (int c = 0; c < 3; ++c)
                                    o[c] = (IndexT)dup_edge_id(mb, db, W, iso_case_edge(tl, 3 * q + c), ci >> 5, ci & 31);
                            }
                        }
                        tcur += ntb;
                    }
                    __syncwarp();  // the vertex list below reuses the triangle list
                    {
                        // ---- MC vertices owned by the batch's cells: cell order, then order of
                        // first appearance in the cell's triangle list
                        const int ci = (int)(rec & 0xffffu);
                        const uint32_t own = live ? (mc_owned_edges(ci == 0, j == 0, k == 0) & s_cut[cs]) : 0u;
                        const uint32_t no = __popc(own);
                        const uint32_t io = warp_incl_scan(no, lane);
                        const uint32_t nob = __shfl_sync(0xffffffffu, io, 31);
                        uint16_t* vl = reinterpret_cast<uint16_t*>(list);
                        if (own) {
                            const uint64_t ord = s_order[cs];
                            uint32_t o = io - no;
                            for (int q = 0; q < iso_case_ntris(ord); ++q) {
                                const int ed = iso_case_edge(ord, q);
                                if ((own >> ed) & 1u) vl[o++] = (uint16_t)(lane | (ed << 5));
                            }
                        }
                        __syncwarp();
                        for (uint32_t vb = 0; vb < nob; vb += 32) {
                            const uint32_t v = vb + lane;
                            if (v < nob) {
                                const uint32_t vr = vl[v];
                                const uint32_t cr = cell[vr & 31u];
                                const int e12 = (int)(vr >> 5);
                                const int i = (int)(cr & 0xffffu);
                                // the edge's place in the global-edge-index order
                                const unsigned long long id = dup_edge_id(mb, db, W, e12, i >> 5, i & 31);
                                int dx, dy, dz, axis;
                                cube_edge_geometry(e12, dx, dy, dz, axis);
                                // the record kernel (k_vertices) computes the vertex from its record
                                put_mc_record(points, id, (uint32_t)(i + dx), (uint32_t)axis,
                                              (uint32_t)(dx | (dy << 1) | (dz << 2)), (uint32_t)(j + dy),
                                              (uint32_t)(k + dz));
                            }
                        }
                    }
                    __syncwarp();  // the next batch overwrites the lists
                }
            }
            __syncwarp();  // the next step overwrites mb
            wA = wC;
            wB = wD;
            wC = nC;
            wD = nD;
            st = nst;
        }
    }  // work items
}

// The duplicate-free order over the whole grid.
template <typename IndexT>
void launch_gen_dup(const Grid& g, const CaseTables* cases, const FeBuffers& b, const CountPlan& cp, const GenPlan& p,
                    long long capV, long long capT, float* points, IndexT* tris, int reverse, cudaStream_t s)
{
    // items of KC planes: about eight per warp of one wave, at least 2 planes
    const long long warps = (long long)p.nsm * kGenCtasPerSm * kGenRows;
    long long KC = ((long long)g.ny * g.nz + 8 * warps - 1) / (8 * warps);
    if (KC < 2) KC = 2;
    while ((long long)g.ny * ((g.nz + KC - 1) / KC) >= (1ll << 31)) KC *= 2;  // item numbers stay below 2^31
    if (KC > g.nz) KC = g.nz;
    const int nkc = (int)((g.nz + KC - 1) / KC);
    const long long nitems = (long long)g.ny * nkc;
    const long long blocks = std::min((nitems + kGenRows - 1) / kGenRows, (long long)p.nsm * kGenCtasPerSm);
    unsigned int* work = reinterpret_cast<unsigned int*>(b.totals + 7);
    const int ws_bytes = (int)gen_warp_scratch_bytes(g.W);
    const size_t smem = (size_t)kGenRows * ws_bytes;
    auto kern = k_gen_warps<IndexT>;
    allow_smem(kern, smem);
    kern<<<(unsigned)blocks, kThreads, smem, s>>>(b.bits, g, (int)KC, nkc, ws_bytes, cases, row_starts(g, cp, b),
                                                  b.totals, work, capV, capT, points, tris, reverse);
}

}  // namespace iso
