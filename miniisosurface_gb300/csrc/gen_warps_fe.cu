// Flying Edges pass 4 (gen_cells.cuh), its vertices from the records
// (vertices.cuh), and the plan of the generate kernels.
#include "../../include/miniiso.h"
#include "gen_cells.cuh"

namespace iso {

// The generate kernels take rows of up to 32 words (1024 points) whose warps
// number their vertices in 32 bits relative to one row's first one; wider grids
// use the row-wise kernels.
GenPlan gen_plan(const Grid& g, int nsm)
{
    GenPlan p;
    p.nsm = nsm;
    const bool rel32 = 6.0 * g.nx * g.ny < 4294967295.0;  // two planes of vertices
    // vertex records pack i < 2^10, j < 2^27, k < 2^22
    p.fits = g.W <= 32 && rel32 && g.ny < (1 << 27) && g.nz < (1 << 22);
    p.kbeg = g.kr;
    p.kend = g.ke;
    p.kemit = g.kr;
    return p;
}

template <typename IndexT>
void launch_fe_gen_warps(const float* vol, const Grid& g, float iso, const CaseTables* cases, const FeBuffers& b,
                         const CountPlan& cp, const GenPlan& p, long long capV, long long capT, float* points,
                         float* normals, IndexT* tris, int reverse, cudaStream_t s)
{
    launch_gen_cells<IndexT, kGenFE>(g, cases, b, cp, p, capV, capT, points, tris, reverse, s);
}

bool launch_fe_vertices(const float* vol, const Grid& g, float iso, const FeBuffers& b, const GenPlan& p,
                        long long capV, long long capT, float* points, float* normals, cudaStream_t s)
{
    if (p.nsm <= 0) return false;
    launch_vertices_impl<false, 0>(vol, g, iso, b, p.kbeg, p.kend, p.nsm, capV, capT, points, normals, s);
    return true;
}

bool launch_fe_vertices_narrow(const void* vol, int dtype, const Grid& g, float iso, const FeBuffers& b,
                               const GenPlan& p, long long capV, long long capT, float* points, float* normals,
                               cudaStream_t s)
{
    if (p.nsm <= 0) return false;
    switch (dtype) {
        case ISO_INT8:
            launch_vertices_impl<false, 0, int8_t>(static_cast<const int8_t*>(vol), g, iso, b, p.kbeg, p.kend, p.nsm,
                                                   capV, capT, points, normals, s);
            break;
        case ISO_UINT8:
            launch_vertices_impl<false, 0, uint8_t>(static_cast<const uint8_t*>(vol), g, iso, b, p.kbeg, p.kend, p.nsm,
                                                    capV, capT, points, normals, s);
            break;
        case ISO_INT16:
            launch_vertices_impl<false, 0, int16_t>(static_cast<const int16_t*>(vol), g, iso, b, p.kbeg, p.kend, p.nsm,
                                                    capV, capT, points, normals, s);
            break;
        default:
            launch_vertices_impl<false, 0, uint16_t>(static_cast<const uint16_t*>(vol), g, iso, b, p.kbeg, p.kend,
                                                     p.nsm, capV, capT, points, normals, s);
            break;
    }
    return true;
}

// The Flying Edges vertices of a list of requests (batch_kernels.cuh), one launch over the concatenation of
// their slots: slot v belongs to request list[q] for vfirst[q] <= v < vfirst[q + 1].  A CTA takes chunks of
// kVertexChunk consecutive slots (chunk c, c + gridDim.x, ...) and walks the requests a chunk overlaps -- one,
// nearly always -- with the request's parameters in shared memory (every thread sees the same requests, so
// the barriers are uniform); each thread loads its next slot's record before it works on the current one.
constexpr int kVertexChunk = 4 * kThreads;

__global__ void __launch_bounds__(kThreads, vertex_ctas_per_sm(false))
    k_vertices_batch(const BatchReq* __restrict__ reqs, const int* __restrict__ list,
                     const unsigned long long* __restrict__ vfirst, int m)
{
    __shared__ BatchReq s_d;
    constexpr int kReqWords = (int)(sizeof(BatchReq) / 4);
    const unsigned long long n = __ldg(&vfirst[m]);
    for (unsigned long long base = (unsigned long long)blockIdx.x * kVertexChunk; base < n;
         base += (unsigned long long)gridDim.x * kVertexChunk) {
        const unsigned long long end = min(base + kVertexChunk, n);
        int q = 0, hi = m - 1;  // the last q with vfirst[q] <= base
        while (q < hi) {
            const int mid = (q + hi + 1) >> 1;
            if (__ldg(&vfirst[mid]) <= base) q = mid;
            else hi = mid - 1;
        }
        for (; q < m; ++q) {
            const unsigned long long v0 = __ldg(&vfirst[q]);
            if (v0 >= end) break;
            const unsigned long long lo = max(v0, base), v1 = min(__ldg(&vfirst[q + 1]), end);
            if (v1 <= lo) continue;  // no slots of request q in the chunk
            __syncthreads();         // the previous request's reads of s_d are done
            if (threadIdx.x < kReqWords)
                reinterpret_cast<uint32_t*>(&s_d)[threadIdx.x] =
                    __ldg(reinterpret_cast<const uint32_t*>(reqs + __ldg(&list[q])) + threadIdx.x);
            __syncthreads();
            float* points = s_d.points;
            unsigned long long v = lo + threadIdx.x;
            uint2 next = v < v1 ? vertex_record(points, v - v0) : make_uint2(0u, 0u);
            for (; v < v1; v += kThreads) {
                const uint2 r = next;
                if (v + kThreads < v1) next = vertex_record(points, v + kThreads - v0);
                vertex_of_record<false, float>(s_d.vol, s_d.g, s_d.gs, s_d.iso, s_d.g.kr, s_d.g.ke, r, v - v0,
                                               points, s_d.normals);
            }
        }
    }
}

int gen_batch_ws_bytes(int W) { return gen_cells_scratch(W, 32 / W, kGenFE); }

int gen_batch_rows(int W) { return gen_group_rows(32 / W, false); }

void launch_gen_batch(int index_bytes, const BatchReq* reqs, const int* list, const unsigned* first, int m,
                      unsigned nitems, const CaseTables* cases, unsigned* work, int ws_bytes, int reverse, int nsm,
                      cudaStream_t s)
{
    const int warps = std::min(kGenBatchWarps, gen_cells_warps(ws_bytes, sizeof(GenCellTables<kGenFE>) + 16 * kGenBatchWarps));
    const long long blocks = std::min(((long long)nitems + warps - 1) / warps, 2ll * nsm);
    if (blocks < 1) return;
    const size_t smem = (size_t)warps * ws_bytes;
    if (index_bytes == 4) {
        allow_smem(k_gen_cells_batch<uint32_t>, smem);
        k_gen_cells_batch<uint32_t><<<(unsigned)blocks, 32 * warps, smem, s>>>(reqs, list, first, m, cases, work,
                                                                               ws_bytes, reverse);
    } else {
        allow_smem(k_gen_cells_batch<uint64_t>, smem);
        k_gen_cells_batch<uint64_t><<<(unsigned)blocks, 32 * warps, smem, s>>>(reqs, list, first, m, cases, work,
                                                                               ws_bytes, reverse);
    }
}

void launch_vertices_batch(const BatchReq* reqs, const int* list, const unsigned long long* vfirst, int m, int nsm,
                           cudaStream_t s)
{
    k_vertices_batch<<<(unsigned)(nsm * vertex_ctas_per_sm(false)), kThreads, 0, s>>>(reqs, list, vfirst, m);
}

template void launch_fe_gen_warps<uint32_t>(const float*, const Grid&, float, const CaseTables*, const FeBuffers&,
                                            const CountPlan&, const GenPlan&, long long, long long, float*, float*,
                                            uint32_t*, int, cudaStream_t);
template void launch_fe_gen_warps<uint64_t>(const float*, const Grid&, float, const CaseTables*, const FeBuffers&,
                                            const CountPlan&, const GenPlan&, long long, long long, float*, float*,
                                            uint64_t*, int, cudaStream_t);

}  // namespace iso

ISO_WAIT_STATS_ACCESSOR(iso_dbg_gen_waits)
