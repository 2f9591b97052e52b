"""GPU: a context whose scratch first grows within a stream capture.  Nothing of a capture has run until its graph is
launched, so the device status of the calls after it must not come from memory that the capture was to zero."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

DIMS = (40, 33, 27)


def cudart():
    import torch

    torch.cuda.init()
    for line in open("/proc/self/maps"):
        if "libcudart" in line:
            return C.CDLL(line.split()[-1])
    pytest.skip("no shared libcudart in the process")


class WrittenBlocks:
    """Device blocks of nbytes written full of ones and given back but for two, so that the driver keeps the memory
    they came from and hands it out again."""

    def __init__(self, nbytes, n=24):
        self.rt, blocks = cudart(), []
        for _ in range(n):
            p = C.c_void_p()
            assert self.rt.cudaMalloc(C.byref(p), C.c_size_t(nbytes)) == 0
            assert self.rt.cudaMemset(p, 255, C.c_size_t(nbytes)) == 0
            blocks.append(p)
        assert self.rt.cudaDeviceSynchronize() == 0
        self.kept = [blocks.pop(n // 2), blocks.pop(0)]
        for p in blocks:
            assert self.rt.cudaFree(p) == 0

    def close(self):
        for p in self.kept:
            assert self.rt.cudaFree(p) == 0


def test_scratch_first_allocated_in_a_capture(cuda):
    import torch
    import miniisosurface_gb300 as M
    from miniisosurface_gb300 import _lib, api

    lib = _lib.load()
    vol = torch.from_numpy(M.generate_blobs(DIMS, nblobs=8, seed=7).reshape(-1)).cuda()
    grid = api.make_grid(DIMS)
    points, normals = (torch.zeros((20000, 3), device="cuda") for _ in range(2))
    tris = torch.zeros((40000, 3), dtype=torch.int32, device="cuda")
    m = _lib.IsoMesh()
    m.points, m.normals, m.tris = points.data_ptr(), normals.data_ptr(), tris.data_ptr()
    m.index_bytes, m.cap_points, m.cap_tris = 4, 20000, 40000
    res = torch.zeros(4, dtype=torch.int64).pin_memory()

    def extract(ctx, stream):
        return lib.iso_extract_device_async(ctx.handle, M.FLYING_EDGES, C.c_void_p(vol.data_ptr()), C.byref(grid),
                                            C.c_float(0.5), C.byref(m), C.cast(C.c_void_p(res.data_ptr()),
                                                                               C.POINTER(C.c_int64)),
                                            C.c_void_p(stream))

    first = M.Context(0)
    assert extract(first, torch.cuda.current_stream().cuda_stream) == _lib.ISO_OK
    torch.cuda.synchronize()
    want, nbytes = res.tolist(), first.scratch_bytes()
    assert want[0] > 0 and want[3] == 0
    first.close()

    written = WrittenBlocks(nbytes)
    ctx = M.Context(0)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="relaxed"):
        st = extract(ctx, torch.cuda.current_stream().cuda_stream)
    assert st == _lib.ISO_OK
    # not launched: calls that wait for their counts see their own status
    mesh = M.extract_device(vol, DIMS, 0.5, M.FLYING_EDGES, ctx=ctx)
    assert (mesh.n_points, mesh.n_tris) == tuple(want[:2])
    assert M.count_device(vol, DIMS, 0.5, M.FLYING_EDGES, ctx=ctx) == tuple(want[:2])
    res.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert res.tolist()[:2] == want[:2] and res.tolist()[3] == 0
    ctx.close()
    written.close()


@pytest.mark.parametrize("algo", ["FLYING_EDGES", "MARCHING_CUBES"])
def test_waiting_calls_after_scratch_grows(cuda, algo):
    """Scratch that grew over written memory between two waiting calls."""
    import torch
    import miniisosurface_gb300 as M

    a = getattr(M, algo)
    ctx = M.Context(0)
    for dims in ((20, 9, 8), (90, 60, 50)):
        written = WrittenBlocks(1 << 17)
        vol = torch.from_numpy(M.generate_value_noise(dims, 3, 8, seed=4).reshape(-1)).cuda()
        other = M.Context(0)
        want = M.count_device(vol, dims, 0.0, a, ctx=other)
        mesh = M.extract_device(vol, dims, 0.0, a, ctx=ctx)
        assert (mesh.n_points, mesh.n_tris) == want
        other.close()
        written.close()
    ctx.close()
