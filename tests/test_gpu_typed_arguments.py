"""GPU: iso_extract_device_typed refuses an unknown algorithm whatever the rows: those read as they are (up to 1024
points, any byte length) and those converted first."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [61, 64, 600, 1100])
@pytest.mark.parametrize("algo", [-1, 3, 7])
def test_unknown_algorithm(cuda, nx, algo):
    import torch
    import miniisosurface_gb300 as M
    from miniisosurface_gb300 import _lib, api

    dims = (nx, 5, 4)
    vol = (torch.arange(nx * 20, device="cuda") % 7).to(torch.uint8)
    cap = 16 * nx * 20
    points, normals = (torch.full((cap, 3), -1.0, device="cuda") for _ in range(2))
    tris = torch.full((cap, 3), 7, dtype=torch.int32, device="cuda")
    m = _lib.IsoMesh()
    m.points, m.normals, m.tris = points.data_ptr(), normals.data_ptr(), tris.data_ptr()
    m.index_bytes, m.cap_points, m.cap_tris = 4, cap, cap
    ctx = M.default_context(0)
    st = _lib.load().iso_extract_device_typed(ctx.handle, algo, C.c_void_p(vol.data_ptr()), api._dtype_code(vol.dtype),
                                              C.byref(api.make_grid(dims)), C.c_float(2.5), C.byref(m),
                                              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert st == _lib.ISO_ERR_INVALID_ARG
    assert bool((points == -1).all()) and bool((normals == -1).all()) and bool((tris == 7).all())
