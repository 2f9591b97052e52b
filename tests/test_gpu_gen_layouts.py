"""The generate pass in the layouts that large grids, slabs and the streamed host path select: all rows that fit side by
side (short rows), rows of 11 to 32 words with vertex and triangle offsets, and runs of planes of two lengths there.
And the duplicate-free order, whose four scans nothing else checks past 4,096 rows, vertex by vertex."""
import numpy as np
import pytest

import oracle_lib

pytestmark = pytest.mark.gpu


def mesh_np(m):
    return [t[:n].cpu().numpy() for t, n in ((m.points, m.n_points), (m.normals, m.n_points), (m.tris, m.n_tris))]


def same(got, want, what):
    assert got[0].shape == want[0].shape and got[2].shape == want[2].shape, what
    assert np.array_equal(got[2].astype(np.uint64), want[2].astype(np.uint64)), what
    for a, b in zip(got[:2], want[:2]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), what


# words per row -> points; 32 / words rows side by side, in two slots, the last of which is the row after the group:
# groups of 2 * (32 / words) - 1 rows (halved on grids that leave a quarter of the GPU's warps without a step)
@pytest.mark.parametrize("nx", [20, 50, 120, 180, 210])
@pytest.mark.parametrize("rest", [-1, 0, 1])
@pytest.mark.parametrize("algo", ["fe", "mc"])
def test_all_rows_side_by_side(cuda, nx, rest, algo):
    import torch
    import miniisosurface_gb300 as M

    side = 32 // ((nx + 31) // 32)
    ny = 20 * (2 * side - 1) + 1 + rest  # 20 groups of cell rows, and one cell row less or more
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 32  # the most that a wave can hold
    nz = 3 * warps // (4 * 20) + 2
    vol = M.generate_value_noise((nx, ny, nz), 3, 16, seed=nx + rest)
    code, ref = {"fe": (M.FLYING_EDGES, oracle_lib.fe), "mc": (M.MARCHING_CUBES, oracle_lib.mc)}[algo]
    want = ref(vol, 0.25)
    dev = torch.from_numpy(np.ascontiguousarray(vol)).cuda().reshape(-1)
    for ib in (4, 8):
        same(mesh_np(M.extract_device(dev, (nx, ny, nz), 0.25, code, index_bytes=ib)), want, (nx, ny, nz, ib))


@pytest.mark.parametrize("dims", [(352, 23, 17), (511, 14, 19), (513, 9, 21), (700, 11, 13), (1024, 10, 12)])
@pytest.mark.parametrize("algo", ["fe", "mc"])
def test_slabs_of_long_rows(cuda, dims, algo):
    import torch
    import miniisosurface_gb300 as M
    from miniisosurface_gb300 import slabs

    code, ref = {"fe": (M.FLYING_EDGES, oracle_lib.fe), "mc": (M.MARCHING_CUBES, oracle_lib.mc)}[algo]
    vol = np.random.default_rng(dims[0]).standard_normal(dims[::-1]).astype(np.float32)
    want = ref(vol, 0.3)
    dev = torch.from_numpy(vol).cuda().reshape(-1)
    for n in (1, 3, dims[2]):
        for ib in (4, 8):
            got = mesh_np(slabs.extract_multislab(dev, dims, 0.3, code, n, index_bytes=ib))
            same(got, want, (dims, n, ib))


# planes x groups of rows enough for long runs of planes and short ones after them within a slab
@pytest.mark.parametrize("dims", [(330, 2200, 140), (513, 1200, 140)])
@pytest.mark.parametrize("algo", ["FLYING_EDGES", "MARCHING_CUBES"])
def test_slabs_with_runs_of_two_lengths(cuda, dims, algo):
    import torch
    import miniisosurface_gb300 as M
    from miniisosurface_gb300 import slabs

    nx, ny, nz = dims
    i, j, k = (torch.arange(n, device="cuda", dtype=torch.float32) for n in (nx, ny, nz))
    vol = (torch.sin(0.21 * i)[None, None, :] + torch.sin(0.17 * j)[None, :, None] * torch.cos(0.3 * k)[:, None, None])
    vol = vol.contiguous().reshape(-1)
    whole = M.extract_device(vol, dims, 0.4, getattr(M, algo))
    parts = slabs.extract_multislab(vol, dims, 0.4, getattr(M, algo), 2)
    assert (whole.n_points, whole.n_tris) == (parts.n_points, parts.n_tris) and whole.n_tris > 10 ** 6
    for a, b, n in ((whole.points, parts.points, whole.n_points), (whole.normals, parts.normals, whole.n_points),
                    (whole.tris, parts.tris, whole.n_tris)):
        assert torch.equal(a[:n].view(torch.int32), b[:n].view(torch.int32))


@pytest.mark.parametrize("dims", [(352, 20, 131), (600, 12, 140), (1024, 9, 129)])
@pytest.mark.parametrize("algo", ["fe", "mc"])
def test_streamed_host_of_long_rows(cuda, dims, algo):
    import miniisosurface_gb300 as M

    code, ref = {"fe": (M.FLYING_EDGES, oracle_lib.fe), "mc": (M.MARCHING_CUBES, oracle_lib.mc)}[algo]
    vol = M.generate_value_noise(dims, 3, 8, seed=dims[0])
    want = ref(vol, 0.1)
    for ib in (4, 8):
        m = M.extract(M.Image3D.from_array(vol), 0.1, code, index_bytes=ib)
        same((m.points, m.normals, m.triangles), want, (dims, ib))


@pytest.mark.parametrize("dims", [(39, 64, 80), (39, 73, 71), (39, 83, 74), (39, 67, 73), (39, 1025, 5), (161, 160, 162)])
@pytest.mark.parametrize("index_bytes", [4, 8])
def test_duplicate_free_order_exactly(cuda, dims, index_bytes):
    """Row counts with every remainder by the four rows of a scan thread."""
    import torch
    import miniisosurface_gb300 as M

    vol = M.generate_value_noise(dims, 4, 8, seed=dims[1])
    dev = torch.from_numpy(np.ascontiguousarray(vol)).cuda().reshape(-1)
    got = mesh_np(M.extract_device(dev, dims, 0.1, M.MC_DUPFREE, index_bytes=index_bytes))
    same(got, oracle_lib.mc_dupfree(vol, 0.1), dims)
