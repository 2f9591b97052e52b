"""The generate pass over rows of up to 32 words: every count of rows side by side, groups that end inside the grid,
runs of planes that end inside it, both index widths, and Marching Cubes through the shared table."""
import numpy as np
import pytest

import oracle_lib

pytestmark = pytest.mark.gpu


def check(vol, iso, algo, index_bytes, spacing=(1, 1, 1), origin=(0, 0, 0)):
    import torch
    import miniisosurface_gb300 as M

    nz, ny, nx = vol.shape
    a = {"fe": M.FLYING_EDGES, "mc": M.MARCHING_CUBES}[algo]
    m = M.extract_device(torch.from_numpy(vol).cuda().reshape(-1), (nx, ny, nz), iso, a, spacing, origin,
                         index_bytes=index_bytes)
    ref = (oracle_lib.fe if algo == "fe" else oracle_lib.mc)(vol, iso, spacing, origin)
    assert (m.n_points, m.n_tris) == (ref[0].shape[0], ref[2].shape[0])
    assert np.array_equal(m.tris[: m.n_tris].cpu().numpy().astype(np.uint64), ref[2])
    for got, want in ((m.points, ref[0]), (m.normals, ref[1])):
        assert np.array_equal(got[: m.n_points].cpu().numpy().view(np.uint32), want.view(np.uint32))


# widths of 1 to 32 words; ny around multiples of the rows of a group (2 * rows side by side)
@pytest.mark.parametrize("nx,ny,nz", [(17, 65, 3), (33, 33, 4), (65, 21, 5), (97, 17, 6), (129, 13, 9), (161, 11, 7),
                                      (200, 9, 8), (257, 7, 5), (300, 6, 6), (352, 5, 13), (500, 9, 6), (513, 3, 9),
                                      (700, 5, 7), (1000, 4, 5), (1024, 2, 3)])
@pytest.mark.parametrize("algo,index_bytes", [("fe", 4), ("fe", 8), ("mc", 4), ("mc", 8)])
def test_widths(cuda, nx, ny, nz, algo, index_bytes):
    rng = np.random.default_rng(nx)
    check(rng.standard_normal((nz, ny, nx)).astype(np.float32), 0.3, algo, index_bytes)


@pytest.mark.parametrize("dims", [(513, 130, 301), (96, 500, 260)])
def test_runs_of_two_lengths(cuda, dims):
    """Enough steps for the long runs of planes and the short ones after them, nearly every cell active in a layer
    and none elsewhere (whole batches, and steps with no cut edge)."""
    nx, ny, nz = dims
    k = np.arange(nz, dtype=np.float32)[:, None, None]
    i = np.arange(nx, dtype=np.float32)[None, None, :]
    j = np.arange(ny, dtype=np.float32)[None, :, None]
    vol = (np.sin(i * 1.3) * np.cos(j * 0.9 + i) * (np.abs(k - nz // 2) < 20) + 0.01 * (k - nz / 3)).astype(np.float32)
    for algo in ("fe", "mc"):
        check(vol, 0.2, algo, 4, (0.5, 0.25, 2.0), (1.0, -2.0, 0.0))
