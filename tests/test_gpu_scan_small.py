"""The one-CTA scan of small grids: rows around a warp's run, a CTA's tiles and its 4,096 rows, in the three numberings."""
import numpy as np
import pytest

import oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz", [(2, 2), (31, 4), (32, 4), (129, 2), (63, 65), (64, 64), (4096 // 8, 8), (17, 241)])
@pytest.mark.parametrize("algo", ["fe", "mc", "dup"])
def test_rows(cuda, ny, nz, algo):
    import torch
    import miniisosurface_gb300 as M

    vol = np.random.default_rng(ny * nz).standard_normal((nz, ny, 35)).astype(np.float32)
    a = {"fe": M.FLYING_EDGES, "mc": M.MARCHING_CUBES, "dup": M.MC_DUPFREE}[algo]
    d = torch.from_numpy(vol).cuda().reshape(-1)
    m = M.extract_device(d, (35, ny, nz), 0.4, a)
    ref = {"fe": oracle_lib.fe, "mc": oracle_lib.mc, "dup": oracle_lib.mc_dupfree}[algo](vol, 0.4)
    assert (m.n_points, m.n_tris) == (ref[0].shape[0], ref[2].shape[0])
    assert np.array_equal(m.tris[: m.n_tris].cpu().numpy().astype(np.uint64), ref[2])
    assert np.array_equal(m.points[: m.n_points].cpu().numpy().view(np.uint32), ref[0].view(np.uint32))
    assert M.count_device(d, (35, ny, nz), 0.4, a) == (m.n_points, m.n_tris)
