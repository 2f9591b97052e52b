"""The row scan over more rows than one CTA takes: every remainder of the rows by the four of a thread, whose starts are
stored together where they lie on a 32-byte boundary."""
import numpy as np
import pytest

import oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz", [(64, 80), (73, 71), (83, 74), (67, 73), (1025, 5)])  # remainders 0, 3, 2, 3, 1
@pytest.mark.parametrize("algo", ["fe", "mc", "dup"])
def test_row_remainders(cuda, ny, nz, algo):
    import torch
    import miniisosurface_gb300 as M

    code = {"fe": M.FLYING_EDGES, "mc": M.MARCHING_CUBES, "dup": M.MC_DUPFREE}[algo]
    vol = M.generate_value_noise((39, ny, nz), 4, 8, seed=ny)
    m = M.extract_device(torch.from_numpy(np.ascontiguousarray(vol)).cuda().reshape(-1), (39, ny, nz), 0.1, code)
    tris = m.tris[: m.n_tris].cpu().numpy().astype(np.uint64)
    ref = oracle_lib.fe(vol, 0.1) if algo == "fe" else oracle_lib.mc(vol, 0.1)
    assert m.n_points == ref[0].shape[0] and tris.shape == ref[2].shape
    if algo != "dup":
        assert np.array_equal(tris, ref[2])
    else:  # the same triangles over vertices in another order
        pts = m.points[: m.n_points].cpu().numpy()
        assert np.array_equal(np.sort(pts[tris.reshape(-1).astype(np.int64)].view(np.uint32), axis=0),
                              np.sort(ref[0][ref[2].reshape(-1).astype(np.int64)].view(np.uint32), axis=0))
