"""The vertex pass on either side of the size up to which it is brought in beside the generate pass: several calls
after one another into the same buffers, bit for bit."""
import numpy as np
import pytest

import oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(33, 31, 17), (161, 160, 162), (163, 161, 160)])  # the last two: 2^22 points, -+ 1%
@pytest.mark.parametrize("algo", ["fe", "mc", "dup"])
def test_either_side_of_the_rule(cuda, dims, algo):
    import torch
    import miniisosurface_gb300 as M

    code = {"fe": M.FLYING_EDGES, "mc": M.MARCHING_CUBES, "dup": M.MC_DUPFREE}[algo]
    vol = M.generate_value_noise(dims, 4, 16, seed=dims[0])
    dev = torch.from_numpy(np.ascontiguousarray(vol)).cuda().reshape(-1)
    first = None
    for iso in (0.2, -0.1, 0.2):
        m = M.extract_device(dev, dims, iso, code)
        got = [t[:n].cpu().numpy() for t, n in ((m.points, m.n_points), (m.normals, m.n_points), (m.tris, m.n_tris))]
        if algo != "dup":
            ref = (oracle_lib.fe if algo == "fe" else oracle_lib.mc)(vol, iso)
            assert np.array_equal(got[2].astype(np.uint64), ref[2])
            assert np.array_equal(got[0].view(np.uint32), ref[0].view(np.uint32))
            assert np.array_equal(got[1].view(np.uint32), ref[1].view(np.uint32))
        if first is None:
            first = got
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(first, got))
