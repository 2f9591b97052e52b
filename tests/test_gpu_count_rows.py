"""The count pass over rows of up to 32 words: rows side by side in a warp at every width class, one, two and four
consecutive rows per lane, and the sign compare at its special isovalues and samples."""
import numpy as np
import pytest

import oracle_lib

pytestmark = pytest.mark.gpu


def extract(vol, iso, algo):
    import torch
    import miniisosurface_gb300 as M

    nz, ny, nx = vol.shape
    m = M.extract_device(torch.from_numpy(np.ascontiguousarray(vol)).cuda().reshape(-1), (nx, ny, nz), iso, algo)
    return m.tris[: m.n_tris].cpu().numpy().astype(np.uint64), m.n_points


@pytest.mark.parametrize("dims", [(31, 37, 5), (32, 33, 6), (65, 29, 5), (96, 41, 4), (97, 23, 7), (161, 19, 5),
                                  (192, 13, 6), (289, 9, 5), (352, 7, 4), (355, 5, 9), (545, 6, 5), (1021, 3, 4),
                                  (33, 701, 121), (160, 470, 90), (150, 470, 90), (513, 261, 381)])
@pytest.mark.parametrize("algo", ["fe", "mc"])
def test_widths_and_rows_per_lane(cuda, dims, algo):
    """The last four have enough rows for two rows per lane (three of them) and four (the last)."""
    import miniisosurface_gb300 as M

    vol = M.generate_value_noise(dims, 3, 16, seed=sum(dims))
    ref = oracle_lib.fe(vol, 0.1, nthreads=8) if algo == "fe" else oracle_lib.mc(vol, 0.1)
    tris, nv = extract(vol, 0.1, M.FLYING_EDGES if algo == "fe" else M.MARCHING_CUBES)
    assert nv == ref[0].shape[0]
    assert np.array_equal(tris, ref[2])


@pytest.mark.parametrize("nx", [40, 43])
@pytest.mark.parametrize("iso", [-np.inf, -np.finfo(np.float32).max, -np.finfo(np.float32).tiny, -1e-45, -0.0, 0.0,
                                 1e-45, 0.5, np.finfo(np.float32).max, np.inf, np.nan])
def test_special_values(cuda, nx, iso):
    """Infinities, NaNs of both signs, denormals and zeros of both signs among the samples: the classification is
    the reference's value >= iso."""
    import miniisosurface_gb300 as M

    rng = np.random.default_rng(nx)
    f = np.finfo(np.float32)
    pick = np.array([-np.inf, -f.max, -1.0, -f.tiny, -1e-45, -0.0, 0.0, 1e-45, f.tiny, 0.5, 1.0, f.max, np.inf, np.nan],
                    np.float32)
    vol = pick[rng.integers(0, pick.size, (7, 11, nx))]
    bits = vol.view(np.uint32)
    bits[np.isnan(vol) & (rng.random(vol.shape) < 0.5)] = 0xFFC12345  # negative NaNs with a payload
    ref = oracle_lib.fe(vol, float(np.float32(iso)))
    tris, nv = extract(vol, float(np.float32(iso)), M.FLYING_EDGES)
    assert nv == ref[0].shape[0]
    assert np.array_equal(tris, ref[2])
