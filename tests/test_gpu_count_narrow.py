"""The count pass over 8- and 16-bit samples: every width class and remainder of a row's bytes, one, two and four rows
per lane, against the same samples converted to float32 first and against the oracle; the compare of several samples
at once at the ends of each type."""
import numpy as np
import pytest

import oracle_lib
from test_gpu_typed_narrow import M, extract, same  # noqa: F401

pytestmark = pytest.mark.gpu

TYPES = [np.int8, np.uint8, np.int16, np.uint16]


def corners(dtype, shape, seed):
    """Samples at the type's ends, around its middle and random ones."""
    rng = np.random.default_rng(seed)
    lo, hi = np.iinfo(dtype).min, np.iinfo(dtype).max
    mid = (lo + hi) // 2
    pick = np.array([lo, lo + 1, mid - 1, mid, mid + 1, mid + 2, hi - 1, hi])
    v = pick[rng.integers(0, pick.size, shape)]
    r = rng.integers(lo, hi + 1, shape)
    return np.where(rng.random(shape) < 0.3, r, v).astype(dtype)


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("dims", [(2, 3, 3), (31, 37, 5), (33, 29, 6), (40, 21, 5), (97, 23, 7), (161, 19, 5), (355, 5, 9),
                                  (520, 9, 5), (545, 6, 5), (1021, 3, 4), (1024, 5, 4)])
def test_widths_against_oracle(M, dtype, dims):  # noqa: F811
    nx, ny, nz = dims
    vol = corners(dtype, (nz, ny, nx), nx)
    f = vol.astype(np.float32)
    iso = float(np.iinfo(dtype).max // 2) + 0.5
    same(extract(M, vol, dims, iso, M.FLYING_EDGES, True), oracle_lib.fe(f, iso)[:3], "FE")
    same(extract(M, vol, dims, iso, M.MARCHING_CUBES, True), oracle_lib.mc(f, iso)[:3], "MC")


@pytest.mark.parametrize("dtype", TYPES)
def test_thresholds(M, dtype):  # noqa: F811
    dims = (43, 11, 7)
    vol = corners(dtype, dims[::-1], 5)
    lo, hi = float(np.iinfo(dtype).min), float(np.iinfo(dtype).max)
    mid = float((np.iinfo(dtype).min + np.iinfo(dtype).max) // 2)
    for iso in (lo - 1, lo, lo + 0.5, lo + 1, -1.0, -0.5, 0.0, 0.5, mid, mid + 1, hi - 0.5, hi, hi + 0.5, 70000.0, -70000.0,
                np.inf, -np.inf, np.nan):
        tris = extract(M, vol, dims, iso, M.FLYING_EDGES, True)[2]
        assert np.array_equal(tris, oracle_lib.fe(vol.astype(np.float32), float(np.float32(iso)))[2]), iso


@pytest.mark.parametrize("dtype", [np.int8, np.uint16])
@pytest.mark.parametrize("dims", [(150, 470, 90), (160, 470, 90), (513, 401, 401), (528, 401, 401)])
def test_rows_per_lane(M, dtype, dims):  # noqa: F811
    """Enough rows for two per lane (the first two) and four (the others)."""
    f = M.generate_value_noise(dims, 4, 16, seed=dims[0])
    scale = 0.9 * (np.iinfo(dtype).max - np.iinfo(dtype).min) / 2
    vol = np.clip(np.round(f * scale) + (0 if np.iinfo(dtype).min else scale), np.iinfo(dtype).min,
                  np.iinfo(dtype).max).astype(dtype)
    iso = float(np.median(vol)) + 0.5
    for algo in (M.FLYING_EDGES, M.MARCHING_CUBES):
        same(extract(M, vol, dims, iso, algo, True), extract(M, vol, dims, iso, algo, False), algo)
