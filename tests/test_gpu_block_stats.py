"""Block statistics of blocks cut off at the far faces in every direction, and of one point of overlap."""
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import mlp_oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 2), (17, 17, 17), (18, 17, 2), (17, 33, 18), (33, 2, 17), (16, 40, 35),
                                  (49, 18, 16), (3, 50, 19)])
def test_block_stats(cuda, dims):
    import torch
    from miniisosurface_gb300 import predictor as P

    rng = np.random.default_rng(sum(dims))
    vol = rng.standard_normal(dims[::-1]).astype(np.float32)
    vol[rng.random(vol.shape) < 0.2] = 0.25  # many equal samples: increments of one bin
    got = P.block_stats(torch.from_numpy(vol).cuda().reshape(-1), dims).cpu().numpy()
    want = mlp_oracle.block_stats(vol)
    assert got.shape == want.shape
    assert np.array_equal(got.view(np.uint32), want.astype(np.float32).view(np.uint32))
