"""The output-size network's sums over several sets in one tile, and its gradients over partial tiles and clusters."""
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import mlp_oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 513, 5000])
def test_gradient_sizes(cuda, n):
    """Within 1e-4 of the largest component of the float64 gradient (sums of n terms in float32, fused)."""
    import torch
    from miniisosurface_gb300 import predictor as P

    rng = np.random.default_rng(n)
    lo = rng.uniform(-1, 0.5, n)
    st = np.concatenate([lo[:, None], (lo + rng.uniform(0.1, 1, n))[:, None], rng.dirichlet(np.ones(32), n)], 1)
    st = st.astype(np.float32)
    iso = (st[:, 0] + (st[:, 1] - st[:, 0]) * rng.uniform(0.1, 0.9, n)).astype(np.float32)
    target = rng.uniform(0, 2, n).astype(np.float32)
    params = P.init_params(3)
    d = [torch.from_numpy(a).cuda() for a in (params, st, iso, target)]
    grads, loss = P.mlp_gradient(*d)
    wloss, want = mlp_oracle.loss_and_gradient(params, mlp_oracle.inputs(st, iso), target)
    assert abs(float(loss) - wloss) <= 1e-5 * wloss
    assert np.abs(grads.cpu().numpy() - want).max() <= 1e-4 * np.abs(want).max()


def test_predict_many_small_sets(cuda):
    """Sets of one block (64 in a tile), of none, and of several tiles, against the forward pass summed in float64."""
    import torch
    from miniisosurface_gb300 import predictor as P

    rng = np.random.default_rng(9)
    net = P.Predictor.load()
    sizes = [1] * 70 + [0, 200, 3, 0, 65] + [2] * 60
    items, want = [], []
    for n in sizes:
        lo = rng.uniform(-1, 0.5, n)
        st = np.concatenate([lo[:, None], (lo + rng.uniform(0.1, 1, n))[:, None], rng.dirichlet(np.ones(32), n)
                             if n else np.zeros((0, 32))], 1).astype(np.float32)
        iso = float(np.float32(rng.uniform(-0.5, 0.5)))
        t = torch.from_numpy(st).cuda()
        y = P.mlp_forward(net.params, t, torch.full((n,), iso, device="cuda")) if n else torch.zeros(0)
        on = (st[:, 0] < np.float32(iso)) & (st[:, 1] >= np.float32(iso))
        want.append(np.maximum(y.double().cpu().numpy()[on], 0).sum() * P.LABEL_SCALE)
        items.append((t, iso))
    got = net.predict(items)
    assert np.allclose(got, want, rtol=1e-5, atol=1e-3)
