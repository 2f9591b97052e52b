"""GPU: the scratch of an extraction stays within 60 bytes per grid row and the bits (rows of few points: more than the
volume itself, so that it decides which grids fit the device), and calls of different orders that share it agree with
calls on contexts of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALGOS = ["FLYING_EDGES", "MARCHING_CUBES", "MC_DUPFREE"]


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("dims", [(2, 700, 600), (33, 300, 200), (1000, 40, 30)])
def test_bytes_per_row(cuda, algo, dims):
    import torch
    import miniisosurface_gb300 as M

    ctx = M.Context(0)
    vol = torch.rand(dims[0] * dims[1] * dims[2], device="cuda")
    M.count_device(vol, dims, 0.5, getattr(M, algo), ctx=ctx)
    rows, words = dims[1] * dims[2], (dims[0] + 31) // 32
    segments = -(-rows // 1024)
    need = (60 + 4 * words) * rows + 32 * segments + 8 * 256  # the parts at 256-byte boundaries
    assert ctx.scratch_bytes() <= need + need // 4
    ctx.close()


def test_orders_share_one_scratch(cuda):
    import torch
    import miniisosurface_gb300 as M

    def mesh(ctx, vol, dims, algo):
        m = M.extract_device(vol, dims, 0.5, getattr(M, algo), ctx=ctx)
        return [t.cpu().numpy() for t in (m.points[: m.n_points], m.normals[: m.n_points], m.tris[: m.n_tris])]

    shared = M.Context(0)
    sizes = [(40, 33, 27), (5, 90, 60), (600, 20, 9)]
    vols = {d: torch.from_numpy(M.generate_value_noise(d, 3, 8, seed=2).reshape(-1)).cuda() + 0.5 for d in sizes}
    for _ in range(2):  # growing, then every order over what the others left
        for d in sizes:
            for algo in ALGOS:
                own = M.Context(0)
                for a, b in zip(mesh(shared, vols[d], d, algo), mesh(own, vols[d], d, algo)):
                    assert a.shape == b.shape and np.array_equal(a.view(np.uint8), b.view(np.uint8)), (d, algo)
                own.close()
    shared.close()
