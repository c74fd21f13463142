"""Parameter gradient of the learned preconditioner against the CPU oracle on grids that end
inside the tiles of the backward kernels (4 x 8 x 8 points and their halo), smaller than a tile,
and with one state or more tiles than persistent blocks. Tolerance as in the other gradient test:
BF16 activations differ at the 1e-3 level, 2e-2 per layer; a misplaced halo point is of order one."""
import numpy as np
import pytest

import oracle.nn_oracle as NN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,ns", [((8, 8, 8), 1), ((8, 4, 4), 2), ((12, 10, 7), 3), ((9, 11, 13), 2), ((20, 18, 22), 5),
                                     ((24, 24, 24), 13)])
def test_gradient_at_tile_edges(cuda_ctx, grid, ns):
    import torch
    from qumasun_b200 import LearnedPreconditioner
    rng = np.random.default_rng(sum(grid) + ns)
    N = grid[0] * grid[1] * grid[2]
    P = rng.normal(0, 0.15, NN.n_params()).astype(np.float32)
    R, Y = rng.normal(size=(ns, N)), rng.normal(size=(ns, N))
    V = -4.0 * np.exp(-rng.uniform(0, 3, size=N))
    nn = LearnedPreconditioner(cuda_ctx)
    nn.set_params(P)
    args = (grid, torch.from_numpy(R).cuda(), torch.from_numpy(V).cuda(), 4.0, torch.from_numpy(Y).cuda())
    loss, g = nn.gradient(*args)
    rl, rg = NN.loss_and_grad(P, grid, R, V, 4.0, Y)
    assert abs(loss - rl) / rl < 5e-3
    off = 0
    for co, ci in ((16, 2), (16, 16), (16, 16), (1, 16)):
        n = co * ci * 27 + co
        a, b = g[off:off + n], rg[off:off + n]
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 2e-2, off
        off += n
    assert np.array_equal(nn.gradient(*args)[1], g)  # sums in a fixed order
    nn.close()


def test_infinite_layer_gradients_stay_infinite(cuda_ctx):
    """Loss gradients near the top of FP32 that overflow on their way back through the last layer: with
    positive weights, activations and inputs every product is +Inf, so every sum is, and none is NaN."""
    import torch
    from qumasun_b200 import LearnedPreconditioner
    rng = np.random.default_rng(11)
    grid = (8, 8, 4)
    N = grid[0] * grid[1] * grid[2]
    layers, first = [], []
    for ci, co, scale in zip(NN.CIN, NN.COUT, (0.02, 0.005, 0.005, 1e4)):
        first.append(sum(a.size for a in layers))
        layers += [scale * rng.uniform(0.5, 1.0, co * ci * 27), 0.01 * rng.uniform(0.5, 1.0, co)]
    P = np.concatenate(layers).astype(np.float32)
    R, V = rng.uniform(0.5, 1.0, (1, N)), 4.0 * rng.uniform(0.5, 1.0, N)
    _, p, rms = NN.forward(P, grid, R, V, 4.0)
    # t = Y / rms constant, 2 max(p) / (N t^2) = 1e35
    Y = np.full((1, N), rms[0] * np.sqrt(2.0 * p.max() / (N * 1e35)))
    nn = LearnedPreconditioner(cuda_ctx)
    nn.set_params(P)
    loss, g = nn.gradient(grid, torch.from_numpy(R).cuda(), torch.from_numpy(V).cuda(), 4.0, torch.from_numpy(Y).cuda())
    nn.close()
    _, rg = NN.loss_and_grad(P, grid, R, V, 4.0, Y)
    last = first[3]
    assert np.linalg.norm(g[last:].astype(float) - rg[last:]) < 2e-2 * np.linalg.norm(rg[last:])
    assert rg[:last].min() > np.finfo(np.float32).max  # the exact values are beyond FP32
    assert np.isposinf(g[:last]).all()
