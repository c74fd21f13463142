"""The k-point stencil kernel at the edges of its dispatch (tiles of two rows, of one row where ny is odd,
tiles smaller than the stencil's radius, spare lanes of the last warp, more k-points than one launch's
arguments hold) against the any-shape kernel, which the other k-point tests hold to the
reference; and the Taylor-4 step on rows that its two-point updates cannot take.

Tolerance: the two kernels add the same ~50 terms per point in different orders: FP64 1e-13, FP32 1e-5
of the state's norm (50 terms of 2^-53 / 2^-24 of sums a few times the result)."""
import numpy as np
import pytest

import oracle as O
from qumasun_b200.cell import build_cell, initial_states

pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a - b).norm(dim=-1) / b.norm(dim=-1)).max().item()


@pytest.mark.parametrize("f64", [True, False], ids=["f64", "f32"])
@pytest.mark.parametrize("order", [2, 6, 8])
@pytest.mark.parametrize("grid", [(16, 15, 12), (20, 14, 9), (40, 8, 8), (24, 62, 16), (36, 40, 33)])
def test_stencil_matches_plain_kernel(cuda_ctx, grid, order, f64):
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(grid=grid, nonlocal_on=False)
    kv = np.array([[0.11, -0.23, 0.31], [0.0, 0.2, 0.0]])
    X = torch.from_numpy(initial_states(10, 2 * cell.N, seed=3).reshape(2, 5, 2 * cell.N)).cuda()
    X = X.to(torch.float64 if f64 else torch.float32)
    H = Hamiltonian(cuda_ctx, cell, fd_order=order)
    got = H.apply_zk(kv, X)
    H.set_stencil_kernel(True)
    ref = H.apply_zk(kv, X)
    H.close()
    assert rel(got.double(), ref.double()) < (1e-13 if f64 else 1e-5)


def test_more_kpoints_than_one_launch_of_coefficients(cuda_ctx):
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(grid=(16, 12, 10))
    nk = 67
    kv = np.random.default_rng(1).uniform(-0.3, 0.3, (nk, 3))
    X = torch.from_numpy(initial_states(nk, 2 * cell.N, seed=5).reshape(nk, 1, 2 * cell.N)).cuda()
    H = Hamiltonian(cuda_ctx, cell)
    many = H.apply_zk(kv, X)
    for k in (0, 31, 32, 63, 64, 66):
        H.set_kvector(kv[k])
        assert torch.equal(H.apply_z(X[k]), many[k])
    H.close()


@pytest.mark.parametrize("grid", [(13, 11, 9), (16, 12, 10)], ids=["odd", "unaligned"])
def test_taylor_step_with_scalar_updates(cuda_ctx, grid):
    import ctypes as C
    import torch
    from qumasun_b200 import Hamiltonian
    from qumasun_b200.engine import lib
    cell = build_cell(grid=grid)
    ns, n2, dt = 3, 2 * cell.N, 0.02
    g = (0.1, -0.2, 0.05)
    X = initial_states(ns, n2, seed=7)
    x = X.copy()  # four terms of exp(-i dt H) x, each from the oracle's H
    w = X.copy()
    for n in range(1, 5):
        hw = O.hamiltonian_kpoint_apply(cell, g, w)
        w = np.concatenate([hw[:, cell.N:], -hw[:, :cell.N]], axis=1) * (dt / n)
        x = x + w
    H = Hamiltonian(cuda_ctx, cell, kvec=g)
    buf = torch.zeros(ns * (n2 + 1) + 1, dtype=torch.float64, device="cuda")
    view = buf[1:].view(ns, n2 + 1)[:, :n2]
    view.copy_(torch.from_numpy(X))
    torch.cuda.synchronize()
    assert lib().qg_td_taylor4_z(H.h, ns, C.c_double(dt), C.c_void_p(view.data_ptr()), n2 + 1) == 0
    cuda_ctx.synchronize()
    H.close()
    # the oracle's powers of H and these lose a few bits per power: the 1e-12 of the other step test
    assert rel(view.cpu(), torch.from_numpy(x)) < 1e-12


@pytest.mark.parametrize("many", [False, True], ids=["one-k", "many-k"])
def test_new_kvectors_inside_a_graph_capture(cuda_ctx, many):
    """An application at k-vectors the operator has not seen is made of launches alone, so that a stream
    capture takes it (the scratch is there after a first call of the same size)."""
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(grid=(16, 12, 10))
    nk = 130 if many else 1  # more than one launch holds as arguments
    kv = np.random.default_rng(2).uniform(-0.3, 0.3, (3, nk, 3))
    X = torch.from_numpy(initial_states(2 * nk, 2 * cell.N, seed=9).reshape(nk, 2, 2 * cell.N)).cuda()
    H = Hamiltonian(cuda_ctx, cell)

    def apply(k, out=None):
        if many:
            return H.apply_zk(kv[k], X, out)
        H.set_kvector(kv[k][0])
        return H.apply_z(X[0], None if out is None else out[0])

    out = torch.empty_like(X)
    apply(0, out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        apply(1, out)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    cuda_ctx.use_torch_stream()
    apply(2)  # other phases in the operator's table
    assert torch.equal(out.reshape(apply(1).shape) if many else out[0], apply(1))
    H.close()
