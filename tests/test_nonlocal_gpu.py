"""Nonlocal projectors through brick tables (cells of more than 16 atoms, every k-point
state) against the CPU oracle, at the edges of the bricks (16 x 8 x 4 points: rows that are no
multiple of 8 or 16, odd rows, layers that end inside a brick, spheres that wrap), of the state
tiles (8 states per warp, 64 per block) and of the row strides and alignments that the
vector loads have to leave to the scalar ones.

Tolerance: a projector sum has at most a few thousand terms in FP64, added pairwise over
bricks: well below 1e-12 of the state's norm, the bound of the other operator tests. The
nonlocal part alone (H x minus the local part, ~1e-3 of the total) is held to 1e-10 of its own size."""
import numpy as np
import pytest

import oracle as O
from qumasun_b200.cell import build_cell, initial_states

pytestmark = pytest.mark.gpu
CELLS = {
    "multiple": dict(reps=(1, 1, 3), grid=(16, 16, 48)),
    "ragged": dict(reps=(1, 1, 3), grid=(20, 18, 50), displacement=0.1, seed=3),
    "odd": dict(reps=(3, 1, 1), grid=(45, 17, 15), displacement=0.1, seed=4),
    "wrap": dict(reps=(1, 3, 1), grid=(12, 34, 10), a0=4.4),
}


def rel(a, b):
    return (np.linalg.norm(a - b, axis=-1) / np.linalg.norm(b, axis=-1)).max()


def padded(X, pad, shift):
    """X as a strided view: rows `pad` elements longer, first element `shift` elements in."""
    import torch
    ns, n = X.shape
    buf = torch.full((ns * (n + pad) + shift,), float("nan"), dtype=X.dtype, device="cuda")
    view = buf[shift:].view(ns, n + pad)[:, :n]
    view.copy_(X)
    return buf, view


@pytest.mark.parametrize("ns", [1, 7, 8, 9, 65])
@pytest.mark.parametrize("name", sorted(CELLS))
def test_real_projection_matches_oracle(cuda_ctx, name, ns):
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(**CELLS[name])
    X = initial_states(ns, cell.N, seed=ns)
    H = Hamiltonian(cuda_ctx, cell)
    Xd = torch.from_numpy(X).cuda()
    out = H.apply(Xd)
    ref = O.hamiltonian_apply(cell, X)
    loc = O.hamiltonian_kpoint_local(cell, (0.0, 0.0, 0.0), np.concatenate([X, 0 * X], 1))[:, :cell.N]
    got = out.cpu().numpy()
    assert rel(got, ref) < 1e-12 and rel(got - loc, ref - loc) < 1e-10
    # the atom-by-atom kernel, and a state's bits whatever its batch
    H.set_nonlocal_blocking(0, 0, 1)
    assert rel(H.apply(Xd).cpu().numpy(), ref) < 1e-12
    H.set_nonlocal_blocking(0, 0, 0)
    if ns > 1:
        assert torch.equal(H.apply(Xd[ns - 1:]), out[ns - 1:])
    # rows of an odd length that start on 8 bytes
    for pad, shift in ((1, 1), (2, 0), (0, 1)):
        xb, xv = padded(Xd, pad, shift)
        hb, hv = padded(torch.zeros_like(Xd), pad, shift)
        torch.cuda.synchronize()
        H.apply_device(ns, xv.data_ptr(), hv.data_ptr(), cell.N + pad, cell.N + pad)
        cuda_ctx.synchronize()
        assert rel(hv.cpu().numpy(), got) < 1e-14, (pad, shift)  # another stencil kernel may run
        del xb, hb
    H.close()


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("ns", [1, 5, 33])
@pytest.mark.parametrize("name", sorted(CELLS))
def test_kpoint_projection_and_scatter_match_oracle(cuda_ctx, name, ns, dtype):
    import ctypes as C
    import torch
    from qumasun_b200 import Hamiltonian
    from qumasun_b200.engine import lib
    f64 = dtype == "complex128"
    cell = build_cell(**CELLS[name])
    n2 = 2 * cell.N
    kv = np.array([[0.11, -0.23, 0.31], [0.0, 0.0, 0.0], [-0.3, 0.07, 0.02]])
    X = initial_states(3 * ns, n2, seed=ns).reshape(3, ns, n2)
    Xd = torch.from_numpy(X).cuda().to(torch.float64 if f64 else torch.float32)
    H = Hamiltonian(cuda_ctx, cell)
    many = H.apply_zk(kv, Xd)
    for k in range(3):
        ref = O.hamiltonian_kpoint_apply(cell, tuple(kv[k]), X[k])
        loc = O.hamiltonian_kpoint_local(cell, tuple(kv[k]), X[k])
        got = many[k].double().cpu().numpy()
        # FP32 states carry 2^-24 of rounding per stencil term: the bound of the complex64 tests
        assert rel(got, ref) < (1e-12 if f64 else 2e-6), k
        if f64:
            assert rel(got - loc, ref - loc) < 1e-10, k
    H.set_kvector(kv[2])
    assert torch.equal(H.apply_z(Xd[2]), many[2])
    fn = lib().qg_hamiltonian_apply_z if f64 else lib().qg_hamiltonian_apply_zf
    for pad, shift in ((1, 1), (2, 0), (0, 1)):
        xb, xv = padded(Xd[2], pad, shift)
        hb, hv = padded(torch.zeros_like(Xd[2]), pad, shift)
        torch.cuda.synchronize()
        assert fn(H.h, ns, C.c_void_p(xv.data_ptr()), n2 + pad, C.c_void_p(hv.data_ptr()), n2 + pad) == 0
        cuda_ctx.synchronize()
        assert rel(hv.double().cpu().numpy(), many[2].double().cpu().numpy()) < (1e-14 if f64 else 1e-6), (pad, shift)
        del xb, hb
    H.close()


@pytest.mark.parametrize("f64", [True, False], ids=["f64", "f32"])
@pytest.mark.parametrize("ns", [1, 5, 37])
@pytest.mark.parametrize("kw", [dict(reps=(1, 1, 3), grid=(40, 38, 100), displacement=0.1, seed=3),
                                dict(grid=(54, 54, 54), a0=4.4)], ids=["ragged", "wrap"])
def test_scatter_by_pairs_matches_oracle(cuda_ctx, kw, ns, f64):
    """Grids large enough for the scatter of two points per thread; rows of odd length go point by
    point (the same entries in the same order)."""
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(**kw)
    X = initial_states(ns, cell.N, seed=ns)
    H = Hamiltonian(cuda_ctx, cell)
    Xd = torch.from_numpy(X).cuda().to(torch.float64 if f64 else torch.float32)
    pairs = H.apply(Xd)
    assert rel(pairs.double().cpu().numpy(), O.hamiltonian_apply(cell, X)) < (1e-12 if f64 else 2e-6)
    for sg in (4, 8):
        H.set_nonlocal_blocking(0, sg, 0)
        assert torch.equal(H.apply(Xd), pairs)
    H.set_nonlocal_blocking(0, 0, 0)
    hb, hv = padded(torch.zeros_like(Xd), 1, 1)
    torch.cuda.synchronize()
    H.apply_device(ns, Xd.data_ptr(), hv.data_ptr(), cell.N, cell.N + 1, "f64" if f64 else "f32")
    cuda_ctx.synchronize()
    assert rel(hv.double().cpu().numpy(), pairs.double().cpu().numpy()) < (1e-14 if f64 else 1e-6)
    H.close()


@pytest.mark.parametrize("kw", [dict(grid=(13, 11, 9)), dict(grid=(27, 17, 15), displacement=0.05, seed=1)],
                         ids=["8-atoms-tiny", "8-atoms"])
@pytest.mark.parametrize("f64", [True, False], ids=["f64", "f32"])
def test_odd_grid_split_scatter_matches_oracle(cuda_ctx, kw, f64):
    """Odd rows: stencil and scatter are two kernels."""
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(**kw)
    X = initial_states(9, cell.N, seed=2)
    H = Hamiltonian(cuda_ctx, cell)
    got = H.apply(torch.from_numpy(X).cuda().to(torch.float64 if f64 else torch.float32)).double().cpu().numpy()
    H.close()
    assert rel(got, O.hamiltonian_apply(cell, X)) < (1e-12 if f64 else 2e-6)


@pytest.mark.parametrize("f64", [True, False], ids=["f64", "f32"])
@pytest.mark.parametrize("kw", [dict(grid=(16, 12, 10)), dict(reps=(1, 1, 3), grid=(16, 16, 48)), dict(grid=(54, 54, 104))],
                         ids=["atoms", "bricks", "pairs"])
def test_projectors_without_a_point(cuda_ctx, kw, f64):
    """All projector values zero: no grid point has an entry, the scatter launched beside the stencil has
    nothing to add, and what follows on the stream still follows the stencil."""
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(**kw)
    cell.cubes = [[(b, s, 0.0 * w) for b, s, w in at] for at in cell.cubes]
    bare = build_cell(**kw, nonlocal_on=False)
    X = torch.from_numpy(initial_states(6, cell.N, seed=8)).cuda().to(torch.float64 if f64 else torch.float32)
    H, H0 = Hamiltonian(cuda_ctx, cell), Hamiltonian(cuda_ctx, bare)
    for _ in range(3):
        ref = H0.apply(X)
        out = torch.full_like(X, float("nan"))
        got = H.apply(X, out).clone()  # the next kernel of the stream reads the result
        assert torch.equal(got, ref)
    H.close()
    H0.close()


def used_by(f):
    """Device memory that f takes (kept alive by its result)."""
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    keep = f()
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0], keep


def test_single_precision_apply_takes_no_brick_scratch(cuda_ctx):
    """FP32 states are projected atom by atom: the scratch is their coefficients, FP32, and no partial sums."""
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(reps=(2, 2, 2), grid=(48, 48, 48))
    ns = 512
    H = Hamiltonian(cuda_ctx, cell)
    H.apply(torch.zeros(16, cell.N, dtype=torch.float32, device="cuda"))
    X = torch.zeros(ns, cell.N, dtype=torch.float32, device="cuda")
    out = torch.empty_like(X)
    taken, _ = used_by(lambda: H.apply_device(ns, X.data_ptr(), out.data_ptr(), cell.N, cell.N, "f32"))
    assert taken <= 4 * ns * cell.n_atoms * 4 + (4 << 20)
    H.close()


def test_small_grids_hold_no_tables_of_point_pairs(cuda_ctx):
    """Grids below the size of the two-points scatter: the tables that it alone reads are not built."""
    from qumasun_b200 import Hamiltonian
    cell = build_cell(reps=(2, 2, 2), grid=(52, 52, 54))  # 146,016 points
    taken, H = used_by(lambda: Hamiltonian(cuda_ctx, cell))
    H.close()
    assert cell.N < 2 * 2 * 148 * 256  # two points per thread, two blocks of 256 per SM
    # sphere points: nonzero in any channel of an atom
    points = sum(int((cell.cubes[a][0][2].reshape(-1) != 0.0).sum()) for a in range(cell.n_atoms))
    # per sphere point: two orders of 4 channels in FP64 and FP32 and their indices; the bricks' blocks,
    # up to twice as many FP64 values; the potential and per-point rows
    assert taken <= points * (2 * 4 * 12 + 2 * 4 + 2 * 4 * 8) + cell.N * 20 + (12 << 20)


def test_autotuner_leaves_a_projection_block_it_does_not_use(cuda_ctx):
    """FP64 states of more than 16 atoms are projected brick by brick: no block size to choose, and the
    operator keeps its own for the kernels that have one (FP32 states, the no-allocation entry point)."""
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(reps=(1, 1, 3), grid=(16, 16, 48))
    X = torch.from_numpy(initial_states(16, cell.N, seed=6)).cuda()
    H = Hamiltonian(cuda_ctx, cell)
    for sb in (0, 1):  # 1: never a candidate
        H.set_nonlocal_blocking(sb, 0, 0)
        assert H.autotune(X)["project_states"] == sb
    H.set_nonlocal_blocking(0, 0, 1)  # atom by atom: the size is used, so it is chosen
    assert H.autotune(X)["project_states"] in (2, 4, 8, 16)
    H.set_nonlocal_blocking(0, 0, 0)
    assert H.autotune(X.float())["project_states"] in (2, 4, 8, 16)
    H.close()


@pytest.mark.parametrize("reps,same", [((1, 1, 1), True), ((2, 1, 1), True), ((3, 1, 1), False)])
def test_noalloc_entry_sums_atom_by_atom(cuda_ctx, reps, same):
    """The no-allocation entry point: the regular one's bits up to 16 atoms, above them another order of the
    projections' sums (a few thousand terms: the bound of the other operator tests), whatever the batch."""
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(reps=reps, grid=(20 * reps[0], 18, 16), displacement=0.05, seed=2)
    X = torch.from_numpy(initial_states(9, cell.N, seed=4)).cuda()
    H = Hamiltonian(cuda_ctx, cell)
    ref, out = H.apply(X), H.apply_noalloc(X, torch.empty_like(X))
    assert torch.equal(out, ref) if same else ((out - ref).norm(dim=1) < 1e-12 * ref.norm(dim=1)).all()
    H.set_nonlocal_blocking(0, 0, 1 if not same else 0)  # the regular entry's atom-by-atom form
    assert torch.equal(H.apply(X), out)
    assert torch.equal(H.apply_noalloc(X[8:], torch.empty_like(X[8:])), out[8:])
    H.close()
