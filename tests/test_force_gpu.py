"""Nonlocal energies and forces against the CPU oracle where the gradient kernel's tiles, the
vector loads and the state chunks end: rows that are no multiple of the tile, odd rows (the
general gradient kernel), strided and 8-byte aligned states, occupied states that are not
neighbours, no occupied state. Tolerance 1e-10 of the largest force or energy, as in the other
force tests (inner products of a gradient and of a state cancel about four digits)."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from qumasun_b200.cell import build_cell, initial_states

pytestmark = pytest.mark.gpu
CELLS = {
    "tiles": dict(grid=(16, 16, 16)),
    "ragged": dict(reps=(1, 1, 2), grid=(22, 18, 34), displacement=0.1, seed=3),
    "rows-of-4": dict(grid=(20, 12, 10), displacement=0.05, seed=5),
    "odd": dict(grid=(17, 13, 15), displacement=0.05, seed=4),
    "wrap": dict(grid=(12, 12, 12), a0=4.4),
}


@pytest.mark.parametrize("ns", [1, 9, 21])
@pytest.mark.parametrize("name", sorted(CELLS))
def test_force_matches_oracle(cuda_ctx, name, ns):
    import torch
    from qumasun_b200 import Hamiltonian
    from qumasun_b200.engine import lib
    cell = build_cell(**CELLS[name])
    X = initial_states(ns, cell.N, seed=ns)
    occ = np.where(np.arange(ns) % 3 == 1, 0.0, 2.0 - 0.05 * np.arange(ns))
    fr, er, evr = O.nonlocal_force(cell, X, occ, impl="port")
    H = Hamiltonian(cuda_ctx, cell)
    Xd = torch.from_numpy(X).cuda()
    f, e, ev = H.nonlocal_force(Xd, occ)
    tf, te = 1e-10 * np.abs(fr).max(), 1e-10 * np.abs(er).max()
    assert np.abs(f - fr).max() < tf and np.abs(e - er).max() < te and abs(ev - evr) < 1e-10 * abs(evr)
    # strided rows that start on 8 bytes
    buf = torch.full((ns * (cell.N + 1) + 1,), float("nan"), dtype=torch.float64, device="cuda")
    buf[1:].view(ns, cell.N + 1)[:, :cell.N].copy_(Xd)
    torch.cuda.synchronize()
    f2, e2 = np.zeros(fr.size), np.zeros(ns)
    dp = C.POINTER(C.c_double)
    assert lib().qg_nonlocal_force_d(H.h, ns, C.c_void_p(buf.data_ptr() + 8), cell.N + 1, occ.ctypes.data_as(dp),
                                     f2.ctypes.data_as(dp), e2.ctypes.data_as(dp), None) == 0
    assert np.abs(f2.reshape(fr.shape) - fr).max() < tf and np.abs(e2 - er).max() < te
    # energies without an occupied state
    f0, e0, ev0 = H.nonlocal_force(Xd, np.zeros(ns))
    assert np.abs(f0).max() == 0.0 and np.abs(e0 - er).max() < te and ev0 == 0.0
    H.close()


@pytest.mark.parametrize("grid", [(130, 56, 8), (130, 100, 8), (146, 40, 9), (128, 40, 8), (144, 24, 10)])
def test_force_on_rows_cut_into_tiles(cuda_ctx, grid):
    """Rows the gradient kernel cuts into tiles of 16 or 24 columns: the last tile 2 columns wide (130 and
    146: the tile before it reads across the row's end too), full ones (128, 144)."""
    import torch
    from qumasun_b200 import Hamiltonian
    cell = build_cell(grid=grid, displacement=0.05, seed=6)
    X = initial_states(5, cell.N, seed=1)
    occ = np.array([2.0, 1.5, 0.0, 1.0, 0.25])
    fr, er, evr = O.nonlocal_force(cell, X, occ, impl="port")
    H = Hamiltonian(cuda_ctx, cell)
    f, e, ev = H.nonlocal_force(torch.from_numpy(X).cuda(), occ)
    H.close()
    assert np.abs(f - fr).max() < 1e-10 * np.abs(fr).max() and np.abs(e - er).max() < 1e-10 * np.abs(er).max()
    assert abs(ev - evr) < 1e-10 * abs(evr)


def test_force_reports_a_wait_that_ran_out(cuda_ctx):
    """With the test hook on, the gradient kernel's producer issues nothing and its consumers give up after
    about a second: the call returns QG_ERR_TIMEOUT and leaves forces and energies alone."""
    import torch
    from qumasun_b200 import Hamiltonian
    from qumasun_b200.engine import lib
    cell = build_cell(grid=(16, 16, 16))
    X = initial_states(3, cell.N, seed=2)
    occ = np.array([2.0, 1.0, 0.5])
    H = Hamiltonian(cuda_ctx, cell)
    Xd = torch.from_numpy(X).cuda()
    good = H.nonlocal_force(Xd, occ)
    f, e, ev = np.full(3 * cell.n_atoms, 7.0), np.full(3, 8.0), C.c_double()
    dp = C.POINTER(C.c_double)

    def call():
        return lib().qg_nonlocal_force_d(H.h, 3, C.c_void_p(Xd.data_ptr()), cell.N, occ.ctypes.data_as(dp),
                                         f.ctypes.data_as(dp), e.ctypes.data_as(dp), C.byref(ev))

    assert lib().qg_hamiltonian_test_stall(H.h, 1) == 0
    assert call() == -5  # QG_ERR_TIMEOUT
    assert (f == 7.0).all() and (e == 8.0).all()
    assert lib().qg_hamiltonian_test_stall(H.h, 0) == 0
    assert call() == 0
    assert np.abs(f - 7.0 - good[0].reshape(-1)).max() < 1e-14 * 8.0 + 1e-13 * np.abs(good[0]).max()
    assert np.array_equal(e, good[1]) and ev.value == good[2]
    assert cuda_ctx.take_device_status() == 0
    H.close()
