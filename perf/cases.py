"""Timed cases of the engine, each one call (or one step's calls) of its public Python API.

Two families of sizes run through them: the synthetic diamond cells of
``qumasun_b200.cell`` (8 to 216 atoms, 40 points per 8-atom cell edge, FD order 8), which the
tests and the benchmark use, and uneven cells of other point counts. A case's operator is
built once per geometry and kept, as a program does between the applications of one SCF
step; the states it works on come from the seed. ``exact`` is the same quantity from plain
torch in 64 bits, from the projector tables and the potential the operator was given.
"""
import math
from collections import OrderedDict

import numpy as np
import torch

from qumasun_b200 import Context, Hamiltonian
from qumasun_b200 import cell as qcell
from qumasun_b200.engine import LearnedPreconditioner, Poisson, density

DEV = "cuda"
F64 = torch.float64
VSCALE = 4.0

# ----------------------------------------------------------------------------- cases


def _hpsi(reps, grid, ns, order=8, dtype="f64", **more):
    return dict(kind="hpsi", rx=reps[0], ry=reps[1], rz=reps[2], nx=grid[0], ny=grid[1], nz=grid[2], ns=ns,
                order=order, dtype=dtype, **more)


def _cubic(kind, r, ns, **more):
    return dict(kind=kind, rx=r, ry=r, rz=r, nx=40 * r, ny=40 * r, nz=40 * r, ns=ns, order=8, **more)


def listed():
    return [
        # one H application of a small solve: 8 atoms, 16 states -- launches and latency
        dict(_hpsi((1, 1, 1), (40, 40, 40), 16), name="hpsi_d8_16"),
        # the batched H application that the benchmark reports
        dict(_hpsi((2, 2, 2), (80, 80, 80), 256), name="hpsi_d64_256"),
        # the same in single precision
        dict(_hpsi((2, 2, 2), (80, 80, 80), 256, dtype="f32"), name="hpsi_d64_256_f32"),
        # an uneven cell with odd point counts (a spacing chosen for the lattice, not for a
        # power of two), the 36 states of 16 atoms with their guard band
        dict(_hpsi((2, 1, 1), (75, 45, 39), 36), name="hpsi_odd_36"),
        # the H application inside the 216-atom solve: 480 states and a guard band of 48
        dict(_hpsi((3, 3, 3), (120, 120, 120), 528), name="hpsi_d216_528"),
        # Bloch states of a 4x4x4 k-point mesh, all k-points in one call, complex64
        dict(_cubic("kpoint", 1, 16, nk=64, dtype="f32"), name="kpoint_d8_64x16_f32"),
        # one step of time propagation (four complex128 H applications)
        dict(_cubic("td", 2, 64), name="td_d64_64"),
        # the density and potential update that closes an SCF step
        dict(_cubic("scf", 2, 256), name="scf_d64_256"),
        # nonlocal energies and forces after the SCF loop
        dict(_cubic("force", 2, 256), name="force_d64_256"),
        # the first iterations of an eigensolve from random states, 2 states per atom + 1/8,
        # and the density of its states, as the SCF loop goes on (each state's own sign or
        # phase is free, so the states themselves are not a result that two solvers share)
        dict(_cubic("lobpcg", 2, 144, iters=4), name="lobpcg_d64_144"),
        # the same over 8 k-points at once
        dict(_cubic("lobpcg_k", 1, 16, nk=8, iters=4), name="lobpcg_k_d8_8x16"),
        # one training batch of the learned preconditioner: forward and backward
        dict(_cubic("learned", 1, 32), name="learned_grad_d8_32"),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _cell_size(rng, most):
    reps = [rng.choice((1, 1, 2, 2, 3)) for _ in range(3)]
    while reps[0] * reps[1] * reps[2] > most:
        k = reps.index(max(reps))
        reps[k] -= 1
    return reps


def draw(rng):
    kind = rng.choice(("hpsi", "hpsi", "hpsi", "hpsi", "kpoint", "kpoint", "td", "scf", "force", "lobpcg",
                       "lobpcg_k", "learned"))
    most = dict(hpsi=27, kpoint=8, td=8, scf=27, force=8, lobpcg=4, lobpcg_k=2, learned=2)[kind]
    reps = _cell_size(rng, most)
    # even point counts in most programs (FFT grids), any count in some
    per = [rng.randint(28, 44) for _ in range(3)]
    grid = [p * r for p, r in zip(per, reps)]
    if rng.random() < 0.6:
        grid = [g + g % 2 for g in grid]
    if kind == "learned":
        grid = [8 * ((g + 7) // 8) if rng.random() < 0.7 else g for g in grid]
    N = grid[0] * grid[1] * grid[2]
    room = 528 * 120 ** 3  # state values of the largest listed case
    order = rng.choice((8, 8, 8, 6, 4, 2))
    c = dict(kind=kind, rx=reps[0], ry=reps[1], rz=reps[2], nx=grid[0], ny=grid[1], nz=grid[2])
    if kind == "hpsi":
        return dict(c, ns=_log(rng, 1, min(528, room // N)), order=order, dtype=rng.choice(("f64", "f64", "f32")))
    if kind == "kpoint":
        nk = _log(rng, 1, 64)
        ns = _log(rng, 1, min(64, max(2, 64 * 16 * 64000 // (nk * N))))
        return dict(c, nk=nk, ns=ns, order=6 if order == 4 else order, dtype=rng.choice(("f64", "f64", "f32")))
    if kind == "td":
        return dict(c, ns=_log(rng, 1, 64), order=6 if order == 4 else order)
    if kind == "scf":
        return dict(c, ns=_log(rng, 4, min(256, room // N)), order=8)
    if kind == "force":
        return dict(c, ns=_log(rng, 4, 256), order=8)
    if kind == "lobpcg":
        return dict(c, ns=_log(rng, 8, 72), order=8, iters=rng.randint(3, 4))
    if kind == "lobpcg_k":
        return dict(c, nk=_log(rng, 1, 8), ns=_log(rng, 4, 18), order=8, iters=rng.randint(3, 4))
    return dict(c, ns=_log(rng, 2, 32), order=8)


# ----------------------------------------------------------------------------- inputs


def _geometry(case):
    return (case["rx"], case["ry"], case["rz"], case["nx"], case["ny"], case["nz"], case["order"])


def _cell(reps, grid, order):
    """A diamond cell with displaced atoms (sigma = 0.05 bohr) and its analytic potential."""
    cell = qcell.build_cell(reps=reps, grid=grid, fd_order=order, displacement=0.05, seed=7, potential_on=False)
    # sum over atoms of a separable Gaussian at the minimum image
    arms = []
    for d, (n, h) in enumerate(((cell.nx, cell.hx), (cell.ny, cell.hy), (cell.nz, cell.hz))):
        x = h * torch.arange(n, dtype=F64, device=DEV)[None, :] - torch.tensor(cell.positions[:, d:d + 1], device=DEV)
        x = x - n * h * torch.round(x / (n * h))
        arms.append(torch.exp(-x * x / (2.0 * qcell.V_SIGMA ** 2)))
    V = qcell.V_DEPTH * torch.einsum("az,ay,ax->zyx", arms[2], arms[1], arms[0])
    cell.V = V.reshape(-1).cpu().numpy()
    return cell


_kept = OrderedDict()  # the operators of the last two geometries: a program keeps its own


def _operator(case):
    key = _geometry(case)
    if key not in _kept:
        while len(_kept) > 1:
            _, old = _kept.popitem(last=False)
            if "poisson" in old:
                old["poisson"].close()
            old["ctx"].close()
        ctx = Context(torch.cuda.current_device())
        ctx.use_torch_stream()
        cell = _cell(key[:3], key[3:6], key[6])
        _kept[key] = dict(ctx=ctx, cell=cell, H=Hamiltonian(ctx, cell))
    _kept.move_to_end(key)
    return _kept[key]


def _k_vectors(cell, nk):
    """The first nk points of a Monkhorst-Pack mesh with at least nk points."""
    m = max(1, math.ceil(round(nk ** (1.0 / 3.0), 9)))
    u = (2.0 * np.arange(1, m + 1) - m - 1) / (2.0 * m)
    L = (cell.nx * cell.hx, cell.ny * cell.hy, cell.nz * cell.hz)
    pts = [(a, b, c) for c in u for b in u for a in u][:nk]
    return np.array([[2.0 * math.pi * f / ll for f, ll in zip(p, L)] for p in pts])


def _random(shape, gen, dtype=F64):
    return torch.rand(shape, generator=gen, device=DEV, dtype=dtype) - 0.5


def _smooth(cell, rows, gen):
    """Smooth normalised states: low-pass filtered noise, sum psi^2 dV = 1 per row."""
    out = torch.empty((rows, cell.N), dtype=F64, device=DEV)
    k2 = 0.0
    for d, (n, h) in enumerate(((cell.nz, cell.hz), (cell.ny, cell.hy), (cell.nx, cell.hx))):
        f = (torch.fft.rfftfreq if d == 2 else torch.fft.fftfreq)(n, device=DEV, dtype=F64) * (2.0 * math.pi / h)
        k2 = k2 + (f * f).reshape([-1 if e == d else 1 for e in range(3)])
    low = 1.0 / (1.0 + 0.25 * k2) ** 2
    grid = (cell.nz, cell.ny, cell.nx)
    for r0 in range(0, rows, 16):
        w = _random((min(16, rows - r0),) + grid, gen)
        w = torch.fft.irfftn(torch.fft.rfftn(w, dim=(1, 2, 3)) * low, s=grid, dim=(1, 2, 3)).reshape(-1, cell.N)
        out[r0:r0 + w.shape[0]] = w / (w.square().sum(1, keepdim=True) * cell.dV).sqrt()
    return out


def _occupations(ns):
    """Two electrons in the lower half of the states, a Fermi tail across the middle."""
    s = np.arange(ns)
    occ = 2.0 / (np.exp(np.minimum((s - (ns // 2 - 0.5)) / 1.5, 80.0)) + 1.0)
    occ[occ < 1.0e-3] = 0.0
    return occ


def prepare(case, seed):
    op = _operator(case)
    cell, kind = op["cell"], case["kind"]
    ns, N = case["ns"], cell.N
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    state = dict(op, case=case)
    if kind == "hpsi":
        state["X"] = _random((ns, N), gen, F64 if case["dtype"] == "f64" else torch.float32)
    elif kind == "kpoint":
        state["k"] = _k_vectors(cell, case["nk"])
        state["X"] = _random((case["nk"], ns, 2 * N), gen, F64 if case["dtype"] == "f64" else torch.float32)
    elif kind == "td":
        state["X"] = _smooth(cell, 2 * ns, gen).reshape(ns, 2 * N)
        state["dt"] = 0.002
    elif kind == "scf":
        state["X"] = _smooth(cell, ns, gen)
        state["occ"] = _occupations(ns)
        state["vext"] = torch.from_numpy(cell.V).to(DEV)
        if "poisson" not in op:
            op["poisson"] = Poisson(op["ctx"], (cell.nx, cell.ny, cell.nz), (cell.hx, cell.hy, cell.hz))
        state["poisson"] = op["poisson"]
    elif kind == "force":
        state["X"] = _smooth(cell, ns, gen)
        state["occ"] = _occupations(ns)
    elif kind == "lobpcg":
        state["X"] = _random((ns, N), gen)
    elif kind == "lobpcg_k":
        state["k"] = _k_vectors(cell, case["nk"])
        state["X"] = _random((case["nk"], ns, 2 * N), gen)
    else:
        state["nn"] = LearnedPreconditioner(op["ctx"])
        w = []
        for ci, co in zip((2, 16, 16, 16), (16, 16, 16, 1)):
            w.append(torch.randn(co * ci * 27, generator=gen, device=DEV) * math.sqrt(2.0 / (ci * 27)))
            w.append(0.05 * torch.randn(co, generator=gen, device=DEV))
        state["params"] = torch.cat(w).cpu().numpy()
        state["nn"].set_params(state["params"])
        state["R"] = 1.0e-3 * _smooth(cell, ns, gen)
        state["Y"] = 0.1 * state["R"] + 1.0e-4 * _smooth(cell, ns, gen)
        state["V"] = torch.from_numpy(cell.V).to(DEV)
    torch.cuda.synchronize()  # inputs are complete before a call on the operator's stream
    return state


# ----------------------------------------------------------------------------- one pass


def run(state):
    case, H = state["case"], state["H"]
    kind = case["kind"]
    if kind == "hpsi":
        return H.apply(state["X"])
    if kind == "kpoint":
        return H.apply_zk(state["k"], state["X"])
    if kind == "td":
        return H.td_taylor4(state["X"], state["dt"])
    if kind == "scf":
        rho = density(state["ctx"], state["X"], state["occ"])
        return rho, state["poisson"].potential(rho, state["vext"])
    if kind == "force":
        return state["H"].nonlocal_force(state["X"], state["occ"])
    if kind == "lobpcg":
        X = state["X"].clone()  # the solver overwrites its starting states
        res = H.lobpcg_device(X, max_iter=case["iters"], precond=1)
        return res["ev"], density(state["ctx"], X, _occupations(case["ns"]))
    if kind == "lobpcg_k":
        X = state["X"].clone()
        res = H.lobpcg_zk(state["k"], X, max_iter=case["iters"], precond=1)
        occ = np.tile(_occupations(case["ns"]), case["nk"])
        return res["ev"], density(state["ctx"], X.reshape(occ.size, -1), occ, complex_states=True)
    nn, cell = state["nn"], state["cell"]
    return nn.gradient((cell.nx, cell.ny, cell.nz), state["R"], state["V"], VSCALE, state["Y"])


# ----------------------------------------------------------------------------- work


def work(case):
    N = case["nx"] * case["ny"] * case["nz"]
    ns, kind = case["ns"], case["kind"]
    atoms = 8 * case["rx"] * case["ry"] * case["rz"]
    length = qcell.A0
    pts = 4.0 / 3.0 * math.pi * qcell.PROJ_CUTOFF ** 3 * N / (length ** 3 * case["rx"] * case["ry"] * case["rz"])
    points = atoms * pts  # sphere points of all projectors
    radius = {2: 1, 4: 3, 6: 3, 8: 4}[case["order"]]
    stencil = 3 * radius * 3 + 3     # per point: per neighbour pair an add and a multiply-add
    nonlocal_ = 2 * 2 * 4 * points   # four channels, gathered and scattered
    tables = (4 * points + 2 * N)
    if kind == "hpsi":
        b = 8 if case["dtype"] == "f64" else 4
        return dict(bytes=b * (2.0 * ns * N + tables), flops=ns * (stencil * N + nonlocal_))
    if kind == "kpoint":
        b = 8 if case["dtype"] == "f64" else 4
        n = case["nk"] * ns
        return dict(bytes=b * (4.0 * n * N + tables), flops=n * (4.0 * stencil * N + 4 * nonlocal_))
    if kind == "td":  # each application waits for the last one's whole result
        return dict(bytes=8.0 * (4 * 4 * ns * N + tables), flops=4 * ns * (4.0 * stencil * N + 4 * nonlocal_))
    if kind == "scf":
        occupied = int((_occupations(ns) > 0).sum())
        return dict(bytes=8.0 * N * (occupied + 3), flops=3.0 * N * occupied + 10.0 * N * math.log2(N))
    if kind == "force":
        return dict(bytes=8.0 * (ns * N + tables), flops=ns * (3 * 12 * N + 4 * nonlocal_))
    if kind == "lobpcg":
        it = case["iters"]  # H of r, x and p; Gram and rotation products; the blocks read and written
        return dict(bytes=8.0 * it * ns * N * 14, flops=it * (3.0 * ns * (stencil * N + nonlocal_) + 18.0 * N * ns * ns))
    if kind == "lobpcg_k":
        it, n = case["iters"], case["nk"] * ns
        return dict(bytes=16.0 * it * n * N * 14,
                    flops=it * (3.0 * n * (4.0 * stencil * N + 4 * nonlocal_) + 72.0 * N * n * ns))
    macs = 27.0 * (2 * 16 + 16 * 16 + 16 * 16 + 16)
    return dict(bytes=8.0 * (2 * ns * N + N), flops=3 * 2 * macs * ns * N)


def tolerance(case):
    kind = case["kind"]
    # measured against exact() and with the projector sums in another order: 2e-16 in 64
    # bits, 7e-8 in 32; a few times that, and more where many terms cancel
    if kind in ("hpsi", "kpoint"):
        return {"rel": 1.0e-14, "max": 1.0e-12} if case["dtype"] == "f64" else {"rel": 1.0e-6, "max": 2.0e-5}
    if kind == "td":
        return {"rel": 1.0e-14, "max": 1.0e-12}
    if kind == "scf":
        return {"rel": 1.0e-13, "max": 1.0e-11}
    if kind == "force":
        return {"rel": 1.0e-12, "max": 1.0e-10}
    if kind in ("lobpcg", "lobpcg_k"):
        # each step multiplies a change in the last bits; the upper states move most
        return {"rel": 1.0e-6, "max": 1.0e-4}
    # activations are rounded to bfloat16, so another order of a 32-bit sum flips some of
    # them: 2.6e-6 between the two forward paths
    return {"rel": 5.0e-5, "max": 5.0e-4}


# ----------------------------------------------------------------------------- in 64 bits

LAP = {2: (-2.0, 1.0), 4: tuple(v / 576.0 for v in (-1460.0, 783.0, -54.0, 1.0)),
       6: tuple(v / 90.0 for v in (-245.0, 135.0, -13.5, 1.0)),
       8: tuple(v / 5040.0 for v in (-14350.0, 8064.0, -1008.0, 128.0, -9.0))}
DER = {2: (0.5,), 6: tuple(v / 60.0 for v in (45.0, -9.0, 1.0)), 8: tuple(v / 840.0 for v in (672.0, -168.0, 32.0, -3.0))}


def _projectors(cell):
    """Per atom: grid index, unwrapped coordinates and channel values of its cube's points, and E."""
    out = []
    for a in range(cell.n_atoms):
        vals, E = [], []
        begin, size, _ = cell.cubes[a][0]  # the cubes of one atom are the same for every l here
        for k, l in enumerate(cell.proj_l):
            w = cell.cubes[a][k][2]
            for m in range(2 * l + 1):
                vals.append(w * (qcell.Y00 if l == 0 else cell.ylm_tabs[a][l * l + m]))
                E.append(cell.proj_E[k])
        u = [np.arange(size[d]) + begin[d] for d in range(3)]
        z, y, x = np.meshgrid(u[2], u[1], u[0], indexing="ij")
        g = x % cell.nx + cell.nx * (y % cell.ny + cell.ny * (z % cell.nz))
        vals = np.stack(vals)
        keep = (vals != 0.0).any(0)
        xyz = np.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)])[:, keep]
        out.append((torch.from_numpy(g.reshape(-1)[keep]).to(DEV), torch.from_numpy(xyz).to(DEV).to(F64),
                    torch.from_numpy(vals[:, keep]).to(DEV), torch.tensor(E, dtype=F64, device=DEV)))
    return out


def _axis(cell, d):
    return 3 - d, (cell.hx, cell.hy, cell.hz)[d]  # the tensor's axis of (s, z, y, x), and the spacing


def _derivative(cell, U, order, d):
    ax, h = _axis(cell, d)
    out = torch.zeros_like(U)
    for j, c in enumerate(DER[order], 1):
        out += (c / h) * (torch.roll(U, -j, ax) - torch.roll(U, j, ax))
    return out


def _h(cell, X, order, proj, g=None):
    """H of (s, N) states: real, or complex with the Bloch vector g."""
    U = X.reshape(-1, cell.nz, cell.ny, cell.nx)
    out = U * torch.from_numpy(cell.V).to(DEV).reshape(U.shape[1:])
    for d in range(3):
        ax, h = _axis(cell, d)
        for j, c in enumerate(LAP[order]):
            out += (-0.5 * c / (h * h)) * (U if j == 0 else torch.roll(U, j, ax) + torch.roll(U, -j, ax))
        if g is not None:
            out += -1j * float(g[d]) * _derivative(cell, U, order, d)
            out += 0.5 * float(g[d]) ** 2 * U
    out = out.reshape(-1, cell.N)
    for idx, xyz, vals, E in proj:
        P = vals
        if g is not None:
            th = sum(float(g[d]) * h * xyz[d] for d, h in enumerate((cell.hx, cell.hy, cell.hz)))
            P = vals * torch.polar(torch.ones_like(th), th)
        c = (X[:, idx] @ P.T) * (E * cell.dV)
        out.index_add_(1, idx, c @ (P.conj() if g is not None else P))
    return out


def _to_complex(X, N):
    return torch.complex(X[..., :N], X[..., N:])


def _from_complex(Z):
    return torch.cat((Z.real, Z.imag), -1)


def _orthonormal_rr(S, HS, dV, n):
    """The n lowest Ritz pairs of the rows of S (with HS = H S)."""
    B = S.conj() @ S.T * dV
    A = S.conj() @ HS.T * dV
    d = B.diagonal().real.rsqrt().to(B.dtype)
    L = torch.linalg.cholesky(B * d[:, None] * d[None, :])
    A = A * d[:, None] * d[None, :]
    A = torch.linalg.solve_triangular(L, A, upper=False)
    A = torch.linalg.solve_triangular(L, A.mH, upper=False).mH
    w, Z = torch.linalg.eigh(0.5 * (A + A.mH))
    return torch.linalg.solve_triangular(L.mH, Z[:, :n], upper=True) * d[:, None]


def _lobpcg(cell, X, order, proj, iters, g=None):
    """Rayleigh quotients and states after `iters` steps of the block iteration, kinetic preconditioner."""
    n = X.shape[0]

    def normal(A):
        return A / (A.abs().square().sum(1, keepdim=True) * cell.dV).sqrt()

    sym = 0.0
    for d, (m, h) in enumerate(((cell.nx, cell.hx), (cell.ny, cell.hy), (cell.nz, cell.hz))):
        th = 2.0 * math.pi * torch.arange(m, dtype=F64, device=DEV) / m
        s = sum((c if j == 0 else 2.0 * c * torch.cos(j * th)) for j, c in enumerate(LAP[order])) / (h * h)
        sym = sym + s.reshape([-1 if e == 2 - d else 1 for e in range(3)])
    T = 1.0 / (1.0 - 0.5 * sym)
    shape = (cell.nz, cell.ny, cell.nx)

    def kinetic(R):
        W = torch.fft.ifftn(torch.fft.fftn(R.reshape((-1,) + shape), dim=(1, 2, 3)) * T, dim=(1, 2, 3))
        return (W if g is not None else W.real).reshape(R.shape)

    def ham(A):
        return torch.cat([_h(cell, A[s:s + 16], order, proj, g) for s in range(0, A.shape[0], 16)])

    X, P = normal(X), None
    HX = ham(X)
    ev = (X.conj() * HX).sum(1).real * cell.dV
    for _ in range(iters):
        W = normal(kinetic(HX - ev[:, None] * X))
        S = torch.cat((X, W) if P is None else (X, W, P))
        Z = _orthonormal_rr(S, ham(S), cell.dV, n)
        P = normal(Z[n:].T @ S[n:])
        X = normal(Z.T @ S)
        HX = ham(X)
        ev = (X.conj() * HX).sum(1).real * cell.dV
    return ev, X


def exact(case, seed):
    state = prepare(case, seed)
    cell, kind, order = state["cell"], case["kind"], case["order"]
    N, ns = cell.N, case["ns"]
    if kind == "learned":
        return _exact_learned(cell, state)
    proj = _projectors(cell)
    X = state["X"]
    if kind == "hpsi":
        out = torch.empty((ns, N), dtype=F64, device=DEV)
        for s in range(0, ns, 16):
            out[s:s + 16] = _h(cell, X[s:s + 16].double(), order, proj)
        return out
    if kind == "kpoint":
        out = torch.empty(X.shape, dtype=F64, device=DEV)
        for k, g in enumerate(state["k"]):
            for s in range(0, ns, 8):
                out[k, s:s + 8] = _from_complex(_h(cell, _to_complex(X[k, s:s + 8].double(), N), order, proj, g))
        return out
    if kind == "td":
        out = torch.empty_like(X)
        for s in range(0, ns, 8):
            term = psi = _to_complex(X[s:s + 8], N)
            for j in range(1, 5):
                term = _h(cell, term, order, proj, (0.0, 0.0, 0.0)) * (-1j * state["dt"] / j)
                psi = psi + term
            out[s:s + 8] = _from_complex(psi)
        return out
    if kind == "scf":
        return _exact_scf(cell, state)
    if kind == "force":
        return _exact_force(cell, state, proj)
    occ, ev, rho = torch.from_numpy(_occupations(ns)).to(DEV), [], 0.0
    for k, g in enumerate(state["k"] if kind == "lobpcg_k" else (None,)):
        Z = X if g is None else _to_complex(X[k], N)
        e, Z = _lobpcg(cell, Z, order, proj, case["iters"], g)
        ev.append(e)
        rho = rho + (occ[:, None] * Z.abs().square()).sum(0)
    ev = torch.cat(ev).cpu().numpy()
    return ev.reshape(case["nk"], ns) if kind == "lobpcg_k" else ev, rho


def _exact_scf(cell, state):
    occ = torch.from_numpy(state["occ"]).to(DEV)
    rho = torch.zeros(cell.N, dtype=F64, device=DEV)
    for s in range(0, occ.numel(), 16):
        rho += (occ[s:s + 16, None] * state["X"][s:s + 16].square()).sum(0)
    grid = (cell.nz, cell.ny, cell.nx)
    k2 = 0.0
    for d, (n, h) in enumerate(((cell.nz, cell.hz), (cell.ny, cell.hy), (cell.nx, cell.hx))):
        j = torch.arange(n, device=DEV, dtype=F64)
        f = torch.where(j < n // 2, j, j - n) * (2.0 * math.pi / (n * h))
        k2 = k2 + (f * f).reshape([-1 if e == d else 1 for e in range(3)])
    kern = torch.where(k2 > 0, 4.0 * math.pi / torch.where(k2 > 0, k2, 1.0), 0.0)
    vh = torch.fft.ifftn(torch.fft.fftn(rho.reshape(grid)) * kern).real.reshape(-1)
    # Perdew-Zunger 1981, unpolarised
    some = rho >= 1.0e-8
    rs = (3.0 / (4.0 * math.pi * torch.where(some, rho, 1.0))) ** (1.0 / 3.0)
    vx = -(9.0 * math.pi / 4.0) ** (1.0 / 3.0) / math.pi / rs  # 4/3 of the exchange energy per electron
    b1, b2, gamma = 1.0529, 0.3334, -0.1423
    sq = rs.sqrt()
    low = gamma * (1.0 + 7.0 / 6.0 * b1 * sq + 4.0 / 3.0 * b2 * rs) / (1.0 + b1 * sq + b2 * rs) ** 2
    A, B, C, D = 0.0311, -0.0480, 0.0020, -0.0116
    high = A * rs.log() + (B - A / 3.0) + 2.0 / 3.0 * C * rs * rs.log() + (2.0 * D - C) / 3.0 * rs
    vc = torch.where(rs >= 1.0, low, high)
    return rho, state["vext"] + vh + torch.where(some, vx + vc, 0.0)


def _exact_force(cell, state, proj):
    occ = torch.from_numpy(state["occ"]).to(DEV)
    ns = occ.numel()
    e = torch.zeros(ns, dtype=F64, device=DEV)
    f = torch.zeros((cell.n_atoms, 3), dtype=F64, device=DEV)
    for s in range(0, ns, 16):
        U = state["X"][s:s + 16]
        G = [_derivative(cell, U.reshape(-1, cell.nz, cell.ny, cell.nx), 8, d).reshape(U.shape) for d in range(3)]
        o = occ[s:s + 16]
        for a, (idx, _, vals, E) in enumerate(proj):
            c = U[:, idx] @ vals.T * cell.dV
            e[s:s + 16] += (E * c * c).sum(1)
            for d in range(3):
                f[a, d] += (-2.0 * o[:, None] * E * c * (G[d][:, idx] @ vals.T * cell.dV)).sum()
    return f.cpu().numpy(), e.cpu().numpy(), float((occ * e).sum())


def _exact_learned(cell, state):
    grid = (cell.nz, cell.ny, cell.nx)
    params = torch.from_numpy(state["params"]).to(DEV).double().requires_grad_(True)
    layers, off = [], 0
    for ci, co in zip((2, 16, 16, 16), (16, 16, 16, 1)):
        w = params[off:off + co * ci * 27].reshape(co, ci, 3, 3, 3)
        layers.append((w, params[off + co * ci * 27:off + co * ci * 27 + co]))
        off += co * ci * 27 + co
    R, Y = state["R"], state["Y"]
    rms = R.square().mean(1, keepdim=True).sqrt()
    target = Y / rms
    norm = target.square().sum()
    loss, grad = 0.0, torch.zeros_like(params)
    for s in range(0, R.shape[0], 2):
        r = R[s:s + 2] / rms[s:s + 2]
        x = torch.stack((r.reshape((-1,) + grid), (state["V"] / VSCALE).reshape((1,) + grid).expand((r.shape[0],) + grid)), 1)
        for i, (w, b) in enumerate(layers):
            x = torch.nn.functional.conv3d(torch.nn.functional.pad(x, (1,) * 6, mode="circular"), w, b)
            x = x.relu() if i < 3 else x
        part = (x.reshape(r.shape) - target[s:s + 2]).square().sum() / norm
        grad += torch.autograd.grad(part, params, retain_graph=True)[0]
        loss += float(part)
    return loss, grad.detach().cpu().numpy()
