"""The batched Hermitian pencil solver at odd sizes and at one row, its pairs' edges, on pencils
with equal eigenvalues and with zero off-diagonals, against LAPACK. Tolerance: the solver stops at an
off-diagonal norm of 1e-13 of the norm; eigenvalues to 1e-11 of the largest, residuals to 1e-10 (the
condition of B, at most 1e3 here, times that)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pencil(k, kind, rng):
    Z = rng.normal(size=(k, k)) + 1j * rng.normal(size=(k, k))
    A = (Z + Z.conj().T) / 2
    if kind == "equal":
        q, _ = np.linalg.qr(Z)
        A = (q * np.where(np.arange(k) % 3 == 0, 2.0, -1.0)) @ q.conj().T
        A = (A + A.conj().T) / 2
    if kind == "diagonal":
        return np.diag(rng.normal(size=k)).astype(complex), np.eye(k, dtype=complex)
    W = rng.normal(size=(k, k)) + 1j * rng.normal(size=(k, k))
    return A, W @ W.conj().T / k + 0.5 * np.eye(k)


@pytest.mark.parametrize("kind", ["full", "equal", "diagonal"])
@pytest.mark.parametrize("k", [1, 2, 3, 5, 31, 33, 55, 56])
def test_hermitian_pairs_and_odd_sizes(cuda_ctx, k, kind):
    import scipy.linalg
    import torch
    from qumasun_b200.engine import hegv_small_batched
    rng = np.random.default_rng(k)
    A, B = pencil(k, kind, rng)
    w, Z, info = hegv_small_batched(cuda_ctx, torch.tensor(A[None]).cuda(), torch.tensor(B[None]).cuda())
    torch.cuda.synchronize()
    assert int(info[0]) == 0
    w, Z = w[0].cpu().numpy(), Z[0].cpu().numpy()
    ref = scipy.linalg.eigh(A, B, eigvals_only=True)
    scale = max(1e-300, np.abs(ref).max())
    assert np.abs(w - ref).max() < 1e-11 * scale
    res = A @ Z - (B @ Z) * w
    assert np.abs(res).max() < 1e-10 * scale * np.abs(B).max() * max(1.0, np.abs(Z).max())


@pytest.mark.parametrize("tiny", [1e-320, 3e-163, 2e-162, 5e-160, 1e-155, 1e-150])
def test_hermitian_pencil_with_tiny_off_diagonals(cuda_ctx, tiny):
    """Off-diagonal elements whose squares are subnormal or zero, next to elements of order one and
    between equal diagonal elements: the eigenvectors stay B-orthonormal."""
    import torch
    from qumasun_b200.engine import hegv_small_batched
    k = 12
    rng = np.random.default_rng(3)
    A = np.diag(np.repeat(np.arange(1.0, 7.0), 2)).astype(complex)
    W = tiny * np.exp(2j * np.pi * rng.uniform(size=(k, k)))
    A += np.triu(W, 1) + np.triu(W, 1).conj().T
    A[0, 5] = 0.3 + 0.4j  # one pair that does turn
    A[5, 0] = A[0, 5].conj()
    w, Z, info = hegv_small_batched(cuda_ctx, torch.tensor(A[None]).cuda(),
                                    torch.eye(k, dtype=torch.complex128)[None].cuda())
    torch.cuda.synchronize()
    assert int(info[0]) == 0
    w, Z = w[0].cpu().numpy(), Z[0].cpu().numpy()
    # a column turns 11 times a sweep, about 2 roundings of 1.1e-16 each, in at most 8 sweeps
    assert np.abs(Z.conj().T @ Z - np.eye(k)).max() < 2e-14
    assert np.abs(w - np.linalg.eigvalsh(A)).max() < 2e-14 * 6 and np.abs(A @ Z - Z * w).max() < 2e-14 * 6
