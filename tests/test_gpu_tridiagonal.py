"""Eigenvalues and eigenvectors of the tridiagonal solver (multisection, inverse iteration, clusters) through the allocation-free entry point, against LAPACK.

Bounds: eigenvalues to a few n eps |A| (backward error of the reduction), residuals likewise; the
vectors of eigenvalues apart by more than ortol = 1e-7 |T|_1 are orthogonal to eps / 1e-7 with a
factor for the residual's few eps, closer ones are re-orthogonalised.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _matrix(kind, n, rng):
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    H = (G + G.conj().T) / 2
    if kind == "random":
        return H
    if kind in ("tiny", "huge"):   # products of two elements beyond the range of the division by FMAs
        return H * {"tiny": 1e-100, "huge": 1e100}[kind]
    Q, _ = np.linalg.qr(G)
    if kind == "pairs":          # every eigenvalue twice: clusters
        w = np.repeat(np.linspace(-1.0, 2.0, (n + 1) // 2), 2)[:n]
    elif kind == "close":        # gaps across ortol, from 1e-12 to 1e-2
        w = np.cumsum(np.logspace(-12, -2, n))
    elif kind == "graded":       # twelve orders of magnitude
        w = np.logspace(-12, 0, n) * np.where(np.arange(n) % 2, 1.0, -1.0)
    elif kind == "blocks":       # decoupled blocks and a repeated diagonal tail
        H = H.copy()
        a = n // 3
        H[a:, :a] = H[:a, a:] = 0.0
        H[2 * a:, :] = H[:, 2 * a:] = 0.0
        H[np.arange(2 * a, n), np.arange(2 * a, n)] = 7.5
        return H
    elif kind == "zero":
        return np.zeros((n, n), complex)
    return (Q * w) @ Q.conj().T


@pytest.mark.parametrize("kind", ["random", "pairs", "close", "graded", "blocks", "zero"])
@pytest.mark.parametrize("n,iu", [(2, 2), (3, 1), (5, 4), (31, 31), (33, 32), (64, 40), (130, 65), (257, 257), (512, 266)])
def test_tridiagonal_solver(kind, n, iu):
    import torch

    import forge_gb300 as fg
    f = fg.load_library().forge_gpu_zheevr_noalloc
    f.argtypes = [C.c_void_p, C.c_int64, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p]
    f.restype = C.c_int
    H = _matrix(kind, n, np.random.default_rng(1000 + n))
    A = torch.from_numpy(np.ascontiguousarray(H.T)).cuda()    # column-major
    w = torch.empty(iu, dtype=torch.float64, device="cuda")
    Z = torch.empty(iu, n, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    assert f(A.data_ptr(), n, iu, w.data_ptr(), Z.data_ptr(), None) == 0
    w, X = w.cpu().numpy(), Z.cpu().numpy().T
    scale = max(np.linalg.norm(H, 2), np.finfo(float).tiny)
    ref = np.linalg.eigvalsh(H)[:iu]
    assert np.max(np.abs(w - ref)) <= 8 * n * EPS * scale
    assert np.max(np.abs(H @ X - X * w)) <= 16 * n * EPS * scale
    assert np.max(np.abs(X.conj().T @ X - np.eye(iu))) <= 64 * EPS / 1e-7


@pytest.mark.parametrize("kind", ["tiny", "huge"])
@pytest.mark.parametrize("n,iu", [(5, 4), (33, 32), (130, 65)])
def test_tridiagonal_solver_far_scales(kind, n, iu):
    test_tridiagonal_solver(kind, n, iu)
