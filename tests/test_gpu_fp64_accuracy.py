"""How far the plain FP64 eigenvalues are from the exact ones of the same matrix, measured below FP64's own rounding.

The reference is the Rayleigh quotient of LAPACK's vectors in extended precision: its error is the square of theirs.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _hermitian(L):
    n = L.shape[0]
    h = np.tril(L) + np.tril(L, -1).conj().T
    h[np.arange(n), np.arange(n)] = h.diagonal().real
    return h


def _quotients(h, X):
    X = X.astype(np.clongdouble)
    Y = h.astype(np.clongdouble) @ X
    return (X.conj() * Y).real.sum(0) / (X.conj() * X).real.sum(0)


@pytest.mark.parametrize("ntheta", [3, 5])
def test_lattice_eigenvalues(ntheta):
    """H(k) of the lattice: the lowest bands' vectors have one sign along the rows, so rounding that is not to nearest
    adds up there (n / 4 units of a tile's last place).  Bound: one EPS |H| of the bisection's bracket and two of the
    reduction, whose roundings are random."""
    import forge_gb300 as fg
    with fg.HartreeFock(fg.Setup(ntheta=ntheta, numk=6)) as hf:
        n, iu = hf.N, hf.N // 2 + 10
        H = hf.HamiltonianHartreeFock(np.zeros(n), np.zeros((n, n, 4), complex, order="F"), 0, 9)[:, :, [0, 8]]
        w, _, info = hf.zheevr_batch(H, iu, vectors=False)
    assert info == 0
    pick = np.unique(np.r_[0:6, 0:iu:max(1, iu // 16)])
    for b in range(2):
        h = _hermitian(H[:, :, b])
        e, X = np.linalg.eigh(h)
        assert np.max(np.abs(w[pick, b] - _quotients(h, X[:, pick]))) <= 3 * EPS * np.max(np.abs(e))


def _graded(n, ratio, rng):
    """A = D B D with a well conditioned B and the entries of D falling from 1 to sqrt(ratio)."""
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    B = np.eye(n) + 0.1 * (G + G.conj().T) / np.sqrt(n)
    d = np.exp2(np.round(np.log2(np.logspace(0, np.log10(ratio) / 2, n))))
    return d[:, None] * B * d[None, :], np.linalg.cond(B)


def _positive_eigenvalues(A):
    """Of a positive definite matrix, each to a few eps cond(B) of itself: one-sided Jacobi on the Cholesky factor
    (J. Demmel and K. Veselic, Jacobi's method is more accurate than QR, SIAM J. Matrix Anal. Appl. 13, 1992)."""
    L = np.linalg.cholesky(A)
    n = L.shape[0]
    for _ in range(30):
        worst = 0.0
        for p in range(n - 1):
            for q in range(p + 1, n):
                a, b, g = np.vdot(L[:, p], L[:, p]).real, np.vdot(L[:, q], L[:, q]).real, np.vdot(L[:, p], L[:, q])
                off = abs(g) / np.sqrt(a * b)
                if off <= EPS:
                    continue
                worst = max(worst, off)
                z = (b - a) / (2 * abs(g))
                t = (1.0 if z >= 0 else -1.0) / (abs(z) + np.hypot(1.0, z))
                c = 1 / np.hypot(1.0, t)
                x, y = L[:, p].copy(), L[:, q] * (g.conjugate() / abs(g))
                L[:, p], L[:, q] = c * x - c * t * y, c * t * x + c * y
        if worst <= 8 * EPS:
            break
    return np.sort(np.sum(np.abs(L) ** 2, 0))


@pytest.mark.parametrize("n,ratio", [(7, 1e-8), (40, 1e-8), (40, 1e-20), (66, 1e-16), (100, 1e-12)])
@pytest.mark.parametrize("unit", [1.0, 1e-60])
def test_graded_matrix(n, ratio, unit):
    """Small eigenvalues of a graded matrix keep their relative accuracy, n^2 eps cond(B) with a factor of four
    (J. Barlow and J. Demmel, Computing accurate eigensystems of scaled diagonally dominant matrices, 1990)."""
    import ctypes as C

    import torch

    import forge_gb300 as fg
    A, cond = _graded(n, ratio, np.random.default_rng(n))
    f = fg.load_library().forge_gpu_zheevr_noalloc
    f.argtypes = [C.c_void_p, C.c_int64, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p]
    f.restype = C.c_int
    dA = torch.from_numpy(np.ascontiguousarray(A.T * unit)).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = torch.empty(n, n, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    assert f(dA.data_ptr(), n, n, w.data_ptr(), Z.data_ptr(), None) == 0
    ref = _positive_eigenvalues(A)
    assert np.max(np.abs(w.cpu().numpy() / unit / ref - 1)) <= 4 * n * n * EPS * cond


def _eigenvalues(A):
    import ctypes as C

    import torch

    import forge_gb300 as fg
    f = fg.load_library().forge_gpu_zheevr_noalloc
    f.argtypes = [C.c_void_p, C.c_int64, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p]
    f.restype = C.c_int
    n = A.shape[0]
    dA = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = torch.empty(n, n, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    assert f(dA.data_ptr(), n, n, w.data_ptr(), Z.data_ptr(), None) == 0
    return w.cpu().numpy()


@pytest.mark.parametrize("ratio", [1e-40, 1e-50, 1e-60])
def test_eigenvalues_far_below_the_norm(ratio):
    """As test_graded_matrix, past the 2^-106 of the norm to which minors with replacements place an eigenvalue."""
    n = 40
    A, cond = _graded(n, ratio, np.random.default_rng(n))
    assert np.max(np.abs(_eigenvalues(A) / _positive_eigenvalues(A) - 1)) <= 4 * n * n * EPS * cond


def test_diagonal_over_many_orders():
    """Eigenvalues that stand on the diagonal come back to the bisection's 2 EPS |lambda|."""
    d = np.array([1e-33, 4.0, -3e-58, 1e-12, 0.0, -2e-31, 7e-31, 5e-45, -1.0, 6e-55])
    w = _eigenvalues(np.diag(d).astype(complex))
    assert np.all(np.abs(w - np.sort(d)) <= np.maximum(2 * EPS * np.abs(np.sort(d)), 1e-75))


@pytest.mark.parametrize("n", [2, 4, 8, 9, 15, 16, 17, 18, 32, 33, 34, 47, 48, 49, 50, 81])
def test_small_matrices(n):
    """The last (here only) block of reflectors ends with its last reflector, and a product's epilogue with the last row
    and column: every pair of matrices around the 16 columns and 32 rows that it goes by.  LAPACK's bounds."""
    import ctypes as C

    import torch

    import forge_gb300 as fg
    f = fg.load_library().forge_gpu_zheevr_noalloc
    f.argtypes = [C.c_void_p, C.c_int64, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p]
    f.restype = C.c_int
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    H = (G + G.conj().T) / 2
    nrm = np.linalg.norm(H, 2)
    for iu in sorted({1, n // 2, n - 1, n} - {0}):
        dA = torch.from_numpy(np.ascontiguousarray(H.T)).cuda()
        w = torch.empty(iu, dtype=torch.float64, device="cuda")
        Z = torch.empty(iu, n, dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        assert f(dA.data_ptr(), n, iu, w.data_ptr(), Z.data_ptr(), None) == 0
        w, X = w.cpu().numpy(), Z.cpu().numpy().T
        assert np.max(np.abs(w - np.linalg.eigvalsh(H)[:iu])) <= 8 * n * EPS * nrm
        assert np.max(np.abs(H @ X - X * w)) <= 16 * n * EPS * nrm
        assert np.max(np.abs(X.conj().T @ X - np.eye(iu))) <= 64 * EPS / 1e-7
