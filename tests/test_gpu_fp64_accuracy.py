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
