"""Batches past the grid's z and y extents for the products of the FP64 path: a small cell on a fine k grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("ntheta,numk", [(1, 182), (2, 128)])
def test_solve_on_a_fine_k_grid(ntheta, numk):
    """numk^2 = 33124 matrices of N = 28 (one block of reflectors) and 16384 of N = 76 (two): 2 x blocks x matrices
    exceeds 65535, and so do the projectors' items.  Every band against LAPACK, the bulk projector against its eigenvectors."""
    import forge_gb300 as fg
    with fg.HartreeFock(fg.Setup(ntheta=ntheta, numk=numk, degfactor_mode="corrected")) as hf:
        N, Nk, s, g = hf.N, hf.Nk, hf.s, hf.geometry
        V = np.random.default_rng(3).standard_normal(N)
        P = np.zeros((N, N, 4), complex, order="F")
        pick = np.r_[0:40, Nk // 2:Nk // 2 + 40, Nk - 40:Nk]
        H = np.concatenate([hf.HamiltonianHartreeFock(V, P, k, 1) for k in pick], 2)
        bands, _, bulk, info = hf.Solve(V, P, bulk=True)
        w_all = hf.HamiltonianHartreeFock(V, P, 0, Nk) if ntheta == 1 else None
    assert info == 0
    lo, up = s.nLower - 1, s.nUpper
    L = np.tril(np.moveaxis(H, 2, 0))
    F = L + np.conj(np.swapaxes(np.tril(L, -1), 1, 2))
    w = np.linalg.eigvalsh(F)
    tol = 8 * N * EPS * np.max(np.abs(w))
    assert np.max(np.abs(bands[:, pick] - w[:, lo:up].T)) <= tol
    # trace of the home cell: the number of bulk states
    assert abs(np.trace(bulk[:, :, 0]) - lo * Nk) <= 64 * N * EPS * Nk
    if w_all is None:
        return
    L = np.tril(np.moveaxis(w_all, 2, 0))
    w, Z = np.linalg.eigh(L + np.conj(np.swapaxes(np.tril(L, -1), 1, 2)))
    assert np.max(np.abs(bands - w[:, lo:up].T)) <= tol
    gap = np.min(w[:, lo] - w[:, lo - 1])
    C = np.einsum("kia,kja->kij", Z[:, :, :lo].conj(), Z[:, :, :lo])
    i1, i2 = (np.asarray(g.nMomentaComponents)[:, q] for q in (0, 1))
    for c in range(4):
        n1, n2 = g.nUnitCell_1[c], g.nUnitCell_2[c]
        ref = np.einsum("k,kij->ij", np.exp(-2j * np.pi * (i1 * n1 + i2 * n1 + i2 * n2) / numk), C)
        assert np.max(np.abs(bulk[:, :, c] - ref)) <= 16 * N * EPS * (1 + 20.0 / gap) * Nk
