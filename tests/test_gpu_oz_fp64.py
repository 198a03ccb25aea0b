"""FP64 products by exact integer slices on the tensor cores (rank-2k update, back-transformation, projectors)
at the edges of their tiles (128 x 128), K blocks (64, 256) and block widths, against numpy.

Bounds: the slices keep 62 bits below a row's maximum, so results are held to what FP64 arithmetic of the
same size gives: n eps times the norms (the factors are those of the LAPACK error bounds, 8 and 16).
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _solve(H, iu):
    import torch

    import forge_gb300 as fg
    f = fg.load_library().forge_gpu_zheevr_noalloc
    f.argtypes = [C.c_void_p, C.c_int64, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p]
    f.restype = C.c_int
    n = H.shape[0]
    A = torch.from_numpy(np.ascontiguousarray(H.T)).cuda()
    w = torch.empty(iu, dtype=torch.float64, device="cuda")
    Z = torch.empty(iu, n, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    assert f(A.data_ptr(), n, iu, w.data_ptr(), Z.data_ptr(), None) == 0
    return w.cpu().numpy(), Z.cpu().numpy().T


@pytest.mark.parametrize("n", [34, 63, 65, 96, 127, 128, 129, 161, 192, 255, 256, 384, 385, 511])
@pytest.mark.parametrize("scale", ["flat", "wild"])
def test_eigenpairs_at_tile_edges(n, scale):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    H = (G + G.conj().T) / 2
    if scale == "wild":           # rows of the update and of V over twelve orders of magnitude
        s = np.logspace(0, -6, n)
        H = s[:, None] * H * s[None, :]
    iu = max(1, n - 3)
    w, X = _solve(H, iu)
    nrm = np.linalg.norm(H, 2)
    assert np.max(np.abs(w - np.linalg.eigvalsh(H)[:iu])) <= 8 * n * EPS * nrm
    assert np.max(np.abs(H @ X - X * w)) <= 16 * n * EPS * nrm


@pytest.mark.parametrize("ntheta,nlayers,numk", [(1, 2, 1), (2, 2, 3), (3, 3, 2), (8, 2, 1)])
def test_bulk_projector(ntheta, nlayers, numk):
    """zFockBulk of a solve = the phase-weighted projectors of LAPACK's eigenvectors of the same H(k)."""
    import forge_gb300 as fg
    S = fg.Setup(ntheta=ntheta, nlayers=nlayers, RotateLayers=(-1, 1, -1)[:nlayers], numk=numk, nfilling=0.0,
                 degfactor_mode="corrected")
    with fg.HartreeFock(S) as hf:
        N, Nk, s = hf.N, hf.Nk, hf.s
        rng = np.random.default_rng(5)
        V = rng.standard_normal(N)      # lifts the degeneracies at the projector's edge
        P = np.zeros((N, N, 4), complex, order="F")
        H = hf.HamiltonianHartreeFock(V, P, 0, Nk)
        _, _, bulk, info = hf.Solve(V, P, bulk=True)
        g = hf.geometry
    assert info == 0
    ref = np.zeros((N, N, 4), complex)
    gap = np.inf
    K = s.nLower - 1
    for k in range(Nk):
        L = np.tril(H[:, :, k])
        w, Z = np.linalg.eigh(L + np.tril(L, -1).conj().T)
        gap = min(gap, w[K] - w[K - 1] if K else np.inf)
        Ck = Z[:, :K].conj() @ Z[:, :K].T
        i1, i2 = g.nMomentaComponents[k]
        for c in range(4):
            n1, n2 = g.nUnitCell_1[c], g.nUnitCell_2[c]
            ref[:, :, c] += Ck * np.exp(-2j * np.pi * (i1 * n1 + i2 * n1 + i2 * n2) / numk)
    # rotation of the occupied space by the backward error n eps |H| over the gap, per k
    tol = 16 * N * EPS * (1 + 20.0 / gap) * Nk
    assert np.max(np.abs(bulk - ref)) <= tol
