"""forge_gpu_zheevr_batch where its workspace serves a part of the batch at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("mode", ["fp64", "mixed", "refined"])
@pytest.mark.parametrize("cap", [1, 3, 7])
def test_batch_in_parts(mode, cap, monkeypatch):
    """Seven matrices, 1, 3 + 3 + 1 or all at a time: the same eigenvalues bit for bit in FP64 (nothing in them depends
    on the batch at this size), to the solver's accuracy in mixed precision, and vectors of their own matrix."""
    import forge_gb300 as fg
    nb = 7
    with fg.HartreeFock(fg.Setup(ntheta=2, numk=1, precision="fp64" if mode == "fp64" else "mixed")) as hf:
        if mode == "refined":
            hf.set_eigen_refinement(1)
        n = hf.N
        iu = n // 2 + 10
        rng = np.random.default_rng(11)
        G = rng.standard_normal((n, n, nb)) + 1j * rng.standard_normal((n, n, nb))
        H = np.asfortranarray((G + G.conj().transpose(1, 0, 2)) / 2)
        monkeypatch.delenv("FORGE_EIG_BATCH", raising=False)
        w0, _, info0 = hf.zheevr_batch(H, iu)
        monkeypatch.setenv("FORGE_EIG_BATCH", str(cap))
        w, X, info = hf.zheevr_batch(H, iu)
    assert info0 == 0 and info == 0
    if mode == "fp64":
        assert np.array_equal(w, w0)
    eps = {"fp64": 16 * n * EPS, "mixed": 16 * n * np.finfo(np.float32).eps, "refined": 1e-8}[mode]
    for b in range(nb):
        nrm = np.linalg.norm(H[:, :, b], 2)
        assert np.max(np.abs(w[:, b] - np.linalg.eigvalsh(H[:, :, b])[:iu])) <= eps * nrm
        assert np.max(np.abs(H[:, :, b] @ X[:, :, b] - X[:, :, b] * w[:, b])) <= eps * nrm


def test_blocks_of_reflectors_formed_together():
    """N = 508: a caller's batch forms V^H and T of all eight blocks in one launch (the allocation-free entry, whose
    array is small, one at a time)."""
    import forge_gb300 as fg
    with fg.HartreeFock(fg.Setup(ntheta=6, numk=1)) as hf:
        n, nb = hf.N, 3
        iu = n // 2 + 10
        rng = np.random.default_rng(6)
        G = rng.standard_normal((n, n, nb)) + 1j * rng.standard_normal((n, n, nb))
        H = np.asfortranarray((G + G.conj().transpose(1, 0, 2)) / 2)
        w, X, info = hf.zheevr_batch(H, iu)
    assert info == 0
    for b in range(nb):
        nrm = np.linalg.norm(H[:, :, b], 2)
        assert np.max(np.abs(w[:, b] - np.linalg.eigvalsh(H[:, :, b])[:iu])) <= 8 * n * EPS * nrm
        assert np.max(np.abs(H[:, :, b] @ X[:, :, b] - X[:, :, b] * w[:, b])) <= 16 * n * EPS * nrm
        assert np.max(np.abs(X[:, :, b].conj().T @ X[:, :, b] - np.eye(iu))) <= 64 * EPS / 1e-7
