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
