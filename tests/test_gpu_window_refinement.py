"""The FP64 window Rayleigh-Ritz (products in FP64 tiles on the CUDA cores, the small problem on the host) for every
parity of the window's width, on three matrices in one launch, against LAPACK."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("width", [1, 2, 3, 17, 31, 32])
@pytest.mark.parametrize("kind", ["random", "degenerate"])
def test_window_rayleigh_ritz(width, kind):
    import forge_gb300 as fg
    with fg.HartreeFock(fg.Setup(ntheta=2, numk=1, precision="mixed")) as hf:
        hf.set_refinement(width)
        n, nb = hf.N, 3
        iu = n // 2 + 10
        rng = np.random.default_rng(width)
        H = np.zeros((n, n, nb), complex, order="F")
        for b in range(nb):
            G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
            if kind == "random":
                H[:, :, b] = (G + G.conj().T) / 2
            else:                                # every level twice
                Q, _ = np.linalg.qr(G)
                H[:, :, b] = (Q * np.repeat(np.linspace(-3.0, 3.0, n // 2), 2)) @ Q.conj().T
        w, X, info = hf.zheevr_batch(H, iu)
    assert info == 0
    for b in range(nb):
        ref = np.linalg.eigvalsh(H[:, :, b])
        nrm = np.max(np.abs(ref))
        Xw, ww = X[:, iu - width:, b], w[iu - width:, b]
        # Ritz values: the FP32 vectors' error squared (n eps_32)^2 over the gaps, plus rounding; the window's
        # edges may cut a degenerate pair, whose values are the same
        assert np.max(np.abs(ww - ref[iu - width:iu])) <= 1e-9 * nrm
        assert np.all(np.diff(ww) >= 0)
        assert np.max(np.abs(Xw.conj().T @ Xw - np.eye(width))) <= 64 * n * EPS
        # the window diagonalises H in its span
        G = Xw.conj().T @ H[:, :, b] @ Xw
        assert np.max(np.abs(G - np.diag(ww))) <= 64 * n * EPS * nrm
