"""A bounded tensor-core wait that gave up: the FP64 eigen-solve and the bulk projector are tried a second time, on matrices
assembled (or copied) anew, and the call reports the error only if that fails as well."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = -5


def _inject(hf, solves, projectors):
    assert hf.lib.forge_gpu_selftest_timeouts(hf.ctx, C.c_int64(solves), C.c_int64(projectors)) == 0


def _solve(hf):
    rng = np.random.default_rng(4)
    V, P = 0.1 * rng.standard_normal(hf.N), np.zeros((hf.N, hf.N, 4), complex, order="F")
    bands, _, bulk, info = hf.Solve(V, P, bulk=True)
    assert info == 0
    return bands, bulk


@pytest.mark.parametrize("c3", [0, 1])
def test_solve(c3, capfd):
    import forge_gb300 as fg
    with fg.HartreeFock(fg.Setup(ntheta=2, numk=3)) as hf:
        if c3:
            hf.set_c3(1)
        ref = _solve(hf)
        _inject(hf, 1, 1)
        got = _solve(hf)
        assert capfd.readouterr().err.count("again") == 2
        assert np.array_equal(ref[0], got[0]) and np.array_equal(ref[1], got[1])
        for twice in ((2, 0), (0, 2)):
            _inject(hf, *twice)
            with pytest.raises(fg.ForgeError) as e:
                _solve(hf)
            assert str(TIMEOUT) in str(e.value)
            got = _solve(hf)
            assert np.array_equal(ref[0], got[0]) and np.array_equal(ref[1], got[1])


def test_iteration_and_group():
    """The group's members have one size: the padding of a smaller one is bounded by sums in no fixed order."""
    import forge_gb300 as fg

    def run(inject):
        with fg.HartreeFock(fg.Setup(ntheta=2, numk=3)) as a, fg.HartreeFock(fg.Setup(ntheta=2, numk=2)) as b:
            E = [a.PlainGuess()[0], b.PlainGuess()[0]]
            if inject:
                _inject(a, 1, 1)
            rep, Ea, _ = a.ScfIteration(E[0])
            if inject:
                _inject(a, 1, 0)
            _, Eg, _ = fg.ScfIterationGroup([a, b], np.array([Ea, E[1]]))
            return np.asarray(Ea), np.asarray(Eg), a.GetState()[0], b.GetState()[0]

    for x, y in zip(run(False), run(True)):
        assert np.array_equal(x, y)


def test_zheevr_batch():
    import forge_gb300 as fg
    with fg.HartreeFock(fg.Setup(ntheta=1, numk=1)) as hf:
        rng = np.random.default_rng(2)
        G = rng.standard_normal((hf.N, hf.N, 3)) + 1j * rng.standard_normal((hf.N, hf.N, 3))
        H = np.asfortranarray((G + G.conj().transpose(1, 0, 2)) / 2)
        ref = hf.zheevr_batch(H, 12)
        _inject(hf, 1, 0)
        got = hf.zheevr_batch(H, 12)
        assert np.array_equal(ref[0], got[0]) and np.array_equal(ref[1], got[1]) and got[2] == 0
        _inject(hf, 2, 0)
        with pytest.raises(fg.ForgeError):
            hf.zheevr_batch(H, 12)
        assert np.array_equal(ref[0], hf.zheevr_batch(H, 12)[0])
