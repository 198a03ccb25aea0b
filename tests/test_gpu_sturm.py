"""The Sturm counts by leading minors where minors vanish: a point exactly on a repeated, uncoupled diagonal replaces
one minor after the other, across every rescale."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _counts(d, e, x):
    import forge_gb300 as fg
    lib = fg.load_library()
    d, e, x = (np.ascontiguousarray(v, np.float64) for v in (d, e, x))
    c = np.zeros((2, x.size), np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    assert lib.forge_gpu_selftest_sturm(C.c_int64(d.size), p(d), p(e), C.c_int64(x.size), p(x), p(c[0]), p(c[1])) == 0
    return c


@pytest.mark.parametrize("n", [1, 2, 4, 5, 6, 9, 10, 33, 100])
@pytest.mark.parametrize("lead", [0, 1, 3])
def test_counts_on_a_repeated_diagonal(n, lead):
    """`lead` entries elsewhere shift the run against the rescales; every eigenvalue equal to x counts."""
    d = np.r_[-0.25 * np.ones(lead), 0.5 * np.ones(n), 0.75]
    c = _counts(d, np.zeros(d.size - 1), [0.5, 0.5 - 2.0**-20, 0.5 + 2.0**-20, 0.75])
    assert c.tolist() == [[lead + n, lead, lead + n, lead + n + 1]] * 2


@pytest.mark.parametrize("n", [3, 64, 257])
def test_counts_of_a_coupled_matrix(n):
    """Away from the eigenvalues (by 1e-4, above the FP32 counts' rounding) both counts are those of LAPACK."""
    rng = np.random.default_rng(n)
    d, e = rng.uniform(-0.4, 0.4, n), rng.uniform(0.05, 0.3, n - 1)
    w = np.linalg.eigvalsh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1))
    x = rng.uniform(-1, 1, 200)
    x = x[np.min(np.abs(x[:, None] - w), 1) > 1e-4]
    c = _counts(d, e, x)
    ref = np.sum(w[None, :] <= x[:, None], 1)
    assert np.array_equal(c[0], ref) and np.array_equal(c[1], ref)


@pytest.mark.parametrize("seed", [1, 2])
def test_division_by_fmas(seed):
    """quot(a, b) against a / b: never off by more than a unit in the last place.  The remainder step leaves the
    quotient within 2^-80 before its rounding, so it rounds the other way for at most one pair in 2^26."""
    import forge_gb300 as fg
    out = (C.c_int64 * 3)()
    assert fg.load_library().forge_gpu_selftest_quot(C.c_int64(seed), C.c_int64(1 << 29), out) == 0
    assert out[0] >= 1 << 29
    assert out[2] == 0 and out[1] <= out[0] >> 26
