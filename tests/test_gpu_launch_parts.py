"""The loops over parts of a batch in the refinement and in the sliced projectors, which a batch of these sizes runs in one
launch: several launches with a remainder give the same bits."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,nfilling", [("fp64", 0.0), ("fp64", 2.0), ("mixed", 2.0)])
def test_parts_of_a_batch(precision, nfilling):
    import forge_gb300 as fg
    out = []
    for per in (None, 1, 2, 4):      # matrices a launch; nine k points
        with fg.HartreeFock(fg.Setup(ntheta=2, numk=3, nfilling=nfilling, degfactor_mode="corrected",
                                     precision=precision)) as hf:
            if precision == "mixed":
                hf.set_eigen_refinement(1)
            if per:
                n, iu = hf.N, (hf.s.nUpper + 7) // 8 * 8
                planes = 2 * (7 if precision == "fp64" else 4)
                proj = per * (planes * n * iu * 2 + 2 * n * n * 8)
                # H and X slices (5 planes, complex, bf16), W and E planes, the transposed vectors; 256-byte rounding
                one = 20 * n * 80 + 20 * hf.s.nUpper * 80 + 48 * hf.s.nUpper * 76 + 16 * n * 76 + 8 * n + 2048
                assert hf.lib.forge_gpu_selftest_launch_bytes(hf.ctx, C.c_int64(per * one), C.c_int64(proj)) == 0
            E, _ = hf.PlainGuess()
            for _ in range(2):
                _, E, _ = hf.ScfIteration(E)
            P, d, V = hf.GetState()
            _, _, bulk, _ = hf.Solve(V, P, bulk=True)
            out.append((np.asarray(E), P, d, V, hf.GetBands(), bulk))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
