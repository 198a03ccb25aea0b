"""Order of the window energies: ranks where all energies differ, the reference's heap sort where some are equal.

The index map has to be the heap sort's restatement on the same bands, entry by entry, and the occupation counts and the
Fermi level those of the restatement; numk = 1 to 9 takes the states from fewer than a warp to more than one a thread.
"""
import numpy as np
import pytest

from oracle import forge_oracle as fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("numk", [1, 3, 9])
@pytest.mark.parametrize("level", [0.0, 1e18])   # at 1e18 the hopping is below the spacing of the energies
def test_sorted_states(numk, level):
    import forge_gb300 as fg
    kw = dict(ntheta=2, numk=numk, nfilling=2.0)
    S, so = fg.Setup(**kw), fo.Setup(**kw)
    g = fo.build_geometry(so)
    with fg.HartreeFock(S) as hf:
        N = hf.N
        P = np.zeros((N, N, 4), complex, order="F")
        B, _, _, _ = hf.Solve(np.full(N, level), P, bands=True)
        e, mom, idx = hf.SortEnergies_1Spin()
        nF, EF, nocc, npart, _ = hf.FermiLevel()
    if level:
        assert np.unique(B).size < B.size
    se, idx_o, mom_o, _, _, _ = fo.sort_energies_1spin(so, g, B)
    assert np.array_equal(e, se)
    assert np.array_equal(idx, idx_o)
    assert np.array_equal(mom, mom_o)
    nFo, EFo, nocco, nparto, _ = fo.fermi_level(so, se)
    assert (nF, nocc, npart) == (nFo, nocco, nparto) and EF == EFo
