"""Failure path of the direct coarse solve (coarse_direct.cu), made without a
device fault: one of its bounded waits is counted as run out (a testing hook), so
that the others give up at once -- in the factor, whose inverses are then not
whole, or in a solve.  The pmgb_solve that meets it fails with an error naming the
waits, and the next one on the same calculation gives the normal answer, with the
factors made again where they were not whole."""
import numpy as np
import pytest

from apbs_b200 import synth
from apbs_b200.vpmg import FP64, PmgbError, Vpmg, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dime,nlev", [(33, 2), (97, 3)])
def test_direct_solve_waits_run_out_and_recover(dime, nlev):
    mol = synth.cluster(60, 4.0, seed=5, net_charge=1.0)
    p = synth.mg_manual(dime, 16.0 / (dime - 1), mol.center(), nlev=nlev)
    with Vpmg(p, FP64) as pmg:
        pmg.fillco(mol)
        pmg.solve()
        u, e = pmg.u, pmg.energy()

    def again(pmg):
        pmg.solve()
        assert np.array_equal(pmg.u, u) and pmg.energy() == e

    with Vpmg(p, FP64) as pmg:
        pmg.fillco(mol)
        for _ in range(2):  # the first factor, and one into the same arrays
            assert lib().pmgb_debug_direct_wait(pmg._h) == 1
            with pytest.raises(PmgbError, match=r"waits ran out \(factor of the direct"):
                pmg.solve()
            again(pmg)
            assert lib().pmgb_debug_direct_wait(pmg._h) == 1
            with pytest.raises(PmgbError, match=r"waits ran out \(direct coarse solve\)"):
                pmg.solve()
            again(pmg)
            pmg.fillco(mol)
