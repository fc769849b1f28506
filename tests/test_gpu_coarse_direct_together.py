"""Calculations with large and small coarsest planes alive together: the direct
solve (coarse_direct.cu) of the large one takes the same route, to the bit, after a
small one was made and solved -- refilled (its factors made anew) and with its
V-cycle captured anew."""
import numpy as np
import pytest

from apbs_b200 import synth
from apbs_b200.vpmg import FP64, TUNE_GS27_LAG, Vpmg, lib

pytestmark = pytest.mark.gpu


def test_large_planes_after_small_ones():
    mol = synth.cluster(60, 4.0, seed=5, net_charge=1.0)

    def calc(n, nlev):
        return Vpmg(synth.mg_manual(n, 16.0 / (n - 1), mol.center(), nlev=nlev), FP64)

    def solve(c, fill=True):
        if fill:
            c.fillco(mol)
        lib().pmgb_launch_count(1)
        c.solve()
        return c.u, lib().pmgb_launch_count(0)

    with calc(97, 3) as large:      # coarsest 25^3: planes of 529
        solve(large)
        u, n = solve(large)
        with calc(33, 2) as small:  # coarsest 17^3: planes of 225
            us, _ = solve(small)
            got = solve(large)
            assert got[1] == n and np.array_equal(got[0], u)
            solve(small)
            large.set_tuning(TUNE_GS27_LAG, 12)  # drops the captured V-cycle
            got = solve(large, fill=False)
            assert np.array_equal(got[0], u)
            got = solve(large)
            assert got[1] == n and np.array_equal(got[0], u)
            assert np.array_equal(solve(small)[0], us)
