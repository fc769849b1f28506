"""The coarsest LPBE level solved by its planes (coarse_direct.cu) against the
reference's banded Cholesky on the same operators: planes of a whole number of
16-row blocks and not, one to many planes, both parities of their number; and
planes too large for it, which the refinement takes."""
import numpy as np
import pytest

from apbs_b200 import synth
from apbs_b200.vpmg import FP64, TUNE_BAND_ALWAYS, Vpmg

pytestmark = pytest.mark.gpu

CASES = [((69, 35, 5), 2), ((67, 35, 7), 2), ((35, 35, 9), 2), ((17, 17, 33), 2),
         ((33, 33, 17), 2), ((33, 33, 33), 2), ((65, 65, 9), 2), ((49, 65, 97), 3),
         ((97, 65, 65), 4)]


@pytest.mark.parametrize("dime,nlev", CASES)
def test_plane_solve_matches_band(dime, nlev):
    mol = synth.cluster(60, 4.0, seed=sum(dime), net_charge=1.0)
    p = synth.mg_manual(dime, tuple(16.0 / (d - 1) for d in dime), mol.center(), nlev=nlev)
    out = []
    for band in (1, 0):
        with Vpmg(p, FP64) as pmg:
            pmg.set_tuning(TUNE_BAND_ALWAYS, band)
            for _ in range(2):  # the second solve refactors into the same arrays
                pmg.fillco(mol)
                pmg.solve()
            out.append((pmg.u, pmg.energy(), pmg.residual_history(), pmg.stats()))
    (ub, eb, hb, sb), (ud, ed, hd, sd) = out
    assert sb["coarse_method"] == 1 and sd["coarse_method"] == 3
    assert len(hb) == len(hd)
    # both solve each coarse system to rounding times its condition number (under
    # 1e4 for these levels), which the V-cycle passes on to u without growth
    assert np.abs(ub - ud).max() <= 1e-11 * np.abs(ub).max()
    assert abs(eb - ed) <= 1e-11 * abs(eb)
