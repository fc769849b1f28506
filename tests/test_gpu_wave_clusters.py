"""The mailbox wavefront (k_gs27_mail) in clusters of every size, down to one CTA
(all neighbours foreign): the same iterates bit for bit as the step-counter
wavefront's, through the same number of launches (a refused launch would show,
as the step-counter route clears x and makes the residual itself).  Row widths
of 8, 24 and 40 slots; planes that fill the last cluster and that do not."""
import numpy as np
import pytest

from apbs_b200 import synth
from apbs_b200.vpmg import FP64, TUNE_GS27_PLANES, Vpmg, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dime,npbe", [((33, 33, 33), False), ((33, 65, 97), True),
                                       ((97, 65, 97), False), ((161, 97, 161), False)])
def test_iterates_do_not_depend_on_the_cluster(dime, npbe):
    m = synth.cluster(150, 7.0, seed=sum(dime), net_charge=1.0)
    p = synth.mg_manual(dime, tuple(26.0 / (d - 1) for d in dime), m.center(), npbe=npbe)
    with Vpmg(p, FP64) as pmg:
        pmg.fillco(m)

        def solve():
            lib().pmgb_launch_count(1)
            pmg.solve()
            return pmg.u, pmg.residual_history(), lib().pmgb_launch_count(0)

        pmg.set_tuning(TUNE_GS27_PLANES, 2)
        u, hist, _ = solve()
        pmg.set_tuning(TUNE_GS27_PLANES, 0)
        solve()                       # with the operators built
        want = solve()[2]
        for cluster in (1, 2, 4, 8, 16):
            assert lib().pmgb_debug_wave_cluster(pmg._h, cluster) == 1
            for _ in range(2):
                got = solve()
                assert np.array_equal(got[0], u) and np.array_equal(got[1], hist), cluster
                assert got[2] == want, cluster
        assert lib().pmgb_debug_wave_cluster(pmg._h, 3) == 0
