"""The mixed path's fine-level smoothing: colour passes, single-pass sweeps and the
size rule between them give the same bits, from no sweep to an odd count (which ends
in the other buffer), on a ragged grid and on one either side of the rule's line."""
import numpy as np
import pytest

from apbs_b200 import synth
from apbs_b200.vpmg import (MIXED, TUNE_GS7_COLOUR_PASSES, TUNE_MIXED_FINE_SWEEPS, Vpmg)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dime,sweeps", [((33, 49, 17), 1), ((33, 49, 17), 3), ((65, 33, 33), 2),
                                         ((129, 129, 161), 2), ((129, 161, 161), 2),
                                         ((129, 161, 161), 1)])
def test_colour_passes_and_single_pass_agree(dime, sweeps):
    m = synth.cluster(60, 5.0, seed=11, net_charge=1.0)
    p = synth.mg_manual(dime, 0.5, m.center())
    got = []
    for passes in (0, 1, 2):
        with Vpmg(p, MIXED) as c:
            c.set_tuning(TUNE_GS7_COLOUR_PASSES, passes)
            c.set_tuning(TUNE_MIXED_FINE_SWEEPS, sweeps)
            c.fillco(m)
            c.solve()
            got.append((c.u.copy(), c.stats()["vcycles"]))
    for u, cycles in got[1:]:
        np.testing.assert_array_equal(u, got[0][0])
        assert cycles == got[0][1]
