"""The one-cluster tail of the mixed-precision V-cycle: where the tail begins is a
launch choice.  A calculation's own solve agrees for every beginning (the damping
sums add up in another order, hence not bit for bit), and the batched kernel, which
always runs its levels in the cluster, gives the same bits whatever the limit says.
Sizes with fewer points than threads, a remainder, and a level above the default."""
import numpy as np
import pytest

from apbs_b200 import synth
from apbs_b200.vpmg import (MIXED, TUNE_MIXED_CHEBYSHEV, TUNE_TAIL_MAX_POINTS, Vpmg, batch_solve)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dime", [(17, 17, 17), (33, 49, 17), (65, 65, 65), (97, 65, 49)])
@pytest.mark.parametrize("cheb", [0, 2, 3])
def test_tail_beginning_is_only_a_launch_choice(dime, cheb):
    m = synth.cluster(60, 5.0, seed=7, net_charge=1.0)
    p = synth.mg_manual(dime, 0.6, m.center())
    alone, batched = [], []
    for limit in (1, 20000, 70000):
        with Vpmg(p, MIXED) as c:
            c.set_tuning(TUNE_TAIL_MAX_POINTS, limit)
            c.set_tuning(TUNE_MIXED_CHEBYSHEV, cheb)
            c.fillco(m)
            c.solve()
            alone.append(c.u.copy())
            c.fillco(m)
            batch_solve([c])
            batched.append(c.u.copy())
    top = np.abs(alone[0]).max()
    for a, b in zip(alone, batched):
        # converged to etol 1e-6 by V-cycles equal up to FP32 rounding
        assert np.abs(a - alone[0]).max() <= 2e-6 * top
        assert np.abs(b - alone[0]).max() <= 2e-6 * top
        np.testing.assert_array_equal(b, batched[0])
