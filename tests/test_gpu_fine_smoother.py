"""pmgb_fine_smoother names the kernel the fine sweeps run in (the benchmark times
it) by the tunable, checked by the launches of a solve -- a single-pass sweep is one launch instead of two."""
import pytest

from apbs_b200 import synth
from apbs_b200.vpmg import (FP64, K_GS7_FP32, K_GS7_FP64, K_GS7_SWEEP_FP32, K_GS7_SWEEP_FP64, MIXED,
                            TUNE_GS7_COLOUR_PASSES, Vpmg, lib)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dime", [65, 161])
def test_mixed_fine_smoother_by_tunable(dime):
    m = synth.cluster(60, 5.0, seed=2, net_charge=1.0)
    p = synth.mg_manual(dime, 30.0 / (dime - 1), m.center())
    per_cycle = {}
    with Vpmg(p, MIXED) as c:
        for value in (0, 1, 2):
            c.set_tuning(TUNE_GS7_COLOUR_PASSES, value)
            c.fillco(m)
            c.solve()
            lib().pmgb_launch_count(1)
            c.solve()
            per_cycle[value] = (lib().pmgb_launch_count(0) - 10.0) / c.stats()["vcycles"]
            want = {0: K_GS7_FP32, 1: K_GS7_FP32, 2: K_GS7_SWEEP_FP32}[value]
            assert c.fine_smoother() == want
    # two sweeps down (the first from zero, in colours either way) and two up: three
    # launches fewer per V-cycle, the solve's other launches aside
    assert per_cycle[1] - per_cycle[2] > 2.0
    assert per_cycle[0] == per_cycle[1]


def test_fp64_fine_smoother():
    p = synth.mg_manual(33, 0.5, (0.0, 0.0, 0.0))
    with Vpmg(p, FP64) as c:
        assert c.fine_smoother() == K_GS7_SWEEP_FP64
        c.set_tuning(TUNE_GS7_COLOUR_PASSES, 1)
        assert c.fine_smoother() == K_GS7_FP64
