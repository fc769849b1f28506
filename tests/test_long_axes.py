"""Axes of more than 1024 points in the one-cluster kernels (apbs_b200/csrc/mixed.cu):
a batched solve and a mixed V-cycle tail of long thin grids against FP64, and the
quotient by multiplication that splits their flat indices, as a host model at its
bounds (the batch's levels have no limit but the caller's)."""
import random

import numpy as np
import pytest

from apbs_b200 import synth
from apbs_b200.vpmg import (FP64, MIXED, TUNE_GS7_COLOUR_PASSES, TUNE_TAIL_MAX_POINTS, Vpmg,
                             batch_solve)


def quotient(q, d):
    bits = (d - 1).bit_length()
    if bits == 0:
        return q
    m = (2**(31 + bits) + d - 1) // d
    assert m < 2**32
    return ((q * m) >> 32) >> (bits - 1)


def test_quotient_is_exact_below_two_to_the_31():
    rng = random.Random(5)
    ds = list(range(1, 300)) + [2**k + e for k in range(8, 31) for e in (-1, 0, 1)] + \
        [rng.randrange(1, 2**31) for _ in range(300)]
    for d in ds:
        top = (2**31 - 1) // d
        for n in [0, 1, 2, top // 2, top - 1, top] + [rng.randrange(0, top + 1) for _ in range(20)]:
            for q in (n * d - 1, n * d, n * d + 1, 2**31 - 1):
                if 0 <= q < 2**31:
                    assert quotient(q, d) == q // d, (q, d)


@pytest.mark.gpu
@pytest.mark.parametrize("dime", [(1089, 17, 17), (2113, 17, 17), (17, 1089, 17),
                                  (17, 2113, 17), (17, 17, 2113)])
def test_long_thin_grids_match_fp64(dime):
    m = synth.cluster(8, 2.5, seed=11, net_charge=1.0)
    axis = int(np.argmax(dime))
    h = tuple(1.0 if a == axis else 12.0 / (dime[a] - 1) for a in range(3))
    center = m.center().copy()
    center[axis] -= 0.5 * dime[axis] - 30  # the molecule 30 points from the far end
    p = synth.mg_manual(dime, h, center, nlev=4, etol=1e-9,
                        ions=((1.0, 0.1, 2.0), (-1.0, 0.1, 2.0)))

    def calc(prec, solve, limit=70000):
        with Vpmg(p, prec) as pmg:
            pmg.set_tuning(TUNE_TAIL_MAX_POINTS, limit)
            # rows of more than 1021 points do not fit the single-pass sweep
            pmg.set_tuning(TUNE_GS7_COLOUR_PASSES, 1)
            pmg.fillco(m)
            solve(pmg)
            return pmg.u, pmg.stats()["vcycles"]

    want, _ = calc(FP64, lambda c: c.solve())
    alone, cycles = calc(MIXED, lambda c: c.solve(), 5000)  # axes up to 529 in the tail
    tail, cycles_tail = calc(MIXED, lambda c: c.solve())
    batch, cycles_batch = calc(MIXED, lambda c: batch_solve([c]))
    # each is solved to a residual of 1e-9 of f; the error of u is that times at most
    # the operator's condition, under 1e3 on the short axes' few points.  A correction
    # that goes to other rows shows in the V-cycles it costs, if not in u
    for u, n in ((alone, cycles), (tail, cycles_tail), (batch, cycles_batch)):
        assert np.abs(u - want).max() <= 1e-6 * np.abs(want).max()
        assert n < 100 and abs(n - cycles) <= 1
