"""pmgb_footprint counts the packed coefficients of the FP64 plane wavefront on the
levels that hold them only: rows of up to 113 points and a CTA per plane on 148 SMs.
A grid whose levels have more planes than that is not charged for them."""
import os

import pytest

from apbs_b200 import serve, synth, vpmg
from apbs_b200.vpmg import FP64


@pytest.mark.skipif(not os.path.exists(vpmg.LIB_PATH), reason="library not built")
def test_levels_with_too_many_planes_are_not_charged():
    def per_plane(dime):
        p = synth.mg_manual(dime, 0.5, (0.0, 0.0, 0.0), nlev=3, npbe=True)
        return serve.footprint(p, FP64, 0) / dime[2]

    held, too_many, too_wide = (65, 65, 289), (65, 65, 449), (65, 65, 4097)
    assert per_plane(too_many) < 0.93 * per_plane(held)
    assert abs(per_plane(too_wide) / per_plane(too_many) - 1) < 0.01
    # level 1 (33, 33, 145): 28 doubles for each of 2 x 16 slots of 143 x 31 rows, and
    # two words for each slot of four half-sweeps; the coarsest level has none
    level = 143 * 31 * 16 * (2 * 28 * 8 + 4 * 2 * 8)
    extra = (per_plane(held) - per_plane(too_many)) * 289
    assert 0.95 * level < extra < 1.05 * level
