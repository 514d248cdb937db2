"""The drainage sweep's waits are bounded by what they wait without any cell
being finished, not by the length of the sweep: a single path of 22,500 cells
(one warp works, all others wait, for some 45 ms) under a bound of 8,192 looks,
of which about one thousand fit between two reports of the working warp."""
import numpy as np
import pytest

import synth
from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


def test_long_path_under_a_short_bound(gpu_lib, oracle_mod):
    import hc
    side = 150
    case = synth.ensemble_member(1, fill=False, side_min=40, side_max=40)
    p = case.params
    p.imax = p.jmax = side
    p.hydro_only = 1
    i, j = np.mgrid[0:side, 0:side]
    along = i * side + np.where(i % 2 == 0, j, side - 1 - j)  # a serpentine
    case.elev = np.round(10 + 0.01 * (side * side - along), 6)
    o = oracle_mod.Oracle(case)
    o.prepare()
    m = hc.Model(case, prepare=False)
    m.test_bounded_waits(1 << 13, 0)
    m.prepare()
    assert_bitwise(m.field("area"), o.field("area"), "area")
