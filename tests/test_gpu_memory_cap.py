"""max_bytes: caps that once held a model with its set-up and a short run with
records go on holding it (small and large grids, square or not, hydro-only or
with erosion, one Manning's n or one per cell)."""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu

# (imax, jmax, hydro_only, spatially_var_mannings), bytes
CAPS = [
    ((3, 700, 0, 0), 6284250),
    ((3, 700, 0, 1), 6284250),
    ((3, 700, 1, 0), 1745820),
    ((3, 700, 1, 1), 1745820),
    ((64, 64, 0, 0), 7795356),
    ((64, 64, 0, 1), 7795356),
    ((64, 64, 1, 0), 1959984),
    ((64, 64, 1, 1), 1959984),
    ((150, 97, 0, 0), 24828192),
    ((150, 97, 0, 1), 24828192),
    ((150, 97, 1, 0), 5371128),
    ((150, 97, 1, 1), 5371128),
    ((400, 400, 0, 0), 268703136),
    ((400, 400, 0, 1), 268703136),
    ((400, 400, 1, 0), 52030452),
    ((400, 400, 1, 1), 52030452),
    ((500, 700, 0, 0), 568404660),
    ((500, 700, 0, 1), 568404660),
    ((500, 700, 1, 0), 112746288),
    ((500, 700, 1, 1), 112746288),
]


@pytest.mark.parametrize("shape,cap", CAPS)
def test_cap_holds(gpu_lib, shape, cap):
    import hc
    imax, jmax, hydro_only, var = shape
    case = synth.ensemble_member(1, fill=False, side_min=40, side_max=40)
    p = case.params
    p.imax, p.jmax, p.hydro_only, p.spatially_var_mannings = imax, jmax, hydro_only, var
    rng = np.random.default_rng(1)
    i = np.mgrid[0:imax, 0:jmax][0]
    case.elev = np.round(50 - 0.1 * i + rng.uniform(0, .05, (imax, jmax)), 6)
    if var:
        case.mannings = np.full((imax, jmax), 0.04)
    m = hc.Model(case, max_bytes=cap)
    assert len(m.run(2)) == 2
    m.close()
