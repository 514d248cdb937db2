"""The drainage area (drainage_area_D8, LSDCatchmentModel.cpp:2091-2271) and
the input points it gives, on grids from 3 x 3 (every cell at an edge, where a
neighbour pushes in several directions) to several blocks; slopes (one long
path, one wide frontier), noise, plateaus (the sort's order among equal
elevations) and no-data cells.  Every term and addition is the oracle's, so
areas are compared bit for bit, twice: a set-up may be repeated."""
import numpy as np
import pytest

import synth
from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


def surface(kind, imax, jmax):
    rng = np.random.default_rng(imax * 1000 + jmax)
    i, j = np.mgrid[0:imax, 0:jmax].astype(float)
    if kind == "noise":
        return np.round(rng.uniform(1, 50, (imax, jmax)), 6)
    if kind == "plateaus":
        return np.round(rng.uniform(1, 6, (imax, jmax)))
    if kind == "path":  # a serpentine: one cell after the other
        z = 10 + 0.01 * (imax * jmax - (i * jmax + np.where(i % 2 == 0, j, jmax - 1 - j)))
        return np.round(z, 6)
    if kind == "holes":
        z = np.round(50 - 0.1 * i + rng.uniform(0, 1, (imax, jmax)), 6)
        z[rng.random((imax, jmax)) < 0.2] = -9999
        return z
    return np.round(50 - 0.1 * i, 6)


@pytest.mark.parametrize("imax,jmax", [(3, 3), (3, 50), (50, 3), (31, 33), (64, 65), (150, 97)])
@pytest.mark.parametrize("kind", ["noise", "plateaus", "path", "holes", "plane"])
def test_area_matches_oracle(gpu_lib, oracle_mod, imax, jmax, kind):
    import hc
    case = synth.ensemble_member(1, fill=False, side_min=40, side_max=40)
    p = case.params
    p.imax, p.jmax = imax, jmax
    p.hydro_only = 1
    p.MIN_Q = 1e-5  # points on small grids too
    case.elev = surface(kind, imax, jmax)
    o = oracle_mod.Oracle(case)
    o.prepare()
    m = hc.Model(case)
    for _ in range(2):
        assert_bitwise(m.field("area"), o.field("area"), "area")
        assert m.scalars().totalinputpoints == o.scalar("totalinputpoints")
        m.upload("elev", m.field("elev"))  # the area is computed again
        m.prepare()
