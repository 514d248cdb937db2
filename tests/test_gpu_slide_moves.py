"""slide_3 where every cell is wet and half the cells stand above their slope:
visits that move in several directions, moves out of and into the clamped
first and last rows, cells with and without a grain record.  Against the
oracle, elevations and record numbers bit for bit, grains and strata to the
member's 1e-12."""
import numpy as np
import pytest

import synth
from helpers import assert_bitwise, assert_close
from test_gpu_members import mid_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 17, 48])
@pytest.mark.parametrize("step", [2.0, 40.0])
def test_slides_match_oracle(gpu_lib, oracle_mod, n, step):
    case = synth.catchment_case(n=n, DX=10.0, hours=72, relief=60.0, lateral=False,
                                storm_start_h=0.1, seed=n)
    case.water_init = np.full((n, n), 0.2)
    o, m = mid_run(oracle_mod, case, 60)
    rng = np.random.default_rng(n)
    e = o.field("elev")
    e[1:-1, 1:-1] += step * (rng.random((n, n)) < 0.5)
    m.upload("elev", e)
    before = np.array(e, copy=True)
    for _ in range(2):
        m.in_channel_landsliding()
        o.lib.hco_in_channel_landsliding(o.h)
    if step > 10:
        assert np.any(o.field("elev") != before)
    assert_bitwise(m.field("elev"), o.field("elev"), "elev")
    assert_bitwise(m.field("index"), o.field("index"), "index")
    for k in ("grain", "strata"):
        assert_close(m.field(k), o.field(k), 1e-12, k, rtol=1e-12)
