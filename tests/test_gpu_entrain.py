"""erode() on grids whose lists of cells with flow lie around the length up to
which 16 lanes share a cell (256 on the smallest launch), for both transport
laws, against the oracle: record numbers bit for bit, the rest within 1e-10
plus 1e-9 relative (the member's bar: exp, log and pow are within 2 ulp of the
host's)."""
import numpy as np
import pytest

import synth
from helpers import assert_bitwise, assert_close
from test_gpu_members import mid_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 15, 16, 17, 20, 40])
@pytest.mark.parametrize("law", ["wilcock", "einstein"])
def test_erode_matches_oracle(gpu_lib, oracle_mod, n, law):
    case = synth.catchment_case(n=n, DX=20.0, hours=72, relief=30.0, lateral=False,
                                storm_start_h=0.1, seed=n)
    case.params.wilcock, case.params.einstein = int(law == "wilcock"), int(law == "einstein")
    case.water_init = np.full((n, n), 0.2)  # every cell flows
    o, m = mid_run(oracle_mod, case, 40)
    for _ in range(2):
        assert_close(m.erode(1.0), o.lib.hco_erode(o.h, 1.0), 0, "tempbmax", rtol=1e-9)
        assert_bitwise(m.field("index"), o.field("index"), "index")
        for k in ("elev", "grain", "strata", "Vsusptot", "Tau", "Vel", "ss", "sr", "sl", "su", "sd"):
            assert_close(m.field(k), o.field(k), 1e-10, k, rtol=1e-9)
