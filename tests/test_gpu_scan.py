"""scan_area (LSDCatchmentModel.cpp:3821-3849) and the wet list built from it,
at grids around the 32-column words and the 8-row strips the device works in,
with few, half and most cells wet: the mask is the oracle's, and flow_route and
depth_update over the list give the oracle's discharges, depths and maximum
(1e-12, the members' bar); then the list is rebuilt from an uploaded mask."""
import numpy as np
import pytest

import synth
from helpers import assert_bitwise, assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("imax,jmax", [(3, 3), (4, 31), (8, 32), (9, 33), (63, 64), (65, 65), (130, 97)])
@pytest.mark.parametrize("wet", [0.002, 0.1, 0.6])
def test_mask_and_list(gpu_lib, oracle_mod, imax, jmax, wet):
    import hc
    case = synth.ensemble_member(1, fill=False, side_min=40, side_max=40)
    p = case.params
    p.imax, p.jmax, p.hydro_only = imax, jmax, 1
    rng = np.random.default_rng(imax * 1000 + jmax)
    case.elev = np.round(rng.uniform(1.0, 3.0, (imax, jmax)), 6)
    o = oracle_mod.Oracle(case)
    o.prepare()
    m = hc.Model(case)
    h = np.zeros((imax + 2, jmax + 2))
    h[1:-1, 1:-1] = np.where(rng.random((imax, jmax)) < wet, rng.uniform(0.01, 1.0, (imax, jmax)), 0.0)
    h[0, 0] = np.nan  # an undefined padding corner counts as dry
    for turn in range(2):
        o.field("water_depth")[...] = h.reshape(o.field("water_depth").shape)
        m.upload("water_depth", h)
        if turn == 0:
            o.lib.hco_scan_area(o.h)
            m.scan_area()
        else:
            ds = np.array(o.field("down_scan"))
            ds[1 + jmax // 2] = 0  # one column taken off the list
            o.field("down_scan")[...] = ds
            m.upload("down_scan", ds)
        assert_bitwise(m.field("down_scan"), o.field("down_scan"), "down_scan")
        m.flow_route()
        o.lib.hco_flow_route(o.h)
        m.depth_update()
        o.lib.hco_depth_update(o.h)
        for k in ("qx", "qy", "water_depth"):
            assert_close(m.field(k), o.field(k), 1e-12, k, rtol=1e-12)
        assert abs(m.scalars().maxdepth - o.scalar("maxdepth")) <= 1e-12
        h = np.array(m.field("water_depth"))
