"""lateral3 (lateral_channel_erode, LSDCatchmentModel.cpp:4850-5291) on
seeded shear-stress fields: sizes at the edges of its loops (the border rows
and the bumped entries make up most of the smallest grids) and of the device's
32-wide tiles, wet cells few, mixed and everywhere, with and without the late
smoothing passes; called twice, so that the second call starts from the border
values the first one left.

The smoothing passes are the oracle's additions and quotients in its order;
the curvature transform's pow is within 2 ulp of the host's, and the
cross-channel means carry such differences on without growing them beyond a
few ulp a pass: 1e-10 relative over the some hundreds of passes."""
import numpy as np
import pytest

import synth
from helpers import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 6, 31, 34, 65])
@pytest.mark.parametrize("wet,passes,shift", [(0.15, 100, 5), (0.5, 3, 2), (0.85, 0, 0), (1.0, 7, 0)])
def test_lateral_matches_oracle(gpu_lib, oracle_mod, n, wet, passes, shift):
    import hc
    case = synth.catchment_case(n=n, DX=20.0, hours=72, relief=30.0, lateral=True, seed=n)
    case.params.edge_smoothing_passes = float(passes)
    case.params.downstream_shift = float(shift)
    rng = np.random.default_rng(n * 1000 + int(100 * wet))
    o = oracle_mod.Oracle(case)
    o.prepare()
    m = hc.Model(case)
    shape = (n + 2, n + 2)
    for _ in range(2):
        tau = np.zeros(shape)
        h = np.zeros(shape)
        wetc = rng.random((n, n)) < wet
        tau[1:-1, 1:-1] = np.where(wetc, rng.uniform(0.05, 5.0, (n, n)), 0.0)
        h[1:-1, 1:-1] = np.where(wetc, rng.uniform(0.0, 0.2, (n, n)), 0.0)
        listed = rng.random((n, n)) < 0.9
        ds = np.zeros((n + 2, n + 2), dtype=np.int32)
        for j in range(1, n + 1):
            rows = 1 + np.flatnonzero(listed[:, j - 1])
            ds[j, 1:1 + len(rows)] = rows
        for k, a in (("Tau", tau), ("water_depth", h), ("down_scan", ds)):
            o.field(k)[...] = a.reshape(o.field(k).shape)
            m.upload(k, a)
        o.lib.hco_lateral_channel_erode(o.h)
        m.lateral_channel_erode()
        assert_close(m.field("edge"), o.field("edge"), 1e-14, "edge", rtol=1e-10)
