"""An error of one ensemble member (here a creep whose waits were made to run
out) is returned, and the members beside it, those of its own host thread
too, run to their end as they would alone."""
import ctypes as C
import os

import pytest

import synth
from helpers import assert_bitwise

pytestmark = pytest.mark.gpu
FIELDS = ["elev", "water_depth", "qx", "qy", "area", "down_scan"]


def test_other_members_run_on(gpu_lib):
    import hc
    case = synth.catchment_case(n=48, DX=20.0, hours=72, relief=60.0, hydro_only=False,
                                lateral=False, storm_start_h=0.5)
    case.params.creep_time_interval = 60
    small = synth.catchment_case(n=24, DX=20.0, hours=72, relief=60.0, hydro_only=False,
                                 lateral=False, storm_start_h=0.2)
    n = 60
    ref = hc.Model(case)
    due, at = ref.scalars().cycle, 0
    for k, cycle in enumerate(ref.run(600)[:, hc.STEP_FIELDS.index("cycle")]):
        if cycle > due:
            due, at = due + 60, k
    lead = at - 20  # a creep falls due in the n iterations after these
    first, alone = hc.Model(case), hc.Model(small)
    first.run(lead + n, records=False)
    alone.run(n, records=False)
    mate = (os.cpu_count() or 1) + 3  # more members than host threads
    ens = [hc.Model(case)] + [hc.Model(small) for _ in range(min(mate, 40))]
    ens[0].run(lead, records=False)
    ens[0].test_bounded_waits(1, 1)
    done = (C.c_int64 * len(ens))()
    st = gpu_lib.hc_run_ensemble((C.c_void_p * len(ens))(*[m.h.value for m in ens]), len(ens), n,
                                 0, done)
    assert hc.STATUS.get(st) == "HC_ERR_TIMEOUT"
    assert list(done[1:]) == [n] * (len(ens) - 1) and done[0] == 0
    for m in ens[1:]:
        for f in FIELDS:
            assert_bitwise(m.field(f), alone.field(f), f)
    ens[0].test_bounded_waits(0, 0)
    k = int(ens[0].scalars().counter)
    assert lead < k < lead + n
    ens[0].run(lead + n - k, records=False)
    for f in FIELDS + ["grain", "index"]:
        assert_bitwise(ens[0].field(f), first.field(f), f)
