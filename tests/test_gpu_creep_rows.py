"""Creep's rows hand their progress down the grid: many rows of few columns
(every row waits for the one above nearly all the time, over more blocks than
one multiprocessor holds), few rows of many, and a grid in between, all cells
with records whose strata move, against the oracle's serial loop, bit for
bit."""
import numpy as np
import pytest

import synth
from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


def creep_case(imax, jmax, oracle_mod):
    """(model, oracle) of a rough surface with a record on every cell."""
    import hc
    case = synth.ensemble_member(1, fill=False, side_min=40, side_max=40)
    case.params.imax, case.params.jmax = imax, jmax
    rng = np.random.default_rng(imax * 10 + jmax)
    case.elev = np.round(rng.uniform(0.0, 30.0, (imax, jmax)), 3)
    o = oracle_mod.Oracle(case)
    o.prepare()
    m = hc.Model(case)
    shape = (imax + 2, jmax + 2)
    n = imax * jmax
    index = np.full(shape, -9999, dtype=np.int32)
    index[1:-1, 1:-1] = 2 + np.arange(n).reshape(imax, jmax)
    grain = np.zeros((shape[0] * shape[1], 11))
    strata = np.zeros((shape[0] * shape[1], 10, 11))
    w = rng.random((n, 9)) ** 4
    grain[2:2 + n, 1:10] = rng.choice([0.2, 0.051, 0.299], (n, 1)) * w / w.sum(1, keepdims=True)
    strata[2:2 + n, :, 0:9] = rng.random((n, 10, 9)) * 0.05
    for k, a in (("index", index), ("grain", grain), ("strata", strata)):
        o.field(k)[...] = a.reshape(o.field(k).shape)
        m.upload(k, a)
    s = m.scalars()
    s.grain_array_tot = float(1 + n)
    m.set_scalars(s)
    o.set_scalar("grain_array_tot", s.grain_array_tot)
    return m, o


def check(m, o):
    for k in ("index", "grain", "strata", "elev"):
        assert_bitwise(m.field(k), o.field(k), k)
    assert m.scalars().grain_array_tot == o.scalar("grain_array_tot")


@pytest.mark.parametrize("imax,jmax", [(1300, 12), (12, 1300), (330, 95)])
def test_many_rows(gpu_lib, oracle_mod, imax, jmax):
    m, o = creep_case(imax, jmax, oracle_mod)
    m.creep(5.0)
    o.lib.hco_creep(o.h, 5.0)
    check(m, o)


@pytest.mark.parametrize("imax,jmax", [(4, 3), (5, 40), (40, 5), (70, 33)])
@pytest.mark.parametrize("spins,beyond", [(1, 1), (40, 1), (3000, 7), (1, 0)])
def test_waits_run_out(gpu_lib, oracle_mod, imax, jmax, spins, beyond):
    """A wait that gives up is reported, and the creep is complete all the
    same; so is the next one, with the built-in bound."""
    import hc
    m, o = creep_case(imax, jmax, oracle_mod)
    m.test_bounded_waits(spins, beyond)
    if beyond:  # the row above never gets there
        with pytest.raises(hc.HCError, match="HC_ERR_TIMEOUT"):
            m.creep(5.0)
    else:  # one look at the row above may or may not be enough
        try:
            m.creep(5.0)
        except hc.HCError as e:
            assert "HC_ERR_TIMEOUT" in str(e)
    o.lib.hco_creep(o.h, 5.0)
    check(m, o)
    m.test_bounded_waits(0, 0)
    m.creep(5.0)
    o.lib.hco_creep(o.h, 5.0)
    check(m, o)


@pytest.mark.parametrize("after", [0, 5])
def test_wait_runs_out_in_a_run(gpu_lib, after):
    """A creep that falls due in a call's last iteration (as always where a
    program runs one iteration a call), or `after` iterations before it: the
    call returns HC_ERR_TIMEOUT after that iteration, and the next one goes on
    as a run that never timed out."""
    import hc
    case = synth.catchment_case(n=48, DX=20.0, hours=72, relief=60.0, hydro_only=False,
                                lateral=False, storm_start_h=0.5)
    case.params.creep_time_interval = 60
    n = 600
    ref = hc.Model(case)
    cycle0 = ref.scalars().cycle
    ra = ref.run(n)
    due, at = cycle0, []
    for k, cycle in enumerate(ra[:, hc.STEP_FIELDS.index("cycle")]):
        if cycle > due:
            due += 60
            at.append(k)
    assert ref.run_stats()["creep"][0] == len(at) >= 2
    k = at[-1]
    assert n - k > 10
    m = hc.Model(case)
    m.run(k)
    assert (m.field("index") != -9999).any(), "no grain to move"
    m.test_bounded_waits(1, 1)
    with pytest.raises(hc.HCError, match="HC_ERR_TIMEOUT creep"):
        m.run(1 + after)
    assert int(m.scalars().counter) == k + 1
    m.test_bounded_waits(0, 0)
    rb = m.run(n - k - 1)
    assert_bitwise(rb, ra[k + 1:], "records")
    for f in ("elev", "index", "grain", "strata", "water_depth", "qx", "area"):
        assert_bitwise(m.field(f), ref.field(f), f)
