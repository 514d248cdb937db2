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
