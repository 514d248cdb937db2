"""Creep's grain transfers (creep, LSDCatchmentModel.cpp:5293-5427) where grain
records exist: the device walks the rows as a wavefront and numbers the new
records afterwards; the oracle's loop is serial.  Grids from a single inner
row or column to several blocks of rows; records on few, some and all cells,
with totals near the strata thresholds, so that strata move and records are
made along the way.  Every operation is the oracle's, so grain, strata,
record numbers and elevations are compared bit for bit."""
import numpy as np
import pytest

import synth
from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("imax,jmax", [(3, 3), (3, 40), (40, 3), (4, 5), (7, 6), (33, 70), (70, 33)])
@pytest.mark.parametrize("share", [0.03, 0.5, 1.0])
def test_creep_with_records(gpu_lib, oracle_mod, imax, jmax, share):
    import hc
    case = synth.ensemble_member(1, fill=False, side_min=40, side_max=40)
    p = case.params
    p.imax, p.jmax = imax, jmax
    rng = np.random.default_rng(imax * 100 + jmax)
    case.elev = np.round(rng.uniform(0.0, 30.0, (imax, jmax)), 3)
    o = oracle_mod.Oracle(case)
    o.prepare()
    m = hc.Model(case)
    shape = (imax + 2, jmax + 2)
    # records on a share of the cells, numbered from 2 in scattered order
    index = np.full(shape, -9999, dtype=np.int32)
    cells = np.argwhere(rng.random((imax, jmax)) < share) + 1
    nrec = shape[0] * shape[1]
    cells = rng.permutation(cells) if len(cells) else np.array([[2, 2]])
    index[tuple(cells.T)] = 2 + np.arange(len(cells))
    grain = np.zeros((nrec, 11))
    strata = np.zeros((nrec, 10, 11))
    used = slice(2, 2 + len(cells))
    size = rng.choice([0.2, 0.3, 0.051, 0.05, 0.299], (len(cells), 1))  # active 0.2: 0.05 and 0.3
    w = rng.random((len(cells), 9)) ** 4
    grain[used, 1:10] = size * w / w.sum(1, keepdims=True)
    strata[used, :, 0:9] = rng.random((len(cells), 10, 9)) * 0.05
    bed = np.full(shape, -9999.0)
    bed[1:-1, 1:-1] = case.elev - rng.uniform(-0.5, 4.0, (imax, jmax))
    for k, a in (("index", index), ("grain", grain), ("strata", strata), ("bedrock", bed)):
        o.field(k)[...] = a.reshape(o.field(k).shape)
        m.upload(k, a)
    s = m.scalars()
    s.grain_array_tot = float(1 + len(cells))
    m.set_scalars(s)
    o.set_scalar("grain_array_tot", s.grain_array_tot)
    for _ in range(2):
        m.creep(5.0)
        o.lib.hco_creep(o.h, 5.0)
        for k in ("index", "grain", "strata", "elev"):
            assert_bitwise(m.field(k), o.field(k), k)
        assert m.scalars().grain_array_tot == o.scalar("grain_array_tot")
