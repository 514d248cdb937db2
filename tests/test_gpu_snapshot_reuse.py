"""Snapshots use the buffers of ended ones again: more of them at once than a
context keeps, fields of two sizes (`edge` is smaller than the padded grid),
and rounds whose fields have changed; every raster is the field as it was when
its snapshot was begun."""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("names", [["elev"], ["edge", "water_depth"],
                                   ["water_depth", "edge", "qx", "qy", "elev", "Tau"]])
def test_buffers_are_used_again(gpu_lib, names):
    import hc
    import torch
    case = synth.catchment_case(n=40, DX=20.0, hours=72, relief=60.0, lateral=False,
                                storm_start_h=0.2)
    m = hc.Model(case)
    for _ in range(3):
        m.run(120, records=False)
        want = {k: m.field(k) for k in names}
        out = {k: torch.empty(v.shape, dtype=torch.float64, pin_memory=True).numpy()
               for k, v in want.items()}
        handles = [m.snapshot_begin(k, out[k]) for k in names]
        m.run(5, records=False)
        for h in handles[::-1]:
            m.snapshot_end(h)
        for k in names:
            assert np.array_equal(out[k].view(np.uint8), want[k].view(np.uint8)), k
