"""A snapshot is its own until it is ended: it may be ended after its model
is closed, and by another thread than the one that runs the model."""
import threading

import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu
NAMES = ["water_depth", "elev", "qx", "qy", "edge", "Tau"]  # more than a context keeps


def model():
    import hc
    return hc.Model(synth.catchment_case(n=40, DX=20.0, hours=72, relief=60.0, lateral=False,
                                         storm_start_h=0.2))


def pinned(want):
    import torch
    return {k: torch.empty(v.shape, dtype=torch.float64, pin_memory=True).numpy()
            for k, v in want.items()}


@pytest.mark.parametrize("ended_before", [0, 2, 6])
def test_end_after_the_model_is_closed(gpu_lib, ended_before):
    for _ in range(4):
        m = model()
        m.run(40, records=False)
        want = {k: m.field(k) for k in NAMES}
        out = pinned(want)
        handles = [m.snapshot_begin(k, out[k]) for k in NAMES]
        for h in handles[:ended_before]:
            m.snapshot_end(h)
        m.close()
        for h in handles[ended_before:]:
            assert gpu_lib.hc_snapshot_end(h) == 0
        for k in NAMES:
            assert np.array_equal(out[k].view(np.uint8), want[k].view(np.uint8)), k


def test_end_on_another_thread(gpu_lib):
    m = model()
    m.run(40, records=False)
    bad = []

    def end(handles, out, want):
        for h in handles:
            if gpu_lib.hc_snapshot_end(h) != 0:
                bad.append("status")
        bad.extend(k for k in want
                   if not np.array_equal(out[k].view(np.uint8), want[k].view(np.uint8)))

    writers = []
    for _ in range(30):
        m.run(2, records=False)
        want = {k: m.field(k) for k in NAMES}
        out = pinned(want)
        handles = [m.snapshot_begin(k, out[k]) for k in NAMES]
        writers.append(threading.Thread(target=end, args=(handles, out, want)))
        writers[-1].start()
    for w in writers:
        w.join()
    m.close()
    assert not bad
