"""Kept snapshot buffers count under a context's max_bytes, make room for its
other allocations, and go with the context."""
import functools

import pytest

import synth

pytestmark = pytest.mark.gpu
NAMES = ["water_depth", "elev", "qx", "qy", "edge", "Tau"]
SIDE = 600


@functools.lru_cache(maxsize=None)
def case():
    return synth.catchment_case(n=SIDE, DX=20.0, hours=24, relief=60.0, hydro_only=True,
                                lateral=False, storm_start_h=0.2)


def make(cap=0):
    import hc
    return hc.Model(case(), max_bytes=cap)


def smallest_cap():
    import hc
    lo, hi = 1, 1 << 31
    while lo < hi:
        mid = (lo + hi) // 2
        try:
            make(mid).close()
            hi = mid
        except hc.HCError:
            lo = mid + 1
    return lo


def take(m):
    import torch
    out = {k: torch.empty(m.field(k).shape, dtype=torch.float64, pin_memory=True).numpy()
           for k in NAMES}
    for h in [m.snapshot_begin(k, out[k]) for k in NAMES]:
        m.snapshot_end(h)


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_kept_buffers_are_bounded_and_counted(gpu_lib):
    import torch
    make().close()
    field = (SIDE + 2) ** 2 * 8
    before = free_bytes()
    m = make()
    with_model = free_bytes()
    take(m)
    assert with_model - free_bytes() <= 4 * (field + (2 << 20))
    m.close()
    assert abs(before - free_bytes()) <= 2 << 20
    # a cap that just holds the model: snapshots go on, none is kept
    cap = smallest_cap()
    m = make(cap)
    with_model = free_bytes()
    take(m)
    assert with_model - free_bytes() < field
    m.close()
    # room for one kept buffer, or for the records of a longer run
    n = 26000
    m = make(cap + field + (1 << 16))
    take(m)
    assert n * 14 * 8 > 1 << 16
    rec = m.run(n)
    assert 0 < len(rec) <= n
    m.close()
