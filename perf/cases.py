"""The work that users of libhc_gpu have it do, as cases to be timed.

Each case is one pass of a program over the public entry points
(hail-caesar_gb300/hc.py, the mirror of include/hc_gpu.h): whole iterations of
the main loop with their records and the rasters a run writes, the
member-by-member drop-in mode, a catchment's set-up, an ensemble, and the
gradient of a discharge misfit.  Sizes follow the benchmark's workloads and
the tests; the inputs are seeded synthetic terrains with the value
distributions of synth.py, made on the GPU.
"""
import math
import os
import sys

# what an ensemble program sets before the CUDA context exists (bench.py)
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hail-caesar_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import hc  # noqa: E402
import synth  # noqa: E402
from hc_abi import default_params  # noqa: E402

# kind: what a pass does.
#   reach      reach mode (one inflow point), erosion with Wilcock transport
#   flow       hydro-only, rain on every cell (distributed TOPMODEL runoff)
#   catchment  catchment mode through input points; erosion with Einstein
#              transport, lateral3 and slide_3, or hydro-only
#   members    the drop-in mode, one reference member per call, flow part
#   sediment   the same, the members of an erosion step
#   hillslope  creep and global landsliding
#   setup      hc_prepare: drainage area, input points, runoff table
#   ensemble   hc_run_ensemble over independent catchments
#   gradient   hc_adj_gradient
_LISTED = [
    # one iteration per call with its record read back, a small reach: the
    # latency a host program pays that drives the loop itself
    dict(name="reach_60x24_step", kind="reach", imax=60, jmax=24, n=1, spin=400),
    # the reach benchmark: 300 x 100 at 10 m, nine fractions
    dict(name="reach_300x100", kind="reach", imax=300, jmax=100, n=100, spin=800),
    # flow-only with every cell wet, a large ragged grid
    dict(name="flow_4001x4103", kind="flow", imax=4001, jmax=4103, n=4, spin=40),
    # a hydro-only catchment fed through its drainage network's input points
    dict(name="catchment_hydro_1024", kind="catchment", imax=1024, jmax=1024, n=40, spin=200,
         erosion=False, showers=False),
    # an ordinary erosion catchment under showers: the baseflow threshold
    # moves, so drainage areas are recomputed as the run goes on
    dict(name="catchment_600_showers", kind="catchment", imax=600, jmax=600, n=100, spin=150,
         erosion=True, showers=True),
    # the headline benchmark's grid in a steady storm
    dict(name="catchment_2000", kind="catchment", imax=2000, jmax=2000, n=20, spin=120,
         erosion=True, showers=False),
    # drop-in use, member by member
    dict(name="members_900x1400", kind="members", imax=900, jmax=1400, n=4),
    dict(name="sediment_512", kind="sediment", imax=512, jmax=512, n=4, spin=100),
    # the hillslope members, which a long run calls every day or ten
    dict(name="hillslope_200", kind="hillslope", imax=200, jmax=200, spin=100),
    # a catchment's set-up, which a storm also repeats when its baseflow moves
    dict(name="setup_1500", kind="setup", imax=1500, jmax=1500, plateaus=True),
    # independent catchments advanced together
    dict(name="ensemble_12", kind="ensemble", members=12, side_min=200, side_max=640, n=32,
         spin=100),
    # one evaluation of a calibration's objective and its gradient
    dict(name="gradient_384", kind="gradient", imax=384, jmax=384, n=160, spin=400, states=64),
]


def listed():
    return [dict(c) for c in _LISTED]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["reach", "flow", "catchment", "catchment", "members", "sediment",
                       "hillslope", "setup", "ensemble", "gradient"])
    if kind == "reach":
        return dict(kind=kind, imax=_side(rng, 60, 300), jmax=_side(rng, 24, 100),
                    n=_side(rng, 1, 60), spin=400)
    if kind == "flow":
        return dict(kind=kind, imax=_side(rng, 64, 2500), jmax=_side(rng, 64, 2500),
                    n=_side(rng, 2, 10), spin=40)
    if kind == "catchment":
        s = _side(rng, 96, 1500)
        return dict(kind=kind, imax=s, jmax=s, n=_side(rng, 8, 60), spin=100,
                    erosion=rng.random() < 0.7, showers=rng.random() < 0.5)
    if kind == "members":
        return dict(kind=kind, imax=_side(rng, 48, 2000), jmax=_side(rng, 48, 2000),
                    n=_side(rng, 1, 6))
    if kind == "sediment":
        s = _side(rng, 64, 800)
        return dict(kind=kind, imax=s, jmax=s, n=_side(rng, 1, 5), spin=60)
    if kind == "hillslope":
        return dict(kind=kind, imax=_side(rng, 40, 200), jmax=_side(rng, 40, 200), spin=60)
    if kind == "setup":
        return dict(kind=kind, imax=_side(rng, 64, 1800), jmax=_side(rng, 64, 1800),
                    plateaus=rng.random() < 0.5)
    if kind == "ensemble":
        lo = _side(rng, 64, 256)
        return dict(kind=kind, members=rng.randint(2, 12), side_min=lo, side_max=2 * lo,
                    n=_side(rng, 8, 40), spin=60)
    return dict(kind=kind, imax=_side(rng, 64, 400), jmax=_side(rng, 64, 400), n=_side(rng, 40, 160),
                spin=200, states=rng.choice([24, 64, 128]))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _spectral(imax, jmax, amp, g):
    """Real noise with the amplitude spectrum amp(k), scaled to [0, 1]."""
    ky = torch.fft.fftfreq(imax, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(jmax, device="cuda", dtype=torch.float64)[None, :]
    w = torch.randn(imax, jmax, generator=g, device="cuda", dtype=torch.float64)
    f = torch.fft.irfft2(torch.fft.rfft2(w) * amp(torch.sqrt(ky * ky + kx * kx)), s=(imax, jmax))
    f = f - f.min()
    return f / f.max()


def _fill(z, eps=1e-4):
    """Pits filled toward the bottom row with a gradient of eps per cell, so
    that every cell drains to that edge (a parallel relaxation from above)."""
    w = torch.full_like(z, 1e9)
    w[-1] = z[-1]
    while True:
        before = w
        for _ in range(48):
            low = -torch.nn.functional.max_pool2d(-w[None, None], 3, 1, 1)[0, 0]
            w = torch.minimum(w, torch.maximum(z, low + eps))
        if torch.equal(before, w):
            return w


def _dem(imax, jmax, relief, seed, tilt=0.5, fill=True):
    """Fractal surface (spectrum of synth.fractal_dem) tilted to the bottom
    edge, pit-filled if asked for, micrometre resolution."""
    f = _spectral(imax, jmax, lambda k: torch.where(k > 0, k.clamp(min=1e-9) ** -1.0, 0.0), _gen(seed))
    ramp = torch.linspace(1.0, 0.0, imax, device="cuda", dtype=torch.float64)[:, None]
    z = (1.0 - tilt) * f + tilt * ramp
    z = z - z.min()
    z = z * (relief / z.max()) + 10.0
    return torch.round(_fill(z) if fill else z, decimals=6)


def _roughness(imax, jmax, seed):
    """Manning's n, a smooth field in [0.03, 0.06]."""
    s = max(2.0, imax / 20.0)
    f = _spectral(imax, jmax, lambda k: torch.exp(-2.0 * (math.pi * s * k) ** 2), _gen(seed + 1000))
    return torch.round(0.03 + 0.03 * f, decimals=6).cpu().numpy()


def _film(imax, jmax, seed):
    """Wet ground at the start: 2 to 8 cm of water that has begun to gather."""
    f = _spectral(imax, jmax, lambda k: torch.where(k > 0, k.clamp(min=1e-9) ** -0.7, 0.0), _gen(seed + 2000))
    return torch.round(0.02 + 0.06 * f, decimals=6)


def _grains(p):
    sizes = synth.geometric_sizes(0.001, 0.256)
    synth.set_grains(p, sizes, synth.lognormal_dprop(sizes, 0.016))


def _case(case, seed):
    """(synth.Case, elevation tensor) of a single-catchment case."""
    imax, jmax, kind = case["imax"], case["jmax"], case["kind"]
    if kind == "reach":
        c = synth.reach_case(imax=imax, jmax=jmax, DX=10.0, seed=int(seed) % (1 << 31), hours=24)
        c.reach[0][:, 1] = np.float32(60.0) + np.float32(0.02) * np.arange(len(c.reach[0]), dtype=np.float32)
        return c, None
    if kind == "flow":
        z = _dem(imax, jmax, 150.0 * max(imax, jmax) / 8192 + 5.0, seed, fill=False)
        p = default_params(imax, jmax, 5.0)
        p.maxcycle, p.max_time_step, p.rain_data_time_step = 72, 300, 60
        p.hydro_only, p.M, p.edgeslope, p.spatially_complex_rainfall = 1, 0.005, 0.005, 1
        rain = np.full((p.maxcycle + 100, 1), 30.0, dtype=np.float32)
        return synth.Case("flow", p, z.cpu().numpy(), rain, water_init=_film(imax, jmax, seed).cpu().numpy()), z
    erosion = case.get("erosion", kind in ("sediment", "hillslope", "setup"))
    z = _dem(imax, jmax, 150.0 * max(imax, jmax) / 2000 + 20.0, seed)
    if case.get("plateaus"):
        # lowlands published in decimetres: many equal elevations
        z = torch.where(z < z.median(), torch.round(z, decimals=1), z)
    p = default_params(imax, jmax, 20.0)
    p.maxcycle, p.max_time_step, p.rain_data_time_step = 72, 300, 10
    p.M, p.spatially_var_mannings, p.edgeslope, p.MIN_Q = 0.01, 1, 0.005, 0.01
    p.hydro_only = 0 if erosion else 1
    p.wilcock, p.einstein, p.active = 0, 1, 0.2
    _grains(p)
    rows = p.maxcycle * 6 + 100
    rain = np.full((rows, 1), 40.0, dtype=np.float32)
    if case.get("showers"):
        rain[1::2] = 1.0
    film = _film(imax, jmax, seed)
    film = torch.where(film > 0.045, film, 0.0) if kind == "members" else film
    c = synth.Case(kind, p, z.cpu().numpy(), rain, mannings=_roughness(imax, jmax, seed),
                   water_init=film.cpu().numpy(),
                   flags=1 if erosion and imax == jmax else 0)
    return c, z


def _pinned(p):
    """A page-locked raster of the padded grid, as the output path takes."""
    return torch.empty((p.imax + 2, p.jmax + 2), dtype=torch.float64, pin_memory=True).numpy()


class State:
    """A model, the rasters its user writes and the buffers they go to."""

    def __init__(self, case, model, names):
        self.case, self.model = case, model
        self.rasters = {k: _pinned(model.p) for k in names}


def _member(case, seed, k):
    sides = np.random.default_rng([case["side_min"], k])  # the case's, not the seed's
    imax, jmax = (int(v) for v in sides.integers(case["side_min"], case["side_max"] + 1, 2))
    r = np.random.default_rng([int(seed), k])
    c, _ = _case(dict(kind="catchment", imax=imax, jmax=jmax, erosion=True), int(seed) * 64 + k)
    c.params.spatially_var_mannings, c.mannings, c.flags = 0, None, 0
    c.params.mannings = float(np.round(r.uniform(0.02, 0.08), 6))
    c.rain[:] = np.float32(r.uniform(5.0, 50.0))
    return c


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        models = [hc.Model(_member(case, seed, k)) for k in range(case["members"])]
        hc.run_ensemble(models, case["spin"])
        return [State(case, m, ("water_depth", "elev")) for m in models]
    c, _ = _case(case, seed)
    m = hc.Model(c)
    if kind == "members":
        m.scan_area()
    elif kind != "setup":
        # the record buffer too is there once a program has made its first run
        m.run(case["spin"])
    if kind == "gradient":
        s = State(case, m, ())
        s.target = np.linspace(0.5, 2.0, 64)
        return s
    if kind == "setup":
        return State(case, m, ("area",))
    return State(case, m, ("water_depth", "qx", "qy") if kind in ("flow", "members") or c.params.hydro_only
                 else ("water_depth", "elev", "Vsusptot"))


# ------------------------------------------------------------------ a pass
def _rasters(states):
    """Writes the rasters of the models, side by side."""
    waiting = [(s, s.model.snapshot_begin(k, a)) for s in states for k, a in s.rasters.items()]
    for s, h in waiting:
        s.model.snapshot_end(h)
    return [dict(s.rasters) for s in states]


def run(state):
    if isinstance(state, list):
        hc.run_ensemble([s.model for s in state], state[0].case["n"])
        return _rasters(state)
    m, case = state.model, state.case
    kind, out = case["kind"], {}
    if kind == "gradient":
        loss, gn, gr, _, ge = m.adj_gradient(case["n"], case["states"], state.target, elev=True)
        return {"loss": loss, "n": gn, "rain": gr, "elev": ge}
    if kind == "setup":
        m.prepare()
        out["points"] = m.scalars().totalinputpoints
    elif kind == "members":
        for _ in range(case["n"]):
            m.set_maximum_timestep()
            m.flow_route()
            m.depth_update()
            m.scan_area()
            m.water_flux_out()
        s = m.scalars()
        out["scalars"] = np.array([s.maxdepth, s.waterOut, s.time_step])
    elif kind == "sediment":
        t = []
        for _ in range(case["n"]):
            m.set_maximum_timestep()
            m.flow_route()
            m.depth_update()
            m.scan_area()
            t.append(m.erode(1.0))
            m.lateral_channel_erode()
            m.water_flux_out()
            m.in_channel_landsliding()
        out["tempbmax"] = np.array(t)
    elif kind == "hillslope":
        m.creep(m.p.creep_coeff)
        out["sweeps"] = m.global_landsliding()
        out["grain"], out["index"] = m.field("grain"), m.field("index")
    else:
        out["records"] = m.run(case["n"])
    out.update(_rasters([state])[0])
    return out


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: per iteration and cell the elevation, depth, discharges and
    Manning's n read and the depth and discharges written once, with erosion
    also the suspended load, its fluxes and the velocities; then the rasters.
    Operations: a face update is about 30, a cell's depth update and inputs
    10, an erosion step about 150 a cell."""
    kind = case["kind"]
    if kind == "ensemble":
        mean = 0.25 * (case["side_min"] + case["side_max"]) ** 2
        cells = case["members"] * mean
    else:
        cells = case["imax"] * case["jmax"]
    if kind == "setup":
        return {"bytes": 24.0 * cells, "flops": 60.0 * cells}
    if kind == "hillslope":  # elevations and records read and written, eight moves a cell
        return {"bytes": 2 * 8 * 13.0 * cells, "flops": 300.0 * cells}
    n = case["n"]
    sed = kind in ("reach", "sediment", "ensemble") or case.get("erosion", False)
    per_b = 64 + (48 if sed else 0)
    per_f = 70 + (150 if sed else 0)
    if kind == "gradient":  # forward, then the reverse pass over the same faces
        per_b, per_f = 3 * per_b, 4 * per_f
    return {"bytes": cells * (n * per_b + 24.0), "flops": float(cells * n * per_f)}


# ------------------------------------------------------------------ 64 bits
_G = 9.81


class _Plain:
    """The hydraulic iteration of a hydro-only run in plain float64 tensors."""

    def __init__(self, c, z):
        p = self.p = c.params
        pad = lambda a, v: torch.nn.functional.pad(torch.as_tensor(a, device="cuda"), (1, 1, 1, 1), value=v)
        self.e = pad(z, -9999.0)
        self.h = pad(c.water_init if c.water_init is not None else torch.zeros_like(z), 0.0)
        self.man = pad(c.mannings, 0.0) if c.mannings is not None else torch.full_like(self.e, p.mannings)
        self.qx, self.qy = torch.zeros_like(self.e), torch.zeros_like(self.e)
        self.mask = torch.zeros_like(self.e, dtype=torch.bool)
        self.inside = torch.zeros_like(self.mask)
        self.inside[1:-1, 1:-1] = True
        self.cycle, self.ts, self.maxdepth, self.counter = 0.0, 1.0, 10.0, 0
        self.win = self.wout = 0.0
        self.time_1, self.j_mean, self.baseflow = 0.0, 0.0, p.baseflow
        self.cells = float((p.imax - 1) * (p.jmax - 1))
        self.table = self._runoff(c.rain)
        self.old_j, self.new_j = self.table[0]
        i = torch.arange(p.imax + 2, device="cuda")[:, None]
        j = torch.arange(p.jmax + 2, device="cuda")[None, :]
        self.edge_x = torch.where(i == p.imax, p.edgeslope, torch.where(i <= 2, -p.edgeslope, math.nan))
        self.edge_y = torch.where(j == p.jmax, p.edgeslope, torch.where(j <= 2, -p.edgeslope, math.nan))
        self.records = []

    def _runoff(self, rain):
        p, rows, j, new, out = self.p, rain.shape[0], 1e-9, 0.0, []
        for t in range(p.maxcycle * 60 + 2000):
            k = int((1.0 if t == 0 else float(t)) / p.rain_data_time_step)
            v = float(rain[k, 0]) if k < rows else 0.0
            r = (v / 1000) / 3600
            old, j0, a = new, j, 60 / p.M
            if r > 0:
                j = r / (((r - j0) / j0) * math.exp(-r * a) + 1)
                new = math.log(((r - j0) + j0 * math.exp(r * a)) / r) / a
            else:
                j = j0 / (1 + j0 * a)
                new = math.log(1 + j0 * a) / a
            new = max(new, 0.0)
            out.append((old, new))
        return out

    def cfl(self):
        return self.p.courant_number * (self.p.DX / math.sqrt(_G * self.maxdepth))

    def set_maximum_timestep(self):
        diff = abs(self.win - self.wout)
        self.maxdepth = max(self.maxdepth, 0.1)
        if self.ts < self.cfl() or (diff > self.p.in_out_difference_allowed and self.ts > self.cfl()):
            self.ts = self.cfl()

    def dt(self):
        return min(self.ts, self.cfl())

    def _face(self, q, dim, edge, dt):
        p, DX = self.p, self.p.DX
        h0, e0 = self.h, self.e
        h1, e1 = torch.roll(h0, 1, dim), torch.roll(e0, 1, dim)
        open_ = self.mask & self.inside & (e0 > -9999) & (e1 > -9999) & ((h0 > 0) | (h1 > 0))
        a0, a1 = e0 + h0, e1 + h1
        hf = torch.maximum(a0, a1) - torch.maximum(e0, e1)
        flows = hf > p.hflow_threshold
        hs = torch.where(flows, hf, 1.0)
        slope = torch.where(torch.isnan(edge), (a1 - a0) / DX, edge)
        ghd = _G * hs * dt
        n = (q - ghd * slope) / (1 + ghd * (self.man * self.man) * q.abs() / (hs * hs * hs))
        lim = hs * (torch.sqrt(_G * hs) * p.froude_limit)
        n = torch.where((n / hs).abs() / torch.sqrt(_G * hs) > p.froude_limit, torch.copysign(lim, n), n)
        n = torch.where((n > 0) & (n * dt / DX > h0 / 4), h0 * DX / 5 / dt, n)
        n = torch.where((n < 0) & ((n * dt / DX).abs() > h1 / 4), -(h1 * DX / 5 / dt), n)
        return torch.where(open_, torch.where(flows, n, 0.0), q)

    def flow_route(self, dt):
        self.qx, self.qy = self._face(self.qx, 0, self.edge_x, dt), self._face(self.qy, 1, self.edge_y, dt)

    def depth_update(self, dt):
        d = dt * (torch.roll(self.qx, -1, 0) - self.qx + torch.roll(self.qy, -1, 1) - self.qy) / self.p.DX
        self.h = torch.where(self.mask, self.h + d, self.h)
        self.maxdepth = max(0.0, float(torch.where(self.mask, self.h, 0.0).max()))

    def scan_area(self):
        wet = (self.h > 0).double()[None, None]
        self.mask = (torch.nn.functional.max_pool2d(wet, 3, 1, 1)[0, 0] > 0) & self.inside

    def water_flux_out(self):
        thr, rim = self.p.water_depth_erosion_threshold, self.inside.clone()
        rim[2:-2, 2:-2] = False
        over = rim & (self.h > thr)
        off = float(torch.where(over, self.h - thr, 0.0).sum())
        self.h = torch.where(over, thr, self.h)
        self.wout = off * self.p.DX * self.p.DX / self.ts
        return off

    def points(self):
        """get_catchment_input_points for the present baseflow."""
        p = self.p
        q = self.area * self.baseflow * 3 * p.DX * p.DX
        self.cin = (q > p.MIN_Q) & (q < p.MIN_Q_MAXVAL)

    def iterate(self):
        p, a2 = self.p, self.p.DX * self.p.DX
        self.set_maximum_timestep()
        self.counter += 1
        self.cycle += self.ts / 60
        fdt, grid = self.dt(), bool(p.spatially_complex_rainfall)
        top = 0.2 / (p.imax * p.jmax * a2)
        if grid:
            amt = min(self.j_mean * fdt, p.ERODEFACTOR)
            self.win = self.cells * self.j_mean * a2 + self.cells * (amt / fdt) * a2
            where = self.inside.clone()
            where[-2], where[:, -2] = False, False
        else:
            self.win = self.j_mean * self.cells * a2
            where = self.cin
            amt = min(self.j_mean * self.cells / max(1, int(where.sum())) * fdt, p.ERODEFACTOR)
        jmm = self.new_j
        stepping = self.cycle >= self.time_1
        while stepping:
            self.time_1 += 1
            self.old_j, self.new_j = self.table[int(self.time_1)]
            if self.ts > p.max_time_step and (jmm if grid else self.new_j) > top:
                self.cycle = self.time_1 + p.max_time_step // 60
                self.ts = float(p.max_time_step)
            stepping = self.time_1 < self.cycle
        self.j_mean = self.old_j + (self.new_j - self.old_j) / 2 * (2 - (self.time_1 - self.cycle))
        moved = False
        if not grid:
            if self.j_mean >= self.baseflow:
                self.baseflow, moved = self.baseflow * 3, True
            if self.baseflow > self.j_mean * 3 and self.baseflow > 0.000001:
                self.baseflow, moved = self.j_mean * 1.25, True
        dt = self.dt()
        self.h = torch.where(where, self.h + amt, self.h)
        vin = amt * float(where.sum())
        self.flow_route(dt)
        edge = self._border(dt)
        self.depth_update(dt)
        deep, vol = self.maxdepth, math.nan
        if self.counter % p.scan_area_interval_iter == 0:
            vol = float(self.h[1:-1, 1:-1].sum()) * a2
            self.scan_area()
        off = self.water_flux_out()
        self.records.append([self.counter, self.cycle, self.ts, deep, self.wout, self.win, 1.0, 0.0, 0.0,
                             self.baseflow, vin * a2, off * a2, edge * a2, vol])
        if moved:
            self.points()

    def _border(self, dt):
        """Depth that crosses the faces between listed and unlisted cells."""
        m, tot = self.mask, 0.0
        for q, dim in ((self.qx, 0), (self.qy, 1)):
            tot += float(torch.where(m & ~torch.roll(m, -1, dim), torch.roll(q, -1, dim), 0.0).sum())
            tot -= float(torch.where(m & ~torch.roll(m, 1, dim), q, 0.0).sum())
        return dt * tot / self.p.DX


def _areas(e, p):
    """Drainage areas: every reached cell hands its area to its lower
    neighbours in proportion to the drops, from the highest cells down, one
    frontier of cells without pending higher neighbours at a time."""
    W, dev = p.jmax + 2, e.device
    inside = torch.zeros_like(e, dtype=torch.bool)
    inside[1:-1, 1:-1] = True
    cells = inside.flatten().nonzero().flatten()
    flat = e.flatten()
    lost = e.numel() - p.imax * p.jmax  # the padding puts this many cells past the sweep
    reached = torch.zeros(e.numel(), dtype=torch.bool, device=dev)
    order = torch.argsort(flat[cells], stable=True)
    reached[cells[order[: len(cells) - lost + 1]]] = True
    row, col = cells // W, cells % W
    dirs = [(0, -1), (1, -1), (1, 0), (1, 1), (0, 1), (-1, 1), (-1, 0), (-1, -1)]
    to, share = [], []
    for di, dj in dirs:
        t = (row + di).clamp(1, p.imax) * W + (col + dj).clamp(1, p.jmax)
        drop = torch.clamp(flat[cells] - flat[t], min=0.0) / (1.414 if di and dj else 1.0)
        to.append(t)
        share.append(drop)
    total = sum(share)
    share = [torch.where(total > 0, s / total.clamp(min=1e-300), 0.0) for s in share]
    slot = torch.zeros(e.numel(), dtype=torch.long, device=dev)
    slot[cells] = torch.arange(len(cells), device=dev)
    to, share = torch.stack(to, 1), torch.stack(share, 1)
    pend = torch.zeros(e.numel(), dtype=torch.int32, device=dev)
    pend.index_add_(0, to[share > 0], torch.ones(int((share > 0).sum()), dtype=torch.int32, device=dev))
    area = torch.zeros(e.numel(), dtype=torch.float64, device=dev)
    area[cells] = reached[cells].double()
    front = cells[pend[cells] == 0]
    while len(front):
        k = slot[front]
        s, t = share[k], to[k]
        on = s > 0
        gift = (area[front][:, None] * s) * reached[front][:, None]
        area.index_add_(0, t[on], torch.where(reached[t[on]], gift[on], 0.0))
        pend.index_add_(0, t[on], torch.full((int(on.sum()),), -1, dtype=torch.int32, device=dev))
        t = torch.unique(t[on])
        front = t[pend[t] == 0]
    return area.view_as(e)


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("flow", "members", "setup") and not (kind == "catchment" and not case["erosion"]):
        return None  # serial orders over grain records and strata, or thousands of reverse steps
    c, z = _case(case, seed)
    s = _Plain(c, z)
    p = c.params
    if kind == "setup":
        s.area = _areas(s.e, p)
        s.points()
        return {"points": float(max(1, int(s.cin.sum()))), "area": s.area.cpu().numpy()}
    if kind == "members":
        s.scan_area()
        for _ in range(case["n"]):
            s.set_maximum_timestep()
            s.flow_route(s.dt())
            s.depth_update(s.dt())
            s.scan_area()
            s.water_flux_out()
        out = {"scalars": np.array([s.maxdepth, s.wout, s.ts])}
    else:
        if not p.spatially_complex_rainfall:
            s.area = _areas(s.e, p)
            s.points()
        for _ in range(case["spin"]):
            s.iterate()
        s.records = []
        for _ in range(case["n"]):
            s.iterate()
        out = {"records": np.array(s.records)}
    out.update(water_depth=s.h.cpu().numpy(), qx=s.qx.cpu().numpy(), qy=s.qy.cpu().numpy())
    return out
