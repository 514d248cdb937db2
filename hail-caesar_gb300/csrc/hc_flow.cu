// Hydraulic part of one iteration: the driver's scalar logic (timestep,
// counters, water inputs, TOPMODEL), flow_route, depth_update, scan_area and
// water_flux_out.
//
// Reference: src/catchmentmodel/LSDCatchmentModel.cpp (line numbers below)
// and src/main.cpp:139-204.  Every expression that produces model state keeps
// the reference's operand order and roundings (the library is compiled with
// --fmad=false, so nothing is contracted into an FMA unless written so): the
// hydraulic state is bit-identical to the reference's serial build.

#include "hc_internal.cuh"

#include <math.h>
#include <algorithm>

namespace {

constexpr double kG = 9.81;  // gravity, LSDCatchmentModel.hpp:438

__device__ __forceinline__ double cfl_dt(const hc_params& p, double maxdepth) {
  // courant_friedrichs_lewy_condition :1884-1887
  return p.courant_number * (p.DX / sqrt(kG * (maxdepth)));
}

__device__ __forceinline__ double flow_dt_of(const hc_params& p, const hc_scalars& s) {
  // get_flow_timestep :1913-1923
  double f = s.time_step;
  double c = cfl_dt(p, s.maxdepth);
  if (f > c) f = c;
  return f;
}

// ---------------------------------------------------------------------------
// control: set_loop_cycle .. catchment_waterinputs (main.cpp:142-158), one
// warp.  Also decides which members run in this iteration.
//
// Every lane forms the scalars (the same values) and lane 0 stores them; lane
// z holds rain zone z, and lane n the grain fraction n + 1 of a reach's
// sediment input, whose sums run over the lanes in the reference's order.
// The kernel runs alone, once an iteration, so its time is latency: dependent
// FP64 operations (divisions on the integer pipe), loads, and the fetch of its
// instructions, which no other launch has left in the cache.  Hence one copy
// of each long operation and rolled loops (ncu, cold caches: 65 -> 16 us for a
// reach, one point and nine fractions, 18 -> 7.3 us without; one thread before).
// ---------------------------------------------------------------------------
static __device__ __noinline__ double cdiv(double a, double b) { return ddiv_rn(a, b); }
static __device__ __noinline__ double csqrt(double x) { return isqrt_rn(x); }

// (long long)x % m for a counter x >= 0, m >= 1
__device__ __forceinline__ bool divides(double x, int m) {
  if (x < 2147483647.0) return (unsigned)x % (unsigned)m == 0;
  return (long long)x % m == 0;
}

// sediment input of a reach point (:3310-3396): the fractions' amounts, one
// per lane, then the sums in fraction order
__device__ __noinline__ void reach_sediment(const hc_view& c, hc_dev* d, int n, int row,
                                            double time_step) {
  const hc_params& p = c.p;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const size_t cell = (size_t)p.inpoints[n][0] * c.W + p.inpoints[n][1];
  if (!(c.h[cell] > p.water_depth_erosion_threshold) || row >= c.reach_rows[n]) return;
  const int rdt = p.reach_input_data_timestep, div = p.div_inputs;
  const double a2 = p.DX * p.DX, secs = (double)(rdt * 60);
  const bool mine = lane < HC_NFRAC;  // fraction lane + 1, column lane + 5
  const float r = mine ? fabsf(c.reach[n][(size_t)row * c.reach_cols[n] + 5 + lane]) : 0.0f;
  const float q = r / div;  // float / int in the reference
  const double part = cdiv(cdiv((double)q, a2), secs) * time_step;
  double added_tot = 0, adding_factor = 1;
#pragma unroll 1
  for (int k = 0; k < HC_NFRAC; k++) added_tot += __shfl_sync(FULL, part, k);
  if (cdiv(added_tot, (double)p.number_of_points) > p.ERODEFACTOR * 0.75)
    adding_factor = cdiv(p.ERODEFACTOR * 0.75, cdiv(added_tot, (double)p.number_of_points));
  if (c.index[cell] == -9999) {  // addGS :3949, serial position: now
    __syncwarp();
    if (lane == 0) {
      d->grain_tot++;
      c.index[cell] = d->grain_tot;
      grain_record_init(c, cell, c.elev[cell], c.bed[cell]);
    }
    __syncwarp();
  }
  const double amt =
      cdiv(cdiv(cdiv(adding_factor * (double)r, (double)div), a2), secs) * time_step;
  if (mine && !p.isSuspended[lane + 1]) grain_at(c, cell, lane + 1) += amt;
  double e = c.elev[cell], vs = c.vs[cell];
#pragma unroll 1
  for (int k = 0; k < HC_NFRAC; k++) {
    const double a = __shfl_sync(FULL, amt, k);
    if (p.isSuspended[k + 1]) vs += a;
    else e += a;
  }
  __syncwarp();
  if (lane == 0) {
    c.elev[cell] = e;
    c.vs[cell] = vs;
  }
  __syncwarp();
}

__global__ void __launch_bounds__(32) k_control(const hc_view c, hc_dev* d, hc_iter_handles hh) {
  const hc_params& p = c.p;
  hc_scalars& s = d->s;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool l0 = lane == 0;
  int pause = d->pause;
  const int64_t budget = d->budget;
  if (pause || budget <= 0) {
    // skipped iteration: every gated kernel of it returns at once; the
    // switches of the iteration that paused stay as they are, for the host
    // to finish that iteration
    __syncwarp();
    if (l0) {
      if (budget <= 0) d->pause = pause | HC_PAUSE_BUDGET;
      d->it_active = 0;
      if (hh.has) {  // no step of it runs, and no iteration follows
        cudaGraphSetConditional(hh.loop, 0u);
        cudaGraphSetConditional(hh.scan, 0u);
        if (!p.hydro_only)
          for (const cudaGraphConditionalHandle h :
               {hh.erode, hh.retry2, hh.retry3, hh.retry4, hh.erode_fin, hh.slide})
            cudaGraphSetConditional(h, 0u);
      }
    }
    return;
  }
  // everything the scalar logic reads, before the first store
  double time_step = s.time_step, maxdepth = s.maxdepth, cycle = s.cycle, time_1 = s.time_1;
  double vin = d->vin_step, baseflow = s.baseflow;
  const double counter = s.counter + 1, erode_call = s.erode_call, erode_mult = s.erode_mult;
  const double previous = cycle;
  const double diff = fabs(s.waterinput - s.waterOut);  // set_inputoutput_diff :1879
  const int rf = p.rfnum;
  const bool zone = lane <= rf;  // rf <= HC_MAX_RF < 32
  double jm = zone ? s.j_mean[lane] : 0.0, oldj = zone ? s.old_j_mean[lane] : 0.0,
         newj = zone ? s.new_j_mean[lane] : 0.0;
  const double cells = zone ? s.nActualGridCells[lane] : 0.0,
               points = zone ? s.catchment_input_counter[lane] : 1.0;
  int err = 0;

  if (maxdepth <= 0.1) maxdepth = 0.1;                    // set_maximum_timestep :1890
  // courant_friedrichs_lewy_condition :1884: the depth does not change here
  const double cfl = p.courant_number * cdiv(p.DX, csqrt(kG * maxdepth));
  if (time_step < cfl) time_step = cfl;
  if (diff > p.in_out_difference_allowed && time_step > cfl) time_step = cfl;
  // adjoint runs record the time steps, or impose recorded ones
  const bool adj = c.adj_dt && d->adj_mode && d->adj_i < d->adj_n;
  const bool impose = adj && d->adj_mode == 2;
  double* arec = adj ? c.adj_dt + (size_t)d->adj_i * HC_ADJ_REC : nullptr;
  if (impose) time_step = arec[0];
  else if (adj && l0) arec[0] = time_step;
  cycle += cdiv(time_step, 60.0);                         // increment_counters :1925
  // get_flow_timestep :1913-1923
  const double fdt = time_step > cfl ? cfl : time_step;

  const double DX = p.DX;
  // reach_water_and_sediment_input :3301-3452
  if (p.reach_mode) {
    const int rdt = p.reach_input_data_timestep;
    const int row = (int)cdiv(cycle, (double)rdt);
    if (!p.hydro_only)
#pragma unroll 1
      for (int n = 0; n <= p.number_of_points - 1; n++) reach_sediment(c, d, n, row, time_step);
#pragma unroll 1
    for (int n = 0; n <= p.number_of_points - 1; n++) {
      const int x = p.inpoints[n][0], y = p.inpoints[n][1];
      const size_t cell = (size_t)x * c.W + y;
      if (row + 1 >= c.reach_rows[n]) {
        err = 102;
        pause |= HC_PAUSE_ERROR;
        continue;
      }
      double i1 = c.reach[n][(size_t)row * c.reach_cols[n] + 1];
      double i2 = c.reach[n][(size_t)(row + 1) * c.reach_cols[n] + 1];
      double prop = cdiv(((row + 1) * rdt) - cycle, (double)rdt);
      double input = i1 + ((i2 - i1) * (1 - prop));
      const double add = cdiv(cdiv(input, (double)p.div_inputs), DX * DX) * fdt;
      const double h = c.h[cell] + add;
      __syncwarp();
      if (l0) c.h[cell] = h;
      __syncwarp();
      if (x >= 1 && x <= c.imax && y >= 1 && y <= c.jmax) vin += add;
    }
  }

  // catchment_waterinputs :2027 -> catchment_water_input_and_hydrology :3455
  double waterinput = 0, fdt2 = fdt;
  if (impose) fdt2 = arec[1];
  else if (adj && l0) arec[1] = fdt2;
  const bool grid = p.spatially_complex_rainfall != 0;
  const int z0 = grid ? 0 : 1;  // the first zone that takes part
  if (zone) d->j_mean_in[lane] = jm;
  double amt, jmm = 0;
  if (grid) {
    // catchment_water_input_and_hydrology(flow_timestep, runoff) :3544-3607.
    // A cell's runoff recurrence (runoffGrid::calculate_runoff) depends only
    // on its rain, i.e. on its rain state: the zone (zones 1 .. rfnum-1, or
    // column 0 for all cells when rfnum is 1) or none (state 0: zone rfnum
    // and others get no rain, rainGrid::create, LSDRainfallRunoff.cpp:33-66),
    // so every cell of a state holds the
    // same values; the host tabulates them per state with glibc.
    amt = jm * fdt2;
    if (amt > p.ERODEFACTOR) amt = p.ERODEFACTOR;
    // the two sums over the cells (:3547-3571), formed state by state, and
    // the ledger (k_runoff_inputs adds amt to each computed cell of state z);
    // new_jmeanmax (:3575-3586) over the states that hold a computed cell
    const double got = cdiv(amt, fdt2);
#pragma unroll 1
    for (int z = 0; z <= rf; z++)
      waterinput += c.runoff_count[z] * (__shfl_sync(FULL, jm, z) * DX * DX);
#pragma unroll 1
    for (int z = 0; z <= rf; z++) {
      const double n = c.runoff_count[z];
      waterinput += n * (__shfl_sync(FULL, got, z) * DX * DX);
      const double a = __shfl_sync(FULL, amt, z), v = __shfl_sync(FULL, newj, z);
      if (n > 0) vin += n * a;
      if (((c.runoff_present >> z) & 1u) && v > jmm) jmm = v;
    }
  } else {
    const double flow = jm * cells;
#pragma unroll 1
    for (int i = 1; i <= rf; i++) waterinput += __shfl_sync(FULL, flow, i) * DX * DX;
    // what each input point of a zone receives (:3463-3477), the same for all
    // points of the zone
    amt = cdiv(flow, points) * fdt2;
    if (amt > p.ERODEFACTOR) amt = p.ERODEFACTOR;
    if (arec && lane <= HC_MAX_RF) arec[3 + lane] = zone ? jm : 0.0;
  }
  if (zone) d->input_amt[lane] = amt;
  if (cycle >= time_1) {
    do {
      time_1++;
      // topmodel_runoff(time_1) :3649-3715: the recurrence depends only on
      // the rain table, so the host evaluates it once (host_topmodel_table)
      // and the device steps through the rows
      const int t = (int)time_1;
      if (t < 0 || t >= c.topm_rows) {
        err = 101;
        pause |= HC_PAUSE_ERROR;
      } else if (zone && lane >= z0) {
        const double* row = c.topm + (size_t)t * 2 * (rf + 1);
        oldj = row[lane];
        newj = row[(rf + 1) + lane];
      }
      if (time_step > p.max_time_step) {
        if (!grid) {
          jmm = 0;
#pragma unroll 1
          for (int n = 1; n <= rf; n++) {
            const double v = __shfl_sync(FULL, newj, n);
            if (v > jmm) jmm = v;
          }
        }
        if (jmm > cdiv(0.2, (unsigned)p.imax * (unsigned)p.jmax * DX * DX)) {
          cycle = time_1 + (p.max_time_step / 60);
          time_step = p.max_time_step;
        }
      }
    } while (time_1 < cycle && !(pause & HC_PAUSE_ERROR));
  }
  // calchydrograph :3718 and (time, runoff) :3728-3740 (x / 2 == x * 0.5)
  if (zone && lane >= z0) jm = oldj + (((newj - oldj) * 0.5) * (2 - (time_1 - cycle)));
  bool recalc = false;  // no drainage area or input points with grid runoff
  if (!grid) {
    if (arec && l0) {
      arec[HC_ADJ_T1] = time_1;
      arec[HC_ADJ_T1 + 1] = cycle;
    }
    double jmeanmax = 0;
#pragma unroll 1
    for (int n = 1; n <= rf; n++) {
      const double v = __shfl_sync(FULL, jm, n);
      if (v > jmeanmax) jmeanmax = v;
    }
    if (jmeanmax >= baseflow) {
      baseflow = baseflow * 3;
      recalc = true;
    }
    if (baseflow > (jmeanmax * 3) && baseflow > 0.000001) {
      baseflow = jmeanmax * 1.25;
      recalc = true;
    }
    // The drainage area and the input-point list are recomputed before the
    // next iteration (the host sorts the elevations, hc_drain.cu does the
    // rest), from the elevations as they are now (k_depth_update copies
    // them before the iteration's erosion); the
    // reference, too, applies the new list from the next iteration on.
    if (recalc) pause |= HC_PAUSE_DRAINAGE;
  }
  if (zone && lane >= z0) {
    s.j_mean[lane] = jm;
    s.old_j_mean[lane] = oldj;
    s.new_j_mean[lane] = newj;
  }

  double flow_timestep = time_step > cfl ? cfl : time_step;
  if (impose) flow_timestep = arec[2];
  const bool scan = divides(counter, p.scan_area_interval_iter);
  const bool erode = !p.hydro_only && counter >= erode_call;
  const bool slide = !p.hydro_only && divides(counter, p.in_channel_landslide_iter_interval);
  if (!l0) return;
  if (adj) {
    if (!impose) arec[2] = flow_timestep;
    d->adj_i++;
  }
  d->budget = budget - 1;
  d->it_active = 1;
  d->rest_active = 1;
  d->erode_passes = 0;
  d->do_lateral = 0;
  d->do_drain = recalc;
  d->do_scan = scan;
  d->do_erode = erode;
  d->erode_retry = erode;
  d->do_slide = slide;
  if (pause) d->pause = pause;
  if (err) d->err_code = err;
  d->input_dt = fdt2;
  d->vin_step = vin;
  s.previous = previous;
  s.input_output_difference = diff;
  s.maxdepth = maxdepth;
  s.counter = counter;
  s.cycle = cycle;
  s.time_1 = time_1;
  s.waterinput = waterinput;
  s.baseflow = baseflow;
  s.flow_timestep = flow_timestep;
  if (erode) {
    // erode()'s start (:4219; k_erode_begin for a direct call): the
    // kernels between here and the erosion block read flow_timestep, set
    // above, not time_step
    time_step = time_step * 1.5;
    d->mult = erode_mult;
    d->tempbmax_bits = 0;
  }
  s.time_step = time_step;
  if (hh.has) {
    // kernels inside the bodies enabled here: scan 3, erosion 5 + 7, slide_3 4
    d->body_kernels += (scan ? 3 : 0) + (erode ? 12 : 0) + (slide ? 4 : 0);
    // the loop goes on when water_flux_out says so; an iteration that stops
    // before it ends the loop
    cudaGraphSetConditional(hh.loop, 0u);
    cudaGraphSetConditional(hh.scan, scan ? 1u : 0u);
    if (!p.hydro_only) {
      cudaGraphSetConditional(hh.retry2, 0u);
      cudaGraphSetConditional(hh.retry3, 0u);
      cudaGraphSetConditional(hh.retry4, 0u);
      cudaGraphSetConditional(hh.erode, erode ? 1u : 0u);
      cudaGraphSetConditional(hh.erode_fin, erode ? 1u : 0u);
      cudaGraphSetConditional(hh.slide, slide ? 1u : 0u);
    }
  }
}

// catchment input points (:3463-3477): one thread per point
// The ledger counts what lands on the grid (rows 1..imax, columns 1..jmax):
// with no point found the reference still visits one (totalinputpoints
// forced to 1, :3765), whose coordinates may be stale or the padding corner.
__global__ void k_inputs(const hc_view c, hc_dev* d) {
  if (!d->it_active) return;
  const hc_scalars& s = d->s;
  const int total = (int)s.totalinputpoints;
  double added = 0;
  for (int z = 1 + blockIdx.x * blockDim.x + threadIdx.x; z <= total;
       z += gridDim.x * blockDim.x) {
    const int i = c.cin_x[z], j = c.cin_y[z];
    const size_t cell = (size_t)i * c.W + j;
    const double a = d->input_amt[c.rfarea[cell]];
    c.h[cell] += a;
    if (i >= 1 && i <= c.imax && j >= 1 && j <= c.jmax) added += a;
  }
  double tot;
  if (grid_sum(added, c.vpart, &d->sum_done, &tot)) d->vin_step += tot;
}

// Distributed runoff (:3560-3573): every computed cell (rows 1 .. imax-1,
// columns 1 .. jmax-1, elevation above no-data) takes its state's amount.
__global__ void k_runoff_inputs(const hc_view c, hc_dev* d) {
  if (!d->it_active) return;
  const int j = 1 + blockIdx.x * blockDim.x + threadIdx.x;
  const int i = 1 + blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= c.imax || j >= c.jmax) return;
  const size_t cell = (size_t)i * c.W + j;
  if (!(dkey(c.elev[cell]) > kNoDataKey)) return;  // j_mean stays 0 there
  const int rf = c.p.rfnum;
  int z = 1;
  if (rf != 1) {
    const int r = c.rfarea[cell];
    z = (r >= 1 && r <= rf - 1) ? r : 0;
  }
  c.h[cell] += d->input_amt[z];
}

__global__ void k_flow_dt(const hc_view c, hc_dev* d) {
  d->s.flow_timestep = flow_dt_of(c.p, d->s);
  d->it_active = 1;
  d->rest_active = 1;
}

// ---------------------------------------------------------------------------
// flow_route :3063-3247.  One thread per cell; cells outside the wet mask keep
// their discharges (the reference does not visit them).
// ---------------------------------------------------------------------------
// The limiters' FP64 tests, for the faces whose float estimates cannot
// decide them: out of line, so that their FP64 instructions (a hardware
// division among them) issue only where they run.
static __device__ __noinline__ bool depth_exceeds(double qn, double dt, double DX, double h) {
  return fabs(qn * dt / DX) > (h / 4);  // :3138, :3144, :3218, :3219
}
static __device__ __noinline__ bool sed_exceeds(double qs, double dt, double v, double DX) {
  return fabs(qs * dt) > (v * DX) / 4;  // :3163, :3169
}

// The limiters' replacement values and the Froude test's exact form, out of
// line as well: they run for few faces, and inlined, their integer-pipe
// divisions and square roots would double the kernel's code, whose
// instruction fetches stall the warps more than anything else.
// (x * DX / 5) / dt, the depth and sediment limits' value (:3140, :3165);
// the divisors 5 (host) and dt (once per block) come prepared
static __device__ __noinline__ double limit_value(double x, const hc_view& c,
                                                  const hc_divisor* dtd) {
  return ddiv_by(ddiv_by(x * c.p.DX, c.fived), *dtd);
}
// |q/hflow| / sqrt(g hflow) > froude_limit, exactly (:3124); gh = g hflow
static __device__ __noinline__ bool froude_exceeds(double qoh, double gh, double fl) {
  return dgt(ddiv_rn(fabs(qoh), isqrt_rn(gh)), fl);
}
// hflow * (sqrt(g hflow) * froude_limit), the Froude limit's value (:3127)
static __device__ __noinline__ double froude_value(double hflow, double gh, double fl) {
  return hflow * (isqrt_rn(gh) * fl);
}

// Three-way test of A > B from float estimates a, b, each within a relative
// 2^-18 of A, B (or flushed to 0 below 2^-126, inf above the float range):
// +1 surely greater, -1 surely not, 0 too close to call (the caller then
// evaluates the reference's FP64 expression).  Tiny pairs, where a flushed
// estimate carries no relative bound, are never decided here.
__device__ __forceinline__ int decide_gt(float a, float b) {
  const float m = 1e-4f * (fabsf(a) + fabsf(b));
  if (!(m >= 1e-34f) || !(m < 1e30f)) return 0;
  const float dd = a - b;
  if (dd > m) return 1;
  if (dd < -m) return -1;
  return 0;
}

// One face of the inertial scheme (:3096-3191 / :3193-3242).  e0,h0: this
// cell; e1,h1: the upstream neighbour (x-1 for qx, y-1 for qy); a0, a1 the
// water surfaces e+h.  `edge_slope` is 0 for interior faces, +1 / -1 where
// the reference replaces the slope by +/-edgeslope.
//
// The FP64 pipe (1.2 TFLOP/s on GB300) bounds this kernel, and compares
// occupy it as much as arithmetic does.  So every test runs on the integer
// pipe (dgt0, dlt, ...: IEEE results for non-NaN operands), and the limiter
// tests, which only pick a branch, are first decided on float estimates; the
// reference's FP64 expression is evaluated only when the estimate is within
// 1e-4 of the threshold.  The branch taken - and so the result - is always
// the reference's.
// The face past the hflow gate: hflow (> hflow_threshold) and dA = a1 - a0
// (the surface difference) as the gate formed them.
// The face update's divisions: inline, or (kCall) through one out-of-line
// copy, which keeps the kernel's code small (its instruction fetches stall
// the warps) at the cost of a call per division; a launch-shape choice of
// the face-compacted kernel.
static __device__ __noinline__ double ddiv_rn_call(double a, double b) { return ddiv_rn(a, b); }
template <bool kCall>
__device__ __forceinline__ double fdiv(double a, double b) {
  if (kCall) return ddiv_rn_call(a, b);
  return ddiv_rn(a, b);
}

template <bool kSusp, bool kVel, bool kCall = false>
__device__ __forceinline__ void inertial_face_core(double& q, double& qs, double& vel_out,
                                                   int& vdir, double hflow, double dA, double h0,
                                                   double h1, double v0, double v1, double c0,
                                                   double nn, double dt, int edge_slope,
                                                   const hc_view& c, const hc_divisor* dtd) {
  const hc_params& p = c.p;
  const double DX = p.DX;
  vdir = 0;
  double slope = ddiv_by(dA, c.dxd);
  if (edge_slope == 1) slope = p.edgeslope;
  if (edge_slope == -1) slope = zero_minus(p.edgeslope);
  const double gh = kG * hflow;
  const double ghd = gh * dt;
  // the numerator once for both branches (a branch apiece would issue its
  // FP64 instructions twice in a warp that holds both)
  double qn = q - (ghd * slope);
  // q = 0: (0 - ghd*slope) / (1 + (ghd*nn*0)/h^3) = (0 - ghd*slope) / 1
  if (!deq0(q)) {
    const double aq = bits_d(dbits(q) & 0x7fffffffffffffffLL);  // fabs
    qn = fdiv<kCall>(qn, 1 + fdiv<kCall>(ghd * nn * aq, icube_rn(hflow)));
  }
  const float hf = approx_abs_f(hflow);
  const float dtf = approx_abs_f(dt);
  // q/hflow: exact when the face velocity is kept (erosion runs), where it
  // also serves the Froude test
  double qoh = 0;
  bool qoh_valid = false;
  // Froude limit: |q/hflow| / sqrt(g*hflow) > froude_limit
  if (!deq0(qn)) {
    float fr;
    if (kVel) {
      qoh = fdiv<kCall>(qn, hflow);
      qoh_valid = true;
      fr = approx_abs_f(qoh) / sqrtf(9.81f * hf);
    } else {
      fr = approx_abs_f(qn) / (hf * sqrtf(9.81f * hf));
    }
    int t = decide_gt(fr, c.flf);
    if (t == 0) {
      if (!qoh_valid) qoh = fdiv<kCall>(qn, hflow);
      t = froude_exceeds(qoh, gh, p.froude_limit) ? 1 : -1;
    }
    if (t > 0) {
      const double lim = froude_value(hflow, gh, p.froude_limit);
      qn = dgt0(qn) ? lim : zero_minus(lim);
      qoh_valid = false;
    }
  }
  // depth limit: |q*dt/DX| > (depth of the giving cell)/4.  The reference
  // tests q > 0, then q < 0 on what that left; a limited q keeps its sign
  // when its depth is not negative, so one test of the giving cell serves
  // both, and a warp issues the limit's operations once.  Only a negative
  // depth lets the first test's result reach the second.
  auto depth_limit = [&](double h, bool pos) {
    int t = decide_gt(approx_abs_f(qn) * dtf / c.DXf, approx_f(h) * 0.25f);
    if (t == 0) t = depth_exceeds(qn, dt, DX, h) ? 1 : -1;
    if (t > 0) {
      const double lim = limit_value(h, c, dtd);
      qn = pos ? lim : zero_minus(lim);
      qoh_valid = false;
    }
  };
  if (!deq0(qn)) {
    const bool pos = dgt0(qn);
    depth_limit(pos ? h0 : h1, pos);
    if (pos && dlt0(qn)) depth_limit(h1, false);
  }
  const bool qpos = dgt0(qn), qneg = dlt0(qn);
  if (kSusp) {
    // qs = q * (V/h) of the giving cell; V = 0 gives 0 * q (a signed zero)
    // (one product for both signs: h1 > 0 here, as h0 above)
    if (qpos || qneg) qs = qn * (qpos ? c0 : (deq0(v1) ? v1 : fdiv<kCall>(v1, h1)));
    // qs*dt > V*DX/4 (giving cell) caps the sediment flux, the two signs'
    // tests as one like the depth limit's
    auto sed_limit = [&](double v, bool pos) {
      int t = decide_gt(approx_abs_f(qs) * dtf, approx_f(v) * c.DXf * 0.25f);
      if (t == 0) t = sed_exceeds(qs, dt, v, DX) ? 1 : -1;
      if (t > 0) {
        const double lim = limit_value(v, c, dtd);
        qs = pos ? lim : zero_minus(lim);
      }
    };
    if (!deq0(qs)) {
      const bool pos = dgt0(qs);
      sed_limit(pos ? v0 : v1, pos);
      if (pos && dlt0(qs)) sed_limit(v1, false);
    }
  }
  if (kVel) {
    // (0 - q)/hflow = -(q/hflow) exactly: division rounds symmetrically
    if ((qpos || qneg) && !qoh_valid) qoh = fdiv<kCall>(qn, hflow);
    if (qpos) {
      vel_out = qoh;
      vdir = 1;
    }
    if (qneg) {
      vel_out = zero_minus(qoh);
      vdir = -1;
    }
  }
  q = qn;
}

template <bool kSusp, bool kVel>
__device__ __forceinline__ void inertial_face(double& q, double& qs, double& vel_out, int& vdir,
                                              double e0, double h0, double a0, double e1,
                                              double h1, double a1, double v0, double v1,
                                              double c0, double nn, double dt, int edge_slope,
                                              const hc_view& c, const hc_divisor* dtd) {
  vdir = 0;
  double hflow = xmax_d(a0, a1) - xmax_d(e1, e0);
  if (!(xkey(hflow) > c.thr_xkey)) {  // hflow > hflow_threshold
    q = 0;
    qs = 0;
    return;
  }
  inertial_face_core<kSusp, kVel>(q, qs, vel_out, vdir, hflow, a1 - a0, h0, h1, v0, v1, c0, nn,
                                  dt, edge_slope, c, dtd);
}

template <bool kSed>
__device__ __forceinline__ void flow_cell(const hc_view& c, const hc_dev* __restrict__ d,
                                          size_t cell, const hc_divisor* dtd) {
  const size_t W = c.W, N2 = c.N2;
  const int i = (int)(cell / W), j = (int)(cell % W);
  const double e0 = c.elev[cell];
  // e > -9999 (no-data and below are skipped)
  auto above_nodata = [](double e) { return xkey(e) > kNoDataXKey; };
  if (!above_nodata(e0)) return;
  const hc_params& p = c.p;
  const double dt = d->s.flow_timestep;
  const double nn = p.spatially_var_mannings ? c.man2[cell] : c.nn;  // n * n
  const bool susp = kSed && p.isSuspended[1] != 0;
  const double h0 = c.h[cell];
  const double a0 = e0 + h0;
  const double v0 = susp ? c.vs[cell] : 0.0;
  // V/h of this cell, shared by both faces.  Only used where q > 0 after
  // the depth limit, which implies h > 0, so a zero V gives V itself (with
  // its sign) without the division.
  const double c0 = (susp && !deq0(v0)) ? ddiv_rn(v0, h0) : v0;
  const bool wet0 = dgt0(h0);
  // x face (rows i-1, i)
  {
    const size_t up = cell - W;
    const double h1 = c.h[up], e1 = c.elev[up];
    if ((wet0 || dgt0(h1)) && above_nodata(e1)) {
      double q = c.qx[cell], qs = kSed ? c.qxs[cell] : 0.0, vel = 0;
      int vdir;
      const int es = (i == c.imax) ? 1 : ((i <= 2) ? -1 : 0);
      if (susp)
        inertial_face<true, kSed>(q, qs, vel, vdir, e0, h0, a0, e1, h1, e1 + h1, v0, c.vs[up],
                                  c0, nn, dt, es, c, dtd);
      else
        inertial_face<false, kSed>(q, qs, vel, vdir, e0, h0, a0, e1, h1, e1 + h1, v0, 0.0, c0,
                                   nn, dt, es, c, dtd);
      c.qx[cell] = q;
      if (kSed) {
        c.qxs[cell] = qs;
        if (vdir == 1) c.vd[3 * N2 + cell] = vel;  // vel_dir[x][y][7]
        if (vdir == -1) c.vd[1 * N2 + up] = vel;   // vel_dir[x-1][y][3]
      }
    }
  }
  // y face (columns j-1, j).  The reference takes max(e0, e1) with the
  // operands the other way round (:3197-3198); for ordered values max is
  // symmetric, so one face routine serves both.
  {
    const size_t lf = cell - 1;
    const double h1 = c.h[lf], e1 = c.elev[lf];
    if ((wet0 || dgt0(h1)) && above_nodata(e1)) {
      double q = c.qy[cell], qs = kSed ? c.qys[cell] : 0.0, vel = 0;
      int vdir;
      const int es = (j == c.jmax) ? 1 : ((j <= 2) ? -1 : 0);
      if (susp)
        inertial_face<true, kSed>(q, qs, vel, vdir, e0, h0, a0, e1, h1, e1 + h1, v0, c.vs[lf],
                                  c0, nn, dt, es, c, dtd);
      else
        inertial_face<false, kSed>(q, qs, vel, vdir, e0, h0, a0, e1, h1, e1 + h1, v0, 0.0, c0,
                                   nn, dt, es, c, dtd);
      c.qy[cell] = q;
      if (kSed) {
        c.qys[cell] = qs;
        if (vdir == 1) c.vd[0 * N2 + cell] = vel;  // vel_dir[x][y][1]
        if (vdir == -1) c.vd[2 * N2 + lf] = vel;   // vel_dir[x][y-1][5]
      }
    }
  }
}

// One thread per wet cell, grid-stride over the wet list: cells outside the
// mask are never touched, as in the reference's down_scan loops.  MINB,
// the blocks of 256 a multiprocessor must hold, sets the register budget
// (3: 80 registers, 4: 64, 5: 48, 6: 40; the autotuner picks one).
template <bool kSed, int MINB>
__global__ void __launch_bounds__(256, MINB) k_flow_route(const hc_view c,
                                                          const hc_dev* __restrict__ d, int gated) {
  if (gated && !d->it_active) return;
  __shared__ hc_divisor dtd;  // dt as a divisor, for the limits
  if (threadIdx.x == 0) dtd = ddiv_prep(d->s.flow_timestep);
  __syncthreads();
  const int n = d->wet_count;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
    flow_cell<kSed>(c, d, (size_t)c.wet[k], &dtd);
}

// Face-compacted flow_route.  In a storm about half the listed cells are dry
// and two faces in three fail the gate (both cells dry) or the hflow
// threshold, so a warp evaluating its 32 cells' faces in turn issues the
// FP64 instructions of a face with a third of its lanes.  Here each lane
// first classifies its cell's two faces (the gate and hflow: two additions
// and compares) and writes q = qs = 0 for gated faces below the threshold;
// the faces that go on are queued in the warp's shared-memory queue (cell,
// face, hflow, a1 - a0), and whenever 32 are queued the warp evaluates them
// together, one per lane, the rest carried over to the next cells.  Every
// face is evaluated from the same inputs by the same expressions as in
// k_flow_route, so the results are the same bit for bit.
constexpr int kFaceQ = 96;  // queue entries per warp: < 32 carried + 64 new

template <bool kSed, bool kCall>
__device__ __forceinline__ void face_work(const hc_view& c, const hc_divisor* dtd,
                                          uint32_t f, double hflow, double dA, double dt) {
  const size_t W = c.W, N2 = c.N2;
  const size_t cell = f >> 1;
  const bool yface = f & 1u;
  const size_t nb = yface ? cell - 1 : cell - W;
  const int i = (int)(cell / W), j = (int)(cell - (size_t)i * W);
  const hc_params& p = c.p;
  const double nn = p.spatially_var_mannings ? c.man2[cell] : c.nn;  // n * n
  const bool susp = kSed && p.isSuspended[1] != 0;
  const double h0 = c.h[cell], h1 = c.h[nb];
  const double v0 = susp ? c.vs[cell] : 0.0;
  const double c0 = (susp && !deq0(v0)) ? fdiv<kCall>(v0, h0) : v0;
  double* qa = yface ? c.qy : c.qx;
  double* qsa = yface ? c.qys : c.qxs;
  double q = qa[cell], qs = kSed ? qsa[cell] : 0.0, vel = 0;
  int vdir;
  const int es = yface ? ((j == c.jmax) ? 1 : ((j <= 2) ? -1 : 0))
                       : ((i == c.imax) ? 1 : ((i <= 2) ? -1 : 0));
  if (susp)
    inertial_face_core<true, kSed, kCall>(q, qs, vel, vdir, hflow, dA, h0, h1, v0, c.vs[nb], c0, nn,
                                          dt, es, c, dtd);
  else
    inertial_face_core<false, kSed, kCall>(q, qs, vel, vdir, hflow, dA, h0, h1, v0, 0.0, c0, nn, dt,
                                           es, c, dtd);
  qa[cell] = q;
  if (kSed) {
    qsa[cell] = qs;
    // x face: vel_dir[x][y][7] / vel_dir[x-1][y][3]; y face: [x][y][1] / [x][y-1][5]
    if (vdir == 1) c.vd[(yface ? 0 : 3) * N2 + cell] = vel;
    if (vdir == -1) c.vd[(yface ? 2 : 1) * N2 + nb] = vel;
  }
}

template <bool kSed, int MINB, bool kCall = false>
__global__ void __launch_bounds__(256, MINB) k_flow_route_q(const hc_view c,
                                                            const hc_dev* __restrict__ d,
                                                            int gated) {
  __shared__ uint32_t qf[8][kFaceQ];
  __shared__ double qh[8][kFaceQ], qa[8][kFaceQ];
  __shared__ hc_divisor dtd;  // dt as a divisor, for the limits
  if (gated && !d->it_active) return;
  if (threadIdx.x == 0) dtd = ddiv_prep(d->s.flow_timestep);
  __syncthreads();
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* Q = qf[warp];
  double* HF = qh[warp];
  double* DA = qa[warp];
  const int n = d->wet_count;
  const double dt = d->s.flow_timestep;
  const size_t W = c.W;
  const int warps = gridDim.x * (blockDim.x >> 5);
  int qn = 0;  // the same on every lane
  // the list entry of the warp's next turn is fetched a turn ahead (its
  // cell's loads then need not wait for it)
  int base = (blockIdx.x * (blockDim.x >> 5) + warp) * 32;
  uint32_t next = (base + lane < n) ? (uint32_t)c.wet[base + lane] : 0u;
  for (; base < n; base += warps * 32) {
    const int k = base + lane;
    bool fx = false, fy = false;
    double hx = 0, hy = 0, ax = 0, ay = 0;
    uint32_t cell = 0;
    const uint32_t mine = next;
    if (k + warps * 32 < n) next = (uint32_t)c.wet[k + warps * 32];
    if (k < n) {
      cell = mine;
      const double e0 = c.elev[cell];
      if (xkey(e0) > kNoDataXKey) {  // e > -9999
        const double h0 = c.h[cell];
        const double a0 = e0 + h0;
        const bool wet0 = dgt0(h0);
        {
          const size_t up = cell - W;
          const double h1 = c.h[up], e1 = c.elev[up];
          if ((wet0 || dgt0(h1)) && xkey(e1) > kNoDataXKey) {
            const double a1 = e1 + h1;
            hx = xmax_d(a0, a1) - xmax_d(e1, e0);
            ax = a1 - a0;
            fx = xkey(hx) > c.thr_xkey;
            if (!fx) {
              c.qx[cell] = 0;
              if (kSed) c.qxs[cell] = 0;
            }
          }
        }
        {
          const size_t lf = cell - 1;
          const double h1 = c.h[lf], e1 = c.elev[lf];
          if ((wet0 || dgt0(h1)) && xkey(e1) > kNoDataXKey) {
            const double a1 = e1 + h1;
            hy = xmax_d(a0, a1) - xmax_d(e1, e0);
            ay = a1 - a0;
            fy = xkey(hy) > c.thr_xkey;
            if (!fy) {
              c.qy[cell] = 0;
              if (kSed) c.qys[cell] = 0;
            }
          }
        }
      }
    }
    const unsigned bx = __ballot_sync(FULL, fx), by = __ballot_sync(FULL, fy);
    const unsigned below = (1u << lane) - 1u;
    const int nx = __popc(bx);
    if (fx) {
      const int s = qn + __popc(bx & below);
      Q[s] = cell << 1;
      HF[s] = hx;
      DA[s] = ax;
    }
    if (fy) {
      const int s = qn + nx + __popc(by & below);
      Q[s] = (cell << 1) | 1u;
      HF[s] = hy;
      DA[s] = ay;
    }
    qn += nx + __popc(by);
    __syncwarp();
    while (qn >= 32) {
      qn -= 32;
      const uint32_t f = Q[qn + lane];
      const double hf = HF[qn + lane], da = DA[qn + lane];
      __syncwarp();  // the entries are read before the next cells' are written
      face_work<kSed, kCall>(c, &dtd, f, hf, da, dt);
    }
  }
  if (lane < qn) face_work<kSed, kCall>(c, &dtd, Q[lane], HF[lane], DA[lane], dt);
}

// ---------------------------------------------------------------------------
// depth_update :3259-3299 with the maxdepth reduction (warp shuffle, block,
// then the last block publishes the grid result).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256, 6) k_depth_update(const hc_view c, hc_dev* d, int gated) {
  __shared__ long long warp_max[8];
  __shared__ bool last;
  if (gated && !d->it_active) return;
  const size_t W = c.W;
  const double dt = d->s.flow_timestep;
  const bool susp = c.p.isSuspended[1] && !c.p.hydro_only;
  const int nw = d->wet_count;
  // the running maximum is kept as the bits of a non-negative double, which
  // order like the values; tests run on the integer pipe (dgt0 etc.)
  long long m = 0;
  bool nonfinite = false;
  double lost = 0;  // water zeroed at no-data cells (the ledger's `lost`)
  // The ledger's mask-edge term: a face between a listed cell and one
  // outside the wet list changes only the listed cell's depth (the other is
  // not updated), so the water crossing it appears or vanishes.  The same
  // expression as the update, over those faces only.
  double edge = 0;
  // The discharges, fluxes, mask, border and elevations are not written by
  // this kernel: they are read through the read-only path (__ldg).  The next
  // list entry is fetched a turn ahead, so that its cell's loads do not wait
  // for the index behind them.
  const int stride = gridDim.x * blockDim.x;
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  int next = (k < nw) ? __ldg(c.wet + k) : 0;
  for (; k < nw; k += stride) {
    const size_t cell = (size_t)next;
    if (k + stride < nw) next = __ldg(c.wet + k + stride);
    if (__ldg(c.border + cell)) {  // k_wet_write marks the listed cells on the border
      const uint8_t mu = __ldg(c.mask + cell - W), md = __ldg(c.mask + cell + W),
                    ml = __ldg(c.mask + cell - 1), mr = __ldg(c.mask + cell + 1);
      const double ux1 = md ? 0.0 : __ldg(c.qx + cell + W), ux0 = mu ? 0.0 : __ldg(c.qx + cell);
      const double uy1 = mr ? 0.0 : __ldg(c.qy + cell + 1), uy0 = ml ? 0.0 : __ldg(c.qy + cell);
      edge += ddiv_by(dt * (ux1 - ux0 + uy1 - uy0), c.dxd);
    }
    // Where the four fluxes are zero (either sign) the update adds a signed
    // zero, which leaves any value but -0 as it is: the FP64 work is skipped
    // then (dry pockets of the list; cells without suspended load).
    constexpr long long kNegZero = (long long)0x8000000000000000ULL;
    double h = c.h[cell];
    {
      const double a = __ldg(c.qx + cell + W), b = __ldg(c.qx + cell),
                   e = __ldg(c.qy + cell + 1), f = __ldg(c.qy + cell);
      if (((dbits(a) | dbits(b) | dbits(e) | dbits(f)) << 1) != 0 || dbits(h) == kNegZero)
        h += ddiv_by(dt * (a - b + e - f), c.dxd);
    }
    // hydro-only runs keep Vsusptot at zero (no sediment source exists)
    if (susp) {
      const double a = __ldg(c.qxs + cell + W), b = __ldg(c.qxs + cell),
                   e = __ldg(c.qys + cell + 1), f = __ldg(c.qys + cell);
      const double v = c.vs[cell];
      if (((dbits(a) | dbits(b) | dbits(e) | dbits(f)) << 1) != 0 || dbits(v) == kNegZero)
        c.vs[cell] = v + ddiv_by(dt * (a - b + e - f), c.dxd);
    }
    nonfinite |= disnan(h);
    if (dgt0(h)) {
      if (dbits(__ldg(c.elev + cell)) == kNoDataBits) {
        lost += h;
        h = 0;
      } else {
        m = max(m, dbits(h));
      }
    }
    c.h[cell] = h;
  }
  // no flux enters a no-data cell, so this is empty in practice (its order
  // of addition is not fixed)
  // the elevations the drainage recomputation after this iteration starts
  // from (flow and depth_update leave them unchanged; erosion comes later);
  // only erosion runs keep the copy (hydro-only elevations never change)
  if (gated && d->do_drain && c.drain_snap)
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < c.N2;
         k += (size_t)gridDim.x * blockDim.x)
      c.drain_snap[k] = c.elev[k];
  if (!deq0(lost)) atomicAdd(&d->vlost_step, lost);
  if (nonfinite) {
    d->err_code = 301;  // a NaN water depth: the run cannot continue
    atomicOr((unsigned int*)&d->pause, HC_PAUSE_ERROR);
  }
  const double esum = block_sum(edge);
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  const int t = threadIdx.x;
  if ((t & 31) == 0) warp_max[t >> 5] = m;
  __syncthreads();
  if (t == 0) {
    long long b = 0;
    for (int w = 0; w < (int)blockDim.x / 32; w++) b = max(b, warp_max[w]);
    if (b > 0) atomicMax(&d->maxdepth_bits, (unsigned long long)b);
    c.vpart[blockIdx.x] = esum;
    __threadfence();
    last = (atomicAdd(&d->depth_done, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (last) {
    __threadfence();
    // the blocks' mask-edge sums, added in block order
    double a = 0;
    for (int k = t; k < (int)gridDim.x; k += blockDim.x) a += ((volatile double*)c.vpart)[k];
    const double etot = block_sum(a);
    if (t == 0) {
      unsigned long long bits = atomicExch(&d->maxdepth_bits, 0ull);
      d->s.maxdepth = bits_d((long long)bits);
      d->maxdepth_step = d->s.maxdepth;
      d->vmask_step += etot;
      d->depth_done = 0;
    }
  }
}

// ---------------------------------------------------------------------------
// scan_area :3821-3849 (every scan_area_interval_iter iterations)
// ---------------------------------------------------------------------------
// A warp takes 32 columns of kScanRows rows: each row's wet cells as one
// ballot (with a bit from either side), a cell is listed when its own bit or
// one of the eight around it is set, so three rows' words combine to the
// mask's word.  The words, 32 cells each, are what the list is counted and
// written from.
// Also the ledger's volume: the depth sum of its block (rows 1..imax,
// columns 1..jmax) into vpart, added up in order by k_wet_count's last block;
// a lane adds its rows first, which costs one FP64 instruction per 32 cells
// where a tree per row cost five.  The scan and the list, a thread per cell
// before: 503 -> 127 us at 4001 x 4103; with the launches of a step that is
// not due, 50 -> 22 us an iteration at 2000^2.
constexpr int kScanRows = 8;

// words of 32 columns in a row of the mask (columns 1..jmax)
__host__ __device__ __forceinline__ int mask_words(int jmax) { return (jmax + 31) / 32; }

__global__ void __launch_bounds__(256) k_scan_area(const hc_view c, const hc_dev* __restrict__ d,
                                                    int gated) {
  if (gated && !(d->it_active && d->do_scan)) return;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x, w = blockIdx.x, wpr = gridDim.x;
  const int i0 = 1 + (blockIdx.y * blockDim.y + threadIdx.y) * kScanRows;
  const size_t W = c.W;
  const int j = 1 + 32 * w + lane;  // columns 0 and jmax+1 are padding, and neighbours
  const int js = lane == 0 ? j - 1 : j + 1;
  const bool in = j <= c.jmax + 1, side = (lane == 0 || lane == 31) && js <= c.jmax + 1;
  double v = 0;
  if (i0 <= c.imax) {
    double h[kScanRows + 2], x[kScanRows + 2];
#pragma unroll
    for (int q = 0; q < kScanRows + 2; q++) {
      const int i = i0 - 1 + q;
      const bool row = i <= c.imax + 1;
      h[q] = row && in ? c.h[(size_t)i * W + j] : 0.0;
      x[q] = row && side ? c.h[(size_t)i * W + js] : 0.0;
    }
    const unsigned cols = c.jmax - 32 * w >= 32 ? FULL : (1u << (c.jmax - 32 * w)) - 1u;
    unsigned m2 = 0, m1 = 0;  // the two rows before, each with its neighbours in the row
#pragma unroll
    for (int q = 0; q < kScanRows + 2; q++) {
      const unsigned b = __ballot_sync(FULL, dpos(h[q])), e = __ballot_sync(FULL, dpos(x[q]));
      const unsigned m0 = b | (b << 1) | (b >> 1) | (e & 0x80000001u);
      const int i = i0 - 2 + q;  // the row between the three
      if (q >= 2 && i <= c.imax) {
        const unsigned wet = (m2 | m1 | m0) & cols;
        if (j <= c.jmax) {
          c.mask[(size_t)i * W + j] = (uint8_t)((wet >> lane) & 1u);
          v += h[q - 1];
        }
        if (lane == 0) c.wet_bits[(size_t)(i - 1) * wpr + w] = wet;
      }
      m2 = m1;
      m1 = m0;
    }
  }
  const double bsum = block_sum(v);
  if (threadIdx.x == 0 && threadIdx.y == 0) c.vpart[blockIdx.x + blockIdx.y * gridDim.x] = bsum;
}

// the words of a mask that was uploaded
__global__ void __launch_bounds__(256) k_mask_words(const hc_view c) {
  const int w = blockIdx.x, i = 1 + blockIdx.y * blockDim.y + threadIdx.y;
  const int j = 1 + 32 * w + threadIdx.x;
  const bool on = i <= c.imax && j <= c.jmax && c.mask[(size_t)i * c.W + j];
  const unsigned b = __ballot_sync(0xffffffffu, on);
  if (threadIdx.x == 0 && i <= c.imax) c.wet_bits[(size_t)(i - 1) * gridDim.x + w] = b;
}

// The wet list: the mask's words counted per block of 1024, the counts
// scanned, the cell numbers written in ascending order.
// The block counts, then, in the block that finishes last, their exclusive
// scan (the wet list's offsets per block) and the list's length.  nvol:
// blocks of the k_scan_area launch before it, whose volume partials the same
// block adds up (0: none, the list is rebuilt from a mask kept as it was).
__global__ void __launch_bounds__(1024) k_wet_count(const hc_view c, hc_dev* d, int gated,
                                                    int nvol) {
  __shared__ int ws[32];
  if (gated && !(d->it_active && d->do_scan)) return;
  const size_t n = (size_t)c.imax * mask_words(c.jmax);
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int v = __reduce_add_sync(0xffffffffu, (i < n) ? __popc(c.wet_bits[i]) : 0);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int s = __reduce_add_sync(0xffffffffu, ws[threadIdx.x]);
    if (threadIdx.x == 0) c.wet_sums[blockIdx.x] = s;
  }
  if (!last_to_arrive(&d->wet_arrive)) return;
  if (nvol > 0) {
    double a = 0;
    for (int k = threadIdx.x; k < nvol; k += blockDim.x) a += c.vpart[k];
    const double tot = block_sum(a);
    if (threadIdx.x == 0) {
      d->vol_scan = tot;
      d->vol_scan_counter = d->s.counter;
    }
  }
  const int total = scan_block_counts(c.wet_sums, (int)gridDim.x);
  if (threadIdx.x == 0) d->wet_count = total;
}

// A thread's word gives its place in the list and its border cells (those
// with an unlisted one of the four neighbours); then each warp writes its 32
// words' cells, a word at a time.
__global__ void __launch_bounds__(1024) k_wet_write(const hc_view c, const hc_dev* d, int gated) {
  __shared__ int ws[32];
  if (gated && !(d->it_active && d->do_scan)) return;
  const unsigned FULL = 0xffffffffu;
  const int wpr = mask_words(c.jmax);
  const size_t n = (size_t)c.imax * wpr;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned m = 0, border = 0;
  int first = 0, cols = 0;  // the word's first cell, its columns
  if (i < n) {
    const int r = (int)((unsigned)i / (unsigned)wpr), w = (int)i - r * wpr;
    m = c.wet_bits[i];
    const unsigned up = r > 0 ? c.wet_bits[i - wpr] : 0u;
    const unsigned down = r < c.imax - 1 ? c.wet_bits[i + wpr] : 0u;
    const unsigned left = (m << 1) | (w > 0 ? c.wet_bits[i - 1] >> 31 : 0u);
    const unsigned right = (m >> 1) | (w < wpr - 1 ? c.wet_bits[i + 1] << 31 : 0u);
    border = m & ~(up & down & left & right);
    first = (int)((size_t)(r + 1) * c.W) + 1 + 32 * w;
    cols = min(32, c.jmax - 32 * w);
  }
  const int cnt = __popc(m);
  int incl = cnt;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) ws[warp] = incl;
  __syncthreads();
  int place = c.wet_sums[blockIdx.x] + incl - cnt;
#pragma unroll
  for (int k = 0; k < 32; k++) place += k < warp ? ws[k] : 0;
#pragma unroll 4
  for (int k = 0; k < 32; k++) {
    const unsigned mk = __shfl_sync(FULL, m, k), bk = __shfl_sync(FULL, border, k);
    const int at = __shfl_sync(FULL, place, k), f = __shfl_sync(FULL, first, k);
    if ((mk >> lane) & 1u) c.wet[at + __popc(mk & ((1u << lane) - 1u))] = f + lane;
    if (lane < __shfl_sync(FULL, cols, k)) c.border[f + lane] = (uint8_t)((bk >> lane) & 1u);
  }
}

// ---------------------------------------------------------------------------
// water_flux_out :3005-3047.  Each edge cell is clamped at its first visit in
// the reference's loop order; the outflow sum is a fixed-order tree
// (deterministic, equal to the serial sum up to rounding).
// Also writes the iteration record and the end-of-loop test of main.cpp:204.
//
// The blocks clamp the cells and leave each one's outflow and depth in
// c.flux; the block that finishes last adds them.  One block did it all
// before, and the cells' FP64 operations (a division among them) waited for
// one multiprocessor's FP64 pipe (ncu, cold caches: 23 -> 12 us at 1024^2,
// 30 -> 15 us at 1400^2).  The sum's order is that of the
// one block of 1024 threads (thread t: t, t + 1024, ...; then the tree).
// ---------------------------------------------------------------------------
constexpr int kFluxSums = 1024, kFluxThreads = 512;

__global__ void __launch_bounds__(kFluxThreads) k_flux_out(const hc_view c, hc_dev* d, int gated, int record,
                                                   hc_step_record* rec, int64_t rec_cap,
                                                   cudaGraphConditionalHandle loop, int has_loop) {
  __shared__ double part[kFluxSums];
  __shared__ double vpart[kFluxSums];
  if (gated && !(d->it_active && d->rest_active)) return;
  const hc_params& p = c.p;
  const int imax = c.imax, jmax = c.jmax;
  const double thr = p.water_depth_erosion_threshold, DX = p.DX;
  const hc_divisor fdt = ddiv_prep(d->s.time_step);
  const int n1 = 2 * imax, n2 = n1 + 2 * jmax;
  const bool solo = gridDim.x == 1;
  double* rates = c.flux;      // the outflow rate per edge cell
  double* depths = c.flux + n2;  // and the depth taken off
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n2; k += gridDim.x * blockDim.x) {
    int i, j;
    bool first = true;
    if (k < n1) {
      i = 1 + k / 2;
      if ((k & 1) == 0) {
        j = jmax;
      } else {
        j = 1;
        if (jmax == 1) first = false;  // same cell as the right-hand edge
      }
    } else {
      const int kk = k - n1;
      j = 1 + kk / 2;
      if (j == 1 || j == jmax) first = false;  // already visited by the row loop
      if ((kk & 1) == 0) {
        i = 1;
      } else {
        i = imax;
        if (imax == 1) first = false;
      }
    }
    double rate = 0, off = 0;
    if (first) {
      double& h = c.h[(size_t)i * c.W + j];
      const double h0 = h;
      if (h0 > thr) {
        off = h0 - thr;
        rate = ddiv_by(off * DX * DX, fdt);
        h = thr;
      }
    }
    if (solo) {  // at most kFluxSums cells: each is a sum of its own
      part[k] = rate;
      vpart[k] = off;
    } else {
      rates[k] = rate;
      depths[k] = off;
    }
  }
  if (!solo && !last_to_arrive(&d->flux_arrive)) return;
  // what the record takes, on its way while the sums are formed
  hc_scalars& s = d->s;
  hc_step_record r;
  double vin = 0, vlost = 0, vmask = 0, vin_tot = 0, vout_tot = 0, vlost_tot = 0, vmask_tot = 0;
  double vol = 0, vol_counter = 0, creep1 = 0, creep2 = 0;
  if (threadIdx.x == 0) {
    r.counter = s.counter;
    r.cycle = s.cycle;
    r.time_step = s.time_step;
    r.maxdepth = d->maxdepth_step;
    r.waterinput = s.waterinput;
    r.erode_mult = s.erode_mult;
    r.sediQ = s.sediQ;
    r.globalsediq = s.globalsediq;
    r.baseflow = s.baseflow;
    creep1 = s.creep_time;
    creep2 = s.creep_time2;
    vin = d->vin_step;
    vlost = d->vlost_step;
    vmask = d->vmask_step;
    vin_tot = d->vin_tot;
    vout_tot = d->vout_tot;
    vlost_tot = d->vlost_tot;
    vmask_tot = d->vmask_tot;
    vol = d->vol_scan;
    vol_counter = d->vol_scan_counter;
  }
  // nothing flowed off a cell whose entry is zero (rates and depths are never
  // negative, so leaving a +0 out changes no sum)
  for (int t = threadIdx.x; t < kFluxSums; t += blockDim.x) {
    if (solo) {
      if (t >= n2) part[t] = vpart[t] = 0;
      continue;
    }
    double acc = 0, vacc = 0;
    for (int k0 = t; k0 < n2; k0 += 4 * kFluxSums) {
      double rt[4], of[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int k = k0 + q * kFluxSums;
        of[q] = k < n2 ? __ldcg(depths + k) : 0.0;
        rt[q] = k < n2 ? __ldcg(rates + k) : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (dbits(of[q]) != 0) {
          acc += rt[q];
          vacc += of[q];
        }
    }
    part[t] = acc;
    vpart[t] = vacc;
  }
  __syncthreads();
  for (int w = kFluxSums / 2; w > 0; w >>= 1) {
    for (int t = threadIdx.x; t < w; t += blockDim.x)
      if (dbits(vpart[t + w]) != 0) {
        part[t] += part[t + w];
        vpart[t] += vpart[t + w];
      }
    if (w > 32) __syncthreads();
    else __syncwarp();
  }
  if (threadIdx.x == 0) {
    s.temptot = part[0];
    s.waterOut = part[0];
    if (record && rec && d->rec_index < rec_cap) {
      r.waterOut = part[0];
      const double a2 = DX * DX;
      r.vol_in = vin * a2;
      r.vol_out = (vpart[0] + vlost) * a2;
      r.vol_mask = vmask * a2;
      r.volume = (vol_counter == r.counter) ? vol * a2 : bits_d(0x7ff8000000000000LL);
      rec[d->rec_index] = r;
    }
    if (record) d->rec_index++;
    if (gated) d->wet_steps += (unsigned long long)d->wet_count;
    // the ledger: this iteration's terms join the totals
    d->vin_tot = vin_tot + vin;
    d->vout_tot = vout_tot + vpart[0];
    d->vlost_tot = vlost_tot + vlost;
    d->vmask_tot = vmask_tot + vmask;
    d->vin_step = 0;
    d->vlost_step = 0;
    d->vmask_step = 0;
    if (gated) {
      if (!p.hydro_only && !(d->flags & HC_RUN_NOHILL) && (r.cycle > creep1 || r.cycle > creep2))
        d->pause |= HC_PAUSE_HOSTSTEP;
      if (!(r.cycle / 60 < p.maxcycle)) d->pause |= HC_PAUSE_FINISHED;
      if (has_loop) cudaGraphSetConditional(loop, d->pause == 0 && d->budget > 0 ? 1u : 0u);
    }
  }
}

// The depth sum of the grid (rows 1..imax, columns 1..jmax) now, in a fixed
// order (hc_mass_balance; the ledger's start).
__global__ void __launch_bounds__(256) k_volume(const hc_view c, hc_dev* d) {
  const size_t n = (size_t)c.imax * c.jmax;
  double a = 0;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    const size_t i = 1 + k / c.jmax, j = 1 + k % c.jmax;
    a += c.h[i * c.W + j];
  }
  double tot;
  if (grid_sum(a, c.vpart, &d->sum_done, &tot)) d->vol_now = tot;
}

__global__ void k_mass_reset(hc_dev* d) {
  d->vol0 = d->vol_now;
  d->vin_tot = d->vout_tot = d->vlost_tot = d->vmask_tot = 0;
  d->vin_step = d->vlost_step = d->vmask_step = 0;
}

}  // namespace

// ------------------------------------------------------------------ launches
static dim3 grid2d(const hc_ctx* c, dim3 b) {
  return dim3((c->v.jmax + b.x - 1) / b.x, (c->v.imax + b.y - 1) / b.y);
}

void launch_control(hc_ctx* c) {
  k_control<<<1, 32, 0, c->cs>>>(c->v, c->dev, c->hcur);
  count_launch(c, 1);
}

void launch_inputs(hc_ctx* c) {
  if (c->v.p.spatially_complex_rainfall) {
    dim3 b(32, 8), g((c->v.jmax + 31) / 32, (c->v.imax + 7) / 8);
    k_runoff_inputs<<<g, b, 0, c->cs>>>(c->v, c->dev);
    count_launch(c, 1);
    return;
  }
  // grid-stride over the current list (its length lives on the device):
  // four blocks per SM on large grids, fewer on small ones, whose lists are
  // short (ensembles run many small members' launches side by side)
  int n = c->v.cin_cap;
  const int cap = std::min(c->sms * 4, std::max(c->sms, (int)(c->v.N2 / 4096)));
  int blocks = std::min((n + 255) / 256, std::min(cap, c->v.vpart_cap));
  if (blocks < 1) blocks = 1;
  k_inputs<<<blocks, 256, 0, c->cs>>>(c->v, c->dev);
  count_launch(c, 1);
}

void launch_flow_dt(hc_ctx* c) {
  k_flow_dt<<<1, 1, 0, c->cs>>>(c->v, c->dev);
  count_launch(c, 1);
}

// grid-stride kernels over the wet list: enough blocks to fill the GPU, no
// more (the list length lives on the device)
static int list_blocks(const hc_ctx* c) {
  const size_t need = (c->v.N2 + 255) / 256;
  return (int)std::min<size_t>(need, 152 * 8);
}

// The launch shapes of k_flow_route the autotuner chooses from: blocks per
// multiprocessor (the register budget) and waves of the grid (grid = SMs x
// blocks per SM x waves; one wave: every block resident at once).
const FlowShape kFlowShapes[kFlowShapeCount] = {
    {4, 0, 0}, {3, 1, 0}, {4, 1, 0}, {5, 1, 0}, {6, 1, 0}, {3, 4, 0}, {4, 4, 0}, {5, 4, 0},
    {6, 4, 0}, {3, 1, 1}, {4, 1, 1}, {5, 1, 1}, {3, 4, 1}, {4, 4, 1}, {5, 4, 1},
    {3, 1, 2}, {4, 1, 2}, {5, 1, 2}};

template <bool kSed>
static void flow_launch(hc_ctx* c, int gated, int shape) {
  const FlowShape f = kFlowShapes[shape];
  int blocks = f.waves ? c->sms * f.minb * f.waves : list_blocks(c);
  blocks = std::max(1, std::min(blocks, (int)((c->v.N2 + 255) / 256)));
  if (f.compact == 2) {  // divisions through one out-of-line copy
    switch (f.minb) {
      case 3: k_flow_route_q<kSed, 3, true><<<blocks, 256, 0, c->cs>>>(c->v, c->dev, gated); break;
      case 5: k_flow_route_q<kSed, 5, true><<<blocks, 256, 0, c->cs>>>(c->v, c->dev, gated); break;
      default: k_flow_route_q<kSed, 4, true><<<blocks, 256, 0, c->cs>>>(c->v, c->dev, gated); break;
    }
    return;
  }
  if (f.compact) {
    switch (f.minb) {
      case 3: k_flow_route_q<kSed, 3><<<blocks, 256, 0, c->cs>>>(c->v, c->dev, gated); break;
      case 5: k_flow_route_q<kSed, 5><<<blocks, 256, 0, c->cs>>>(c->v, c->dev, gated); break;
      default: k_flow_route_q<kSed, 4><<<blocks, 256, 0, c->cs>>>(c->v, c->dev, gated); break;
    }
    return;
  }
  switch (f.minb) {
    case 3: k_flow_route<kSed, 3><<<blocks, 256, 0, c->cs>>>(c->v, c->dev, gated); break;
    case 5: k_flow_route<kSed, 5><<<blocks, 256, 0, c->cs>>>(c->v, c->dev, gated); break;
    case 6: k_flow_route<kSed, 6><<<blocks, 256, 0, c->cs>>>(c->v, c->dev, gated); break;
    default: k_flow_route<kSed, 4><<<blocks, 256, 0, c->cs>>>(c->v, c->dev, gated); break;
  }
}

void launch_flow_route_shape(hc_ctx* c, int gated, int shape) {
  if (shape < 0 || shape >= kFlowShapeCount) shape = 0;
  if (c->v.p.hydro_only) flow_launch<false>(c, gated, shape);
  else flow_launch<true>(c, gated, shape);
  count_launch(c, 1);
}

void launch_flow_route(hc_ctx* c, int gated) { launch_flow_route_shape(c, gated, c->flow_shape); }

void launch_depth_update(hc_ctx* c, int gated) {
  // one wave of the six blocks a multiprocessor holds (list_blocks, a wave and
  // a third: 266 -> 205 us at 4000^2, 68 -> 57 in a storm at 1400^2, 31 -> 27 at
  // 1024^2)
  k_depth_update<<<std::min(list_blocks(c), c->sms * 6), 256, 0, c->cs>>>(c->v, c->dev, gated);
  count_launch(c, 1);
}

static void wet_list(hc_ctx* c, int gated, int nvol);

void launch_scan_area(hc_ctx* c, int gated) {
  dim3 b(32, 8);
  const int rows = 8 * kScanRows;
  const dim3 g(mask_words(c->v.jmax), (c->v.imax + rows - 1) / rows);
  k_scan_area<<<g, b, 0, c->cs>>>(c->v, c->dev, gated);
  count_launch(c, 1);
  wet_list(c, gated, (int)(g.x * g.y));
}

void launch_wet_list(hc_ctx* c, int gated) {
  const dim3 g(mask_words(c->v.jmax), (c->v.imax + 7) / 8);
  k_mask_words<<<g, dim3(32, 8), 0, c->cs>>>(c->v);
  count_launch(c, 1);
  wet_list(c, gated, 0);
}

static void wet_list(hc_ctx* c, int gated, int nvol) {
  const size_t words = (size_t)c->v.imax * mask_words(c->v.jmax);
  const int nb = (int)((words + 1023) / 1024);
  k_wet_count<<<nb, 1024, 0, c->cs>>>(c->v, c->dev, gated, nvol);
  k_wet_write<<<nb, 1024, 0, c->cs>>>(c->v, c->dev, gated);
  count_launch(c, 2);
}

void launch_flux_out(hc_ctx* c, int gated, int record) {
  const int n = 2 * (c->v.imax + c->v.jmax);
  // one block while every cell can be a sum of its own: nothing goes through
  // memory then, and no block waits for another's arrival
  const int blocks = n <= kFluxSums ? 1 : std::min((n + kFluxThreads - 1) / kFluxThreads, 64);
  k_flux_out<<<blocks, kFluxThreads, 0, c->cs>>>(c->v, c->dev, gated, record, c->v.rec,
                                                 c->v.rec_cap, c->hcur.loop, c->capturing ? 1 : 0);
  count_launch(c, 1);
}

// grid of the grid_sum kernels: at most the SMs x 4 blocks of 256 (the
// partials array holds vpart_cap entries)
static int sum_blocks(const hc_ctx* c, size_t n) {
  const size_t need = (n + 255) / 256;
  return (int)std::max<size_t>(1, std::min<size_t>(need, (size_t)std::min(152 * 4, c->v.vpart_cap)));
}

void launch_volume(hc_ctx* c) {
  k_volume<<<sum_blocks(c, (size_t)c->v.imax * c->v.jmax), 256, 0, c->cs>>>(c->v, c->dev);
  count_launch(c, 1);
}

void launch_mass_reset(hc_ctx* c) {
  launch_volume(c);
  k_mass_reset<<<1, 1, 0, c->cs>>>(c->dev);
  count_launch(c, 1);
}
