// lateral_channel_erode :4850-5291 ("lateral3"): the channel-edge curvature
// field `edge` that erode() uses for lateral bank erosion.
//
// The reference indexes its scratch arrays and `edge` with x < jmax+1 and
// y < imax+1, which only describes the grid for square domains; the library
// runs lateral3 on square grids and reports HC_ERR_UNSUPPORTED otherwise.
//
// Passes of the reference:
//   L1  water_depth2 from Tau with isolated cells removed       :4863-4890
//   L2  edge cells and the 2x upscaled wet/dry grid              :4894-4939
//   L3  edge marks on the upscaled grid                          :4942-4958
//   L4  inside/outside tally on the upscaled grid                :4961-4991
//   L5  edge values from the tally                               :4994-5009
//   L6  edge_smoothing_passes + downstream_shift smoothing       :5011-5208
//   L7  curvature transform                                      :5210-5227
//   L8  cross-channel smoothing until converged                  :5229-5288
//
// Here: k_wet2 (L1), k_edges (L2-L5: a cell's four upscaled quarters are
// functions of water_depth2 within two cells, so the upscaled grids are never
// stored), k_lists, then one small kernel per smoothing pass, k_curve (L7)
// and one small kernel per pass of L8.
//
// What bounds it is the number of passes, 105 of L6 and some dozens of L8:
// a pass moves little data.  Which neighbours join a cell's mean depends only
// on water_depth2, on the water surface (the last passes) and on which cells
// hold an edge value, and none of these change from pass to pass.  So k_lists
// writes, once, the cells that L6 and L8 change with the neighbours of each
// as a bit mask, and a pass is one kernel over that list from one copy of the
// edge field into another.  L8's test runs on the device: a pass whose
// predecessor changed nothing by more than the tolerance returns at once,
// and the host looks at the changes once per kSmoothBatch passes.  Before,
// a pass was three kernels over the whole grid (L8: and a read by the host):
// 9.3 -> 1.3 ms a call at 512 x 512 (36,000 edge cells, 4.5 us a pass), 39 ->
// 5.6 ms at 2000 x 2000.
//
// In L6 and L8 a down_scan entry of row 1 or row jmax is processed at row 2
// or jmax-1 (the reference bumps x).  In L6 that never shows: such an entry
// writes the value that the entry of row 2 (jmax-1) writes too, or a value
// that no copy reads, and its own row takes 0.  In L8 it makes the cell of
// row 2 (jmax-1) a visited one.

#include "hc_grain.cuh"

#include <math.h>
#include <algorithm>

namespace {

__constant__ int kLx[9] = {0, 0, 1, 1, 1, 0, -1, -1, -1};
__constant__ int kLy[9] = {0, -1, -1, 0, 1, 1, 1, 0, -1};

constexpr double kMft = 0.1;
constexpr int kSmoothBatch = 32;  // passes of L8 between two looks of the host

// L6 cells: bits 0-7 the neighbours (kLx, kLy 1..8) of the early passes,
// 8-15 those of the late ones, bit 16: the value is 0 whatever they hold.
// L8 cells: bits 0-3 the neighbours 1, 3, 5, 7.
constexpr uint32_t kZeroed = 1u << 16;

struct LatCount {
  unsigned int n6, n8;
  double diff[kSmoothBatch + 1];  // largest change of each pass of a batch
};

struct LatBufs {
  double* et;      // edge_temp: the edge field's other copy, (jmax+1)(imax+1)
  double* wd2;     // water_depth2
  uint32_t *cell6, *bits6, *cell8, *bits8;
  LatCount* n;
};

// the divisors of a mean over 1..9 values
struct SmallDivisors {
  hc_divisor d[10];
};

__device__ __forceinline__ size_t L(const hc_view& c, int x, int y) {
  return (size_t)x * (c.imax + 1) + y;
}
__device__ __forceinline__ double& EDG(const hc_view& c, int x, int y) {
  return c.edge[(size_t)x * (c.jmax + 1) + y];
}
// the cell (x, y) is visited by the entry of its own row or by a bumped one
__device__ __forceinline__ bool visited(const hc_view& c, int x, int y) {
  return c.mask[(size_t)x * c.W + y] || (x == 2 && c.mask[(size_t)1 * c.W + y]) ||
         (x == c.jmax - 1 && c.mask[(size_t)c.jmax * c.W + y]);
}
__device__ __forceinline__ bool inner(const hc_view& c, int x, int y) {
  return x >= 2 && x <= c.jmax - 1 && y >= 2 && y <= c.imax - 1;
}

// L1, every cell of the array
__global__ void k_wet2(const hc_view c, LatBufs b) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  const int x = blockIdx.y * blockDim.y + threadIdx.y;
  if (y > c.imax || x > c.jmax) return;
  double w = 0;
  if (inner(c, x, y) && visited(c, x, y)) {
    const double t = c.tau[(size_t)x * c.W + y];
    if (t > kMft) {
      int tc = 0;
      for (int dir = 1; dir <= 8; dir++)
        if (c.tau[(size_t)(x + kLx[dir]) * c.W + (y + kLy[dir])] < kMft) tc++;
      w = (tc > 6) ? 0.0 : t;
    }
  }
  b.wd2[L(c, x, y)] = w;
}

// the upscaled grid's quarter (X, Y), 1 where its cell is wet (L2); quarters
// of cells outside rows 2..jmax-1, columns 2..imax-1 stay 0
__device__ __forceinline__ bool up_wet(const hc_view& c, const LatBufs& b, int X, int Y) {
  const int x = (X + 1) >> 1, y = (Y + 1) >> 1;
  return inner(c, x, y) && b.wd2[L(c, x, y)] >= kMft;
}
// after L3: 1 wet, 2 dry next to a wet quarter, else 0
__device__ __forceinline__ int up_mark(const hc_view& c, const LatBufs& b, int X, int Y) {
  if (up_wet(c, b, X, Y)) return 1;
  if (Y < 2 || Y > 2 * c.imax - 1 || X < 2 || X > 2 * c.jmax - 1) return 0;
  return (up_wet(c, b, X, Y - 1) || up_wet(c, b, X - 1, Y) || up_wet(c, b, X + 1, Y) ||
          up_wet(c, b, X, Y + 1))
             ? 2
             : 0;
}
// L4: wet minus dry quarters around a marked one
__device__ __forceinline__ int up_tally(const hc_view& c, const LatBufs& b, int X, int Y) {
  if (Y < 2 || Y > 2 * c.imax - 1 || X < 2 || X > 2 * c.jmax - 1) return 0;
  if (up_mark(c, b, X, Y) != 2) return 0;
  int wet = 0, dry = 0, ecc = 1;
#pragma unroll 1
  for (int dir = 1; dir <= 7; dir += 2) {
    const int v = up_mark(c, b, X + kLx[dir], Y + kLy[dir]);
    if (v == 1) wet += 1;
    if (v == 0) dry += 1;
    if (v == 2) ecc += 1;
  }
  if (ecc > 3) dry += ecc - 2;
  return wet - dry;
}

// L2 and L5
__global__ void k_edges(const hc_view c, LatBufs b) {
  const int y = 1 + blockIdx.x * blockDim.x + threadIdx.x;
  const int x = 1 + blockIdx.y * blockDim.y + threadIdx.y;
  if (y > c.imax || x > c.jmax) return;
  double e;
  if (inner(c, x, y)) {
    e = -9999;
    if (b.wd2[L(c, x, y)] < kMft) {
      const double a = b.wd2[L(c, x, y - 1)], bb = b.wd2[L(c, x - 1, y)],
                   cc = b.wd2[L(c, x + 1, y)], dd = b.wd2[L(c, x, y + 1)];
      if (a > kMft || bb > kMft || cc > kMft || dd > kMft) e = 0;
      if (a > kMft && bb > kMft && cc > kMft && dd > kMft) {
        e = -9999;
        c.edge2[(size_t)x * (c.jmax + 1) + y] = -9999;
      }
    }
  } else {
    e = EDG(c, x, y);
  }
  if (e == 0) {
    int t = 0;
#pragma unroll 1
    for (int k = 0; k < 4; k++) t += up_tally(c, b, 2 * x - (k >> 1), 2 * y - (k & 1));
    e = (double)t;
    if (e > 2) e = 2;
    if (e < -2) e = -2;
  }
  EDG(c, x, y) = e;
}

// whether neighbour dir of (x,y) joins the smoothing mean (:5061-5196)
__device__ __forceinline__ bool joins(const hc_view& c, const LatBufs& b, int x, int y, int dir) {
  const int dx = kLx[dir], dy = kLy[dir];
  const double* w = b.wd2;
  if ((abs(dx) + abs(dy)) != 2) {
    if (dx == 1 && dy == 0) return w[L(c, x + 1, y - 1)] > kMft || w[L(c, x + 1, y + 1)] > kMft;
    if (dx == 0 && dy == 1) return w[L(c, x + 1, y + 1)] > kMft || w[L(c, x - 1, y + 1)] > kMft;
    if (dx == -1 && dy == 0) return w[L(c, x - 1, y - 1)] > kMft || w[L(c, x - 1, y + 1)] > kMft;
    if (dx == 0 && dy == -1) return w[L(c, x - 1, y - 1)] > kMft || w[L(c, x + 1, y - 1)] > kMft;
  } else {
    if (dx == -1 && dy == -1) return w[L(c, x, y - 1)] < kMft || w[L(c, x - 1, y)] < kMft;
    if (dx == 1 && dy == -1) return w[L(c, x, y - 1)] < kMft || w[L(c, x + 1, y)] < kMft;
    if (dx == 1 && dy == 1) return w[L(c, x + 1, y)] < kMft || w[L(c, x, y + 1)] < kMft;
    if (dx == -1 && dy == 1) return w[L(c, x, y + 1)] < kMft || w[L(c, x - 1, y)] < kMft;
  }
  return false;
}

// the edge value of (x, y) after L7 lies above -9999: it did before, or the
// cell is under water there
__device__ __forceinline__ bool edge_after_l7(const hc_view& c, int x, int y) {
  return EDG(c, x, y) > -9999 || c.h[(size_t)x * c.W + y] > c.p.water_depth_erosion_threshold;
}
__device__ __forceinline__ bool in_l8(const hc_view& c, const LatBufs& b, int x, int y) {
  return inner(c, x, y) && b.wd2[L(c, x, y)] > kMft && visited(c, x, y);
}

// appends the warp's flagged lanes to a list (one atomic per warp)
__device__ __forceinline__ void append(bool on, unsigned int* count, uint32_t* cells,
                                       uint32_t* bits, uint32_t cell, uint32_t word) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xffffffffu, on);
  if (!m) return;
  unsigned base = 0;
  if (lane == 0) base = atomicAdd(count, (unsigned)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (!on) return;
  const unsigned k = base + __popc(m & ((1u << lane) - 1u));
  cells[k] = cell;
  bits[k] = word;
}

// The cells that L6 and L8 change, with the neighbours that join each mean,
// and the edge field's second copy.  blockDim.x is 32: a warp is one run of
// columns, so the lists keep runs of neighbouring cells together.
__global__ void k_lists(const hc_view c, LatBufs b, int late_passes) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  const int x = blockIdx.y * blockDim.y + threadIdx.y;
  const bool in = y <= c.imax && x <= c.jmax;
  bool on6 = false, on8 = false;
  uint32_t w6 = 0, w8 = 0;
  const uint32_t cell = in ? (uint32_t)L(c, x, y) : 0u;
  if (in) {
    const double e = EDG(c, x, y);
    b.et[cell] = e;
    if (x >= 1 && y >= 2 && y <= c.imax - 1) {
      on6 = c.mask[(size_t)x * c.W + y] && e > -9999;
      if (on6) {
        // rows and columns this close to the border take 0 (:5199-5203)
        if (x < 3 || x > (c.jmax - 3) || y < 3 || y > (c.imax - 3)) {
          w6 = kZeroed;
        } else {
          const double ws0 = late_passes ? mean_ws_elev_dev(c, x, y) : 0.0;
#pragma unroll 1
          for (int dir = 1; dir <= 8; dir++) {
            const int x2 = x + kLx[dir], y2 = y + kLy[dir];
            if (!(EDG(c, x2, y2) > -9999 && b.wd2[L(c, x2, y2)] < kMft)) continue;
            if (!joins(c, b, x, y, dir)) continue;
            w6 |= 1u << (dir - 1);
            if (late_passes && mean_ws_elev_dev(c, x2, y2) > ws0) w6 |= 1u << (dir + 7);
          }
        }
      }
      on8 = in_l8(c, b, x, y);
      if (on8)
#pragma unroll 1
        for (int k = 0; k < 4; k++) {
          const int x2 = x + kLx[1 + 2 * k], y2 = y + kLy[1 + 2 * k];
          // a wet cell's -9999 is turned into 0 right before it is read
          if (edge_after_l7(c, x2, y2) || b.wd2[L(c, x2, y2)] > kMft) w8 |= 1u << k;
        }
    }
  }
  append(on6, &b.n->n6, b.cell6, b.bits6, cell, w6);
  append(on8, &b.n->n8, b.cell8, b.bits8, cell, w8);
}

// One pass of L6: the mean of the cell and its joining neighbours, summed in
// their order; a zero sum gives 0 (edge_temp's initial value).
__global__ void __launch_bounds__(256) k_smooth(const double* __restrict__ src,
                                                double* __restrict__ dst,
                                                const uint32_t* __restrict__ cells,
                                                const uint32_t* __restrict__ bits, unsigned n,
                                                int pitch, int late,
                                                const __grid_constant__ SmallDivisors dv) {
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t cell = cells[k], w = bits[k];
  double v = 0;
  if (!(w & kZeroed)) {
    const unsigned m = (w >> (late ? 8 : 0)) & 0xffu;
    const double* s = src + cell;
    const int P = pitch;
    // every joining value is loaded before the first is added
    const int off[8] = {-1, P - 1, P, P + 1, 1, -P + 1, -P, -P - 1};
    double e[8];
#pragma unroll
    for (int q = 0; q < 8; q++) e[q] = ((m >> q) & 1u) ? s[off[q]] : 0.0;
    double mean = 0.0 + s[0];
#pragma unroll
    for (int q = 0; q < 8; q++)
      if ((m >> q) & 1u) mean += e[q];
    if (!deq0(mean)) v = ddiv_by(mean, dv.d[1 + __popc(m)]);
  }
  dst[cell] = v;
}

// L7 from the smoothed copy into `edge` and its second copy, with L8's first
// reads: a wet cell's -9999 becomes 0 where an entry of L8 reads it
__global__ void k_curve(const hc_view c, LatBufs b, const double* src) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  const int x = blockIdx.y * blockDim.y + threadIdx.y;
  if (y > c.imax || x > c.jmax) return;
  double e = src[L(c, x, y)];
  if (x >= 1 && y >= 1) {
    if (e > -9999) {
      if (e > 0) e = 0;
      e = 0 - e;
      e = 1 / ((2.131 * pow(e, -1.0794)) * c.p.DX);
    }
    if (c.h[(size_t)x * c.W + y] > c.p.water_depth_erosion_threshold && e == -9999) e = 0;
    if (e == -9999 && b.wd2[L(c, x, y)] > kMft &&
        (in_l8(c, b, x, y) || in_l8(c, b, x - 1, y) || in_l8(c, b, x + 1, y) ||
         in_l8(c, b, x, y - 1) || in_l8(c, b, x, y + 1)))
      e = 0;
  }
  EDG(c, x, y) = e;
  b.et[L(c, x, y)] = e;
}

// Pass p of a batch of L8: skipped when the pass before it changed nothing by
// more than tol (pass 0 always runs: the host has looked).
__global__ void __launch_bounds__(256) k_cross(const double* __restrict__ src,
                                               double* __restrict__ dst, LatBufs b, unsigned n,
                                               int pitch, int p, double tol,
                                               const __grid_constant__ SmallDivisors dv) {
  __shared__ double wmax[8];
  if (p > 0 && !(*(volatile double*)&b.n->diff[p - 1] > tol)) return;
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
  double m = 0;
  if (k < n) {
    const uint32_t cell = b.cell8[k], w = b.bits8[k];
    const double* s = src + cell;
    const double e0 = s[0];
    double t = e0;
    if (e0 > -9999) {  // not a NaN of an earlier pass
      const int off[4] = {-1, pitch, 1, -pitch};
      double e[4];
#pragma unroll
      for (int q = 0; q < 4; q++) e[q] = ((w >> q) & 1u) ? s[off[q]] : 0.0;
      double mean = 0;
      int num = 0;
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (((w >> q) & 1u) && e[q] > -9999) {
          mean += e[q];
          num++;
        }
      t = num > 0 ? ddiv_by(mean, dv.d[num]) : mean / num;
      m = fabs(e0 - t);
      if (!(m == m)) m = 0;  // a NaN change never raises the reference's max
    }
    dst[cell] = t;
  }
  for (int o = 16; o > 0; o >>= 1) m = smax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double bm = 0;
    for (int q = 0; q < 8; q++) bm = smax(bm, wmax[q]);
    if (bm > 0) atomic_max_pos((unsigned long long*)&b.n->diff[p], bm);
  }
}

// the listed cells of the copy that holds the result, into `edge`
__global__ void __launch_bounds__(256) k_cross_out(const hc_view c, LatBufs b, unsigned n) {
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) c.edge[b.cell8[k]] = b.et[b.cell8[k]];
}

}  // namespace

size_t lateral_scratch_bytes(int imax, int jmax) {
  const size_t n1 = (size_t)(jmax + 1) * (imax + 1);
  return 2 * n1 * 8 + 4 * n1 * 4 + sizeof(LatCount) + 256;
}

hc_status run_lateral(hc_ctx* c) {
  const hc_view& v = c->v;
  if (v.imax != v.jmax) return hc_fail(c, HC_ERR_UNSUPPORTED, "lateral3 needs a square grid");
  extern double* lateral_buffer(hc_ctx*);
  const size_t n1 = (size_t)(v.jmax + 1) * (v.imax + 1);
  LatBufs b;
  b.et = lateral_buffer(c);
  b.wd2 = b.et + n1;
  b.n = (LatCount*)(b.wd2 + n1);
  b.cell6 = (uint32_t*)(b.n + 1);
  b.bits6 = b.cell6 + n1;
  b.cell8 = b.bits6 + n1;
  b.bits8 = b.cell8 + n1;
  SmallDivisors dv;
  for (int k = 0; k < 10; k++) dv.d[k] = host_divisor(k > 0 ? (double)k : 1.0);
  cudaStream_t s = c->s;
  const int J = v.jmax, P = v.imax + 1;
  dim3 bl(32, 8);
  const dim3 all((P + 31) / 32, (J + 1 + 7) / 8);
  const double esp = v.p.edge_smoothing_passes, passes = esp + v.p.downstream_shift;
  cudaMemsetAsync(b.n, 0, sizeof(LatCount), s);
  k_wet2<<<all, bl, 0, s>>>(v, b);
  k_edges<<<dim3((v.imax + 31) / 32, (J + 7) / 8), bl, 0, s>>>(v, b);
  int early = 0, total = 0;
  for (int n = 1; n <= passes; n++) {
    total++;
    if (!(n > esp)) early++;
  }
  k_lists<<<all, bl, 0, s>>>(v, b, total > early ? 1 : 0);
  count_launch(c, 3);
  LatCount h;
  cudaError_t e = cudaMemcpyAsync(&h, b.n, sizeof h, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return hc_cuda(c, e, "lateral3");
  double* buf[2] = {v.edge, b.et};
  const unsigned g6 = (h.n6 + 255) / 256, g8 = (h.n8 + 255) / 256;
  int cur = 0;
  for (int n = 0; n < total && h.n6 > 0; n++) {
    k_smooth<<<g6, 256, 0, s>>>(buf[cur], buf[1 - cur], b.cell6, b.bits6, h.n6, P,
                                n >= early ? 1 : 0, dv);
    count_launch(c, 1);
    cur ^= 1;
  }
  k_curve<<<all, bl, 0, s>>>(v, b, buf[cur]);
  count_launch(c, 1);
  const double tol = v.p.lateral_cross_channel_smoothing;
  cur = 0;
  bool more = h.n8 > 0;
  for (int guard = 0; more; guard++) {
    if (guard > 10000000 / kSmoothBatch)
      return hc_fail(c, HC_ERR_TIMEOUT, "lateral3 did not converge");
    cudaMemsetAsync(b.n->diff, 0, sizeof h.diff, s);
    for (int p = 0; p < kSmoothBatch; p++)
      k_cross<<<g8, 256, 0, s>>>(buf[(cur + p) & 1], buf[(cur + p + 1) & 1], b, h.n8, P, p, tol, dv);
    count_launch(c, kSmoothBatch);
    e = cudaMemcpyAsync(&h, b.n, sizeof h, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return hc_cuda(c, e, "lateral3");
    // passes that ran: up to the first that changed nothing by more than tol
    int ran = 0;
    while (ran < kSmoothBatch && h.diff[ran] > tol) ran++;
    more = ran == kSmoothBatch;
    cur = (cur + (more ? kSmoothBatch : ran + 1)) & 1;
  }
  if (cur) {
    k_cross_out<<<g8, 256, 0, s>>>(v, b, h.n8);
    count_launch(c, 1);
  }
  return hc_cuda(c, cudaGetLastError(), "lateral3");
}
