// Drainage area and catchment input points, recomputed when the baseflow
// threshold moves (catchment_water_input_and_hydrology :3524-3539):
// zero_and_calc_drainage_area :2072-2089, drainage_area_D8 :2091-2271 and
// get_catchment_input_points :3741-3767.
//
// The reference sweeps all cells once from the highest to the lowest (an
// order fixed by a sort, hc_sort.cu) and pushes each cell's area to
// its lower neighbours.  A cell's final area is therefore its initial value
// plus the pushes of its higher neighbours, added in the order those were
// swept.  Here the same sums are pulled instead: a cell is ready once all
// its higher neighbours are done (Kahn's algorithm on the "higher than"
// graph), and it adds its neighbours' terms in their sweep order (the
// position in the sort, so equal elevations keep the reference's order).
// Every term and every addition is the reference's, so the areas are
// bit-identical.  Cells the reference's loop never reaches (sorted position 0
// and above imax*jmax, where the sort's padding pairs push them) keep area 0
// and push nothing, as there.
//
// The sort itself is needed only where its order among equal elevations can
// show: two higher neighbours of one cell at the same elevation (the order
// of their pushes), or a group of equal elevations that straddles the first
// or the last reached position.  The device checks for those (a radix
// selection finds the last reached position); when none occurs, "reached" is
// a threshold on the elevation, the pushes are ordered by elevation, and no
// sort runs at all.  Otherwise the device sorts (hc_sort.cu; the host's
// exact sort where that declines).
//
// The elevations are those at the start of the iteration that moved the
// threshold (k_depth_update copies them before the iteration's erosion).

#include "hc_internal.cuh"

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <vector>

namespace {

__constant__ int kDrX[9] = {0, 0, 1, 1, 1, 0, -1, -1, -1};
__constant__ int kDrY[9] = {0, -1, -1, 0, 1, 1, 1, 0, -1};

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// unsigned key that orders like the elevations (std::sort's `<`: +0 == -0)
__host__ __device__ __forceinline__ unsigned long long ukey_bits(long long b) {
  const long long s = b >> 63;
  const long long k = ((b & 0x7fffffffffffffffLL) ^ s) - s;
  return (unsigned long long)k ^ 0x8000000000000000ULL;
}
__device__ __forceinline__ unsigned long long ukey(double x) {
  return ukey_bits(dbits(x));
}
constexpr unsigned long long kZeroKey = 0x8000000000000000ULL;  // ukey(0.0)

__device__ __forceinline__ bool interior_ij(const hc_view& c, int& i, int& j) {
  j = 1 + blockIdx.x * blockDim.x + threadIdx.x;
  i = 1 + blockIdx.y * blockDim.y + threadIdx.y;
  return i <= c.imax && j <= c.jmax;
}

// smallest elevation key
__global__ void k_drain_min(const hc_view c, const double* __restrict__ el) {
  int i, j;
  unsigned long long u = ~0ull;
  if (interior_ij(c, i, j)) u = ukey(el[(size_t)i * c.W + j]);
  for (int o = 16; o > 0; o >>= 1) u = min(u, __shfl_xor_sync(0xffffffffu, u, o));
  if ((threadIdx.x & 31) == 0) atomicMin(&c.drain_aux->min_u, u);
}

// how many cells share the smallest elevation, and whether any of them can
// receive area (an in-catchment cell, or a no-data cell below a neighbour)
__global__ void k_drain_mincount(const hc_view c, const double* __restrict__ el) {
  int i, j;
  if (!interior_ij(c, i, j)) return;
  const size_t W = c.W;
  const double e = el[(size_t)i * W + j];
  if (ukey(e) != c.drain_aux->min_u) return;
  atomicAdd(&c.drain_aux->min_count, 1u);
  bool matters = !(e == -9999);
  for (int dx = -1; dx <= 1; dx++)
    for (int dy = -1; dy <= 1; dy++) {
      const int i2 = i + dx, j2 = j + dy;
      if ((dx == 0 && dy == 0) || i2 < 1 || i2 > c.imax || j2 < 1 || j2 > c.jmax) continue;
      if (el[(size_t)i2 * W + j2] > e) matters = true;
    }
  if (matters) atomicOr(&c.drain_aux->min_matters, 1u);
}

// radix selection (8 bits a pass, most significant first) of the P-th
// largest key of the reference's sorted vector: the interior cells plus
// P = (imax+2)(jmax+2) - imax*jmax padding zeros
__global__ void k_sel_hist(const hc_view c, const double* __restrict__ el, int shift) {
  __shared__ unsigned int h[256];
  const int t = threadIdx.y * blockDim.x + threadIdx.x;
  const int nt = blockDim.x * blockDim.y;
  for (int k = t; k < 256; k += nt) h[k] = 0;
  __syncthreads();
  int i, j;
  const hc_drain_aux* a = c.drain_aux;
  if (interior_ij(c, i, j)) {
    const unsigned long long u = ukey(el[(size_t)i * c.W + j]);
    if ((u & a->mask) == a->prefix) atomicAdd(&h[(u >> shift) & 255], 1u);
  }
  __syncthreads();
  for (int k = t; k < 256; k += nt)
    if (h[k]) atomicAdd(&c.drain_aux->hist[k], h[k]);
}

// one block of 256 threads, a digit each: the suffix sums of the counts, then
// the digit whose sum is the first to reach k
__global__ void __launch_bounds__(256) k_sel_pick(const hc_view c, int shift,
                                                  unsigned long long padding) {
  __shared__ unsigned long long sum[256];
  hc_drain_aux* a = c.drain_aux;
  const int d = threadIdx.x;
  const unsigned long long zero_digit = (kZeroKey >> shift) & 255;
  const bool zero_in = (kZeroKey & a->mask) == a->prefix;
  const unsigned long long k = a->k;
  const unsigned real = a->hist[d];
  const unsigned long long n = real + ((zero_in && (unsigned)d == zero_digit) ? padding : 0);
  sum[d] = n;
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {
    const unsigned long long v = d + o < 256 ? sum[d + o] : 0;
    __syncthreads();
    sum[d] += v;
    __syncthreads();
  }
  const unsigned long long above = sum[d] - n;  // keys with a larger digit
  // k is at most the number of keys left, so one digit takes it
  if (above < k && sum[d] >= k) {
    a->real_eq = real;
    a->k = k - above;
    a->gt += above;
    a->prefix |= (unsigned long long)d << shift;
    a->mask |= 255ull << shift;
  }
  a->hist[d] = 0;
}

// sorted position of every cell the sweep reaches (1 .. imax*jmax); 0 = not
// reached
__global__ void k_drain_pos(const hc_view c, const uint32_t* __restrict__ order) {
  const size_t M = (size_t)c.imax * c.jmax;
  for (size_t n = 1 + (size_t)blockIdx.x * blockDim.x + threadIdx.x; n <= M;
       n += (size_t)gridDim.x * blockDim.x) {
    const uint32_t cell = order[n];
    if (cell != 0) c.drain_pos[cell] = (uint32_t)n;
  }
}

// per interior cell: the sum of downhill drops (difftot, the
// reference's clamped 8-neighbour loop in its order), the number of higher
// neighbours to wait for, whether
// the sweep reaches the cell (drain_pos 1/0: below the selected last
// position, and not the unique lowest cell), and whether two higher
// neighbours share an elevation
__global__ void k_drain_init(const hc_view c, const double* __restrict__ el) {
  int i, j;
  if (!interior_ij(c, i, j)) return;
  const size_t W = c.W;
  const size_t cell = (size_t)i * W + j;
  const double e = el[cell];
  double difftot = 0;
  for (int dir = 1; dir <= 8; dir++) {
    const int i2 = clampi(i + kDrX[dir], 1, c.imax), j2 = clampi(j + kDrY[dir], 1, c.jmax);
    const double e2 = el[(size_t)i2 * W + j2];
    if (dir % 2 != 0) {
      if (e2 < e) difftot += e - e2;
    } else {
      if (e2 < e) difftot += ddiv_by(e - e2, c.diagd);
    }
  }
  c.drain_dt[cell] = difftot;
  int higher = 0;
  double eh[8];
  bool tie = false;
  for (int dx = -1; dx <= 1; dx++)
    for (int dy = -1; dy <= 1; dy++) {
      const int i2 = i + dx, j2 = j + dy;
      if ((dx == 0 && dy == 0) || i2 < 1 || i2 > c.imax || j2 < 1 || j2 > c.jmax) continue;
      const double e2 = el[(size_t)i2 * W + j2];
      if (e2 > e) {
        for (int k = 0; k < higher; k++) tie |= (eh[k] == e2);
        eh[higher++] = e2;
      }
    }
  c.drain_pend[cell] = higher;
  if (tie) atomicOr(&c.drain_aux->contrib_tie, 1u);
  const hc_drain_aux* a = c.drain_aux;
  const unsigned long long u = ukey(e);
  const bool reached = !(u > a->prefix) &&
                       !(a->min_u < kZeroKey && a->min_count == 1 && u == a->min_u);
  c.drain_pos[cell] = reached ? 1u : 0u;
}

// A cell's terms, before the sweep: its higher neighbours that the sweep
// reaches, in sweep order (higher elevation first, equal elevations by sorted
// position), each with the share of its area that comes here: the
// reference's term (e_q - e)/difftot_q, or its diagonal form
// ((e_q - e)/1.414)/difftot_q, per direction of q whose (clamped) step lands
// here, in the order of the directions (one for an interior q, possibly two
// at the edges; never more than eight terms in all).  The sweep then adds
// area_q * share, the reference's operations on the same values, and its
// critical path has no division (about 600 cycles each on this GPU's FP64
// pipe, against 128 for a multiply and an add) and no ordering to find.
//
// drain_head of a cell: 4 bits per term with the neighbour's number
// 3*(di+1) + (dj+1), their count at bit 32, the mask of its lower neighbours
// (by number) at bit 36, bit 45 when the sweep reaches it, bit 46 when its
// own unit of area counts (not no-data).
constexpr int kHeadCount = 32, kHeadLower = 36, kHeadReached = 45, kHeadOwn = 46;

// Elevations are compared as integer keys (a NaN, below and above nothing, as
// the cell's own key), and quotients run on the integer pipe: a pick of the
// next higher neighbour is up to nine compares, which as FP64 instructions
// took most of the kernel's time: 1912 -> 232 us at 1500^2.
__global__ void __launch_bounds__(256) k_drain_terms(const hc_view c,
                                                     const double* __restrict__ el) {
  int i, j;
  if (!interior_ij(c, i, j)) return;
  const size_t W = c.W;
  const size_t cell = (size_t)i * W + j;
  const double e = el[cell];
  const long long ke = dkey(e);
  unsigned left = 0, lower = 0;
  long long kn[9];
  uint32_t pn[9];
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const int iq = i + k / 3 - 1, jq = j + k % 3 - 1;
    const bool in = k != 4 && iq >= 1 && iq <= c.imax && jq >= 1 && jq <= c.jmax;
    const size_t q = (size_t)iq * W + jq;
    const double en = in ? el[q] : e;
    kn[k] = disnan(en) || disnan(e) ? ke : dkey(en);
    pn[k] = in ? c.drain_pos[q] : 0u;
    if (kn[k] > ke && pn[k] != 0) left |= 1u << k;
    if (kn[k] < ke) lower |= 1u << k;
  }
  const bool reached = c.drain_pos[cell] != 0;
  unsigned long long head = ((unsigned long long)lower << kHeadLower) |
                            ((unsigned long long)reached << kHeadReached) |
                            ((unsigned long long)(ke != kNoDataKey) << kHeadOwn);
  int n = 0;
  if (reached) {
    double* share = c.drain_share + cell * 8;
#pragma unroll 1
    while (left) {
      int best = -1;
      long long bk = 0;
      uint32_t bp = 0;
#pragma unroll
      for (int k = 0; k < 9; k++) {
        if (!((left >> k) & 1u)) continue;
        if (best < 0 || kn[k] > bk || (kn[k] == bk && pn[k] > bp)) {
          best = k;
          bk = kn[k];
          bp = pn[k];
        }
      }
      left &= ~(1u << best);
      const int di = best / 3 - 1, dj = best - 3 * (di + 1) - 1;
      const int iq = i + di, jq = j + dj;
      const size_t q = (size_t)iq * W + jq;
      const double drop = el[q] - e;
      const double dq = c.drain_dt[q];
      if (iq > 1 && iq < c.imax && jq > 1 && jq < c.jmax) {  // one direction of q lands here
        share[n] = ddiv_rn(di != 0 && dj != 0 ? ddiv_by(drop, c.diagd) : drop, dq);
        head |= (unsigned long long)best << (4 * n);
        n++;
        continue;
      }
#pragma unroll 1
      for (int dir = 1; dir <= 8; dir++) {
        const int i3 = clampi(iq + kDrX[dir], 1, c.imax), j3 = clampi(jq + kDrY[dir], 1, c.jmax);
        if (i3 != i || j3 != j) continue;
        share[n] = ddiv_rn(dir % 2 != 0 ? drop : ddiv_by(drop, c.diagd), dq);
        head |= (unsigned long long)best << (4 * n);
        n++;
      }
    }
  }
  c.drain_head[cell] = head | ((unsigned long long)n << kHeadCount);
  // not yet summed: no area is a NaN
  c.area[cell] = bits_d(-1LL);
}

// The sweep's shared state, all zero at the start.
struct DrainSync {
  unsigned long long done;  // cells finished
  unsigned int tail;        // queue entries appended
  unsigned int taken;       // queue entries handed out
  unsigned int hops;        // cells on the longest chain of releases
  unsigned int err;         // a wait ran out
};

constexpr int kSweepThreads = 128;
constexpr int kSweepBlocks = 2;  // per multiprocessor
constexpr unsigned kReportTurns = 256;  // about half a millisecond
constexpr int kSpareMax = 32 * 8;  // per lane: 8 released but one it keeps, and a queue entry

// The first frontier's cells (no higher neighbour), as queue entries: a warp
// takes 32 columns of kSeedRows rows, and a block's eight warps one atomic (a
// set-up at 1500^2 took 50 us longer with one per warp and row).
constexpr int kSeedRows = 8;

__global__ void __launch_bounds__(256) k_drain_seed(const hc_view c, DrainSync* g,
                                                    unsigned long long* queue) {
  __shared__ unsigned count[8], base;
  const unsigned lane = threadIdx.x, warp = threadIdx.y;
  const int j = 1 + blockIdx.x * 32 + lane;
  const int i0 = 1 + (blockIdx.y * 8 + warp) * kSeedRows;
  unsigned m[kSeedRows], n = 0;
#pragma unroll
  for (int r = 0; r < kSeedRows; r++) {
    const bool in = i0 + r <= c.imax && j <= c.jmax;
    m[r] = __ballot_sync(0xffffffffu, in && c.drain_pend[(size_t)(i0 + r) * c.W + j] == 0);
    n += __popc(m[r]);
  }
  if (lane == 0) count[warp] = n;
  __syncthreads();
  if (lane == 0 && warp == 0) {
    unsigned all = 0;
    for (int w = 0; w < 8; w++) all += count[w];
    base = all ? atomicAdd(&g->tail, all) : 0u;
  }
  __syncthreads();
  unsigned at = base;
  for (unsigned w = 0; w < warp; w++) at += count[w];
#pragma unroll
  for (int r = 0; r < kSeedRows; r++) {
    if ((m[r] >> lane) & 1u)
      queue[at + __popc(m[r] & ((1u << lane) - 1u))] =
          (1ull << 32) | (uint32_t)((size_t)(i0 + r) * c.W + j);
    at += __popc(m[r]);
  }
}

__device__ __forceinline__ unsigned long long ld_relaxed(const void* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// Predicated forms, without a branch around each: a lane's loads (or atomics)
// are issued one behind the other and their latencies overlap.
__device__ __forceinline__ unsigned long long ld_relaxed_if(bool on, const void* p) {
  unsigned long long v;
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n mov.u64 %0, 0;\n"
      " @p ld.relaxed.gpu.global.u64 %0, [%1];\n}"
      : "=l"(v)
      : "l"(p), "r"((unsigned)on)
      : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_const_if(bool on, const void* p) {
  unsigned long long v;
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n mov.u64 %0, 0;\n"
      " @p ld.global.nc.u64 %0, [%1];\n}"
      : "=l"(v)
      : "l"(p), "r"((unsigned)on));
  return v;
}
__device__ __forceinline__ int count_down_if(bool on, int* p) {  // the old count, 0 when off
  int v;
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n mov.u32 %0, 0;\n"
      " @p atom.relaxed.gpu.global.add.s32 %0, [%1], -1;\n}"
      : "=r"(v)
      : "l"(p), "r"((unsigned)on)
      : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(void* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The accumulation, without frontiers or barriers: a lane sums a ready cell,
// stores its area, counts down its lower neighbours and goes on with one that
// this made ready; the others go to a queue, from which lanes without a cell
// take theirs in turn.  The areas themselves tell when they are there (a NaN
// until then), so no fence stands between a cell's sum and its neighbours'
// counts; a lane that was handed a cell before the last area arrived asks
// again.  Lanes never wait for a block that is not running: an entry's lane
// took its number while it ran.
//
// What bounds it is the longest path down the terrain (2,000 to 3,200 cells
// at 1024^2 to 2000^2) times one cell's latency.  A cell costs two round trips
// to L2: one for its shares and its neighbours' areas, one for the counts of
// its lower neighbours, whose heads come along with it, so that the next
// cell's terms are known when its count is; the loads and atomics of a
// round trip are predicated instructions in a row (as branches they ran one
// after the other: 4,300 cycles for the counts instead of 1,400).  The
// queue's loads are issued with the first round trip and its entries written
// behind it; cells that a lane releases beyond one go to idle lanes of its
// warp before the queue.
// Frontier by frontier (grid barriers, or one block alone on small frontiers)
// a cell of the path took 9-10 us, now 2 us: 18.1 -> 4.0 ms at 1024^2,
// 32 -> 7.0 ms at 2000^2.  More or fewer warps than two blocks of 128 per
// multiprocessor are slower (one: 7.1, four: 7.7 ms at 2000^2).
__global__ void __launch_bounds__(kSweepThreads) k_drain_sweep(const hc_view c, DrainSync* g,
                                                               unsigned long long* queue) {
  const unsigned FULL = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31;
  const int W = (int)c.W;
  const bool test = c.wait_spins > 0;  // a test shortens the waits and has them run out
  const unsigned limit = test ? (unsigned)c.wait_spins : 1u << 24;
  const unsigned long long M =
      (unsigned long long)c.imax * c.jmax + (test ? (unsigned)c.barrier_extra : 0u);
  uint32_t cell = 0;             // 0: none (cell 0 is a padding cell)
  unsigned long long head = 0;   // of `cell`
  unsigned hop = 0, most = 0;
  unsigned slot = 0;
  bool ticket = false;           // the lane waits for queue entry `slot`
  unsigned finished = 0;         // cells finished by the lane since the last report
  unsigned turn = 0;
  unsigned waited = 0;           // turns the lane has waited for its cell's areas
  // lane 0: the cells finished when it last looked, and its looks since then
  unsigned long long done = 0;
  unsigned idle = 0;
  __shared__ uint4 spare[kSweepThreads / 32][kSpareMax];  // released: cell, hop, head
  uint4* mine = spare[threadIdx.x >> 5];
  unsigned out0 = 0, out1 = 0;   // of them, [out0, out1) go to the queue ...
  unsigned base = 0;             // ... at this place (lane 0)
  for (;;) {
    // first round trip: the cell's terms, or the lane's queue entry
    const int n = cell != 0 ? (int)(head >> kHeadCount) & 15 : 0;
    const double* share = c.drain_share + (size_t)cell * 8;
    unsigned long long s[8], a[8];
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const int k = (int)(head >> (4 * t)) & 15;
      s[t] = ld_const_if(t < n, share + t);
      a[t] = ld_relaxed_if(t < n, c.area + ((int)cell + (k / 3 - 1) * W + k % 3 - 1));
    }
    const unsigned long long q = ld_relaxed_if(ticket && slot < (unsigned)c.N2, queue + slot);
    // the last turn's released cells, at the place their atomic gave
    if (out1 > out0) {
      const unsigned m = __shfl_sync(FULL, base, 0);
      for (unsigned k = out0 + lane; k < out1; k += 32)
        st_relaxed(queue + m + (k - out0),
                   ((unsigned long long)mine[k].y << 32) | mine[k].x);
      __syncwarp();
      out1 = out0 = 0;
    }
    bool ready = cell != 0;
#pragma unroll
    for (int t = 0; t < 8; t++) ready = ready && a[t] != ~0ull;
    const int n_warp = (int)__reduce_max_sync(FULL, (unsigned)n);
    uint32_t next = ready ? 0u : cell;
    unsigned long long next_head = head;
    unsigned next_hop = hop, rel = 0;
    unsigned long long hd[9];
    if (ready) {
      double sum = ((head >> kHeadOwn) & 1u) ? 1.0 : 0.0;
#pragma unroll
      for (int t = 0; t < 8; t++)  // the terms past n are +0, which adds nothing
        if (t < n_warp)
          sum += bits_d((long long)a[t]) * bits_d((long long)s[t]);
      if (!((head >> kHeadReached) & 1u) || !(sum > 0)) sum = 0;
      st_relaxed(c.area + cell, (unsigned long long)dbits(sum));
      // second round trip: the lower neighbours' counts and heads
      const unsigned lower = (unsigned)(head >> kHeadLower) & 0x1ffu;
      int old[9];
#pragma unroll
      for (int k = 0; k < 9; k++) {
        const int nb = (int)cell + (k / 3 - 1) * W + k % 3 - 1;
        const bool low = k != 4 && ((lower >> k) & 1u);
        old[k] = count_down_if(low, &c.drain_pend[nb]);
        hd[k] = ld_const_if(low, c.drain_head + nb);
      }
#pragma unroll
      for (int k = 8; k >= 0; k--)
        if (old[k] == 1) {
          rel |= 1u << k;
          next = (uint32_t)((int)cell + (k / 3 - 1) * W + k % 3 - 1);
          next_head = hd[k];
        }
      rel &= rel - 1;  // the lane goes on with the lowest of them itself
      next_hop = hop + 1;
      finished++;
      waited = 0;
      most = max(most, hop);
    } else if (cell != 0) {
      waited++;  // an area still on its way
    }
    // the lane's queue entry: its own when it is idle (it may have been given
    // a cell by another lane since it took its number), else one more to share
    bool extra = false;
    unsigned long long q_head = 0;
    if (q) {
      q_head = __ldg(c.drain_head + (uint32_t)q);
      ticket = false;
      if (next == 0) {
        next = (uint32_t)q;
        next_hop = (unsigned)(q >> 32);
        next_head = q_head;
      } else {
        extra = true;
      }
    }
    const unsigned cnt = __popc(rel) + (extra ? 1u : 0u);
    if (__any_sync(FULL, cnt != 0)) {
      // cells beyond one per lane: to the warp's idle lanes first (a cell that
      // goes by the queue loses two more round trips), the rest to the queue
      unsigned incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(FULL, incl, o);
        if (lane >= (unsigned)o) incl += y;
      }
      const unsigned total = __shfl_sync(FULL, incl, 31);
      unsigned m = incl - cnt;
#pragma unroll
      for (int k = 0; k < 9; k++)
        if ((rel >> k) & 1u)
          mine[m++] = make_uint4((unsigned)((int)cell + (k / 3 - 1) * W + k % 3 - 1), hop + 1,
                                 (unsigned)hd[k], (unsigned)(hd[k] >> 32));
      if (extra)
        mine[m] = make_uint4((unsigned)q, (unsigned)(q >> 32), (unsigned)q_head,
                             (unsigned)(q_head >> 32));
      __syncwarp();
      const unsigned free = __ballot_sync(FULL, next == 0);
      const unsigned take = min(total, (unsigned)__popc(free));
      const unsigned r = __popc(free & ((1u << lane) - 1u));
      if (next == 0 && r < take) {
        const uint4 e = mine[r];
        next = e.x;
        next_hop = e.y;
        next_head = ((unsigned long long)e.w << 32) | e.z;
      }
      out0 = take;
      out1 = total;
      if (lane == 0 && total > take) base = atomicAdd(&g->tail, total - take);
    }
    cell = next;
    head = next_head;
    hop = next_hop;
    // a queue number for each lane that needs one, one atomic per warp
    const unsigned want = __ballot_sync(FULL, cell == 0 && !ticket);
    if (want) {
      unsigned first = 0;
      const int leader = __ffs(want) - 1;
      if ((int)lane == leader) first = atomicAdd(&g->taken, (unsigned)__popc(want));
      first = __shfl_sync(FULL, first, leader);
      if ((want >> lane) & 1u) {
        slot = first + __popc(want & ((1u << lane) - 1u));
        ticket = true;
      }
    }
    // Report what was finished: with nothing to do, and every kReportTurns
    // turns of work, so that the warps that wait see the sweep move.  With
    // nothing to do, leave when every cell is finished, or when none was for
    // as many looks as the bound allows.
    const bool quiet = out1 == out0 && !__any_sync(FULL, cell != 0);
    if (quiet || ++turn == kReportTurns) {
      turn = 0;
      unsigned f = finished;
      for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(FULL, f, o);
      finished = 0;
      unsigned stop = 0;
      if (lane == 0) {
        if (f) atomicAdd(&g->done, (unsigned long long)f);
        if (quiet) {
          const unsigned long long now = ld_relaxed(&g->done);
          if (now != done) idle = 0;
          done = now;
          if (now >= M) {
            stop = 1;
          } else if (++idle > limit || *(volatile unsigned*)&g->err) {
            atomicExch(&g->err, 1u);
            stop = 1;
          } else {
            __nanosleep(64);
          }
        }
      }
      if (__any_sync(FULL, waited > limit)) {
        if (lane == 0) atomicExch(&g->err, 1u);
        break;
      }
      if (__shfl_sync(FULL, stop, 0)) break;
    }
  }
  for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(FULL, most, o));
  if (lane == 0) atomicMax(&g->hops, most);
}

// the sweep's outcome into the control block
__global__ void k_drain_end(hc_dev* d, const DrainSync* g) {
  d->drain_done = (unsigned)g->done;
  d->drain_levels = g->hops;
  if (g->err) {
    d->err_code = 401;
    d->pause |= HC_PAUSE_ERROR;
  }
}

// get_catchment_input_points: cells in row-major order whose
// area*baseflow*3*DX*DX lies strictly between MIN_Q and MIN_Q_MAXVAL
__device__ __forceinline__ bool input_point(const hc_view& c, const hc_dev* d, size_t cell) {
  const int i = (int)(cell / c.W), j = (int)(cell % c.W);
  if (i < 1 || i > c.imax || j < 1 || j > c.jmax) return false;
  const double DX = c.p.DX;
  const double q = c.area[cell] * d->s.baseflow * 3 * DX * DX;
  return q > c.p.MIN_Q && q < c.p.MIN_Q_MAXVAL;
}

__global__ void __launch_bounds__(1024) k_points_count(const hc_view c, const hc_dev* d) {
  __shared__ int ws[32];
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  int v = (k < c.N2 && input_point(c, d, k)) ? 1 : 0;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int w = 0; w < 32; w++) s += ws[w];
    c.wet_sums[blockIdx.x] = s;
  }
}

__global__ void __launch_bounds__(1024) k_points_scan(const hc_view c, hc_dev* d, int nblocks) {
  __shared__ int buf[1024];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nblocks; base += 1024) {
    const int k = base + threadIdx.x;
    const int v = (k < nblocks) ? c.wet_sums[k] : 0;
    buf[threadIdx.x] = v;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
      const int t = (threadIdx.x >= (unsigned)off) ? buf[threadIdx.x - off] : 0;
      __syncthreads();
      buf[threadIdx.x] += t;
      __syncthreads();
    }
    if (k < nblocks) c.wet_sums[k] = carry + buf[threadIdx.x] - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += buf[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) d->drain_points = (unsigned)carry;
}

__global__ void __launch_bounds__(1024) k_points_write(const hc_view c, hc_dev* d) {
  __shared__ int ws[32], wb[32];
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool v = k < c.N2 && input_point(c, d, k);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v ? 1 : 0;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) ws[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int w = 0; w < 32; w++) {
      wb[w] = s;
      s += ws[w];
    }
  }
  __syncthreads();
  if (v) {
    const int t = 1 + c.wet_sums[blockIdx.x] + wb[warp] + incl - 1;  // 1-based, as the reference
    c.cin_x[t] = (int32_t)(k / c.W);
    c.cin_y[t] = (int32_t)(k % c.W);
    const int rf = c.rfarea[k];
    const unsigned same = __match_any_sync(__activemask(), rf);  // one atomic per warp and zone
    if (rf >= 0 && rf <= HC_MAX_RF && lane == __ffs(same) - 1)
      atomicAdd(&d->drain_rf[rf], (unsigned)__popc(same));
  }
}

// totalinputpoints and catchment_input_counter (entries 1..rfnum restart
// from zero; an rfarea of 0 keeps adding to entry 0, as in the reference)
__global__ void k_points_finish(const hc_view c, hc_dev* d) {
  hc_scalars& s = d->s;
  for (int n = 1; n <= c.p.rfnum && n <= HC_MAX_RF; n++) s.catchment_input_counter[n] = 0;
  for (int n = 0; n <= HC_MAX_RF; n++) {
    if (n <= c.p.rfnum) s.catchment_input_counter[n] += (double)d->drain_rf[n];
    d->drain_rf[n] = 0;
  }
  const unsigned t = d->drain_points;
  s.totalinputpoints = (t == 0) ? 1.0 : (double)t;
}

// count_catchment_gridcells :2813: the cells of rows 1 .. imax-1, columns
// 1 .. jmax-1 above no-data, by zone; bad: the first cell whose zone is out
// of range
__global__ void __launch_bounds__(256) k_zone_count(const hc_view c, unsigned int* counts,
                                                    unsigned int* bad) {
  __shared__ unsigned int h[HC_MAX_RF + 1];
  for (int k = threadIdx.x; k <= HC_MAX_RF; k += blockDim.x) h[k] = 0;
  __syncthreads();
  const size_t n = (size_t)(c.imax - 1) * c.W;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    const size_t cell = c.W + k;
    const int j = (int)(k % c.W);
    const double e = c.elev[cell];
    if (j < 1 || j >= c.jmax || !(e > -9999)) continue;
    const int r = c.rfarea[cell];
    if (r < 0 || r > c.p.rfnum) {
      atomicMin(bad, (unsigned)cell);
      continue;
    }
    const unsigned same = __match_any_sync(__activemask(), r);
    if ((int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&h[r], (unsigned)__popc(same));
  }
  __syncthreads();
  for (int k = threadIdx.x; k <= HC_MAX_RF; k += blockDim.x)
    if (h[k]) atomicAdd(&counts[k], h[k]);
}

}  // namespace

// nActualGridCells per zone (HC_MAX_RF + 1 entries) by the device; *bad_zone
// receives an out-of-range zone (of the first such cell) and *ok tells.
hc_status count_zone_cells(hc_ctx* c, double* cells, bool* ok, int* bad_zone) {
  unsigned int* n = (unsigned int*)c->v.drain_aux->hist;  // scratch until the next selection
  unsigned int h[HC_MAX_RF + 2];
  cudaStream_t s = c->s;
  cudaError_t e = cudaMemsetAsync(n, 0, (HC_MAX_RF + 1) * 4, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(n + HC_MAX_RF + 1, 0xff, 4, s);
  if (e == cudaSuccess) {
    k_zone_count<<<c->sms * 4, 256, 0, s>>>(c->v, n, n + HC_MAX_RF + 1);
    count_launch(c, 1);
    e = cudaMemcpyAsync(h, n, sizeof h, cudaMemcpyDeviceToHost, s);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return hc_cuda(c, e, "prepare");
  c->d2h_bytes += sizeof h;
  for (int k = 0; k <= HC_MAX_RF; k++) cells[k] = (double)h[k];
  *ok = h[HC_MAX_RF + 1] == 0xffffffffu;
  if (!*ok) {
    e = cudaMemcpy(bad_zone, c->v.rfarea + h[HC_MAX_RF + 1], 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return hc_cuda(c, e, "prepare");
  }
  return HC_OK;
}

// The drainage area for the elevations `el` (device), then the input points.
// `sort_order` is called, and its order used, only when the sort's order
// among equal elevations can show (see the top of the file).  Returns HC_OK,
// or HC_ERR_CUDA; *sorted tells which way it went.
hc_status run_drainage_device(hc_ctx* c, const double* el, bool area_valid,
                              hc_status (*sort_order)(hc_ctx*, const double*, uint32_t*),
                              bool* sorted) {
  hc_view& v = c->v;
  const size_t N2 = v.N2;
  cudaStream_t s = c->s;
  *sorted = false;
  if (!area_valid) {
    const unsigned long long M = (unsigned long long)v.imax * v.jmax;
    const unsigned long long P = N2 - M;
    hc_drain_aux a0;
    std::memset(&a0, 0, sizeof a0);
    a0.min_u = ~0ull;
    a0.k = P;
    if (cudaMemcpyAsync(v.drain_aux, &a0, sizeof a0, cudaMemcpyHostToDevice, s) != cudaSuccess)
      return HC_ERR_CUDA;
    dim3 b(32, 8);
    dim3 g((v.jmax + 31) / 32, (v.imax + 7) / 8);
    k_drain_min<<<g, b, 0, s>>>(v, el);
    k_drain_mincount<<<g, b, 0, s>>>(v, el);
    for (int shift = 56; shift >= 0; shift -= 8) {
      k_sel_hist<<<g, b, 0, s>>>(v, el, shift);
      k_sel_pick<<<1, 256, 0, s>>>(v, shift, P);
    }
    k_drain_init<<<g, b, 0, s>>>(v, el);
    c->launches += 19;
    hc_drain_aux a;
    if (cudaMemcpyAsync(&a, v.drain_aux, sizeof a, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return HC_ERR_CUDA;
    c->d2h_bytes += sizeof a;
    const bool top_ok = a.gt == P - 1 || (a.prefix == kZeroKey && a.real_eq == 0);
    const bool bottom_ok =
        a.min_u > kZeroKey || (a.min_u < kZeroKey && (a.min_count == 1 || !a.min_matters));
    if (a.contrib_tie || !top_ok || !bottom_ok) {
      uint32_t* order = (uint32_t*)v.drain_share;  // free until the terms are formed
      if (sort_order(c, el, order) != HC_OK) return HC_ERR_CUDA;
      if (cudaMemsetAsync(v.drain_pos, 0, N2 * 4, s) != cudaSuccess) return HC_ERR_CUDA;
      k_drain_pos<<<152 * 4, 256, 0, s>>>(v, order);
      c->launches += 1;
      *sorted = true;
    }
    k_drain_terms<<<g, b, 0, s>>>(v, el);
    // the queue takes the place of difftot, which only the terms needed; the
    // sweep's state that of the selection's histogram, which is finished
    static_assert(sizeof(DrainSync) <= sizeof(hc_drain_aux::hist), "sweep state fits");
    DrainSync* gs = (DrainSync*)((char*)v.drain_aux + offsetof(hc_drain_aux, hist));
    unsigned long long* queue = (unsigned long long*)v.drain_dt;
    if (cudaMemsetAsync(gs, 0, sizeof(DrainSync), s) != cudaSuccess ||
        cudaMemsetAsync(queue, 0, N2 * 8, s) != cudaSuccess)
      return HC_ERR_CUDA;
    const int seed_rows = 8 * kSeedRows;
    k_drain_seed<<<dim3((v.jmax + 31) / 32, (v.imax + seed_rows - 1) / seed_rows), b, 0, s>>>(
        v, gs, queue);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    const int nblocks = (int)std::max<size_t>(
        1, std::min<size_t>((size_t)c->sms * kSweepBlocks, (M + 1023) / 1024));
    k_drain_sweep<<<nblocks, kSweepThreads, 0, s>>>(v, gs, queue);
    cudaEventRecord(e1, s);
    k_drain_end<<<1, 1, 0, s>>>(c->dev, gs);
    c->launches += 4;
    if (cudaEventSynchronize(e1) == cudaSuccess) {
      float ms = 0;
      cudaEventElapsedTime(&ms, e0, e1);
      c->stat_n[HC_STAT_DRAINAGE_SWEEP]++;
      c->stat_ms[HC_STAT_DRAINAGE_SWEEP] += ms;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }
  const int nb = (int)((N2 + 1023) / 1024);
  k_points_count<<<nb, 1024, 0, s>>>(v, c->dev);
  k_points_scan<<<1, 1024, 0, s>>>(v, c->dev, nb);
  k_points_write<<<nb, 1024, 0, s>>>(v, c->dev);
  k_points_finish<<<1, 1, 0, s>>>(v, c->dev);
  c->launches += 4;
  return cudaGetLastError() == cudaSuccess ? HC_OK : HC_ERR_CUDA;
}
