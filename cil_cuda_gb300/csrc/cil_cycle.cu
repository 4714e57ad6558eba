// The single-element cell-cycle model on the GPU (include/cil_cycle.h).
//
// Layout: structure of arrays in index order (cell i at i), FP64. Two complete state sets;
// a removal (apoptosis, drain) compacts the survivors stably into the other set and the host
// flips the set index. The pair passes read copies in bin order (CyOrdered), so they update the
// state in place.
//
// A step (no host synchronisation; the cell count lives on the device):
//   bins       k_cy_keys / scan / k_cy_scatter / k_cy_place: a counting sort of the cells into
//              bins (width set per call from the largest diameter), ascending cell index
//              inside a bin, with copies of the positions and diameters in that order; the pair
//              search walks +-k bins with k from the colony's largest diameter of the previous
//              step, so growing cells never outgrow the search;
//   forces     k_cy_force: Hertz contacts with adhesion and the pressure sum, motility along the
//              velocity, passive noise, the position update with the pressure-dependent friction,
//              and the cell's cycle (ODEs, division test);
//   divisions  k_cy_divide (daughters appended in mother order; the step's counts);
//   apoptosis  k_cy_mark / scan / k_cy_compact (only with apoptosis on).
// The DPD integrator: k_cy_keys makes the first half kick and the drift, k_dpd_forces the conservative
// forces and the pressure, the pair dissipative and random forces and the second half kick (into the
// spare velocity buffer), k_dpd_dis background and pair dissipation
// at the new velocities and the cell's cycle; then the same divisions and apoptosis.
// The file is compiled without FMA contraction: outside the forms of "FP64 arithmetic" (cil_internal.cuh), the
// arithmetic is that of the host restatement the tests compare with, to a few units of the last place.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "cil_cycle.h"
#include "cil_internal.cuh"

// Axis loops: unrolled to three with a guard, so that per-axis arrays stay in registers (the
// dimension is a run-time value)
#define CY_AXES(d, D) _Pragma("unroll") for (int d = 0; d < 3; ++d) if (d < (D))

namespace {

using cil::kTile;
using cil::finite_bits;
using cil::mid_range;
using cil::philox4x32_10;
using cil::rcp_normal;
using cil::rsqrt_pos;
using cil::sqrt_from;
using cil::u32x4;

constexpr double kPi = 3.14159265358979323846;
constexpr double kLn2 = 0.69314718055994530942;
constexpr int kScanTile = 1024;  // elements per block of the scans

// Philox purposes (third counter word)
constexpr uint32_t kCyNoise = 11, kCyDir = 12, kCyDiv = 13, kCyApo = 14, kCyInit = 15;
// DPD pair normals: counter (lower cell index, step, purpose, higher cell index)
constexpr uint32_t kCyDpd0 = 16, kCyDpd1 = 17;

struct CyConst {
  int D;
  int periodic[3];
  double box[3];
  double dt;
  int ns[3];
  double bw[3];       // bin width per axis
  float bwf[3], boxf[3], halff[3];  // FP32 copies for the range tests and FP32 separations
  double half[3];     // box / 2
  float inv_bwf[3];   // bins per length, rounded up
  float scalef[3];    // and to the nearest
  double inv_bw[3];
  double sigma_core;
  double hz_c;        // (1 - nu^2) / E
  float c2f, adhf, gdf, srf;  // FP32: 2 hz_c, adhesion, gamma_d, sigma_r
  double adhesion;
  double motility, zeta, zeta_p, zeta_p_beta;
  double noise_amp;   // sqrt(2 D) / sqrt(dt)
  int divide;
  int apoptosis;
  double tau_div_mu, tau_div_sigma, tau_mig_mu, tau_mig_sigma;
  double v1, tau_r, tau_v, tau_p;   // tau_* in steps
  double v_s;
  double growth, inv_vs_tau_v, inv_tau_r, inv_tau_r_neg, inv_p0;  // (v1 - 1) / tau_v, reciprocals
  double inv_hz;          // 1 / (0.75 c2), c2 = 2 (1 - nu^2) / E
  double div_mu2, div_s2; // log-normal parameters of the cycle time
  double p0, beta_vs, rho_ratio, r_maxed_inv, p_shift, p_shift_tau_inv, osm;
  double apop_pressure, apop_duration, apop_rate_step, extr_gamma;
  double apop_steps;  // apop_duration / dt
  double extr_rate;
  // DPD
  int dpd;
  double kick_f, kick_r;  // dt and sqrt(dt) over 2 (2 m), updateVel's divisor with the mass argument 2 m
  double gamma_d, gamma_b, sigma_r;  // DISDIFCEL, DISBG, sqrt(2 DISDIFCEL kT)
  uint32_t seed_lo, seed_hi;
  int capacity;
};

struct CySet {
  double *x;      // [D][cap]
  double *v;      // [D][cap]
  double *sig, *sigt, *theta, *rho, *om, *p;
  int *tp, *t0, *tsw;
  double *fc, *fd, *fr;  // [D][cap], DPD only (conservative, dissipative, random forces)
};

// The cells in bin order, written by k_cy_place for the pair kernels: [q] is the cell at place q.
struct CyOrdered {
  double *x;    // [D][cap]
  double *rad;  // radius (sigma / 2, exact)
  float4 *rec;  // FP32 position (z 0 in 2D) and diameter, for the range tests
  float4 *vel;  // FP32 velocity (DPD, precision 1)
  float4 *loc;  // FP32 position relative to the origin of the cell's bin (z 0 in 2D) and diameter (DPD, precision 1)
  ushort4 *cell;  // the bin's place along each axis (DPD, precision 1)
  int *idx;     // the cell's index
  int *bin;
};

struct CyCounters {
  int n;
  int err;
  long long ndiv_total;
  long long napo_total;
  unsigned long long sigma_max_bits;  // largest diameter (non-negative doubles order like their bits)
  unsigned long long sigma_next_bits;  // the same, of the step under way (k_cy_divide)
  int ndiv_step;
  int nrem_step;
  int ndue;   // cells at phase 1, of the step under way
  int ndone;  // blocks of k_cy_divide that have finished
};

constexpr int kErrCapacity = 1;
constexpr int kErrNonFinite = 2;
constexpr int kErrOutOfBox = 4;
constexpr int kErrCrowded = 8;     // a bin holds more than kBinSortMax cells
constexpr int kDueMax = 1024;      // dividing cells ranked from a queue (more: by a scan of the cells)
constexpr int kBinSortMax = 256;   // cells a bin may hold (about 1 at the bin width used)

// ---------------------------------------------------------------- draws
__host__ __device__ inline double u53(uint32_t a, uint32_t b) {
  const uint64_t m = (static_cast<uint64_t>(a) << 21) ^ (static_cast<uint64_t>(b) >> 11);
  return static_cast<double>(m & ((1ull << 53) - 1)) * 1.1102230246251565e-16;
}

// Two standard normals (Box-Muller, FP64) from the four words of one Philox block.
__device__ inline void normal2(const u32x4 &r, double *n0, double *n1) {
  const double a = 1.0 - u53(r.v[0], r.v[1]);  // (0, 1]
  const double b = u53(r.v[2], r.v[3]);
  const double rad = sqrt(-2.0 * log(a));
  const double ang = 6.283185307179586 * b;
  *n0 = rad * cos(ang);
  *n1 = rad * sin(ang);
}

__device__ inline u32x4 draw(const CyConst &C, uint32_t cell, int ts, uint32_t purpose, uint32_t sub) {
  return philox4x32_10(cell, static_cast<uint32_t>(ts), purpose, sub, C.seed_lo, C.seed_hi);
}

__device__ inline int nint(double a) { return a >= 0.0 ? static_cast<int>(a + 0.5) : static_cast<int>(a - 0.5); }

// max(Nint(x / dt), 1) (randomTimeSpan, MD.cuh:434-436)
__device__ inline int span_steps(double x, double dt) {
  const int s = nint(x / dt);
  return s > 1 ? s : 1;
}

// ---------------------------------------------------------------- geometry (Utils.hpp:223-256)
__device__ inline double area_of(double s) { return kPi * ((s / 2) * (s / 2)); }
__device__ inline double volume_of(double s) { return 4 * kPi * ((s / 2) * (s / 2) * (s / 2)) / 3; }
__device__ inline double sigma_of_area(double a) { return 2 * sqrt(a / kPi); }
__device__ inline double sigma_of_volume(double v) { return 2 * cbrt(3 * v / (4 * kPi)); }

__device__ inline double contact_area(double r, double a, double b) {
  const double ra = a / 2, rb = b / 2;
  const double u = r * r - rb * rb + ra * ra;
  const double t = sqrt(4 * (r * r) * (ra * ra) - u * u) / (2 * r);
  return t > 0 ? kPi * (t * t) : 0.0;
}

__device__ inline double wrap(double t, double L) { return cil::wrap_bits(t, L); }  // fmod(t + L, L)

__device__ inline int bin_of(const CyConst &C, const double *xd) {
  int b = 0;
  CY_AXES(d, C.D) {
    int v = cil::floor_scaled(xd[d], C.scalef[d], [&] { return xd[d] * C.inv_bw[d]; });
    v = v < 0 ? 0 : (v >= C.ns[d] ? C.ns[d] - 1 : v);
    b = b * C.ns[d] + v;
  }
  return b;
}

__device__ inline float f4c(const float4 &v, int d) { return d == 0 ? v.x : (d == 1 ? v.y : v.z); }

// ---------------------------------------------------------------- block scan
// Exclusive scan over the block (any multiple of 32 threads up to kTile)
__device__ inline int block_excl_scan(int v, int *total) {
  __shared__ int ws[kTile / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) ws[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    int w = lane < nw ? ws[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    if (lane < nw) ws[lane] = w;
  }
  __syncthreads();
  const int base = wid > 0 ? ws[wid - 1] : 0;
  *total = ws[nw - 1];
  __syncthreads();
  return base + inc - v;
}

// Exclusive scan of `count[0..m)` in place by one block; count[m] receives the total.
__global__ void k_cy_scan_small(int *count, int m) {
  int carry = 0;
  for (int base = 0; base < m; base += kTile) {
    const int i = base + threadIdx.x;
    const int v = i < m ? count[i] : 0;
    int tot;
    const int ex = block_excl_scan(v, &tot);
    if (i < m) count[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) count[m] = carry;
}

// Block sums of kScanTile-sized chunks (4 per thread)
__global__ void k_cy_chunk_sums(const int *count, int m, int *part) {
  cil::enter_step_kernel();
  const int b0 = blockIdx.x * kScanTile + threadIdx.x * 4;
  int s = 0;
  for (int q = 0; q < 4; ++q) s += (b0 + q < m) ? count[b0 + q] : 0;
  int tot;
  block_excl_scan(s, &tot);
  if (threadIdx.x == 0) part[blockIdx.x] = tot;
}

// Exclusive scan of count[0..m) into start[0..m] (start[m] = total; the chunks cover index m,
// count[m] reads as 0); count is left at zero. part: the chunk sums, scanned when `scanned`, otherwise
// each block adds those before it itself (a few loads per thread, cheaper than a launch).
__global__ void k_cy_chunk_apply(int *count, int m, const int *part, int *start, int scanned) {
  cil::enter_step_kernel();
  const int b0 = blockIdx.x * kScanTile + threadIdx.x * 4;
  int c[4], s = 0;
  for (int q = 0; q < 4; ++q) {
    c[q] = (b0 + q < m) ? count[b0 + q] : 0;
    if (b0 + q < m) count[b0 + q] = 0;
    s += c[q];
  }
  int before = 0;
  if (scanned) {
    before = part[blockIdx.x];
  } else {
    int v = 0;
    for (int u = threadIdx.x; u < static_cast<int>(blockIdx.x); u += kTile) v += part[u];
    block_excl_scan(v, &before);
  }
  int tot;
  int e = before + block_excl_scan(s, &tot);
  for (int q = 0; q < 4; ++q) {
    if (b0 + q <= m) start[b0 + q] = e;
    e += c[q];
  }
}

// ---------------------------------------------------------------- bins
// A counting sort of the cells into bins: k_cy_keys counts (a cell's arrival rank in its bin comes
// with the count), the scan gives the bins' starts and leaves the counts at zero for the next call,
// k_cy_scatter fills the bins in arrival order, k_cy_place gives each cell its place by index in its
// bin and writes the bin-ordered copies that the pair kernels read.

// DPD's first half kick and drift (updateVelocities then updatePositions, CIL.cu:871-897, 849-866;
// DPD step, CIL.cu:1055-1056) of the keys' own cells: no pass of its own over the positions.
__device__ inline double kick(const CyConst &C, double v, double fc, double fd, double fr) {
  // updateVel (Utils.hpp:568-571): v + (fc dt + fd dt + fr sqrt(dt)) / (2 (2 m))
  return __fma_rn(fr, C.kick_r, __fma_rn(fc + fd, C.kick_f, v));
}

__global__ void __launch_bounds__(kTile) k_cy_keys(CyConst C, CySet S, const CyCounters *cnt, int *key, int *arrival,
                                                   int *count, int *dblk, int drift) {
  cil::enter_step_kernel();
  if (threadIdx.x == 0) dblk[blockIdx.x] = 0;  // the coming step's divisions per block of cells
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt->n) return;
  double xd[3];
  CY_AXES(d, C.D) {
    const size_t k = static_cast<size_t>(d) * C.capacity + i;
    xd[d] = S.x[k];
    if (drift) {
      const double v = kick(C, S.v[k], S.fc[k], S.fd[k], S.fr[k]);
      S.v[k] = v;
      const double t = __fma_rn(C.dt, v, xd[d]);
      xd[d] = C.periodic[d] ? wrap(t, C.box[d]) : t;  // BoundingBox::updatePos
      S.x[k] = xd[d];
    }
  }
  const int b = bin_of(C, xd);
  key[i] = b;
  arrival[i] = atomicAdd(count + b, 1);
}

__global__ void __launch_bounds__(kTile) k_cy_scatter(const CyCounters *cnt, const int *key, const int *arrival,
                                                      const int *start, int2 *tmp) {
  cil::enter_step_kernel();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt->n) return;
  const int b = key[i];
  tmp[start[b] + arrival[i]] = make_int2(i, b);
}

// The bin order: a cell's place is its bin's start plus the number of smaller indices in the bin
// (bins hold a few cells; a bin with more than kBinSortMax means overlapping cells and is reported,
// its cells in arrival order). Written at the place: the index, the bin, the FP64 position and
// radius, and the FP32 record (absolute position and diameter) of the range tests. Threads take the
// cells in arrival order, next to their places: the state is gathered (32 bytes a value where the
// index order is not the bin order) and the copies are written in full lines (DPD, 0.15M cells: 6.8 us;
// from the index order, with the copies scattered, 8.2 us; without `loc` and `cell`).
__global__ void __launch_bounds__(kTile) k_cy_place(CyConst C, CySet S, CyCounters *cnt, const int *start,
                                                    const int2 *tmp, CyOrdered O, int with_vel) {
  cil::enter_step_kernel();
  const int at = blockIdx.x * blockDim.x + threadIdx.x;
  if (at >= cnt->n) return;
  const int2 ib = tmp[at];
  const int i = ib.x, b = ib.y, lo = start[b], hi = start[b + 1];
  const size_t cap = C.capacity;
  double x[3] = {0.0, 0.0, 0.0};
  float vf[3] = {0.0f, 0.0f, 0.0f};
  CY_AXES(d, C.D) {
    x[d] = S.x[d * cap + i];
    if (with_vel) vf[d] = static_cast<float>(S.v[d * cap + i]);
  }
  const double sg = S.sig[i];
  int q = at;
  if (hi - lo > kBinSortMax) {
    atomicOr(&cnt->err, kErrCrowded);
  } else {
    q = lo;
    for (int k = lo; k < hi; ++k) q += tmp[k].x < i ? 1 : 0;
  }
  CY_AXES(d, C.D) O.x[d * cap + q] = x[d];
  O.rad[q] = 0.5 * sg;
  O.idx[q] = i;
  O.bin[q] = b;
  O.rec[q] = make_float4(static_cast<float>(x[0]), static_cast<float>(x[1]), static_cast<float>(x[2]),
                         static_cast<float>(sg));
  if (with_vel) {
    O.vel[q] = make_float4(vf[0], vf[1], vf[2], 0.0f);
    int v[3] = {0, 0, 0}, r = b;
    float u[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int d = 2; d >= 0; --d) {
      if (d >= C.D) continue;
      v[d] = d > 0 ? r % C.ns[d] : r;
      r /= C.ns[d];
      u[d] = static_cast<float>(x[d] - v[d] * C.bw[d]);
    }
    O.loc[q] = make_float4(u[0], u[1], u[2], static_cast<float>(sg));
    O.cell[q] = make_ushort4(static_cast<unsigned short>(v[0]), static_cast<unsigned short>(v[1]),
                             static_cast<unsigned short>(v[2]), 0);
  }
}

// ---------------------------------------------------------------- the pair walk
// 2^lane_bits lanes per cell in bin order, no block cooperation. What bounds the pair kernels is the
// FP64 pipe, so FP64 runs for the pairs in range only, with full warps:
//   walk    the candidates of the stencil's rows of bins along the last axis (consecutive bins hold
//           consecutive places), tested in FP32 against a reach widened by the rounding of the
//           records; a cell's lanes take consecutive candidates and a ballot keeps the survivors in
//           walk order, so that the sums do not depend on the lane count;
//   pairs   the warp's survivors as one flattened range, a pair per lane;
//   sums    a cell's first lane adds its pairs in walk order.
// The contacts and the cycle of 1M cells (2.6 contacts a cell, FP64) take 515 us (caches flushed), with
// the FP64 pipe 83 % busy (260 FP64 instructions a warp of 32 cells); one thread per cell with each contact
// evaluated where it was met took 1079 us, and the cycle's own pass 258 us.
constexpr int kPairBlock = 128;
constexpr int kPairNear = 384;  // survivors held per warp (12 per cell at one lane each)
constexpr int kPairAhead = 4;   // candidates a lane has in flight (one lane per cell)

template <int D, int NRES, typename R>
struct PairWarp {
  static constexpr int kSeg = NRES > 6 ? 64 : 128;  // pairs evaluated before their sums are taken
  R res[kSeg * NRES];
  double x[32 * D];
  R v[32 * D];  // velocities (DPD)
  // CyOrdered::loc and ::cell, of DPD with FP32 pair terms (the others keep the 2 KB a block: 1 % of a step of
  // 1024 cells)
  static constexpr int kLoc = sizeof(R) == sizeof(float) && NRES != D + 1 ? 32 * D : 1;
  float u[kLoc];
  int cell[kLoc];
  double rad[32];
  float dia[32];
  int idx[32];
  int tt[kPairNear];
  unsigned char own[kPairNear];
};

// r_j - r_i at the nearest image (|dd| < L, so Nint(dd / L) is -1, 0 or 1; the two forms differ
// only at |dd| = L/2), the comparison on bit patterns
__device__ inline double nearest(double dd, double L, double half) {
  const long long b = __double_as_longlong(dd);
  if ((b & 0x7fffffffffffffffll) > __double_as_longlong(half)) return b < 0 ? dd + L : dd - L;
  return dd;
}

// DPD's FP32 pair terms take the displacement from coordinates relative to the bins' origins and the
// bins' offset. Not from the FP64 positions, although those would round better: the random force's
// sqrt(1 - r / rc) of a pair at the end of its range follows the last bits of r, so with another rounding
// a velocity differs by up to 2e-3 of their root mean square (0.15M cells, 12 steps) from what this
// form has always given.
// Bit d: the search covers axis d whole (each bin once), and an offset may span the axis.
template <int D>
__device__ __forceinline__ int whole_axes(const CyConst &C, float radius) {
  int m = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float kk = ceilf(__fmul_ru(radius, C.inv_bwf[d]));
    const int k = (kk >= 0.0f && kk < static_cast<float>(C.ns[d])) ? static_cast<int>(kk) : C.ns[d];
    if (2 * k + 1 >= C.ns[d]) m |= 1 << d;
  }
  return m;
}

// the warp's cell o to the cell at place tt, at the nearest image on periodic axes
template <int D, int NRES, typename R>
__device__ __forceinline__ void local_separation(const CyConst &C, const CyOrdered &O, const PairWarp<D, NRES, R> &W,
                                                 int whole, int o, int tt, float *df) {
  const float4 uj = O.loc[tt];
  const ushort4 cj = O.cell[tt];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    int off = (d == 0 ? cj.x : (d == 1 ? cj.y : cj.z)) - W.cell[o * D + d];
    if (C.periodic[d] && !(whole >> d & 1)) {
      if (2 * off > C.ns[d]) off -= C.ns[d];
      if (2 * off < -C.ns[d]) off += C.ns[d];
    }
    float v = f4c(uj, d) + static_cast<float>(off) * C.bwf[d] - W.u[o * D + d];
    if (C.periodic[d]) {
      if (v > C.halff[d])
        v -= C.boxf[d];
      else if (v < -C.halff[d])
        v += C.boxf[d];
    }
    df[d] = v;
  }
}

// reach2(me, p): the squared range of a pair in FP32 (an upper bound up to rounding);
// pair(o, tt, out): the terms of the pair of the warp's cell o and the cell at place tt (in range or
// not: the exact test is the callee's, which writes zeros out of range); acc: the cell's sums,
// complete in its first lane. radius: no pair farther apart is in range. Whole warp.
template <int D, int NRES, typename R, class Reach, class Pair>
__device__ __forceinline__ void walk_pairs(const CyConst &C, PairWarp<D, NRES, R> &W, const CyOrdered &O,
                                           const int *start, bool live, int q, int lane_bits, float radius,
                                           Reach reach2, Pair pair, R *acc) {
  const int lane = threadIdx.x & 31, L = 1 << lane_bits;
  const int sub = lane & (L - 1), el = lane >> lane_bits;
  const unsigned gmask = (L == 32 ? 0xffffffffu : (1u << L) - 1u) << (lane & ~(L - 1));
  const unsigned below = gmask & ((1u << lane) - 1u);
  const int cap = kPairNear >> (5 - lane_bits);
  const int nb0 = el * cap;
  int cnt = 0;
  auto flush = [&]() {
    int inc = sub == 0 ? cnt : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    const int total = __shfl_sync(0xffffffffu, inc, 31);
    const int end = __shfl_sync(0xffffffffu, inc, lane & ~(L - 1));
    const int off = end - cnt;
    for (int k = sub; k < cnt; k += L) W.own[off + k] = static_cast<unsigned char>(el);
    __syncwarp();
    constexpr int kSeg = PairWarp<D, NRES, R>::kSeg;
    for (int S = 0; S < total; S += kSeg) {
      const int E = min(total, S + kSeg);
      for (int f0 = S; f0 < E; f0 += 32) {  // uniform
        const int f = f0 + lane;
        const int o = f < E ? W.own[f] : 0;
        const int offo = __shfl_sync(0xffffffffu, off, o << lane_bits);
        if (f < E) pair(o, W.tt[o * cap + (f - offo)], &W.res[(f - S) * NRES]);
      }
      __syncwarp();
      if (sub == 0) {
        for (int f = max(off, S); f < min(end, E); ++f)
#pragma unroll
          for (int k = 0; k < NRES; ++k) acc[k] += W.res[(f - S) * NRES + k];
      }
      __syncwarp();
    }
    cnt = 0;
  };
  // the cell's bin and the bins to search on each side: k = ceil(radius / bin width) (FP32, rounded
  // up), the whole axis (each bin once) when 2k + 1 covers it, clipped at open walls
  int bi[D], lo[D], hi[D];
  {
    int b = live ? O.bin[q] : 0;
#pragma unroll
    for (int d = D - 1; d >= 0; --d) {
      bi[d] = d > 0 ? b % C.ns[d] : b;
      b /= C.ns[d];
      const float kk = ceilf(__fmul_ru(radius, C.inv_bwf[d]));
      const int k = (kk >= 0.0f && kk < static_cast<float>(C.ns[d])) ? static_cast<int>(kk) : C.ns[d];
      if (2 * k + 1 >= C.ns[d]) {
        lo[d] = -bi[d];
        hi[d] = C.ns[d] - 1 - bi[d];
      } else if (C.periodic[d]) {
        lo[d] = -k;
        hi[d] = k;
      } else {
        lo[d] = bi[d] - k < 0 ? -bi[d] : -k;
        hi[d] = bi[d] + k >= C.ns[d] ? C.ns[d] - 1 - bi[d] : k;
      }
    }
  }
  const float4 me = live ? O.rec[q] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  // FP32 rounds both positions, the box and the differences, each by 2^-24 of a value within
  // max(box, |x|) or so: 2^-21 of their sum bounds a separation's error along an axis
  float margin[D];
#pragma unroll
  for (int d = 0; d < D; ++d) margin[d] = 4.76837158e-07f * (C.boxf[d] + fabsf(f4c(me, d)));
  const int nl = C.ns[D - 1], ahead = lane_bits == 0 ? kPairAhead : 1;
  // rows of bins over the other axes; the loop runs to the warp's longest stencil
  const int n0 = live ? hi[0] - lo[0] + 1 : 0, n1 = D == 3 ? hi[D - 2] - lo[D - 2] + 1 : 1;
  const int rows = n0 * n1;
  const int rows_w = __reduce_max_sync(0xffffffffu, rows);
  // a row's span [a, z] of the last axis is up to three pieces of consecutive bins: inside, below 0 and
  // at or past the end; the piece inside is loaded a row ahead
  const int a = bi[D - 1] + lo[D - 1], z = bi[D - 1] + hi[D - 1];
  const int a1 = max(a, 0), z1 = min(z, nl - 1) + 1;
  const bool wraps = __any_sync(0xffffffffu, live && (a < 0 || z >= nl));
  auto row_start = [&](int row) {
    int v = bi[0] + lo[0] + (D == 3 ? row / n1 : row);
    if (v < 0) v += C.ns[0];
    if (v >= C.ns[0]) v -= C.ns[0];
    if (D == 3) {
      int u = bi[1] + lo[1] + row % n1;
      if (u < 0) u += C.ns[1];
      if (u >= C.ns[1]) u -= C.ns[1];
      v = v * C.ns[1] + u;
    }
    return start + static_cast<size_t>(v) * nl;
  };
  const int *rs = start;
  int st = 0, en = 0;
  if (rows > 0) {
    rs = row_start(0);
    st = rs[a1];
    en = rs[z1];
  }
  for (int row = 0; row < rows_w; ++row) {
    const int *rs_next = start;
    int st_next = 0, en_next = 0;
    if (row + 1 < rows) {
      rs_next = row_start(row + 1);
      st_next = rs_next[a1];
      en_next = rs_next[z1];
    }
    for (int piece = 0; piece < (wraps ? 3 : 1); ++piece) {
      if (piece == 1) {
        st = en = 0;
        if (row < rows && a < 0) {
          st = rs[a + nl];
          en = rs[nl];
        }
      } else if (piece == 2) {
        st = en = 0;
        if (row < rows && z >= nl) {
          st = rs[0];
          en = rs[z - nl + 1];
        }
      }
      // candidates in flight: kPairAhead of a lane alone with its cell, or one each of several lanes
      for (int tt0 = st; __any_sync(0xffffffffu, tt0 < en); tt0 += ahead * L) {
        float4 p[kPairAhead];
        bool there[kPairAhead];
#pragma unroll
        for (int u = 0; u < kPairAhead; ++u) {
          const int tt = tt0 + u * L + sub;
          there[u] = u < ahead && tt < en && tt != q;
          p[u] = there[u] ? O.rec[tt] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int u = 0; u < kPairAhead; ++u) {
          if (u >= ahead) break;
          float r2 = 0.0f;
#pragma unroll
          for (int d = 0; d < D; ++d) {
            float dx = fabsf(f4c(p[u], d) - f4c(me, d));
            if (C.periodic[d] && dx > C.halff[d]) dx = fabsf(dx - C.boxf[d]);
            dx = fmaxf(dx - margin[d], 0.0f);
            r2 += dx * dx;
          }
          const bool near = there[u] && !(r2 > 1.00001f * reach2(me, p[u]));
          const unsigned m = __ballot_sync(0xffffffffu, near);
          if (near) W.tt[nb0 + cnt + __popc(m & below)] = tt0 + u * L + sub;
          cnt += __popc(m & gmask);
        }
        if (__any_sync(0xffffffffu, cnt + ahead * L > cap)) {
          __syncwarp();
          flush();
        }
      }
    }
    rs = rs_next;
    st = st_next;
    en = en_next;
  }
  __syncwarp();
  flush();
}

// the colony's largest diameter of the last step, rounded up
__device__ inline float sigma_max_f(const CyCounters *cnt) {
  return __double2float_ru(__longlong_as_double(static_cast<long long>(cnt->sigma_max_bits)));
}

// ---------------------------------------------------------------- the cell cycle of one cell
// The cycle ODEs at the step's end with pressure p; a cell at phase 1 is counted for k_cy_divide
// (by its block of kTile cells, so that daughters come in mother order). Returns the bits of the
// cell's diameter.
__device__ inline unsigned long long cycle_update(const CyConst &C, const CySet &S, CyCounters *cnt, int *dblk,
                                                  int *dueq, int i, int ts, double p, double rad) {
  // every load before the first store, which the compiler could not move them across
  const int tp = S.tp[i];
  const double om = S.om[i], st = S.sigt[i], theta0 = S.theta[i];
  double rho = S.rho[i];
  // cellTPressure (CIL.cu:493-494): every cell is in the dividing state when the species divides
  S.tp[i] = p < C.apop_pressure ? 0 : tp + 1;
  double pp = p;
  if (C.p_shift != 0.0) pp += C.p_shift * exp(-ts * C.p_shift_tau_inv);
  double pnd = 0.0;
  if (__double_as_longlong(pp) > 0 && !(__double2hiint(pp) > 0x7ff00000)) {  // fmax(0, p) / p0
    pnd = pp * C.inv_p0;
    if (finite_bits(pnd)) pnd = __fma_rn(__fma_rn(-pnd, C.p0, pp), C.inv_p0, pnd);
  }
  const double theta = theta0 + om * fmin(C.r_maxed_inv * rho, 1.0);
  S.theta[i] = theta;
  const bool d3 = C.D == 3;
  double vt = d3 ? volume_of(st) : (kPi / 4) * (st * st);
  const double vt_prime = __fma_rn(__fma_rn(om, kLn2, C.growth), rho, -((vt - C.v_s) * C.inv_vs_tau_v));
  vt = __fma_rn(vt_prime, vt, vt);
  double v = vt;  // CYCLE_TAU_P 0 takes the target at once
  if (C.tau_p != 0) {
    v = d3 ? volume_of(2 * rad) : area_of(2 * rad);
    v += -(v - (vt / (1 + C.beta_vs * (C.osm + pnd)))) / C.tau_p;
  }
  double sn;
  if (d3) {
    S.sigt[i] = sigma_of_volume(vt);
    sn = sigma_of_volume(v);
  } else {
    const double a = vt * (4 / kPi);  // 2 sqrt(vt / pi)
    const double s = mid_range(a) ? sqrt_from(a, rsqrt_pos(a)) : sigma_of_area(vt);
    S.sigt[i] = s;
    sn = C.tau_p == 0 ? s : sigma_of_area(v);
  }
  S.sig[i] = sn;
  const double r_np = (1 - rho - pnd);
  rho = __fma_rn(r_np * (__double2hiint(r_np) >= 0 ? C.inv_tau_r : C.inv_tau_r_neg), rho, rho);
  S.rho[i] = rho;
  if (theta >= 1) {
    atomicAdd(dblk + i / kTile, 1);
    const int at = atomicAdd(&cnt->ndue, 1);
    if (at < kDueMax) dueq[at] = i;
  }
  return static_cast<unsigned long long>(__double_as_longlong(sn));
}

// the largest diameter of the warp's cells, for k_cy_divide (all the warps of a colony that fits the
// chip at once would meet at one address)
__device__ inline void warp_sigma(unsigned long long *part, unsigned long long s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, s, o);
    s = v > s ? v : s;
  }
  if ((threadIdx.x & 31) == 0) part[(blockIdx.x * kPairBlock + threadIdx.x) >> 5] = s;
}

// ---------------------------------------------------------------- forces + update
// The contact of cells a and b (radii, a the lower index) at distance r with overlap h = ra + rb - r
// and half the reciprocal distance hy = 1 / (2 r), the device draft's Hertz law with adhesion and its pressure
// (MD.cu:302-366): the force along the separation f0 = -fel + adhesion A, fel = h^1.5 / (0.75 c2
// sqrt(1/ra + 1/rb)), and 2 f0 / (contact volume). 2D: the contact length A = 2 sqrt(ra^2 - q^2),
// q = ra - h (2 rb - h) / (2 r), is 2 sqrt(w (2 ra - w)), w = h (2 rb - h) / (2 r) (no cancellation for
// small h); the elastic term is h^2 ra rb / (0.75 c2 sqrt(h (ra + rb) ra rb)). With the separation's,
// three reciprocal square roots and about 40 FP64 instructions per pair.
template <int D>
__device__ inline void contact(const CyConst &C, double r, double h, double hy, double cut, double ra, double rb,
                               double *f0, double *pr2) {
  const double u = h * (ra * rb), g = u * cut;
  const double fel = mid_range(g) ? u * h * (rsqrt_pos(g) * C.inv_hz) : h * sqrt(h / (1.0 / ra + 1.0 / rb)) * C.inv_hz;
  if (D == 3) {
    const double A = contact_area(r, 2 * ra, 2 * rb);
    const double vol = (A == 0 ? 0 : (4 * kPi * (ra * ra) / 3));
    *f0 = -fel + C.adhesion * A;
    *pr2 = vol != 0.0 ? 2 * (*f0 / vol) : 0.0;
    return;
  }
  const double w = h * hy * __fma_rn(2.0, rb, -h);
  const double t2 = w * __fma_rn(2.0, ra, -w);
  if (mid_range(t2)) {  // A is also the contact's volume in 2D
    const double z = rsqrt_pos(t2);
    *f0 = __fma_rn(2 * C.adhesion, t2 * z, -fel);
    *pr2 = *f0 * z;
  } else {
    const double t = 2 * sqrt(t2);
    const double A = isnan(t) ? 2 * (ra <= rb ? ra : rb) : t;
    *f0 = -fel + C.adhesion * A;
    *pr2 = A != 0.0 ? 2 * (*f0 / A) : 0.0;
  }
}

// The terms of the pair at displacement rij (FP64, or FP32 with FP32 pair terms; r2 its square, FP64
// form): the contact force on the cell, and in out[D] the pressure term, -f0 / volume doubled (FP64) or
// f0 / volume (MIXED); zeros out of contact. The warp's cell o and the cell at place tt; first: the cell
// has the lower index.
template <int D, bool MIXED, int NRES, typename R, typename X>
__device__ __forceinline__ void contact_terms(const CyConst &C, const CyOrdered &O, const PairWarp<D, NRES, R> &W, int o,
                                              int tt, const X *rij, double r2, bool first, R *out) {
  // the pair's first cell is the one of lower index (the contact length is not symmetric in
  // the two diameters)
#pragma unroll
  for (int k = 0; k <= D; ++k) out[k] = R(0);
  if (MIXED) {
    float df[D], r2f = 0.0f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      df[d] = static_cast<float>(rij[d]);
      r2f += df[d] * df[d];
    }
    const float sif = W.dia[o], sjf = O.rec[tt].w;
    const float cut = 0.5f * (sif + sjf);
    if (!(r2f <= cut * cut) || r2f == 0.0f) return;
    const float r = sqrtf(r2f);
    const float sa = first ? sif : sjf, sb = first ? sjf : sif;
    const float h = fmaxf(cut - r, 0.0f);
    const float fel = (h * sqrtf(h)) / (0.75f * C.c2f * sqrtf(2.0f / sif + 2.0f / sjf));
    const float ra = 0.5f * sa, rb = 0.5f * sb;
    float A, vol;
    if (D == 3) {
      const float u = r2f - rb * rb + ra * ra;
      const float t = sqrtf(4.0f * r2f * (ra * ra) - u * u) / (2.0f * r);
      A = t > 0.0f ? static_cast<float>(kPi) * (t * t) : 0.0f;
      vol = A == 0.0f ? 0.0f : (4.0f * static_cast<float>(kPi) * (ra * ra) / 3.0f);
    } else {
      const float w = h * (sb - h) / (2.0f * r);
      const float t = 2.0f * sqrtf(w * (sa - w));
      A = isnan(t) ? fminf(sa, sb) : t;
      vol = A;
    }
    const float f0 = -fel + C.adhf * A;
#pragma unroll
    for (int d = 0; d < D; ++d) out[d] = static_cast<R>(f0 * df[d]);
    out[D] = static_cast<R>(vol != 0.0f ? f0 / vol : 0.0f);
  } else {
    const double ro = W.rad[o], rj = O.rad[tt];
    double hy, r;
    if (mid_range(r2)) {
      const double y = rsqrt_pos(r2);
      r = sqrt_from(r2, y);
      hy = 0.5 * y;
    } else {
      r = sqrt(r2);
      hy = 0.5 / r;
    }
    const double cut = ro + rj, h = cut - r;
    // h >= 0 and finite (sign and exponent bits), r not 0
    if (__double2hiint(h) < 0 || !finite_bits(h) || __double_as_longlong(r) == 0) return;
    double f0, pr2;
    contact<D>(C, r, h, hy, cut, first ? ro : rj, first ? rj : ro, &f0, &pr2);
#pragma unroll
    for (int d = 0; d < D; ++d) out[d] = static_cast<R>(f0 * rij[d]);
    out[D] = static_cast<R>(pr2);
  }
}

// Motility along the velocity and passive noise of cell i
template <int D>
__device__ __forceinline__ void own_force(const CyConst &C, const CySet &S, int i, int ts, double *F) {
  const size_t cap = C.capacity;
  // ---- motility along the velocity (singleCellForce, MD.cu:600-646)
  {
    double vi[D], v2 = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      vi[d] = S.v[d * cap + i];
      v2 = d == 0 ? vi[d] * vi[d] : __fma_rn(vi[d], vi[d], v2);
    }
    if (mid_range(v2)) {
      const double m = C.motility * rsqrt_pos(v2);
#pragma unroll
      for (int d = 0; d < D; ++d) F[d] = m * vi[d];
    } else {
      double vl = sqrt(v2);
      if (vl == 0.0) {  // a direction at random, length 1e-11 (BIG_TOL_MP)
        const u32x4 r = draw(C, i, ts, kCyDir, 0);
        if (D == 2) {
          const double ang = 6.283185307179586 * u53(r.v[0], r.v[1]);
          vi[0] = 1e-11 * cos(ang);
          vi[1] = 1e-11 * sin(ang);
        } else {
          const double z = 2.0 * u53(r.v[0], r.v[1]) - 1.0;
          const double ang = 6.283185307179586 * u53(r.v[2], r.v[3]);
          const double s = sqrt(1.0 - z * z);
          vi[0] = 1e-11 * (s * cos(ang));
          vi[1] = 1e-11 * (s * sin(ang));
          vi[D - 1] = 1e-11 * z;
        }
        v2 = 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) v2 += vi[d] * vi[d];
        vl = sqrt(v2);
      }
#pragma unroll
      for (int d = 0; d < D; ++d) F[d] = C.motility * (vi[d] / vl);
    }
  }
  // ---- passive noise (CIL.cu:84-97)
  if (C.noise_amp > 0.0) {
    double nz[4];
    normal2(draw(C, i, ts, kCyNoise, 0), &nz[0], &nz[1]);
    if (D == 3) normal2(draw(C, i, ts, kCyNoise, 1), &nz[2], &nz[3]);
#pragma unroll
    for (int d = 0; d < D; ++d) F[d] += C.zeta * (C.noise_amp * nz[d]);
  }
}

// MIXED: the contact arithmetic in FP32 on the FP64 displacement; the forces and the pressure are
// summed in FP32 over the contacts and added to the FP64 motility and noise; the position update and
// the cell state stay FP64.
// Blocks an SM: 8 (64 registers) with FP32 pair terms, where the walk's loads need the warps (10 steps of
// 0.6M cells 3.17 -> 3.06 ms against the compiler's 95 registers); 7 (72) in FP64, which is bound by the
// FP64 pipe (more registers and fewer blocks: 1M cells 7.44 -> 8.34 ms).
// mode 0 (Euler): the position update with the pressure-dependent friction follows (in place: the
// other cells read the bin-ordered copies), then the cell cycle; mode 1: the forces go to frc and
// nothing moves. Draws are keyed by the device step counter.
template <int D, bool MIXED>
__global__ void __launch_bounds__(kPairBlock, MIXED ? 8 : 7) k_cy_force(CyConst C, CySet S, double *frc, CyCounters *cnt,
                                                         const int *start, const int *ts_dev, int mode, CyOrdered O, int lane_bits, int *dblk, int *dueq,
                                                         unsigned long long *sig_part) {
  cil::enter_step_kernel();
  using R = typename std::conditional<MIXED, float, double>::type;
  __shared__ PairWarp<D, D + 1, R> s_warp[kPairBlock / 32];
  PairWarp<D, D + 1, R> &W = s_warp[threadIdx.x >> 5];
  const int t = blockIdx.x * kPairBlock + threadIdx.x;
  const int n = cnt->n;
  const int L = 1 << lane_bits;
  const int q = t >> lane_bits, lane = threadIdx.x & 31, sub = lane & (L - 1), el = lane >> lane_bits;
  if ((t & ~31) >> lane_bits >= n) return;  // uniform per warp
  const bool live = q < n;
  const size_t cap = C.capacity;
  const int i = live ? O.idx[q] : 0;
  double xi[D];
#pragma unroll
  for (int d = 0; d < D; ++d) xi[d] = live ? O.x[d * cap + q] : 0.0;
  const double ri = live ? O.rad[q] : 1.0;
  if (sub == 0) {
#pragma unroll
    for (int d = 0; d < D; ++d) W.x[el * D + d] = xi[d];
    W.rad[el] = ri;
    W.dia[el] = live ? O.rec[q].w : 1.0f;
    W.idx[el] = i;
  }
  __syncwarp();
  R acc[D + 1];
#pragma unroll
  for (int k = 0; k <= D; ++k) acc[k] = R(0);
  walk_pairs<D, D + 1, R>(
      C, W, O, start, live, q, lane_bits, sigma_max_f(cnt),
      [](const float4 &a, const float4 &b) {
        const float cut = 0.5f * (a.w + b.w);
        return cut * cut;
      },
      [&](int o, int tt, R *out) {
        double rij[D], r2 = 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          double v = O.x[d * cap + tt] - W.x[o * D + d];
          if (C.periodic[d]) v = nearest(v, C.box[d], C.half[d]);
          rij[d] = v;
          if (!MIXED) r2 = d == 0 ? v * v : __fma_rn(v, v, r2);
        }
        contact_terms<D, MIXED>(C, O, W, o, tt, rij, r2, W.idx[o] < O.idx[tt], out);
      },
      acc);
  unsigned long long sbits = 0ull;
  if (live && sub == 0) {
    const int ts = *ts_dev;
    double F[D];
    own_force<D>(C, S, i, ts, F);
    bool finite = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      F[d] += static_cast<double>(acc[d]);
      finite = finite && finite_bits(F[d]);
    }
    const double pres = MIXED ? -static_cast<double>(acc[D]) : -0.5 * static_cast<double>(acc[D]);
    S.p[i] = pres;
    if (!finite) atomicOr(&cnt->err, kErrNonFinite);
    if (mode == 1) {
#pragma unroll
      for (int d = 0; d < D; ++d) frc[d * cap + i] = F[d];
    } else {
      // ---- position update with the pressure-dependent friction (CIL.cu:902-939)
      // pow(x, 0) is 1 for every x
      const double pw = C.zeta_p_beta == 0.0 ? 1.0 : pow(pres / C.p0, C.zeta_p_beta);
      const double den = (C.zeta + C.zeta_p * pw) * (kPi * (ri * ri));
      const double mu = mid_range(den) ? rcp_normal(den) : 1.0 / den;
      const double temp = C.dt * mu;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const double x = __fma_rn(temp, F[d], xi[d]);
        S.x[d * cap + i] = C.periodic[d] ? wrap(x, C.box[d]) : x;
        S.v[d * cap + i] = F[d] * mu;
      }
      if (C.divide) sbits = cycle_update(C, S, cnt, dblk, dueq, i, ts + 1, pres, ri);
    }
  }
  if (mode == 0 && C.divide) warp_sigma(sig_part, sbits);
}

// ---------------------------------------------------------------- DPD
// Two standard normals in FP32 (Box-Muller on 24-bit uniforms) from the four words of one
// Philox block, the FP32 counterpart of normal2: its uniforms are normal2's rounded to 24 bits
// (1 - u from the first word, u from the third), so the two agree to FP32 rounding.
__device__ inline void normal2f(const u32x4 &r, float *n0, float *n1) {
  const float u1 = static_cast<float>((1u << 24) - (r.v[0] >> 8)) * 5.9604644775390625e-08f;  // (0, 1]
  const float u2 = static_cast<float>(r.v[2] >> 8) * 5.9604644775390625e-08f;
  const float rad = sqrtf(-2.0f * __logf(u1));
  float sn, cs;
  __sincosf(6.2831853071795865f * u2, &sn, &cs);
  *n0 = rad * cs;
  *n1 = rad * sn;
}

// The conservative forces and the pressure (k_cy_force's) and the pair dissipative and random forces
// (cellCellDisRanForce, MD.cu:861-905) over the pairs closer than the lower-index cell's diameter, in
// one walk (a contact's range, the mean diameter, is within the larger one); then, with `kick`, the
// second half kick into v_out. In two walks 0.15M cells with FP32 pair terms took 25.4 and 22.6 us; in
// one about 32. 8 blocks an SM with FP32 pair terms (12 steps of 0.15M cells 1.87 -> 1.82 ms against 95
// registers); FP64 keeps its registers (10 steps 4.19 -> 4.04 ms).
// MIXED: the pair terms in FP32 on the separations of local_separation, FP32 velocities and normals, summed in FP32
// per cell; the kick stays FP64, and the new velocities' records go to vel_out for k_dpd_dis.
template <int D, bool MIXED>
__global__ void __launch_bounds__(kPairBlock, MIXED ? 8 : 1) k_dpd_forces(CyConst C, CySet S, double *v_out, CyCounters *cnt,
                                                         const int *start, const int *ts_dev, int key_off, int kick_on,
                                                         CyOrdered O, float4 *vel_out, int lane_bits) {
  cil::enter_step_kernel();
  using R = typename std::conditional<MIXED, float, double>::type;
  using X = R;  // displacements
  __shared__ PairWarp<D, 3 * D + 1, R> s_warp[kPairBlock / 32];
  PairWarp<D, 3 * D + 1, R> &W = s_warp[threadIdx.x >> 5];
  const int t = blockIdx.x * kPairBlock + threadIdx.x;
  const int n = cnt->n;
  const int L = 1 << lane_bits;
  const int q = t >> lane_bits, lane = threadIdx.x & 31, sub = lane & (L - 1), el = lane >> lane_bits;
  if ((t & ~31) >> lane_bits >= n) return;  // uniform per warp
  const bool live = q < n;
  const uint32_t ts = static_cast<uint32_t>(*ts_dev + key_off);
  const size_t cap = C.capacity;
  const int i = live ? O.idx[q] : 0;
  double vi[D];
#pragma unroll
  for (int d = 0; d < D; ++d) vi[d] = live ? S.v[d * cap + i] : 0.0;
  if (sub == 0) {
    if constexpr (MIXED) {
      const float4 u = live ? O.loc[q] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const ushort4 b = live ? O.cell[q] : make_ushort4(0, 0, 0, 0);
#pragma unroll
      for (int d = 0; d < D; ++d) {
        W.u[el * D + d] = f4c(u, d);
        W.cell[el * D + d] = d == 0 ? b.x : (d == 1 ? b.y : b.z);
      }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (!MIXED) W.x[el * D + d] = live ? O.x[d * cap + q] : 0.0;
      W.v[el * D + d] = static_cast<R>(vi[d]);
    }
    W.rad[el] = live ? O.rad[q] : 1.0;
    W.dia[el] = live ? O.rec[q].w : 1.0f;
    W.idx[el] = i;
  }
  __syncwarp();
  const float radius = sigma_max_f(cnt);
  const int whole = MIXED ? whole_axes<D>(C, radius) : 0;
  R acc[3 * D + 1];  // conservative, pressure, dissipative, random
#pragma unroll
  for (int k = 0; k < 3 * D + 1; ++k) acc[k] = R(0);
  walk_pairs<D, 3 * D + 1, R>(
      C, W, O, start, live, q, lane_bits, radius,
      [](const float4 &a, const float4 &b) {
        const float s = fmaxf(a.w, b.w);
        return s * s;
      },
      [&](int o, int tt, R *out) {
        X rij[D];
        double r2 = 0.0;
        if constexpr (MIXED) {
          local_separation<D>(C, O, W, whole, o, tt, rij);
        } else {
#pragma unroll
          for (int d = 0; d < D; ++d) {
            double v = O.x[d * cap + tt] - W.x[o * D + d];
            if (C.periodic[d]) v = nearest(v, C.box[d], C.half[d]);
            rij[d] = v;
            r2 = d == 0 ? v * v : __fma_rn(v, v, r2);
          }
        }
        const int io = W.idx[o], j = O.idx[tt];
        const uint32_t a = static_cast<uint32_t>(io < j ? io : j), z = static_cast<uint32_t>(io < j ? j : io);
        contact_terms<D, MIXED>(C, O, W, o, tt, rij, r2, io < j, out);
        out += D + 1;
#pragma unroll
        for (int k = 0; k < 2 * D; ++k) out[k] = R(0);
        if (MIXED) {
          float r2f = 0.0f;
#pragma unroll
          for (int d = 0; d < D; ++d) r2f += rij[d] * rij[d];
          const float rc = io < j ? W.dia[o] : O.rec[tt].w;
          if (!(r2f < rc * rc) || r2f == 0.0f) return;
          const float4 vj4 = O.vel[tt];
          const float rinv = rsqrtf(r2f);
          // within the range by a few units of the last place, r2f rinv may pass rc: not below 0
          const float w = fmaxf(1.0f - r2f * rinv / rc, 0.0f);
          float xf[4];
          normal2f(philox4x32_10(a, ts, kCyDpd0, z, C.seed_lo, C.seed_hi), &xf[0], &xf[1]);
          if (D == 3) normal2f(philox4x32_10(a, ts, kCyDpd1, z, C.seed_lo, C.seed_hi), &xf[2], &xf[3]);
          const float sw = sqrtf(w);
#pragma unroll
          for (int d = 0; d < D; ++d) {
            const float nd = rij[d] * rinv;
            const float dv = static_cast<float>(W.v[o * D + d]) - f4c(vj4, d);
            out[d] = static_cast<R>(-(C.gdf * w * (dv * nd) * nd));
            out[D + d] = static_cast<R>(C.srf * sw * nd * xf[d]);
          }
        } else {
          const double rc = 2 * (io < j ? W.rad[o] : O.rad[tt]);
          double ir, r;
          if (mid_range(r2)) {
            ir = rsqrt_pos(r2);
            r = sqrt_from(r2, ir);
          } else {
            r = sqrt(r2);
            ir = 1.0 / r;
          }
          if (!(r < rc) || r == 0.0) return;
          const double w = 1 - r / rc;
          double xn[4];
          normal2(philox4x32_10(a, ts, kCyDpd0, z, C.seed_lo, C.seed_hi), &xn[0], &xn[1]);
          if (D == 3) normal2(philox4x32_10(a, ts, kCyDpd1, z, C.seed_lo, C.seed_hi), &xn[2], &xn[3]);
          const double gw = C.gamma_d * w, sw = C.sigma_r * sqrt(w);
#pragma unroll
          for (int d = 0; d < D; ++d) {
            const double nd = rij[d] * ir;
            const double vj = S.v[d * cap + j];
            out[d] = static_cast<R>(-(gw * ((W.v[o * D + d] - vj) * nd) * nd));
            out[D + d] = static_cast<R>(sw * nd * xn[d]);
          }
        }
      },
      acc);
  if (!live || sub != 0) return;
  bool finite = true;
  float vf[3] = {0.0f, 0.0f, 0.0f};
  double F[D];
  own_force<D>(C, S, i, static_cast<int>(ts), F);
  S.p[i] = MIXED ? -static_cast<double>(acc[D]) : -0.5 * static_cast<double>(acc[D]);
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const size_t k = d * cap + i;
    F[d] += static_cast<double>(acc[d]);
    finite = finite && finite_bits(F[d]);
    S.fc[k] = F[d];
    const double fd = static_cast<double>(acc[D + 1 + d]), fr = static_cast<double>(acc[2 * D + 1 + d]);
    S.fd[k] = fd;
    S.fr[k] = fr;
    if (kick_on) {
      const double v = kick(C, vi[d], F[d], fd, fr);
      v_out[k] = v;
      vf[d] = static_cast<float>(v);
      finite = finite && finite_bits(v);
    }
  }
  if (MIXED && kick_on) vel_out[q] = make_float4(vf[0], vf[1], vf[2], 0.0f);
  if (!finite) atomicOr(&cnt->err, kErrNonFinite);
}

// Background and pair dissipation at the new velocities (calculDisForces, CIL.cu:294-364:
// sameCellDisForce zeroes a single-element cell's Fd, cellBackDisForce subtracts gamma_bg v,
// cellCellDisForce, MD.cu:951-985, with w = 1 - r^2 / sigma_core for r < sigma_core), then the cell
// cycle.
template <int D, bool MIXED>
__global__ void __launch_bounds__(kPairBlock) k_dpd_dis(CyConst C, CySet S, CyCounters *cnt, const int *start,
                                                        const int *ts_dev, CyOrdered O, const float4 *vel,
                                                        int lane_bits, int *dblk, int *dueq,
                                                         unsigned long long *sig_part) {
  cil::enter_step_kernel();
  using R = typename std::conditional<MIXED, float, double>::type;
  using X = R;  // displacements
  __shared__ PairWarp<D, D, R> s_warp[kPairBlock / 32];
  PairWarp<D, D, R> &W = s_warp[threadIdx.x >> 5];
  const int t = blockIdx.x * kPairBlock + threadIdx.x;
  const int n = cnt->n;
  const int L = 1 << lane_bits;
  const int q = t >> lane_bits, lane = threadIdx.x & 31, sub = lane & (L - 1), el = lane >> lane_bits;
  if ((t & ~31) >> lane_bits >= n) return;  // uniform per warp
  const bool live = q < n;
  const size_t cap = C.capacity;
  const int i = live ? O.idx[q] : 0;
  double vi[D];
#pragma unroll
  for (int d = 0; d < D; ++d) vi[d] = live ? S.v[d * cap + i] : 0.0;
  if (sub == 0) {
    if constexpr (MIXED) {
      const float4 u = live ? O.loc[q] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const ushort4 b = live ? O.cell[q] : make_ushort4(0, 0, 0, 0);
#pragma unroll
      for (int d = 0; d < D; ++d) {
        W.u[el * D + d] = f4c(u, d);
        W.cell[el * D + d] = d == 0 ? b.x : (d == 1 ? b.y : b.z);
      }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (!MIXED) W.x[el * D + d] = live ? O.x[d * cap + q] : 0.0;
      W.v[el * D + d] = static_cast<R>(vi[d]);
    }
  }
  __syncwarp();
  const double rc = C.sigma_core;
  const float rcf = static_cast<float>(rc);
  const float radius = fmaxf(sigma_max_f(cnt), __double2float_ru(rc));
  const int whole = MIXED ? whole_axes<D>(C, radius) : 0;
  R acc[D];
#pragma unroll
  for (int d = 0; d < D; ++d) acc[d] = R(0);
  walk_pairs<D, D, R>(
      C, W, O, start, live, q, lane_bits, radius,
      [&](const float4 &, const float4 &) { return rcf * rcf; },
      [&](int o, int tt, R *out) {
        X rij[D];
        double r2 = 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) out[d] = R(0);
        if constexpr (MIXED) {
          local_separation<D>(C, O, W, whole, o, tt, rij);
        } else {
#pragma unroll
          for (int d = 0; d < D; ++d) {
            double v = O.x[d * cap + tt] - W.x[o * D + d];
            if (C.periodic[d]) v = nearest(v, C.box[d], C.half[d]);
            rij[d] = v;
            r2 = d == 0 ? v * v : __fma_rn(v, v, r2);
          }
        }
        if (MIXED) {
          float r2f = 0.0f;
#pragma unroll
          for (int d = 0; d < D; ++d) r2f += rij[d] * rij[d];
          if (!(r2f < rcf * rcf) || r2f == 0.0f) return;
          const float4 vj4 = vel[tt];
          const float rinv = rsqrtf(r2f);
          const float w = 1.0f - r2f / rcf;
#pragma unroll
          for (int d = 0; d < D; ++d) {
            const float nd = -rij[d] * rinv;
            const float dv = static_cast<float>(W.v[o * D + d]) - f4c(vj4, d);
            out[d] = static_cast<R>(-(C.gdf * w * (dv * nd) * nd));
          }
        } else {
          const int j = O.idx[tt];
          double ir, r;
          if (mid_range(r2)) {
            ir = rsqrt_pos(r2);
            r = sqrt_from(r2, ir);
          } else {
            r = sqrt(r2);
            ir = 1.0 / r;
          }
          if (!(r < rc) || r == 0.0) return;
          const double gw = C.gamma_d * (1 - r2 / rc);
#pragma unroll
          for (int d = 0; d < D; ++d) {
            const double nd = rij[d] * ir;
            out[d] = static_cast<R>(-(gw * ((W.v[o * D + d] - S.v[d * cap + j]) * nd) * nd));
          }
        }
      },
      acc);
  unsigned long long sbits = 0ull;
  if (live && sub == 0) {
#pragma unroll
    for (int d = 0; d < D; ++d) S.fd[d * cap + i] = static_cast<double>(acc[d]) - C.gamma_b * vi[d];
    if (C.divide) sbits = cycle_update(C, S, cnt, dblk, dueq, i, *ts_dev + 1, S.p[i], O.rad[q]);
  }
  if (C.divide) warp_sigma(sig_part, sbits);
}

__device__ inline void put_sigma_max(CyCounters *cnt, double s) {
  atomicMax(&cnt->sigma_max_bits, static_cast<unsigned long long>(__double_as_longlong(s)));
}

// Divisions in mother order: daughter of the k-th dividing cell at n + k (calculDivisionsSingle,
// CIL.cu:527-600; singleCellDivision, MD.cu:664-718). Up to kDueMax dividing cells are ranked among
// themselves from their queue; more, by a scan over the cells. The block that finishes last commits the
// step: the cell count, the largest diameter and the step counter (every block has read them by then).
// The division of cell i into i and inew: divide_places (positions, velocities, forces, diameters) and
// divide_times (cycles), which touch different arrays, so that two warps run their chains at once. The
// loads come before the stores, which the compiler could not move them across.
__device__ void divide_places(const CyConst &C, const CySet &S, int ts, int i, int inew) {
  const size_t cap = C.capacity;
  const int D = C.D;
  const double lmom = S.sig[i];
  double x[3] = {0, 0, 0};
  CY_AXES(d, D) x[d] = S.x[d * cap + i];
  double ldau, newsig;
  double dr[3] = {0, 0, 0};
  const u32x4 r0 = draw(C, i, ts, kCyDiv, 0);
  if (D == 2) {
    ldau = lmom / sqrt(2.0);
    newsig = ldau;
    const double rr = (lmom - ldau) / 2;
    const double alpha = u53(r0.v[0], r0.v[1]) * 6.283185307179586;
    dr[0] = rr * sin(alpha);
    dr[1] = rr * cos(alpha);
  } else {
    const double rmom = lmom / 2;
    const double vmom = 4 * kPi * rmom * rmom * rmom / 3;
    const double a = 9 * lmom / 4;
    const double b = -(3 * (lmom * lmom) / 2);
    const double c = lmom * lmom * lmom / 4 - 3 * vmom / (kPi);
    ldau = (-b + sqrt(b * b - 4 * a * c)) / (2 * a);
    newsig = ldau;
    const double rr = (lmom - ldau) / 2;
    const double alpha = u53(r0.v[0], r0.v[1]) * 6.283185307179586;
    const double beta = u53(r0.v[2], r0.v[3]) * 6.283185307179586;
    dr[0] = rr * sin(alpha) * cos(beta);
    dr[1] = rr * sin(alpha) * sin(beta);
    dr[2] = rr * cos(alpha);
  }
  CY_AXES(d, D) {
    const double m = x[d];
    double xd = m + dr[d], xm = m + (-dr[d]);
    if (C.periodic[d]) {
      xd = wrap(xd, C.box[d]);
      xm = wrap(xm, C.box[d]);
    }
    S.x[d * cap + inew] = xd;
    S.x[d * cap + i] = xm;
    S.v[d * cap + inew] = 0.0;
    S.v[d * cap + i] = 0.0;
    if (S.fc) {  // resetFrc (CIL.cu:597-598)
      S.fc[d * cap + inew] = S.fd[d * cap + inew] = S.fr[d * cap + inew] = 0.0;
      S.fc[d * cap + i] = S.fd[d * cap + i] = S.fr[d * cap + i] = 0.0;
    }
  }
  S.sig[inew] = newsig;
  S.sig[i] = newsig;
  S.sigt[inew] = newsig;
  S.sigt[i] = newsig;
}

__device__ void divide_times(const CyConst &C, const CySet &S, int ts, int i, int inew) {
  // cycle times: migration spans (daughter, then mother), log-normal cycle speeds (mother,
  // then daughter), as the reference draws them (a span without spread needs no draw)
  const double p = S.p[i], rho = S.rho[i];
  double z0 = 0.0, z1 = 0.0, z2, z3;
  if (C.tau_mig_sigma != 0.0) normal2(draw(C, i, ts, kCyDiv, 1), &z0, &z1);
  normal2(draw(C, i, ts, kCyDiv, 2), &z2, &z3);
  S.tsw[inew] = ts + span_steps(C.tau_mig_mu + C.tau_mig_sigma * z0, C.dt);
  S.tsw[i] = ts + span_steps(C.tau_mig_mu + C.tau_mig_sigma * z1, C.dt);
  S.om[i] = 1.0 / span_steps(exp(C.div_mu2 + C.div_s2 * z2), C.dt);
  S.om[inew] = 1.0 / span_steps(exp(C.div_mu2 + C.div_s2 * z3), C.dt);
  S.t0[inew] = ts;
  S.t0[i] = ts;
  S.theta[i] = 0;
  S.theta[inew] = 0;
  S.p[inew] = p;
  S.rho[inew] = rho;
  S.tp[inew] = -1;  // an unused slot of the reference's arrays (Colony.cpp:253)
}

__global__ void __launch_bounds__(kTile) k_cy_divide(CyConst C, CySet S, CyCounters *cnt, int *ts_dev,
                                                     const int *dblk, const int *dueq,
                                                     const unsigned long long *sig_part, int lane_bits) {
  cil::enter_step_kernel();
  __shared__ int s_due[kDueMax];
  __shared__ unsigned long long s_sig;
  const int n = cnt->n, ts = *ts_dev + 1, nd = cnt->ndue;
  if (threadIdx.x == 0) s_sig = 0ull;
  __syncthreads();
  {  // the step's largest diameter (before the divisions halve the dividing cells)
    const int nw = static_cast<int>(((static_cast<long long>(n) << lane_bits) + 31) >> 5);
    unsigned long long m = 0ull;
    for (int k = blockIdx.x * kTile + threadIdx.x; k < nw; k += gridDim.x * kTile) m = sig_part[k] > m ? sig_part[k] : m;
    if (m) atomicMax(&s_sig, m);
  }
  if (nd <= kDueMax) {
    // the queue's cells (in no particular order): each one's rank is the number of smaller indices;
    // the block's first half takes the places, the second the times
    constexpr int kHalf = kTile / 2;
    if (blockIdx.x * kHalf < nd) {  // uniform
      for (int k = threadIdx.x; k < nd; k += kTile) s_due[k] = dueq[k];
      __syncthreads();
      for (int r = blockIdx.x * kHalf + threadIdx.x % kHalf; r < nd; r += gridDim.x * kHalf) {
        const int i = s_due[r];
        int rank = 0;
        for (int k = 0; k < nd; ++k) rank += s_due[k] < i ? 1 : 0;
        if (n + rank >= C.capacity)
          atomicOr(&cnt->err, kErrCapacity);
        else if (threadIdx.x < kHalf)
          divide_places(C, S, ts, i, n + rank);
        else
          divide_times(C, S, ts, i, n + rank);
      }
    }
  } else {
    // the blocks of kTile cells in turn, those without a dividing cell passed over
    const int nb = (n + kTile - 1) / kTile;
    for (int cb = blockIdx.x; cb < nb; cb += gridDim.x) {
      if (dblk[cb] == 0) continue;  // uniform
      int before = 0, off, tot;
      for (int u = threadIdx.x; u < cb; u += kTile) before += dblk[u];
      block_excl_scan(before, &tot);
      off = tot;
      const int i = cb * kTile + threadIdx.x;
      const int f = (i < n && S.theta[i] >= 1) ? 1 : 0;
      const int rank = off + block_excl_scan(f, &tot);
      if (f && n + rank >= C.capacity) {
        atomicOr(&cnt->err, kErrCapacity);
      } else if (f) {
        divide_places(C, S, ts, i, n + rank);
        divide_times(C, S, ts, i, n + rank);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_sig) atomicMax(&cnt->sigma_next_bits, s_sig);
    __threadfence();
    if (atomicAdd(&cnt->ndone, 1) == static_cast<int>(gridDim.x) - 1) {
      const int nd = cnt->ndue, room = C.capacity - n;
      const int add = nd < room ? nd : (room > 0 ? room : 0);
      cnt->n = n + add;
      cnt->ndiv_total += add;
      cnt->ndiv_step = add;
      cnt->sigma_max_bits = atomicExch(&cnt->sigma_next_bits, 0ull);
      cnt->ndue = 0;
      cnt->ndone = 0;
      *ts_dev = ts;
    }
  }
}

__global__ void k_cy_advance(int *ts) { *ts += 1; }

// ---------------------------------------------------------------- removals
// mode 1: apoptosis (the law of C.apoptosis, one Philox block per cell and step); mode 2:
// outside the box (drain)
__global__ void __launch_bounds__(kTile) k_cy_mark(CyConst C, CySet S, CyCounters *cnt, const int *ts_dev,
                                                   int mode, int *keep, int *block_count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = cnt->n;
  int k = 0;
  if (i < n) {
    k = 1;
    if (mode == 1) {
      const int ts = *ts_dev;
      const u32x4 r = draw(C, i, ts, kCyApo, 0);
      const double u = u53(r.v[0], r.v[1]);
      const double rho = S.rho[i];
      if (C.apoptosis == CIL_APOP_CYCLE_PRESSURE) {
        const double p = S.p[i];
        const double rate = C.apop_rate_step * pow((1 - (rho / C.apop_pressure)), C.apop_duration) *
                            pow(p / (p + C.p0), C.extr_gamma);
        if (u <= rate) k = 0;
      } else if (C.apoptosis == CIL_APOP_PRESSURE_TIME) {
        if (((C.apop_duration > 0) && (S.tp[i] >= C.apop_steps)) || ((C.apop_rate_step > 0) && (u <= C.apop_rate_step)))
          k = 0;
      } else if (C.apoptosis == CIL_APOP_RATE) {
        if (u <= C.apop_rate_step) k = 0;
      } else if (C.apoptosis == CIL_APOP_CYCLE) {
        if (rho < 1 && u <= C.apop_rate_step * pow((1 - (rho / C.apop_pressure)), C.apop_duration)) k = 0;
      } else {  // CIL_APOP_CYCLE_EXTRUDE
        if (rho < 1 && u <= C.apop_rate_step) k = 0;
        const double u2 = u53(r.v[2], r.v[3]);
        if (rho <= 0.1 &&
            u2 <= C.extr_rate * pow(((S.p[i] - C.apop_pressure) / C.apop_pressure), C.extr_gamma))
          k = 0;
      }
    } else {
      CY_AXES(d, C.D) {
        const double x = S.x[static_cast<size_t>(d) * C.capacity + i];
        if (!(x >= 0.0 && x < C.box[d])) k = 0;
      }
    }
    keep[i] = k;
  }
  int tot;
  block_excl_scan(k, &tot);
  if (threadIdx.x == 0) block_count[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kTile) k_cy_compact(CyConst C, CySet A, CySet B, const CyCounters *cnt,
                                                      const int *keep, const int *block_start) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = cnt->n;
  const int k = (i < n) ? keep[i] : 0;
  int tot;
  const int dst = block_start[blockIdx.x] + block_excl_scan(k, &tot);
  if (!k) return;
  const size_t cap = C.capacity;
  CY_AXES(d, C.D) {
    B.x[d * cap + dst] = A.x[d * cap + i];
    B.v[d * cap + dst] = A.v[d * cap + i];
    if (A.fc) {
      B.fc[d * cap + dst] = A.fc[d * cap + i];
      B.fd[d * cap + dst] = A.fd[d * cap + i];
      B.fr[d * cap + dst] = A.fr[d * cap + i];
    }
  }
  B.sig[dst] = A.sig[i];
  B.sigt[dst] = A.sigt[i];
  B.theta[dst] = A.theta[i];
  B.rho[dst] = A.rho[i];
  B.om[dst] = A.om[i];
  B.p[dst] = A.p[i];
  B.tp[dst] = A.tp[i];
  B.t0[dst] = A.t0[i];
  B.tsw[dst] = A.tsw[i];
}

__global__ void k_cy_commit_removals(CyCounters *cnt, const int *block_start, int n_blocks, int mode) {
  const int kept = block_start[n_blocks];
  const int removed = cnt->n - kept;
  cnt->n = kept;
  cnt->nrem_step = removed;
  if (mode == 1) cnt->napo_total += removed;
}

// ---------------------------------------------------------------- initial cell status
// initializeCellStatus (CIL.cuh:253-330) for single-element cells, counter-based draws
__global__ void k_cy_init_status(CyConst C, CySet S, const CyCounters *cnt, int ts, int fill_sigma, int fill_cycle) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt->n) return;
  if (fill_sigma) {
    S.sig[i] = C.sigma_core;
    S.sigt[i] = C.sigma_core;
  }
  S.tp[i] = 0;
  S.t0[i] = 0;
  if (!fill_cycle) return;
  S.tsw[i] = -1;
  S.rho[i] = 1;
  if (!C.divide) {
    S.theta[i] = 0;
    S.om[i] = 0;
    return;
  }
  // every cell starts in the dividing state (the migration probability is 0): a cycle length
  // max(Nint(N(tau_div) / dt), 1), the phase U[0, 1), and the elapsed part of the span
  const u32x4 r0 = draw(C, i, ts, kCyInit, 0);
  double z0, z1;
  normal2(draw(C, i, ts, kCyInit, 1), &z0, &z1);
  int span = span_steps(C.tau_div_mu + C.tau_div_sigma * z0, C.dt);
  S.om[i] = 1.0 / span;
  S.theta[i] = u53(r0.v[2], r0.v[3]);
  const u32x4 r2 = draw(C, i, ts, kCyInit, 2);
  span -= nint(u53(r2.v[0], r2.v[1]) * static_cast<double>(span)) - 1;
  S.tsw[i] = S.t0[i] + span;
}

__global__ void k_cy_sigma_max(CyConst C, CySet S, CyCounters *cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  __shared__ unsigned long long smax;
  if (threadIdx.x == 0) smax = 0ull;
  __syncthreads();
  if (i < cnt->n) atomicMax(&smax, static_cast<unsigned long long>(__double_as_longlong(S.sig[i])));
  __syncthreads();
  if (threadIdx.x == 0 && smax) put_sigma_max(cnt, __longlong_as_double(static_cast<long long>(smax)));
}

// ---------------------------------------------------------------- host copies
// The host's vectors are [cell][axis], the device's [axis][cap]: staged as the host has them and
// rearranged here, so that a copy from or into pinned memory runs at the link's rate (a host loop and
// pageable copies took 5.8 of the 13.1 ms of a 1M-cell leg of 10 steps).
__global__ void __launch_bounds__(kTile) k_cy_from_host(const double *staged, int n, int D, size_t cap, double *dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  CY_AXES(d, D) dst[d * cap + i] = staged[static_cast<size_t>(i) * D + d];
}

__global__ void __launch_bounds__(kTile) k_cy_to_host(const double *src, int n, int D, size_t cap, double *staged) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  CY_AXES(d, D) staged[static_cast<size_t>(i) * D + d] = src[d * cap + i];
}

// a staged position outside [0, box) sets *bad
__global__ void __launch_bounds__(kTile) k_cy_check_staged(CyConst C, const double *staged, int n, int *bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  CY_AXES(d, C.D) {
    const double x = staged[static_cast<size_t>(i) * C.D + d];
    if (!(x >= 0.0 && x < C.box[d])) *bad = 1;
  }
}

}  // namespace

// ================================================================ host side
struct cil_cycle {
  cil_cycle_params p{};
  CyConst C{};
  int device = 0;
  int cap = 0;
  cudaStream_t stream = nullptr;
  CySet set[2] = {};
  int cur = 0;
  double *vs = nullptr;   // velocity output buffer of the DPD pair pass
  CyOrdered O{};          // the cells in bin order
  float4 *vel_next = nullptr;  // the new velocities' records (DPD, precision 1)
  double *frc = nullptr;  // forces of the last download (output only)
  // captured steps: keyed by the buffer configuration before the step and the bin grid, each
  // records the configuration after it (a step rotates v / vs and the state sets)
  struct Buffers {
    CySet set[2];
    double *vs;
    int cur;
  };
  struct StepGraph {
    Buffers before, after;
    uint64_t grid;
    cudaGraphExec_t exec;
    int64_t nodes;
  };
  std::vector<StepGraph> graphs;
  uint64_t grid_gen = 0;
  int pair_bs = kTile;  // threads per block of the removal kernels (set per call)
  int lane_bits = 0;    // log2 of the lanes per cell of the pair kernels (set per call)
  CyCounters *cnt = nullptr;
  CyCounters *h_cnt = nullptr;  // pinned
  int *ts_dev = nullptr;
  int *key = nullptr, *arrival = nullptr, *bcount = nullptr, *bstart = nullptr, *part = nullptr;
  int2 *tmp = nullptr;
  int *flag = nullptr, *blk = nullptr, *dblk = nullptr, *dueq = nullptr;
  unsigned long long *sig_part = nullptr;  // the step's largest diameter per warp of the pair kernel
  int nbins = 0, nparts = 0, nblocks = 0;
  long long nbins_cap = 0;  // bins the arrays hold
  int64_t ts = 0;
  bool uploaded = false;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  double t_total = 0.0;
  int64_t launches = 0;
  std::string err;
  std::vector<void *> allocs;

  template <typename T>
  T *alloc(size_t n) {
    void *q = nullptr;
    if (cudaMalloc(&q, n * sizeof(T)) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    allocs.push_back(q);
    return static_cast<T *>(q);
  }
  cil_status fail(cil_status s, const std::string &m) {
    err = m;
    return s;
  }
};

#define CY_TRY(h, call)                                                                      \
  do {                                                                                       \
    cudaError_t e_ = (call);                                                                 \
    if (e_ != cudaSuccess) return (h)->fail(CIL_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

namespace {

cil_status check_params(const cil_cycle_params *p) {
  if (p->dim != 2 && p->dim != 3) return CIL_ERR_CONFIG;
  if (!(p->dt > 0.0) || !(p->sigma_core > 0.0) || !(p->E > 0.0)) return CIL_ERR_CONFIG;
  for (int d = 0; d < p->dim; ++d)
    if (!(p->box[d] > 0.0)) return CIL_ERR_CONFIG;
  if (p->integrator == CIL_CYCLE_EULER) {
    if (!(p->zeta > 0.0)) return CIL_ERR_CONFIG;  // "In Euler, zeta should > 0!!!" (CIL.cu:924)
  } else if (p->integrator == CIL_CYCLE_DPD) {
    // the reference's DPD step draws no passive noise (NOISE_ON is set by the stochastic
    // integrators only, Input.cpp:527-535)
    if (!(p->mass > 0.0) || !(p->kbt >= 0.0) || !(p->dis_diff >= 0.0) || !(p->dis_bg >= 0.0) || p->noise_D != 0.0)
      return CIL_ERR_CONFIG;
  } else {
    return CIL_ERR_CONFIG;
  }
  if (p->apoptosis < CIL_APOP_NONE || p->apoptosis > CIL_APOP_CYCLE_EXTRUDE) return CIL_ERR_CONFIG;
  if (p->precision != 0 && p->precision != 1) return CIL_ERR_CONFIG;
  if (p->divide && (!(p->tau_div_mu > 0.0) || !(p->cycle_p0 != 0.0) || !(p->cycle_sigma_min > 0.0) ||
                    !(p->cycle_tau_r > 0.0) || !(p->cycle_tau_v > 0.0)))
    return CIL_ERR_CONFIG;
  // a migration time (crawling state) takes cells out of the single-element cycle for good in
  // the reference (initializeCellStatus with calculDivisionsSingle); the shipped runs use 0
  if (p->divide && p->tau_mig_mu != 0.0) return CIL_ERR_CONFIG;
  return CIL_OK;
}

int blocks_for(int n) { return n > 0 ? (n + kTile - 1) / kTile : 1; }

constexpr int kNumSMs = 152;  // GB300

// grid of a removal kernel at h->pair_bs threads per block
int pair_grid(const cil_cycle *h) { return (h->cap + h->pair_bs - 1) / h->pair_bs; }

// Lanes per cell of the pair kernels: up to 8, while the colony gives fewer than two warps
// per scheduler of every SM (152 SMs x 4 x 2 x 32 threads), and while the grid over the
// capacity stays within 2^24 threads. The restatement uses the same rule.
int contact_lane_bits(long long ncells, long long capacity) {
  int b = 0;
  while (b < 3 && ncells * (2LL << b) <= 2LL * kNumSMs * 4 * 32 && (capacity << (b + 1)) <= (1LL << 24)) ++b;
  return b;
}

int bins_along(double box, double width) {
  const int ns = static_cast<int>(box / width);
  return ns < 1 ? 1 : (ns > 4096 ? 4096 : ns);
}

// The bin grid of a step call: bins at least 1.05 x max(SIGMA_CORE, the colony's largest
// diameter) wide, so that the pair search spans one bin on each side (3^D bins) unless cells
// grow by more than 5 % within the call (the search then widens by itself). Narrower bins than
// the diameter would make every search span two bins on each side (5^D bins). The host
// restatement picks its grid by the same rule at the start of each call.
void set_bins(cil_cycle *h, double smax, int ncells) {
  CyConst &C = h->C;
  const double w = (smax > h->p.sigma_core ? smax : h->p.sigma_core) * 1.05;
  const int before[3] = {C.ns[0], C.ns[1], C.ns[2]};
  // blocks of the removal kernels (FP64-heavy, no block cooperation): small enough that
  // a small colony still spreads over every SM (two blocks per SM), 32 to kTile threads
  const int bs_before = h->pair_bs, lb_before = h->lane_bits;
  h->lane_bits = contact_lane_bits(ncells, h->cap);
  if (h->lane_bits != lb_before) h->grid_gen += 1;
  h->pair_bs = 32;
  while (h->pair_bs < kTile && static_cast<long long>(h->pair_bs) * 2 * kNumSMs < ncells) h->pair_bs *= 2;
  // the grids cover the capacity: keep them at most 65536 blocks (a large capacity, few cells)
  while (h->pair_bs < kTile && (h->cap + h->pair_bs - 1) / h->pair_bs > 65536) h->pair_bs *= 2;
  if (h->pair_bs != bs_before) h->grid_gen += 1;
  h->nbins = 1;
  for (int d = 0; d < 3; ++d) {
    if (d < h->p.dim) {
      const int ns = bins_along(C.box[d], w);
      C.ns[d] = ns;
      C.bw[d] = C.box[d] / ns;
      C.inv_bw[d] = ns / C.box[d];
    } else {
      C.ns[d] = 1;
      C.bw[d] = 1.0;
      C.inv_bw[d] = 1.0;
    }
    C.bwf[d] = static_cast<float>(C.bw[d]);
    C.scalef[d] = static_cast<float>(C.inv_bw[d]);
    C.inv_bwf[d] = std::nextafter(static_cast<float>(C.inv_bw[d]), INFINITY);
    h->nbins *= C.ns[d];
  }
  if (C.ns[0] != before[0] || C.ns[1] != before[1] || C.ns[2] != before[2]) h->grid_gen += 1;
}

double host_sigma_max(const cil_cycle *h) {
  double s;
  const unsigned long long b = h->h_cnt->sigma_max_bits;
  std::memcpy(&s, &b, sizeof s);
  return s;
}

// scan of count[0..m) into start[0..m] (start[m] = total), count left at zero. Up to 2048 chunks (2M
// bins) each block adds the chunk sums before its own; the quadratic cost of that passes a launch's
// near there.
void scan_into(cil_cycle *h, int *count, int m, int *start) {
  const int nchunks = m / kScanTile + 1;  // covers index m
  const int scanned = nchunks > 2048 ? 1 : 0;
  cil::launch_step(true, nchunks, kTile, 0, h->stream, k_cy_chunk_sums, count, m, h->part);
  if (scanned) k_cy_scan_small<<<1, kTile, 0, h->stream>>>(h->part, nchunks);
  cil::launch_step(true, nchunks, kTile, 0, h->stream, k_cy_chunk_apply, count, m, h->part, start, scanned);
  h->launches += 2 + scanned;
}

// drift: with DPD's first half kick and drift
cil_status bin_cells(cil_cycle *h, int drift) {
  const CySet &S = h->set[h->cur];
  const int g = blocks_for(h->cap);
  cil::launch_step(true, g, kTile, 0, h->stream, k_cy_keys, h->C, S, h->cnt, h->key, h->arrival, h->bcount, h->dblk, drift);
  scan_into(h, h->bcount, h->nbins, h->bstart);
  cil::launch_step(true, g, kTile, 0, h->stream, k_cy_scatter, h->cnt, h->key, h->arrival, h->bstart, h->tmp);
  cil::launch_step(true, g, kTile, 0, h->stream, k_cy_place, h->C, S, h->cnt, h->bstart, h->tmp, h->O,
                                         h->C.dpd && h->p.precision == 1 ? 1 : 0);
  h->launches += 3;
  return CIL_OK;
}

cil_status removals(cil_cycle *h, int mode) {
  const int g = pair_grid(h), bs = h->pair_bs;
  CySet &A = h->set[h->cur];
  CySet &B = h->set[1 - h->cur];
  k_cy_mark<<<g, bs, 0, h->stream>>>(h->C, A, h->cnt, h->ts_dev, mode, h->flag, h->blk);
  k_cy_scan_small<<<1, kTile, 0, h->stream>>>(h->blk, g);
  k_cy_compact<<<g, bs, 0, h->stream>>>(h->C, A, B, h->cnt, h->flag, h->blk);
  k_cy_commit_removals<<<1, 1, 0, h->stream>>>(h->cnt, h->blk, g, mode);
  h->launches += 4;
  h->cur = 1 - h->cur;
  return CIL_OK;
}

// blocks of a pair kernel: 2^lane_bits lanes for every cell of the capacity
int pair_blocks(const cil_cycle *h) {
  const long long threads = static_cast<long long>(h->cap) << h->lane_bits;
  return static_cast<int>((threads + kPairBlock - 1) / kPairBlock);
}

template <int D>
void launch_force_d(cil_cycle *h, CySet &S, double *frc, int mode) {
  const int g = pair_blocks(h);
  if (h->p.precision == 1)
    cil::launch_step(true, g, kPairBlock, 0, h->stream, k_cy_force<D, true>, h->C, S, frc, h->cnt, h->bstart, h->ts_dev, mode,
                                                         h->O, h->lane_bits, h->dblk, h->dueq, h->sig_part);
  else
    cil::launch_step(true, g, kPairBlock, 0, h->stream, k_cy_force<D, false>, h->C, S, frc, h->cnt, h->bstart, h->ts_dev, mode,
                                                          h->O, h->lane_bits, h->dblk, h->dueq, h->sig_part);
}

void launch_force(cil_cycle *h, CySet &S, double *frc, int mode) {
  if (h->C.D == 2)
    launch_force_d<2>(h, S, frc, mode);
  else
    launch_force_d<3>(h, S, frc, mode);
  h->launches += 1;
}

template <int D>
void launch_dpd_forces_d(cil_cycle *h, CySet &S, int key_off, int kick_on) {
  const int g = pair_blocks(h);
  if (h->p.precision == 1)
    cil::launch_step(true, g, kPairBlock, 0, h->stream, k_dpd_forces<D, true>, h->C, S, h->vs, h->cnt, h->bstart, h->ts_dev, key_off, kick_on,
                                                         h->O, h->vel_next, h->lane_bits);
  else
    cil::launch_step(true, g, kPairBlock, 0, h->stream, k_dpd_forces<D, false>, h->C, S, h->vs, h->cnt, h->bstart, h->ts_dev, key_off,
                                                          kick_on, h->O, h->vel_next, h->lane_bits);
}

void launch_dpd_forces(cil_cycle *h, CySet &S, int key_off, int kick_on) {
  if (h->C.D == 2)
    launch_dpd_forces_d<2>(h, S, key_off, kick_on);
  else
    launch_dpd_forces_d<3>(h, S, key_off, kick_on);
  h->launches += 1;
}

template <int D>
void launch_dpd_dis_d(cil_cycle *h, CySet &S) {
  const int g = pair_blocks(h);
  if (h->p.precision == 1)
    cil::launch_step(true, g, kPairBlock, 0, h->stream, k_dpd_dis<D, true>, h->C, S, h->cnt, h->bstart, h->ts_dev, h->O, h->vel_next,
                                                        h->lane_bits, h->dblk, h->dueq, h->sig_part);
  else
    cil::launch_step(true, g, kPairBlock, 0, h->stream, k_dpd_dis<D, false>, h->C, S, h->cnt, h->bstart, h->ts_dev, h->O, h->vel_next,
                                                         h->lane_bits, h->dblk, h->dueq, h->sig_part);
}

void launch_dpd_dis(cil_cycle *h, CySet &S) {
  if (h->C.D == 2)
    launch_dpd_dis_d<2>(h, S);
  else
    launch_dpd_dis_d<3>(h, S);
  h->launches += 1;
}

// Fc, pressure, Fd and Fr at the current positions and velocities (the forces the reference
// evaluates before its first step, CIL.cu:1096), draws keyed by the current step counter
void dpd_initial_forces(cil_cycle *h) {
  CySet &S = h->set[h->cur];
  bin_cells(h, 0);
  launch_dpd_forces(h, S, 0, 0);
}

cil_status enqueue_step(cil_cycle *h) {
  CySet &S = h->set[h->cur];
  bin_cells(h, h->C.dpd);
  if (h->C.dpd) {  // DPD (CIL.cu:1054-1066); this step's draws are keyed by ts + 1
    launch_dpd_forces(h, S, 1, 1);
    std::swap(S.v, h->vs);
    launch_dpd_dis(h, S);
  } else {
    launch_force(h, S, nullptr, 0);
  }
  h->ts += 1;
  if (h->C.divide) {  // also moves the step counter
    cil::launch_step(true, std::min(blocks_for(h->cap), 2 * kNumSMs), kTile, 0, h->stream, k_cy_divide, h->C, S, h->cnt, h->ts_dev,
                                                                                      h->dblk, h->dueq, h->sig_part,
                                                                                      h->lane_bits);
  } else {
    k_cy_advance<<<1, 1, 0, h->stream>>>(h->ts_dev);
  }
  h->launches += 1;
  if (h->C.apoptosis != CIL_APOP_NONE) removals(h, 1);
  CY_TRY(h, cudaGetLastError());
  return CIL_OK;
}

constexpr size_t kMaxStepGraphs = 16;

cil_cycle::Buffers buffers_of(const cil_cycle *h) {
  cil_cycle::Buffers b{};
  b.set[0] = h->set[0];
  b.set[1] = h->set[1];
  b.vs = h->vs;
  b.cur = h->cur;
  return b;
}

bool same_buffers(const cil_cycle::Buffers &a, const cil_cycle::Buffers &b) {
  return std::memcmp(&a.set[0], &b.set[0], sizeof(CySet)) == 0 &&
         std::memcmp(&a.set[1], &b.set[1], sizeof(CySet)) == 0 && a.vs == b.vs && a.cur == b.cur;
}

// One step through the graph of its buffer configuration: captured from enqueue_step the first
// time (the capture leaves the host state as the step leaves it), replayed afterwards
cil_status graph_step(cil_cycle *h) {
  const cil_cycle::Buffers b = buffers_of(h);
  for (const auto &g : h->graphs)
    if (g.grid == h->grid_gen && same_buffers(g.before, b)) {
      CY_TRY(h, cudaGraphLaunch(g.exec, h->stream));
      h->set[0] = g.after.set[0];
      h->set[1] = g.after.set[1];
      h->vs = g.after.vs;
      h->cur = g.after.cur;
      h->ts += 1;
      h->launches += g.nodes;
      return CIL_OK;
    }
  // graphs of earlier grids serve no more (a grid's number never comes back), and none of them is in
  // flight: a grid changes between calls, which end with the stream idle
  for (size_t k = 0; k < h->graphs.size();) {
    if (h->graphs[k].grid != h->grid_gen) {
      cudaGraphExecDestroy(h->graphs[k].exec);
      h->graphs.erase(h->graphs.begin() + static_cast<std::ptrdiff_t>(k));
    } else {
      ++k;
    }
  }
  if (h->graphs.size() >= kMaxStepGraphs) return enqueue_step(h);
  const int64_t l0 = h->launches, ts0 = h->ts;
  if (cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    return enqueue_step(h);
  }
  const cil_status st = enqueue_step(h);
  cudaGraph_t graph = nullptr;
  const cudaError_t ce = cudaStreamEndCapture(h->stream, &graph);
  cudaGraphExec_t exec = nullptr;
  cudaError_t ie = cudaErrorUnknown;
  if (st == CIL_OK && ce == cudaSuccess && graph) ie = cudaGraphInstantiate(&exec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (ie != cudaSuccess) {
    // nothing ran: put the host state back as it was before the capture and launch the step
    cudaGetLastError();
    h->set[0] = b.set[0];
    h->set[1] = b.set[1];
    h->vs = b.vs;
    h->cur = b.cur;
    h->ts = ts0;
    h->launches = l0;
    return enqueue_step(h);
  }
  h->graphs.push_back({b, buffers_of(h), h->grid_gen, exec, h->launches - l0});
  CY_TRY(h, cudaGraphLaunch(exec, h->stream));
  return CIL_OK;
}

// Pageable memory that nobody has touched is faulted in here, on the host, before a copy into it: the
// device faults its pages in one by one (a download of 0.6M cells into new arrays took 51 ms, now 4.2; with a
// host loop over the vectors 30).
void touch_pages(void *dst, size_t bytes) {
  if (bytes < 65536) return;  // a page or two
  cudaPointerAttributes at{};
  const bool pageable = cudaPointerGetAttributes(&at, dst) != cudaSuccess || at.type == cudaMemoryTypeUnregistered;
  cudaGetLastError();
  if (!pageable) return;
  volatile char *p = static_cast<char *>(dst);
  for (size_t k = 0; k < bytes; k += 4096) p[k] = 0;
  p[bytes - 1] = 0;
}

cil_status read_counters(cil_cycle *h) {
  CY_TRY(h, cudaMemcpyAsync(h->h_cnt, h->cnt, sizeof(CyCounters), cudaMemcpyDeviceToHost, h->stream));
  CY_TRY(h, cudaStreamSynchronize(h->stream));
  if (h->h_cnt->err & kErrNonFinite) return h->fail(CIL_ERR_NAN, "non-finite force");
  if (h->h_cnt->err & kErrCapacity) return h->fail(CIL_ERR_CAPACITY, "cell capacity exceeded");
  if (h->h_cnt->err & kErrOutOfBox) return h->fail(CIL_ERR_OUT_OF_BOX, "Particle outside domain!");
  if (h->h_cnt->err & kErrCrowded) return h->fail(CIL_ERR_CAPACITY, "more than 256 cells in one bin (overlapping cells)");
  return CIL_OK;
}

}  // namespace

extern "C" {

cil_status cil_cycle_create(const cil_cycle_params *p, int32_t capacity, uint64_t seed, int32_t device,
                            cil_cycle **out) {
  if (!p || !out || capacity <= 0) return CIL_ERR_CONFIG;
  *out = nullptr;
  if (check_params(p) != CIL_OK) return CIL_ERR_CONFIG;
  if (cudaSetDevice(device) != cudaSuccess) {
    cudaGetLastError();
    return CIL_ERR_CUDA;
  }
  cil_cycle *h = new cil_cycle();
  h->p = *p;
  h->device = device;
  h->cap = capacity;
  CyConst &C = h->C;
  C.D = p->dim;
  C.capacity = capacity;
  C.dt = p->dt;
  for (int d = 0; d < 3; ++d) {
    C.periodic[d] = d < p->dim ? p->periodic[d] : 0;
    C.box[d] = d < p->dim ? p->box[d] : 1.0;
    C.half[d] = 0.5 * C.box[d];
    C.boxf[d] = static_cast<float>(C.box[d]);
    C.halff[d] = static_cast<float>(C.half[d]);
  }
  // bin arrays for the finest grid the colony can use (width SIGMA_CORE); set_bins picks the
  // grid of each call
  h->nbins_cap = 1;
  for (int d = 0; d < p->dim; ++d) h->nbins_cap *= bins_along(C.box[d], p->sigma_core);
  C.sigma_core = p->sigma_core;
  set_bins(h, p->sigma_core, capacity);
  C.hz_c = (1 - p->nu * p->nu) / p->E;
  C.adhesion = p->adhesion;
  C.c2f = static_cast<float>(C.hz_c + C.hz_c);
  C.adhf = static_cast<float>(C.adhesion);
  C.motility = p->motility;
  C.zeta = p->zeta;
  C.zeta_p = p->zeta_p;
  C.zeta_p_beta = p->zeta_p_beta;
  C.noise_amp = p->noise_D > 0.0 ? std::sqrt(2.0 * p->noise_D) * (1.0 / std::sqrt(p->dt)) : 0.0;
  C.divide = p->divide;
  C.apoptosis = p->apoptosis;
  C.tau_div_mu = p->tau_div_mu;
  C.tau_div_sigma = p->tau_div_sigma;
  C.tau_mig_mu = p->tau_mig_mu;
  C.tau_mig_sigma = p->tau_mig_sigma;
  // the cycle time's log-normal exp(mu2 + s2 Z), mu2 = log(mu^2 / sqrt(mu^2 + s^2)),
  // s2 = sqrt(log(1 + s^2 / mu^2)) (Random.hpp:55-60)
  if (p->tau_div_mu != 0.0) {
    const double mu = p->tau_div_mu, sd = p->tau_div_sigma;
    C.div_mu2 = std::log((mu * mu) / std::sqrt(mu * mu + sd * sd));
    C.div_s2 = std::sqrt(std::log(1 + (sd * sd) / (mu * mu)));
  }
  C.inv_hz = 1.0 / (0.75 * (C.hz_c + C.hz_c));
  // cycle times in steps (Input.cpp:176-178, CIL.cuh:225-233)
  C.v1 = p->v1;
  C.tau_r = p->cycle_tau_r * p->tau_div_mu / p->dt;
  C.tau_v = p->cycle_tau_v * p->tau_div_mu / p->dt;
  C.tau_p = p->cycle_tau_p * p->tau_div_mu / p->dt;
  {
    const double r = p->cycle_sigma_min / 2;
    C.v_s = p->dim == 3 ? 4 * kPi * (r * r * r) / 3 : kPi * (r * r);  // Sigma2Volume / Sigma2Area
  }
  C.p0 = p->cycle_p0;
  C.inv_p0 = 1.0 / C.p0;
  C.growth = (C.v1 - 1) / C.tau_v;
  C.inv_vs_tau_v = 1.0 / (C.v_s * C.tau_v);
  C.inv_tau_r = 1.0 / C.tau_r;
  C.inv_tau_r_neg = 1.0 / (C.tau_r * p->cycle_rho_ratio);
  C.beta_vs = p->cycle_beta_vs;
  C.rho_ratio = p->cycle_rho_ratio;
  C.r_maxed_inv = p->cycle_r_maxed > 0.0 ? 1.0 / p->cycle_r_maxed : 1.0;
  C.p_shift = p->cycle_p_shift * p->cycle_p0;
  C.p_shift_tau_inv = p->cycle_p_shift_tau > 0.0 ? 1.0 / (p->cycle_p_shift_tau * p->tau_div_mu) * p->dt : 0.0;
  C.osm = p->osmotic_pressure;
  C.apop_pressure = p->apop_pressure;
  C.apop_duration = p->apop_duration;
  C.apop_rate_step = p->apop_rate * p->dt;
  C.extr_gamma = p->extr_gamma;
  C.apop_steps = p->apop_duration / p->dt;
  C.extr_rate = p->extr_rate;
  C.dpd = p->integrator == CIL_CYCLE_DPD ? 1 : 0;
  C.kick_f = p->dt / (2 * (2 * p->mass));
  C.kick_r = std::sqrt(p->dt) / (2 * (2 * p->mass));
  C.gamma_d = p->dis_diff;
  C.gamma_b = p->dis_bg;
  C.sigma_r = std::sqrt(2 * p->dis_diff * p->kbt);  // Sigma (MD.cu:872)
  C.gdf = static_cast<float>(C.gamma_d);
  C.srf = static_cast<float>(C.sigma_r);
  C.seed_lo = static_cast<uint32_t>(seed);
  C.seed_hi = static_cast<uint32_t>(seed >> 32);

  const size_t cap = capacity, D = p->dim;
  bool ok = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) == cudaSuccess &&
            cudaEventCreate(&h->ev[0]) == cudaSuccess && cudaEventCreate(&h->ev[1]) == cudaSuccess;
  for (int s = 0; ok && s < 2; ++s) {
    CySet &S = h->set[s];
    S.x = h->alloc<double>(D * cap);
    S.v = h->alloc<double>(D * cap);
    S.sig = h->alloc<double>(cap);
    S.sigt = h->alloc<double>(cap);
    S.theta = h->alloc<double>(cap);
    S.rho = h->alloc<double>(cap);
    S.om = h->alloc<double>(cap);
    S.p = h->alloc<double>(cap);
    S.tp = h->alloc<int>(cap);
    S.t0 = h->alloc<int>(cap);
    S.tsw = h->alloc<int>(cap);
    ok = S.x && S.v && S.sig && S.sigt && S.theta && S.rho && S.om && S.p && S.tp && S.t0 && S.tsw;
    if (ok && C.dpd) {
      S.fc = h->alloc<double>(D * cap);
      S.fd = h->alloc<double>(D * cap);
      S.fr = h->alloc<double>(D * cap);
      ok = S.fc && S.fd && S.fr;
    }
  }
  if (ok && C.dpd) {
    h->vs = h->alloc<double>(D * cap);
    ok = h->vs != nullptr;
  }
  if (ok && p->precision == 1 && C.dpd) {
    h->O.vel = h->alloc<float4>(cap);
    h->vel_next = h->alloc<float4>(cap);
    h->O.loc = h->alloc<float4>(cap);
    h->O.cell = h->alloc<ushort4>(cap);
    ok = h->O.vel && h->vel_next && h->O.loc && h->O.cell;
  }
  h->nblocks = (capacity + 31) / 32;  // blocks of the per-cell event kernels at their smallest (32 threads)
  h->nparts = (h->nbins_cap + kScanTile - 1) / kScanTile + 1;
  if (ok) {
    h->frc = h->alloc<double>(D * cap);
    h->O.x = h->alloc<double>(D * cap);
    h->O.rad = h->alloc<double>(cap);
    h->O.rec = h->alloc<float4>(cap);
    h->O.idx = h->alloc<int>(cap);
    h->O.bin = h->alloc<int>(cap);
    h->cnt = h->alloc<CyCounters>(1);
    h->ts_dev = h->alloc<int>(1);
    h->key = h->alloc<int>(cap);
    h->bcount = h->alloc<int>(h->nbins_cap + 1);
    h->bstart = h->alloc<int>(h->nbins_cap + 1);
    h->arrival = h->alloc<int>(cap);
    h->tmp = h->alloc<int2>(cap);
    h->dueq = h->alloc<int>(kDueMax);
    h->sig_part = h->alloc<unsigned long long>(cap / 4 + kPairBlock / 32);  // up to 8 lanes per cell
    h->dblk = h->alloc<int>(blocks_for(capacity));
    h->part = h->alloc<int>(h->nparts + 1);
    h->flag = h->alloc<int>(cap);
    h->blk = h->alloc<int>(h->nblocks + 1);
    ok = h->frc && h->O.x && h->O.rad && h->O.rec && h->O.idx && h->O.bin && h->cnt && h->ts_dev && h->key &&
         h->bcount && h->bstart && h->arrival && h->tmp && h->dblk && h->dueq && h->sig_part &&
         h->part && h->flag && h->blk &&
         cudaHostAlloc(&h->h_cnt, sizeof(CyCounters), cudaHostAllocDefault) == cudaSuccess;
  }
  if (ok) ok = cudaMemsetAsync(h->cnt, 0, sizeof(CyCounters), h->stream) == cudaSuccess &&
               cudaMemsetAsync(h->ts_dev, 0, sizeof(int), h->stream) == cudaSuccess &&
               cudaMemsetAsync(h->bcount, 0, sizeof(int) * (h->nbins_cap + 1), h->stream) == cudaSuccess &&
               cudaStreamSynchronize(h->stream) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    cil_cycle_destroy(h);
    return CIL_ERR_CUDA;
  }
  *out = h;
  return CIL_OK;
}

void cil_cycle_destroy(cil_cycle *h) {
  if (!h) return;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (auto &g : h->graphs) cudaGraphExecDestroy(g.exec);
  for (void *q : h->allocs) cudaFree(q);
  if (h->h_cnt) cudaFreeHost(h->h_cnt);
  for (auto e : h->ev)
    if (e) cudaEventDestroy(e);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

cil_status cil_cycle_upload(cil_cycle *h, const cil_cycle_view *v) {
  if (!h || !v || !v->pos) return CIL_ERR_CONFIG;
  if (v->ncells < 0 || v->ncells > h->cap) return h->fail(CIL_ERR_CAPACITY, "cil_cycle_upload: more cells than the capacity");
  CY_TRY(h, cudaSetDevice(h->device));
  const int n = v->ncells, D = h->C.D, g = blocks_for(n);
  const size_t cap = h->cap, vec = sizeof(double) * static_cast<size_t>(n) * D;
  // staged and checked before any of the state is written (O.x and the outputs of the last download
  // are free between calls)
  double *st_pos = h->O.x, *st_vel = h->frc;
  int bad = 0, *d_bad = h->dueq;
  if (n > 0) {
    CY_TRY(h, cudaMemcpyAsync(st_pos, v->pos, vec, cudaMemcpyHostToDevice, h->stream));
    CY_TRY(h, cudaMemsetAsync(d_bad, 0, sizeof(int), h->stream));
    k_cy_check_staged<<<g, kTile, 0, h->stream>>>(h->C, st_pos, n, d_bad);
    CY_TRY(h, cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    if (v->vel) CY_TRY(h, cudaMemcpyAsync(st_vel, v->vel, vec, cudaMemcpyHostToDevice, h->stream));
    CY_TRY(h, cudaStreamSynchronize(h->stream));
  }
  if (bad) return h->fail(CIL_ERR_OUT_OF_BOX, "Input Positions Out of Bounds!");
  h->cur = 0;
  CySet &S = h->set[0];
  CY_TRY(h, cudaMemsetAsync(S.v, 0, sizeof(double) * D * cap, h->stream));
  if (n > 0) {
    k_cy_from_host<<<g, kTile, 0, h->stream>>>(st_pos, n, D, cap, S.x);
    if (v->vel) k_cy_from_host<<<g, kTile, 0, h->stream>>>(st_vel, n, D, cap, S.v);
  }
  auto up = [&](double *dst, const double *src) -> cudaError_t {
    return src ? cudaMemcpyAsync(dst, src, sizeof(double) * n, cudaMemcpyHostToDevice, h->stream) : cudaSuccess;
  };
  CY_TRY(h, up(S.sig, v->sigma));
  CY_TRY(h, up(S.sigt, v->sigma_t ? v->sigma_t : v->sigma));
  CY_TRY(h, up(S.theta, v->theta));
  CY_TRY(h, up(S.rho, v->rho));
  CY_TRY(h, up(S.om, v->angvel));
  CY_TRY(h, cudaMemsetAsync(S.p, 0, sizeof(double) * cap, h->stream));
  if (v->pressure) CY_TRY(h, up(S.p, v->pressure));
  CyCounters c{};
  c.n = n;
  CY_TRY(h, cudaMemcpyAsync(h->cnt, &c, sizeof(c), cudaMemcpyHostToDevice, h->stream));
  const int ts = v->ts;
  CY_TRY(h, cudaMemcpyAsync(h->ts_dev, &ts, sizeof(int), cudaMemcpyHostToDevice, h->stream));
  h->ts = ts;
  const int fill_sigma = v->sigma ? 0 : 1;
  const int fill_cycle = (v->theta && v->rho && v->angvel) ? 0 : 1;
  k_cy_init_status<<<blocks_for(h->cap), kTile, 0, h->stream>>>(h->C, S, h->cnt, ts, fill_sigma, fill_cycle);
  if (v->tpressure) {
    CY_TRY(h, cudaMemcpyAsync(S.tp, v->tpressure, sizeof(int) * n, cudaMemcpyHostToDevice, h->stream));
  }
  k_cy_sigma_max<<<blocks_for(h->cap), kTile, 0, h->stream>>>(h->C, S, h->cnt);
  CY_TRY(h, cudaGetLastError());
  const cil_status st = read_counters(h);
  if (st != CIL_OK) return st;
  set_bins(h, host_sigma_max(h), h->h_cnt->n);
  h->uploaded = true;
  if (!h->C.dpd) return CIL_OK;
  dpd_initial_forces(h);
  CY_TRY(h, cudaGetLastError());
  return read_counters(h);
}

cil_status cil_cycle_step(cil_cycle *h, int32_t nsteps, int64_t *ts) {
  if (!h) return CIL_ERR_CONFIG;
  if (!h->uploaded) return h->fail(CIL_ERR_STATE, "cil_cycle_step before cil_cycle_upload");
  if (nsteps < 0) return h->fail(CIL_ERR_CONFIG, "negative step count");
  CY_TRY(h, cudaSetDevice(h->device));
  // the counters of the last call (every entry point ends by reading them)
  set_bins(h, host_sigma_max(h), h->h_cnt->n);
  h->launches = 0;
  CY_TRY(h, cudaEventRecord(h->ev[0], h->stream));
  const bool graphs = !(h->p.flags & CIL_CYCLE_NO_GRAPH);
  for (int k = 0; k < nsteps; ++k) {
    const cil_status st = graphs ? graph_step(h) : enqueue_step(h);
    if (st != CIL_OK) return st;
  }
  CY_TRY(h, cudaEventRecord(h->ev[1], h->stream));
  const cil_status st = read_counters(h);
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, h->ev[0], h->ev[1]);
  h->t_total = ms;
  if (ts) *ts = h->ts;
  return st;
}

cil_status cil_cycle_check_positions(cil_cycle *h) {
  if (!h) return CIL_ERR_CONFIG;
  if (!h->uploaded) return h->fail(CIL_ERR_STATE, "not uploaded");
  CY_TRY(h, cudaSetDevice(h->device));
  if (h->p.drain) {
    removals(h, 2);
    CY_TRY(h, cudaGetLastError());
    return read_counters(h);
  }
  // without drain any cell off the box is an error (run_assert, CIL.cu:956)
  const int g = pair_grid(h);
  k_cy_mark<<<g, h->pair_bs, 0, h->stream>>>(h->C, h->set[h->cur], h->cnt, h->ts_dev, 2, h->flag, h->blk);
  k_cy_scan_small<<<1, kTile, 0, h->stream>>>(h->blk, g);
  CY_TRY(h, cudaGetLastError());
  cil_status st = read_counters(h);
  if (st != CIL_OK) return st;
  int kept = 0;
  CY_TRY(h, cudaMemcpy(&kept, h->blk + g, sizeof(int), cudaMemcpyDeviceToHost));
  if (kept != h->h_cnt->n) return h->fail(CIL_ERR_OUT_OF_BOX, "Particle outside domain!");
  return CIL_OK;
}

cil_status cil_cycle_download(cil_cycle *h, cil_cycle_view *v) {
  if (!h || !v) return CIL_ERR_CONFIG;
  CY_TRY(h, cudaSetDevice(h->device));
  if (h->uploaded && !h->C.dpd) {
    const int64_t launches = h->launches;  // cil_cycle_timings reports the last cil_cycle_step
    // the forces and pressures at the current state, which the reference's Euler step
    // evaluates at its end (CIL.cu:1019) and writes out; the next step's force pass computes
    // the same values again (same positions, velocities and step key)
    bin_cells(h, 0);
    launch_force(h, h->set[h->cur], h->frc, 1);
    h->launches = launches;
    CY_TRY(h, cudaGetLastError());
  }
  const cil_status st = read_counters(h);
  const int n = h->h_cnt->n, D = h->C.D;
  v->ncells = n;
  v->ts = static_cast<int32_t>(h->ts);
  if (n > v->capacity) return h->fail(CIL_ERR_CAPACITY, "cil_cycle_download: host arrays too small");
  const CySet &S = h->set[h->cur];
  const size_t cap = h->cap;
  // rearranged in O.x (free between steps), one vector after the other on the stream
  auto vec = [&](double *dst, const double *src) -> cudaError_t {
    if (!dst || n == 0) return cudaSuccess;
    touch_pages(dst, sizeof(double) * static_cast<size_t>(n) * D);
    k_cy_to_host<<<blocks_for(n), kTile, 0, h->stream>>>(src, n, D, cap, h->O.x);
    return cudaMemcpyAsync(dst, h->O.x, sizeof(double) * static_cast<size_t>(n) * D, cudaMemcpyDeviceToHost, h->stream);
  };
  auto sca = [&](void *dst, const void *src, size_t es) -> cudaError_t {
    if (!dst || n == 0) return cudaSuccess;
    touch_pages(dst, es * n);
    return cudaMemcpyAsync(dst, src, es * n, cudaMemcpyDeviceToHost, h->stream);
  };
  CY_TRY(h, vec(v->pos, S.x));
  CY_TRY(h, vec(v->vel, S.v));
  CY_TRY(h, sca(v->sigma, S.sig, sizeof(double)));
  CY_TRY(h, sca(v->sigma_t, S.sigt, sizeof(double)));
  CY_TRY(h, sca(v->theta, S.theta, sizeof(double)));
  CY_TRY(h, sca(v->rho, S.rho, sizeof(double)));
  CY_TRY(h, sca(v->angvel, S.om, sizeof(double)));
  CY_TRY(h, sca(v->pressure, S.p, sizeof(double)));
  CY_TRY(h, sca(v->tpressure, S.tp, sizeof(int)));
  CY_TRY(h, sca(v->t0, S.t0, sizeof(int)));
  if (h->C.dpd) {
    CY_TRY(h, vec(v->force, S.fc));
    CY_TRY(h, vec(v->force_dis, S.fd));
    CY_TRY(h, vec(v->force_ran, S.fr));
  } else {
    CY_TRY(h, vec(v->force, h->frc));
    for (double *f : {v->force_dis, v->force_ran})
      if (f) std::fill(f, f + static_cast<size_t>(n) * D, 0.0);
  }
  CY_TRY(h, cudaStreamSynchronize(h->stream));
  return st;
}

cil_status cil_cycle_timings(cil_cycle *h, double *total_ms, int64_t *launches) {
  if (!h) return CIL_ERR_CONFIG;
  if (total_ms) *total_ms = h->t_total;
  if (launches) *launches = h->launches;
  return CIL_OK;
}

void cil_cycle_last_error(const cil_cycle *h, char *buf, size_t len) {
  if (!buf || len == 0) return;
  snprintf(buf, len, "%s", h ? h->err.c_str() : "");
}

}  // extern "C"
