// Fused force + integrate kernels over the binned elements.
//
// Per element, in the reference's accumulation order (calculForcesPressure,
// CIL.cu:999-1007):
//   intra-cell spring + motility (binaryCellForce's role, MD.cu:525-598; assigns),
//   one-sided flat Hertz walls (Wall.hpp:80-91's role), passive noise zeta_j W
//   (CIL.cu:84-98), then pair forces from every other cell's elements in the 3^d
//   neighbour bins (calculInterForces + cellCellForce, CIL.cu:177-231, MD.cu:757-790,
//   as a full stencil: each thread accumulates only its own force, so no atomics), and
//   finally the overdamped Euler-Maruyama update with the reference's periodic wrap
//   (updatePositions, CIL.cu:858-875; BoundingBox::updatePos, Utils.hpp:561-566).
//
// FP64 form (k_force_fp64): everything in FP64; the parity path.
// Mixed form (k_force_mixed): GB300 issues FP64 at about 1/64 of the FP32 rate, so every
//   per-element operation runs in FP32 on bin-local coordinates (the element's FP32 offset
//   from its bin origin plus the FP32 offset between bin origins, exact for a periodic
//   image) and only the position accumulation stays FP64: one FP64 add per axis, with the
//   float->double conversion and the wrap test done in integer arithmetic.
#include "cil_internal.cuh"

namespace cil {

namespace {

// nint(v / L) (Utils.hpp:173-175) without a division when |v| < L / 4, where v / L lies in
// (-0.25, 0.25) whatever its rounding: a minimum image leaves v as it is then. L / 4 by its exponent,
// the comparison on bit patterns.
__device__ __forceinline__ double min_image(double v, double L) {
  const long long quarter = __double_as_longlong(L) - 0x0020000000000000ll;
  if ((__double_as_longlong(v) & 0x7fffffffffffffffll) < quarter) return v;
  return v - static_cast<double>(nint(v / L)) * L;
}

// The law of pair_force without its constant factor (pair_scale), with its roots and quotients formed
// from one reciprocal or reciprocal square root (as pair_f0_fast does in FP32), each within a few units
// of the last place; 0 out of range. hi = sigma_i / 2, sj = sigma_j. About 20 FP64 instructions for the
// soft core with the displacement, where the form with sqrt and divisions took 50 and one with the
// library's rsqrt 28.
//   soft core: q = 1 / (r rc) gives r / rc = r2 q and 1 / r = rc q
//   Hertz:     y = 1 / r gives r = r2 y, corrected by one Newton residual because sigma_ij - r
//              cancels; delta^1.5 = delta^2 / sqrt(delta)
//   LJ:        1 / r2
// The other laws, and squares out of those forms' range, take pair_force.
template <int LAW>
__device__ __forceinline__ double pair_scale(double eps) {
  return LAW == CIL_FORCE_LJ_WCA ? 24.0 * eps : (LAW == CIL_FORCE_SC ? 1.0 : -eps);
}

template <int LAW>
__device__ __forceinline__ double pair_force_lean(double r2, double hi, double sj, double eps, double rcs, double em,
                                                  double xi, int shifted) {
  const double sij = __fma_rn(0.5, sj, hi);
  if (LAW == CIL_FORCE_SOFTCORE || LAW == CIL_FORCE_HERTZ) {
    const double rc = rcs * sij;
    const double rc2 = rc * rc;
    if (mid_range(r2) && mid_range(rc2)) {
      if (__double_as_longlong(r2) >= __double_as_longlong(rc2)) return 0.0;
      if (LAW == CIL_FORCE_SOFTCORE) {
        const double q = rsqrt_pos(r2 * rc2);
        const double w = __fma_rn(-r2, q, 1.0);
        return (w * w) * (rc * q);
      }
      const double y = rsqrt_pos(r2);
      const double delta = sij - sqrt_from(r2, y);
      if (mid_range(delta)) return (delta * delta) * (rsqrt_pos(delta) * y);
      return delta * sqrt(delta) * y;
    }
  } else if (LAW == CIL_FORCE_LJ_WCA) {
    const double sij2 = sij * sij;
    const double rc2 = sij2 * (rcs * rcs);
    if (!shifted && mid_range(r2) && mid_range(rc2)) {
      if (__double_as_longlong(r2) > __double_as_longlong(rc2)) return 0.0;
      const double ir2 = rcp_normal(r2);
      const double s2 = sij2 * ir2;
      const double s6 = s2 * s2 * s2;
      return (s6 * ir2) * __fma_rn(-2.0, s6, 1.0);
    }
  }
  double f0 = 0.0;
  const double unit = LAW == CIL_FORCE_LJ_WCA ? 1.0 / 24.0 : (LAW == CIL_FORCE_SC ? eps : -1.0);
  return pair_force<LAW, double>(r2, 2.0 * hi, sj, unit, rcs, f0, em, xi, shifted) ? f0 : 0.0;
}

// Forms without lists: back elements whose cell's cycle ends at the coming events (step ts + 1) put it
// into the colony's due-cell queue, one atomic per warp. Whole warp.
__device__ __forceinline__ void collect_due(const ForceArgs &a, const ColonyConst &C, int c, bool back, int s, int e) {
  if (!a.collect_due || !C.divide) return;  // uniform
  const bool due = back && a.cyc[s].y == a.ts + 1;
  const unsigned dm = __ballot_sync(0xffffffffu, due);
  if (!dm) return;
  const int lane = threadIdx.x & 31, leader = __ffs(dm) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(&a.cnt[c].ndue, __popc(dm));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (due) a.dueq[C.due_base + base + __popc(dm & ((1u << lane) - 1u))] = (e >> 1) - C.cell_base;
}

// The FP64 force pass: 2^lane_bits lanes per binned element, blocks of kF64Block threads.
//
// What bounds it is the FP64 pipe (2 lanes a clock per SM, 1/64 of FP32), so FP64 runs only for
// the pairs inside the cutoff and with full warps:
//   walk    the candidates of the 3^d neighbour bins in rows along the last axis (consecutive bins
//           hold consecutive slots), tested in FP32 on absolute FP32 coordinates (ForceArgs::rec)
//           against a cutoff widened by their rounding; the lanes of an element take consecutive
//           candidates and a ballot keeps the survivors in walk order in shared memory, whatever
//           the number of lanes, so that an element's sum never depends on it;
//   pairs   the warp's survivors as one flattened range, a pair per lane (exact FP64 test and law),
//           results in shared memory;
//   sums    the element's first lane adds its pairs in walk order, then integrates.
// Lanes per element: see set_lane_bits (cil_api.cu). When every candidate's separation was formed
// in FP64 and each lane evaluated its own pairs, a pass took 879 us for 0.5M elements of the 2D
// growth colony, 376 us for 0.12M of the 3D channel and 42 us for 8192 WCA elements; now 161, 62
// and 12.4 us, with the FP64 pipe 77 % active in the first (152 FP64 instructions a warp's 32
// elements); the walk over 9 rows of bins is most of the channel's instructions. Compiled for 8 blocks
// an SM; in 3D a block's 28 KB of shared memory let 7 of them fit.
constexpr int kF64Block = 128;
constexpr int kF64Near = 512;  // survivors held per warp (16 per element at one lane each)
constexpr int kF64Seg = 128;   // pairs evaluated before their sums are taken
template <int D>
struct F64Warp {
  double res[kF64Seg * D];
  double x[32 * D];
  double hs[32];  // half diameters
  int tt[kF64Near];
  unsigned char code[kF64Near];
  unsigned char own[kF64Near];
};

template <int D, int LAW, int AHEAD>
__global__ void __launch_bounds__(kF64Block, 8) k_force_fp64(ForceArgs a_, int lane_bits) {
  enter_step_kernel();
  extern __shared__ __align__(16) unsigned char s_f64[];
  ForceArgs a = a_;
  a.ts = *a_.ts_dev;
  const int per_tile = 2 << lane_bits;  // blocks per tile of kTile elements (kTile = 2 kF64Block)
  const int t = blockIdx.x / per_tile;
  if (t >= a.tiles_live[a.B]) return;  // uniform per block
  F64Warp<D> &W = reinterpret_cast<F64Warp<D> *>(s_f64)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31, L = 1 << lane_bits;
  const int sub = lane & (L - 1), el = lane >> lane_bits;  // lane of the element, element of the warp
  const int c = colony_of_tile(a.tiles_live, a.B, t);
  const ColonyConst &C = a.col[c];
  const int s = C.slot_base + (t - a.tiles_live[c]) * kTile +
                (((blockIdx.x - t * per_tile) * kF64Block + static_cast<int>(threadIdx.x)) >> lane_bits);
  const int nlive = a.cnt[c].nlive;
  const size_t SS = a.SS;
  const int e = s < C.slot_base + nlive ? a.eid[s] : -1;
  const bool live = e >= 0;
  const int g = e >> 1, j = e & 1;
  double xi[D], F[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    xi[d] = live ? a.x_in[d * SS + s] : 0.0;
    F[d] = 0.0;
  }
  const double si = live ? a.sig[s] : 1.0;
  const int ps = live ? a.slot_of[e ^ 1] : -1;
  collect_due(a, C, c, live && sub == 0 && j == 0, s, e);

  if (live && sub == 0) {
    // ---- intra-cell: linear spring to the partner + motility along back->front
    {
      double rij[D];
      double r2 = 0.0;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const double xp = a.x_in[d * SS + ps];
        double v = (j == 0) ? xp - xi[d] : xi[d] - xp;  // r1 - r0
        if (C.periodic[d]) v = min_image(v, C.box[d]);
        rij[d] = v;
        r2 += v * v;
      }
      if (r2 == 0.0) {
#pragma unroll
        for (int d = 0; d < D; ++d) F[d] = 0.0;
      } else if (C.cell_sm && a.cst[g] == kCellDividing) {
        double spring, act[2];
        fene_bond_dividing<double>(r2, fmax(si, a.sig[ps]), C.fene_r2max_div, C.fene_kappa, C.fene_kappa_push,
                                   C.fene_ratio, C.div_r2min, C.growth_k0, C.growth_k1, C.growth_k2, spring, act);
        double rnd[3] = {0.0, 0.0, 0.0};
        if (C.act_noise && a.noise_mode == 2) bond_noise<D, double>(a.noise_act[g], a.noise_act_t[g], rij, sqrt(r2), rnd);
#pragma unroll
        for (int d = 0; d < D; ++d)
          F[d] = (j == 0) ? -(act[0] * rij[d] + spring * rij[d] * 1.0 + rnd[d] * rij[d])
                          : act[1] * rij[d] + spring * rij[d] * 1.0 + rnd[d] * rij[d];
      } else if (C.intra_fene) {
        const double r = sqrt(r2);
        double spring, sc;
        fene_bond<double>(r2, r, fmax(si, a.sig[ps]), C.fene_r2max, C.fene_kappa, C.fene_kappa_push, C.fene_ratio,
                          C.fene_rss, C.cil, spring, sc);
        double rnd[3] = {0.0, 0.0, 0.0};
        if (C.act_noise && a.noise_mode == 2) bond_noise<D, double>(a.noise_act[g], a.noise_act_t[g], rij, r, rnd);
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const double nd = C.cil ? rij[d] : rij[d] * sc;
          F[d] = (j == 0) ? -(C.motility[0] * nd + spring * rij[d] * 2.0 + rnd[d] * rij[d])
                          : C.motility[1] * nd + spring * rij[d] * 2.0 + rnd[d] * rij[d];
        }
      } else {
        double ir, r;
        if (mid_range(r2)) {
          ir = rsqrt_pos(r2);
          r = sqrt_from(r2, ir);
        } else {
          r = sqrt(r2);
          ir = 1.0 / r;
        }
        double rest = C.rest0;
        if (C.divide) {
          const int2 cy = a.cyc[s];
          const int span = cy.y - cy.x, age = a.ts - cy.x;
          double frac = 1.0;  // age / span within [0, 1], the quotient by its residual
          if (span > 0 && age < span) {
            const double m = static_cast<double>(span), p = static_cast<double>(age > 0 ? age : 0), im = rcp_normal(m);
            frac = p * im;
            frac = __fma_rn(__fma_rn(-frac, m, p), im, frac);
          }
          rest = __fma_rn(C.rest1 - C.rest0, frac, C.rest0);
        }
        const double sp = C.kappa * (r - rest);
        const double coef = ((j == 0) ? sp - C.motility[0] : C.motility[1] - sp) * ir;
#pragma unroll
        for (int d = 0; d < D; ++d) F[d] = coef * rij[d];
      }
    }
    // ---- walls
    if (C.nwalls > 0) {
      const double rad = 0.5 * si;
      for (int w = 0; w < C.nwalls; ++w) {
        const double dir = static_cast<double>(C.wall_dir[w]);
        const double delta = rad - dir * (xi[D - 1] - C.wall_pos[w]);
        if (delta > 0.0) F[D - 1] += dir * C.wall_E * delta * sqrt(delta);
      }
    }
    // ---- passive noise
    if (a.noise_mode == 2) {
      const size_t base = static_cast<size_t>(C.noise_per_cell ? g : e) * D;
#pragma unroll
      for (int d = 0; d < D; ++d) F[d] += C.zeta[j] * a.noise[base + d];
    } else if (a.noise_mode == 1) {
      uint32_t w[4];
      noise_words<D>(e - 2 * C.cell_base, C.noise_per_cell, noise_index(a.ts, a.heun), C.rng_stream, a.seed_lo, a.seed_hi, w);
      float n[4];
      box_muller(w[0], w[1], n[0], n[1]);
      if (D == 3) box_muller(w[2], w[3], n[2], n[3]);
#pragma unroll
      for (int d = 0; d < D; ++d) F[d] = __fma_rn(C.zeta[j] * C.noise_amp, static_cast<double>(n[d]), F[d]);
    }
  }

  // ---- pair forces
  const double eps = C.epsilon, rcs = C.rcut_scale, hs = 0.5 * si;
  double P[D];  // the pair forces without the law's factor
#pragma unroll
  for (int d = 0; d < D; ++d) P[d] = 0.0;
  if (C.single_bin) {
    if (live && sub == 0) {
      // one bin: all elements, minimum image as BoundingBox::distance (Utils.hpp:536-544)
      for (int tt = C.slot_base; tt < C.slot_base + nlive; ++tt) {
        const int ej = a.eid[tt];
        if (ej < 0 || (ej >> 1) == g) continue;
        double dx[D];
        double r2 = 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          double v = a.x_in[d * SS + tt] - xi[d];
          if (C.periodic[d]) v = min_image(v, C.box[d]);
          dx[d] = v;
          r2 += v * v;
        }
        const double f0 = pair_force_lean<LAW>(r2, hs, a.sig[tt], eps, rcs, C.well_eps, C.well_sigma, C.force_shifted);
#pragma unroll
        for (int d = 0; d < D; ++d) P[d] = __fma_rn(f0, dx[d], P[d]);
      }
    }
  } else {  // uniform per block
    if (sub == 0) {
#pragma unroll
      for (int d = 0; d < D; ++d) W.x[el * D + d] = xi[d];
      W.hs[el] = hs;
    }
    const int cap = kF64Near >> (5 - lane_bits);  // survivors held per element
    const int nb0 = el * cap;
    const unsigned gmask = (L == 32 ? 0xffffffffu : (1u << L) - 1u) << (lane & ~(L - 1));
    const unsigned below = gmask & ((1u << lane) - 1u);
    int cnt = 0;  // the element's survivors so far (the same in all its lanes)
    // the survivors' pairs, the whole warp: flattened, a pair per lane, then the elements' sums
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
      for (int S = 0; S < total; S += kF64Seg) {
        const int E = min(total, S + kF64Seg);
        for (int f0i = S; f0i < E; f0i += 32) {  // uniform
          const int f = f0i + lane;
          const int o = f < E ? W.own[f] : 0;
          const int offo = __shfl_sync(0xffffffffu, off, o << lane_bits);
          if (f < E) {
            const int at = o * cap + (f - offo);
            const int tt = W.tt[at], code = W.code[at];
            double dx[D];
            double r2 = 0.0;
#pragma unroll
            for (int d = 0; d < D; ++d) {
              double xj = a.x_in[d * SS + tt];
              const int k = (code >> (2 * d)) & 3;  // the neighbour's image: 1 below, 2 above
              if (k) xj = __dadd_rn(xj, k == 1 ? -C.box[d] : C.box[d]);
              dx[d] = xj - W.x[o * D + d];
              r2 += dx[d] * dx[d];
            }
            const double f0 = pair_force_lean<LAW>(r2, W.hs[o], a.sig[tt], eps, rcs, C.well_eps, C.well_sigma,
                                                   C.force_shifted);
#pragma unroll
            for (int d = 0; d < D; ++d) W.res[(f - S) * D + d] = f0 * dx[d];
          }
        }
        __syncwarp();
        if (sub == 0) {
          for (int f = max(off, S); f < min(end, E); ++f)
#pragma unroll
            for (int d = 0; d < D; ++d) P[d] += W.res[(f - S) * D + d];
        }
        __syncwarp();
      }
      cnt = 0;
    };
    int bi[D];
    bin_decode<D>(C, live ? a.sbin[s] : 0, bi);
    const float4 me = live ? a.rec[s] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // FP32 rounds both coordinates, an image's shift and two sums, each by 2^-24 of a value within
    // max(box, |coordinate|) or so: 2^-21 of their sum bounds a separation's error along an axis
    float margin[D];
#pragma unroll
    for (int d = 0; d < D; ++d) margin[d] = 4.76837158e-07f * (static_cast<float>(C.box[d]) + fabsf(pk_c(me, d)));
    const float rcsf = C.rcs_f, xif = C.well_sigma_f;
    // the rows of bins (all axes but the last), and per row one range of the last axis where its three
    // bins are consecutive, each bin of its own at the ends of the axis. A row's range is loaded a row
    // ahead (of the piece inside, at the ends: the element's own bin and its neighbours inside).
    constexpr int NROW = D == 2 ? 3 : 9;
    const int last = bi[D - 1], nl = C.ns[D - 1];
    const bool wraps = __any_sync(0xffffffffu, live && (last == 0 || last == nl - 1));
    const int lo = max(last - 1, 0), hi = min(last + 1, nl - 1);
    struct Row {
      const int2 *rng;
      int st, en, code;
      bool ok;
    };
    auto load_row = [&](int row) {
      const int oo[2] = {(D == 2 ? row : row / 3) - 1, row % 3 - 1};
      Row r;
      r.ok = live && row < NROW;
      r.code = 0;
      int rowbin = 0;
#pragma unroll
      for (int d = 0; d < D - 1; ++d) {
        int v = bi[d] + oo[d];
        if (v < 0) {
          r.ok = r.ok && C.periodic[d];
          v += C.ns[d];
          r.code |= 1 << (2 * d);
        } else if (v >= C.ns[d]) {
          r.ok = r.ok && C.periodic[d];
          v -= C.ns[d];
          r.code |= 2 << (2 * d);
        }
        rowbin = rowbin * C.ns[d] + v;
      }
      r.rng = a.range + C.bin_base + rowbin * nl;
      r.st = r.en = 0;
      if (r.ok) {
        r.st = r.rng[lo].x;
        r.en = r.rng[hi].y;
      }
      return r;
    };
    Row next = load_row(0);
    for (int row = 0; row < NROW; ++row) {
      const Row r = next;
      next = load_row(row + 1);
      for (int piece = 0; piece < (wraps ? 2 : 1); ++piece) {
        // piece 0: the bins inside the axis; piece 1: the bin past its end, through the boundary
        int st = r.st, en = r.en, code = r.code;
        if (piece == 1) {
          st = en = 0;
          if (r.ok && C.periodic[D - 1] && (last == 0 || last == nl - 1)) {
            const int2 q = r.rng[last == 0 ? nl - 1 : 0];
            st = q.x;
            en = q.y;
            code |= (last == 0 ? 1 : 2) << (2 * (D - 1));
          }
        }
        float sh[D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const int k = (code >> (2 * d)) & 3;
          sh[d] = k == 0 ? 0.0f : (k == 1 ? -static_cast<float>(C.box[d]) : static_cast<float>(C.box[d]));
        }
        for (int tt0 = st; __any_sync(0xffffffffu, tt0 < en); tt0 += AHEAD * L) {
          float4 p[AHEAD];
          bool there[AHEAD];
#pragma unroll
          for (int u = 0; u < AHEAD; ++u) {
            const int tt = tt0 + u * L + sub;
            there[u] = tt < en && tt != s && tt != ps;
            p[u] = there[u] ? a.rec[tt] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          }
#pragma unroll
          for (int u = 0; u < AHEAD; ++u) {
            float r2f = 0.0f;
#pragma unroll
            for (int d = 0; d < D; ++d) {
              const float dx = fmaxf(fabsf((pk_c(p[u], d) + sh[d]) - pk_c(me, d)) - margin[d], 0.0f);
              r2f += dx * dx;
            }
            const bool near = there[u] && pair_maybe_reaches<LAW>(r2f, me.w, p[u].w, rcsf, xif);
            const unsigned m = __ballot_sync(0xffffffffu, near);
            if (near) {
              const int at = nb0 + cnt + __popc(m & below);
              W.tt[at] = tt0 + u * L + sub;
              W.code[at] = static_cast<unsigned char>(code);
            }
            cnt += __popc(m & gmask);
          }
          if (__any_sync(0xffffffffu, cnt + AHEAD * L > cap)) {
            __syncwarp();
            flush();
          }
        }
      }
    }
    __syncwarp();
    flush();
  }
  if (!live || sub != 0) return;
#pragma unroll
  for (int d = 0; d < D; ++d) F[d] = __fma_rn(pair_scale<LAW>(eps), P[d], F[d]);

  // ---- checks, integration, outputs
  bool finite = true;
#pragma unroll
  for (int d = 0; d < D; ++d) finite = finite && finite_bits(F[d]);
  if (!finite) atomicOr(&a.cnt[c].err, kErrNan);
  if (a.frc) {
#pragma unroll
    for (int d = 0; d < D; ++d) a.frc[d * SS + s] = F[d];
  }
  if (a.integrate) {
    const double temp = a.heun ? 0.5 * C.temp[j] : C.temp[j];  // (dt/2) / zeta is exact
    bool inside = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const double tnew = __dadd_rn(xi[d], __dmul_rn(temp, F[d]));
      double xn;
      if (C.periodic[d]) {
        xn = wrap_bits(tnew, C.box[d]);
      } else {
        xn = tnew;
        inside = inside && (xn >= 0.0 && xn < C.box[d]);
      }
      a.x_out[d * SS + s] = xn;
    }
    if (!inside) atomicOr(&a.cnt[c].err, kErrBox);
    if (a.vel) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const double v = F[d] * C.mu_eff[j];
        a.vel[d * SS + s] = a.heun == 2 ? 0.5 * ((a.vel_prev ? a.vel_prev : a.vel)[d * SS + s] + v) : v;
      }
    }
  }
}

// ---------------------------------------------------------------- mixed-precision pieces

// Intra-cell spring + motility, walls and passive noise of one element (FP32), in the
// reference's order. ui / bi: the element's packed coordinates and home bin.
template <int D>
__device__ __forceinline__ void mixed_own_forces(const ForceArgs &a, const ColonyConst &C, int s, int e,
                                                 const float *ui, const int *bi, float si, float *F) {
  const int g = e >> 1, j = e & 1;
  {
    const int ps = a.slot_of[e ^ 1];
    const float4 pp = a.pk[ps];
    int bp[D];
    bin_decode<D>(C, a.sbin[ps], bp);
    float rij[D];
    float r2 = 0.0f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      float v = pk_c(pp, d) - ui[d];
      if (C.single_bin) {
        if (C.periodic[d]) v -= rintf(v * C.inv_bwf[d]) * C.bwf[d];
      } else {
        int db = bp[d] - bi[d];
        if (C.periodic[d]) {
          if (db > (C.ns[d] >> 1)) db -= C.ns[d];
          if (db < -(C.ns[d] >> 1)) db += C.ns[d];
        }
        v += static_cast<float>(db) * C.bwf[d];
      }
      rij[d] = (j == 0) ? v : -v;  // r1 - r0
      r2 += rij[d] * rij[d];
    }
#pragma unroll
    for (int d = 0; d < D; ++d) F[d] = 0.0f;
    if (r2 > 0.0f && C.cell_sm && a.cst[g] == kCellDividing) {
      float spring, act[2];
      fene_bond_dividing<float>(r2, fmaxf(si, fabsf(pp.w)), C.fene_r2max_div_f, C.fene_kappa_f, C.fene_kappa_push_f,
                                C.fene_ratio_f, C.div_r2min_f, C.growth_k0_f, C.growth_k1_f, C.growth_k2_f, spring, act);
      const float coef = (j == 0) ? -(act[0] + spring) : act[1] + spring;
      float rnd[3] = {0.0f, 0.0f, 0.0f};
      if (C.act_noise && a.noise_mode == 2)
        bond_noise<D, float>(static_cast<float>(a.noise_act[g]), static_cast<float>(a.noise_act_t[g]), rij, sqrtf(r2), rnd);
#pragma unroll
      for (int d = 0; d < D; ++d) F[d] = coef * rij[d] + (j == 0 ? -rnd[d] : rnd[d]) * rij[d];
    } else if (r2 > 0.0f && C.intra_fene) {
      const float rinv = rsqrtf(r2);
      float spring, sc;
      fene_bond<float>(r2, r2 * rinv, fmaxf(si, fabsf(pp.w)), C.fene_r2max_f, C.fene_kappa_f, C.fene_kappa_push_f,
                       C.fene_ratio_f, C.fene_rss_f, C.cil, spring, sc);
      const float coef = (j == 0) ? -(C.motility_f[0] * sc + 2.0f * spring) : C.motility_f[1] * sc + 2.0f * spring;
      float rnd[3] = {0.0f, 0.0f, 0.0f};
      if (C.act_noise && a.noise_mode == 2)
        bond_noise<D, float>(static_cast<float>(a.noise_act[g]), static_cast<float>(a.noise_act_t[g]), rij, r2 * rinv, rnd);
#pragma unroll
      for (int d = 0; d < D; ++d) F[d] = coef * rij[d] + (j == 0 ? -rnd[d] : rnd[d]) * rij[d];
    } else if (r2 > 0.0f) {
      const float rinv = rsqrtf(r2);
      float rest = C.rest0_f;
      if (C.divide) {
        const int2 cy = a.cyc[s];
        const int span = cy.y - cy.x;
        float frac = span > 0 ? __fdividef(static_cast<float>(a.ts - cy.x), static_cast<float>(span)) : 1.0f;
        frac = fminf(1.0f, fmaxf(0.0f, frac));
        rest = C.rest0_f + (C.rest1_f - C.rest0_f) * frac;
      }
      const float sp = C.kappa_f * (r2 * rinv - rest);
      const float coef = ((j == 0) ? (sp - C.motility_f[0]) : (C.motility_f[1] - sp)) * rinv;
#pragma unroll
      for (int d = 0; d < D; ++d) F[d] = coef * rij[d];
    }
  }
  if (C.nwalls > 0) {
    const float z = static_cast<float>(bi[D - 1]) * C.bwf[D - 1] + ui[D - 1];
    const float rad = 0.5f * si;
    for (int w = 0; w < C.nwalls; ++w) {
      const float dir = static_cast<float>(C.wall_dir[w]);
      const float delta = rad - dir * (z - C.wall_pos_f[w]);
      if (delta > 0.0f) F[D - 1] += dir * C.wall_E_f * delta * (delta * rsqrtf(delta));
    }
  }
  if (a.noise_mode == 1) {
    // Box-Muller with the fast log / sincos
    uint32_t w[4];
    noise_words<D>(e - 2 * C.cell_base, C.noise_per_cell, noise_index(a.ts, a.heun), C.rng_stream, a.seed_lo, a.seed_hi, w);
    const float amp = C.zeta_f[j] * C.amp_f;
#pragma unroll
    for (int h = 0; h < (D + 1) / 2; ++h) {
      const float u1 = static_cast<float>((w[2 * h] >> 8) + 1u) * 5.9604644775390625e-08f;
      const float u2 = static_cast<float>(w[2 * h + 1] >> 8) * 5.9604644775390625e-08f;
      const float m = fmaxf(-2.0f * __logf(u1), 0.0f);
      const float rad = m * rsqrtf(fmaxf(m, 1e-30f));  // sqrt(m), 0 when u1 == 1
      float sn, cs;
      __sincosf(6.2831853071795865f * u2, &sn, &cs);
      F[2 * h] += amp * rad * cs;
      if (2 * h + 1 < D) F[2 * h + 1] += amp * rad * sn;
    }
  } else if (a.noise_mode == 2) {
    const size_t base = static_cast<size_t>(C.noise_per_cell ? g : e) * D;
#pragma unroll
    for (int d = 0; d < D; ++d) F[d] += C.zeta_f[j] * static_cast<float>(a.noise[base + d]);
  }
}

// Checks, outputs and the Euler-Maruyama update of one element: one FP64 add per axis, the
// float->double conversion and the periodic wrap in integer arithmetic. Writes the next
// packed record (w carried over) and returns the FP32 step in dx.
template <int D>
__device__ __forceinline__ void mixed_integrate(const ForceArgs &a, const ColonyConst &C, int c, int s, int j,
                                                const float *ui, float w, const float *F, float *dx) {
  bool finite = true;
#pragma unroll
  for (int d = 0; d < D; ++d) finite = finite && isfinite(F[d]);
  if (!finite) atomicOr(&a.cnt[c].err, kErrNan);
  if (a.frc) {
#pragma unroll
    for (int d = 0; d < D; ++d) a.frc[d * a.SS + s] = static_cast<double>(F[d]);
  }
  if (!a.integrate) return;
  const float temp = a.heun ? 0.5f * C.temp_f[j] : C.temp_f[j];
  bool inside = true;
  float4 pn = make_float4(0.0f, 0.0f, 0.0f, w);
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float dxf = temp * F[d];
    double xn = a.x_in[d * a.SS + s] + f2d_exact(dxf);
    const long long xb = __double_as_longlong(xn);
    const long long lb = __double_as_longlong(C.box[d]);
    const bool lo = xb < 0, hi = xb >= lb;
    if (C.periodic[d]) {
      // non-negative doubles order like their bit patterns: wrap tests without FP64
      // compares; a tiny negative x + L that rounds to L ends at 0 like fmod(x + L, L). The
      // wrap runs only in warps where some element crossed 0 or L.
      if (__any_sync(__activemask(), lo || hi)) {
        if (lo) xn = (xb & 0x7fffffffffffffffll) ? xn + C.box[d] : 0.0;
        if (__double_as_longlong(xn) >= lb) xn -= C.box[d];
      }
    } else {
      inside = inside && !lo && !hi;
    }
    a.x_out[d * a.SS + s] = xn;
    pk_set(pn, d, ui[d] + dxf);
    dx[d] = dxf;
  }
  a.pk_next[s] = pn;
  if (!inside) atomicOr(&a.cnt[c].err, kErrBox);
  if (a.vel) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const double v = static_cast<double>(F[d] * C.mu_f[j]);
      a.vel[d * a.SS + s] = a.heun == 2 ? 0.5 * ((a.vel_prev ? a.vel_prev : a.vel)[d * a.SS + s] + v) : v;
    }
  }
}

// Mixed-precision step without lists, one thread per binned element: its intra-cell, wall and noise
// force, then the pair forces over the rows of bins around it, summed in slot order, then the update.
// The three bins of a row along the last axis hold consecutive slots, so a row is one range of records
// (kMixedAhead in flight) that the warp's elements, neighbours in bin order, share in L1; which of the
// three bins a candidate is in follows from its slot. The law is branch-free and costs about what the
// record's load does, so candidates out of range are evaluated and masked, and the cell's own two
// elements are told by their slots. 0.4M elements of the 2D growth colony: 26 us; staging the bin
// ranges in shared memory and sharing out a block's candidates evenly (element ids loaded per
// candidate, partial sums by shared atomics) took 49.6 us.
constexpr int kMixedAhead = 4;

template <int D, int LAW>
__global__ void __launch_bounds__(kTile, 4) k_force_mixed(ForceArgs a_) {
  enter_step_kernel();
  ForceArgs a = a_;
  a.ts = *a_.ts_dev;
  const int t = blockIdx.x;
  if (t >= a.tiles_live[a.B]) return;  // uniform per block
  const int c = colony_of_tile(a.tiles_live, a.B, t);
  const ColonyConst &C = a.col[c];
  const int s = C.slot_base + (t - a.tiles_live[c]) * kTile + static_cast<int>(threadIdx.x);
  const int nlive = a.cnt[c].nlive;
  const int e = s < C.slot_base + nlive ? a.eid[s] : -1;
  const bool live = e >= 0;
  const int j = e & 1;
  collect_due(a, C, c, live && j == 0, s, e);
  if (!live) return;
  const float4 pi = a.pk[s];
  float ui[D], F[D];
#pragma unroll
  for (int d = 0; d < D; ++d) ui[d] = pk_c(pi, d);
  const float si = fabsf(pi.w);
  int bi[D];
  bin_decode<D>(C, a.sbin[s], bi);
  mixed_own_forces<D>(a, C, s, e, ui, bi, si, F);
  const float eps = C.eps_f, rcs = C.rcs_f;
  if (C.single_bin) {
    // one bin only (tiny boxes): every element, FP32 minimum image
    const int g = e >> 1;
    for (int tt = C.slot_base; tt < C.slot_base + nlive; ++tt) {
      const int ej = a.eid[tt];
      const float4 pj = a.pk[tt];
      float dx[D];
      float r2 = 0.0f;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        float v = pk_c(pj, d) - ui[d];
        if (C.periodic[d]) v -= rintf(v * C.inv_bwf[d]) * C.bwf[d];
        dx[d] = v;
        r2 += v * v;
      }
      const float f0 = pair_f0_fast<LAW>(r2, si, pj.w, eps, rcs, ej >= 0 && (ej >> 1) != g, C.well_eps_f, C.well_sigma_f, C.force_shifted);
#pragma unroll
      for (int d = 0; d < D; ++d) F[d] += f0 * dx[d];
    }
  } else {
    const int ps = a.slot_of[e ^ 1];
    float acc[D];
#pragma unroll
    for (int d = 0; d < D; ++d) acc[d] = 0.0f;
    constexpr int NROW = D == 2 ? 3 : 9;
    const int last = bi[D - 1], nl = C.ns[D - 1];
    const bool inner = last > 0 && last < nl - 1;
    const float bwl = C.bwf[D - 1];
    for (int row = 0; row < NROW; ++row) {
      const int oo[3] = {(D == 2 ? row : row / 3) - 1, (D == 2 ? 0 : row % 3) - 1, 0};
      int rowbin = 0;
      bool ok = true;
      float ofs[D];  // the row's bin origins relative to the element
#pragma unroll
      for (int d = 0; d < D - 1; ++d) {
        int v = bi[d] + oo[d];
        if (v < 0) {
          ok = ok && C.periodic[d];
          v += C.ns[d];
        } else if (v >= C.ns[d]) {
          ok = ok && C.periodic[d];
          v -= C.ns[d];
        }
        rowbin = rowbin * C.ns[d] + v;
        ofs[d] = static_cast<float>(oo[d]) * C.bwf[d] - ui[d];
      }
      ofs[D - 1] = -ui[D - 1];
      if (!ok) continue;
      const int2 *rng = a.range + C.bin_base + rowbin * nl;
      for (int piece = 0; piece < (inner ? 1 : 3); ++piece) {
        // [st, en) with the bins' bounds: below m0 the bin before the element's, from m1 on the one after
        int st, en, m0, m1;
        if (inner) {
          const int2 r0 = rng[last - 1], r1 = rng[last + 1];
          st = r0.x;
          m0 = r0.y;
          m1 = r1.x;
          en = r1.y;
        } else {
          int v = last + piece - 1;
          if (v < 0 || v >= nl) {
            if (!C.periodic[D - 1]) continue;
            v += v < 0 ? nl : -nl;
          }
          const int2 r = rng[v];
          st = r.x;
          en = r.y;
          m0 = piece == 0 ? en : st;
          m1 = piece == 2 ? st : en;
        }
        for (int t0 = st; t0 < en; t0 += kMixedAhead) {
          float4 pj[kMixedAhead];
#pragma unroll
          for (int u = 0; u < kMixedAhead; ++u) pj[u] = a.pk[min(t0 + u, en - 1)];
#pragma unroll
          for (int u = 0; u < kMixedAhead; ++u) {
            const int tt = t0 + u;
            const float ol = ofs[D - 1] + (tt < m0 ? -bwl : (tt >= m1 ? bwl : 0.0f));
            float dx[D];
            float r2 = 0.0f;
#pragma unroll
            for (int d = 0; d < D; ++d) {
              dx[d] = pk_c(pj[u], d) + (d == D - 1 ? ol : ofs[d]);
              r2 += dx[d] * dx[d];
            }
            const float f0 = pair_f0_fast<LAW>(r2, si, pj[u].w, eps, rcs, tt < en && tt != s && tt != ps, C.well_eps_f, C.well_sigma_f, C.force_shifted);
#pragma unroll
            for (int d = 0; d < D; ++d) acc[d] += f0 * dx[d];
          }
        }
      }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) F[d] += acc[d];
  }
  float dstep[D];
  mixed_integrate<D>(a, C, c, s, j, ui, pi.w, F, dstep);
}

// Asynchronous global -> shared copies (cp.async, sm_80 and later): issued early, waited for
// where the data is used, so their latency overlaps the work in between. Each thread waits
// for its own copies; a __syncwarp after the wait publishes them to the warp.
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Per-warp shared memory of the cell kernel, for segments of SEG flattened list entries:
//   records of the warp's 64 elements             64 x 16 B
//   FP64 positions of the 64 elements (staged)    64 x D x 8 B, axis-major
//   list entries of the segment                   SEG x 4 B
//   owner (element of the warp) of each entry     SEG x 1 B
//   pair force of each entry                      SEG x D x 4 B
// SEG is the largest multiple of 32 (at most 1024) with which MINB blocks of TILE threads fit
// in the 228 KB of shared memory of an SM, leaving 2 KB per block for the static variables
// and the per-block reservation.
template <int D, int MINB, int TILE>
__host__ __device__ constexpr int pair_seg() {
  return ((233472 / MINB - 2048) / (TILE / 32) - (64 * 16 + 64 * D * 8)) / (5 + 4 * D) / 32 * 32 > 1024
             ? 1024
             : ((233472 / MINB - 2048) / (TILE / 32) - (64 * 16 + 64 * D * 8)) / (5 + 4 * D) / 32 * 32;
}
template <int D, int SEG>
__host__ __device__ constexpr int pair_smem_warp() {
  return 64 * 16 + 64 * D * 8 + SEG * (4 + 1 + 4 * D);
}
template <int D, int SEG>
struct PairSmem {
  float4 *rec;
  double *x;
  unsigned *ent;
  unsigned char *own;
  float *c;
  __device__ __forceinline__ explicit PairSmem(unsigned char *w)
      : rec(reinterpret_cast<float4 *>(w)),
        x(reinterpret_cast<double *>(w + 64 * 16)),
        ent(reinterpret_cast<unsigned *>(w + 64 * 16 + 64 * D * 8)),
        own(w + 64 * 16 + 64 * D * 8 + SEG * 4),
        c(reinterpret_cast<float *>(w + 64 * 16 + 64 * D * 8 + SEG * 5)) {}
};

// Bin-origin offsets by list-entry code (2 bits per axis: bin offset + 1), per block:
// entry k holds ((k >> 2d) & 3) - 1 times the bin width on axis d (exact products).
template <int D>
constexpr int kOffStride = D == 2 ? 2 : 4;
template <int D>
constexpr int kOffCodes = D == 2 ? 16 : 64;

// The warp's range of flattened list entries (k_list_flatten): element 2 lane owns [st0, en0),
// element 2 lane + 1 owns [st1, en1) of the warp's T entries. T and the starts are those of the
// last list build; an element that became fresh or dead since has an empty range (its entries
// are still evaluated, and dropped).
struct PairRange {
  int st0, en0, st1, en1, T;
};

// One segment [S, E) of the warp's range: 16-byte copies of its list entries and their owners
// from the flattened lists. The warp's range starts 16 KB aligned and S is a multiple of 32, so
// every copy is aligned; the copies round E up to 4 entries and 16 owners, which stays inside
// the warp's 64 kListCap entries and inside the segment's shared arrays (SEG is a multiple of 32).
template <int D, int SEG>
__device__ __forceinline__ void pairs_segment_start(const ForceArgs &a, int sw0, const PairRange &R, int S,
                                                    const PairSmem<D, SEG> &sm) {
  const int lane = threadIdx.x & 31;
  const int E = min(R.T, S + SEG);
  const int *le = a.lflat + static_cast<size_t>(sw0) * kListCap + S;
  const unsigned char *lo = a.oflat + static_cast<size_t>(sw0) * kListCap + S;
  const int ne = (E - S + 3) >> 2, no = (E - S + 15) >> 4;
  for (int i = lane; i < ne; i += 32) cp_async16(sm.ent + 4 * i, le + 4 * i);
  for (int i = lane; i < no; i += 32) cp_async16(sm.own + 16 * i, lo + 16 * i);
}

// The start of the pair pass, right after the cell's own loads: the records of the warp's 64
// elements into shared memory, the warp's range, and the copies of the first segment. Every
// lane calls it; lanes without a live cell pass n = (0, 0). ls: the two elements' starts;
// Tw: the warp's entry count at the last build.
template <int D, int SEG>
__device__ __forceinline__ PairRange pairs_begin(const ForceArgs &a, int sw0, int2 nn, ushort2 ls, int Tw,
                                                 const float4 *pr, const PairSmem<D, SEG> &sm) {
  const int lane = threadIdx.x & 31;
  sm.rec[2 * lane] = pr[0];
  sm.rec[2 * lane + 1] = pr[1];
  PairRange R;
  R.T = min(Tw, 64 * kListCap);
  R.st0 = ls.x;
  R.en0 = ls.x + nn.x;
  R.st1 = ls.y;
  R.en1 = ls.y + nn.y;
  pairs_segment_start<D, SEG>(a, sw0, R, 0, sm);
  return R;
}

// The pair forces of a warp's 32 cells (64 elements), whole warp: the elements' Verlet-list
// entries are taken as one flattened range (element by element, each list in order), so every
// lane evaluates a real entry whatever the lengths of the lists; each lane then adds its two
// elements' pair forces in list order (the sums do not depend on scheduling). UNROLL chunks of
// 32 entries have their partner records in flight together.
template <int D, int LAW, int UNROLL, int SEG>
__device__ __forceinline__ void pairs_finish(const ForceArgs &a, const ColonyConst &C, int sw0, const PairRange &R,
                                             float (*F)[D], const PairSmem<D, SEG> &sm, const float *s_off) {
  const int lane = threadIdx.x & 31;
  const float eps = C.eps_f, rcs = C.rcs_f;
  for (int S = 0; S < R.T; S += SEG) {  // uniform
    const int E = min(R.T, S + SEG);
    if (S > 0) {
      __syncwarp();  // the last segment's sums are read
      pairs_segment_start<D, SEG>(a, sw0, R, S, sm);
    }
    cp_async_wait_all();
    __syncwarp();  // every lane's copies (entries, records, owners) are visible to the warp
    for (int base = S; base < E; base += 32 * UNROLL) {  // uniform
      unsigned ent[UNROLL];
      int own[UNROLL];
      float4 pj[UNROLL];
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const int f = base + 32 * u + lane;
        own[u] = f < E ? sm.own[f - S] : -1;
        ent[u] = f < E ? sm.ent[f - S] : 0u;
      }
#pragma unroll
      for (int u = 0; u < UNROLL; ++u)
        pj[u] = own[u] >= 0 ? a.pk[ent[u] & ((1u << kListSlotBits) - 1u)]
                            : make_float4(0.0f, 0.0f, 0.0f, -1.0f);
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        if (own[u] < 0) continue;
        const float4 me = sm.rec[own[u]];
        // the offset between the two home bins' origins, from the entry's bin offset code
        const float *ov = s_off + (ent[u] >> kListSlotBits) * kOffStride<D>;
        float dx[D];
        float r2 = 0.0f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          dx[d] = pk_c(pj[u], d) + (ov[d] - pk_c(me, d));
          r2 += dx[d] * dx[d];
        }
        const float f0 = pair_f0_fast<LAW>(r2, fabsf(me.w), pj[u].w, eps, rcs, pj[u].w > 0.0f, C.well_eps_f, C.well_sigma_f, C.force_shifted);
        float *cf = sm.c + (base + 32 * u + lane - S) * D;
#pragma unroll
        for (int d = 0; d < D; ++d) cf[d] = f0 * dx[d];
      }
    }
    __syncwarp();
    // each element adds its entries of the segment, in list order
    for (int f = max(R.st0, S); f < min(R.en0, E); ++f)
#pragma unroll
      for (int d = 0; d < D; ++d) F[0][d] += sm.c[(f - S) * D + d];
    for (int f = max(R.st1, S); f < min(R.en1, E); ++f)
#pragma unroll
      for (int d = 0; d < D; ++d) F[1][d] += sm.c[(f - S) * D + d];
  }
  cp_async_wait_all();  // a warp without list entries has waited for nothing yet
}

// Skin-mode step over cell-major slots, one thread per cell. Between slot re-sorts a cell's
// two elements sit in adjacent slots, back element first (s0 = slot_base + 2 p, s1 = s0 + 1):
// the re-sort ranks cells, division appends daughters as slot pairs, apoptosis leaves pairs of
// tombstones. So a thread reads both records, the cycle and the FP64 positions of its cell
// with coalesced loads, evaluates the intra-cell spring once and draws the noise of both
// elements from one Philox block (2D); the warp evaluates its 64 elements' Verlet-list
// entries as one flattened range (pairs_begin / pairs_finish). The list entries and the FP64
// positions are copied into shared memory asynchronously at the start, so they arrive while
// the spring, wall and noise terms are evaluated; in the pair pass only the partner records
// are gathered (UNROLL chunks of 32 entries in flight per warp). Per element: the spring, wall
// and noise terms are the expressions of the other force kernels, the pair terms are summed in
// list order, and pairs with fresh elements (created or moved by a division since the last
// list build, in no list) arrive through facc from k_fresh_pairs.
// One tile of TILE cells, the whole block.
template <int D, int LAW, int UNROLL, int MINB, int TILE>
__device__ __forceinline__ void force_tile(const ForceArgs &a, int t) {
  constexpr int SEG = pair_seg<D, MINB, TILE>();
  extern __shared__ __align__(16) unsigned char s_pairs[];
  __shared__ ColonyConst sC;
  __shared__ unsigned s_dmax, s_smax;  // float bits of non-negative values
  __shared__ float s_ssum;
  __shared__ float s_half2;
  __shared__ int s_nbuilt;
  __shared__ int s_warps_done;
  __shared__ __align__(16) float s_off[kOffCodes<D> * kOffStride<D>];
  const int tid = threadIdx.x;
  const int c = colony_of_tile(a.tiles, a.B, t);
  {
    const int *src = reinterpret_cast<const int *>(a.col + c);
    int *dst = reinterpret_cast<int *>(&sC);
    for (int i = tid; i < static_cast<int>(sizeof(ColonyConst) / sizeof(int)); i += TILE) dst[i] = __ldg(src + i);
    if (tid < kOffCodes<D>) {
#pragma unroll
      for (int d = 0; d < D; ++d)
        s_off[tid * kOffStride<D> + d] = static_cast<float>(((tid >> (2 * d)) & 3) - 1) * __ldg(&a.col[c].bwf[d]);
    }
    if (tid == 0) {
      s_dmax = 0u;
      s_smax = 0u;
      s_ssum = 0.0f;
      s_half2 = a.skin[c].half2;
      s_nbuilt = a.skin[c].nslot_built;
      s_warps_done = 0;
    }
  }
  __syncthreads();
  const ColonyConst &C = sC;
  const int ts = *a.ts_dev;
  const size_t SS = a.SS;
  const int s0 = C.slot_base + 2 * ((t - a.tiles[c]) * TILE + tid);
  // every load of the cell is issued at once, guarded by the colony's slot capacity only (the
  // memory is there; what lies past the used slots is not used), so none waits on another
  const bool incap = s0 < C.slot_base + C.slot_cap;
  int2 ee = make_int2(-1, -1), sb = make_int2(0, 0), nn = make_int2(0, 0), cy = make_int2(0, 0);
  float4 pr[2] = {make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f)};
  ushort2 ls = make_ushort2(0, 0);
  if (incap) {
    ee = *reinterpret_cast<const int2 *>(a.eid + s0);
    pr[0] = a.pk[s0];
    pr[1] = a.pk[s0 + 1];
    sb = *reinterpret_cast<const int2 *>(a.sbin + s0);
    nn = *reinterpret_cast<const int2 *>(a.ncnt + s0);
    ls = *reinterpret_cast<const ushort2 *>(a.lstart + s0);
    if (C.divide) cy = a.cyc[s0];
  }
  // the warp's entry count at the last build (warps past the slots of that build have none)
  const int sw0 = s0 - 2 * (tid & 31);
  const int Tw = sw0 < C.slot_base + s_nbuilt ? a.lwarp[sw0 >> 6] : 0;
  // fresh-pair contributions: one bit per slot; slot bases are 32-aligned and s0 is even, so
  // both bits of the cell sit in one word (16 cells per word)
  const unsigned tword = a.ftouch[s0 >> 5];
  const unsigned tbits = (tword >> (s0 & 31)) & 3u;
  const bool used = s0 < C.slot_base + a.cnt[c].nslot;
  const bool live = used && ee.x >= 0;
  if (!live) nn = make_int2(0, 0);
  if (a.collect_due && C.divide) {  // uniform
    // cells whose cycle ends at the coming events (step ts + 1) join the colony's due-cell
    // queue: one atomic per warp
    const bool due = live && cy.y == ts + 1;
    const unsigned dm = __ballot_sync(0xffffffffu, due);
    if (dm) {
      const int lane = tid & 31, leader = __ffs(dm) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(&a.cnt[c].ndue, __popc(dm));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (due) a.dueq[C.due_base + base + __popc(dm & ((1u << lane) - 1u))] = (ee.x >> 1) - C.cell_base;
    }
  }
  float d2 = 0.0f, st2[2] = {0.0f, 0.0f};
  // ---- the pair pass starts: the warp's records, its flattened list range, and asynchronous
  // copies of its list entries and of the cells' FP64 positions, which arrive while the
  // per-element terms below are evaluated
  PairSmem<D, SEG> sm(s_pairs + (tid >> 5) * pair_smem_warp<D, SEG>());
  const PairRange R = pairs_begin<D, SEG>(a, sw0, nn, ls, Tw, pr, sm);
  if (live) {
#pragma unroll
    for (int d = 0; d < D; ++d) cp_async16(sm.x + d * 64 + 2 * (tid & 31), a.x_in + d * SS + s0);
  }
  // ---- the per-element terms (live cells)
  float F[2][D], ui[2][D];
#pragma unroll
  for (int d = 0; d < D; ++d) F[0][d] = F[1][d] = 0.0f;
  if (live) {
    const int g = ee.x >> 1;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      ui[0][d] = pk_c(pr[0], d);
      ui[1][d] = pk_c(pr[1], d);
    }
    const float si[2] = {fabsf(pr[0].w), fabsf(pr[1].w)};
    int bi[2][D];
    bin_decode<D>(C, sb.x, bi[0]);
    bin_decode<D>(C, sb.y, bi[1]);
    // ---- intra-cell spring + motility (the back element's view r1 - r0; the front
    // element's is the same vector, as -(r0 - r1) is exact)
    {
      float rij[D];
      float r2 = 0.0f;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        float v = ui[1][d] - ui[0][d];
        if (C.single_bin) {
          if (C.periodic[d]) v -= rintf(v * C.inv_bwf[d]) * C.bwf[d];
        } else {
          int db = bi[1][d] - bi[0][d];
          if (C.periodic[d]) {
            if (db > (C.ns[d] >> 1)) db -= C.ns[d];
            if (db < -(C.ns[d] >> 1)) db += C.ns[d];
          }
          v += static_cast<float>(db) * C.bwf[d];
        }
        rij[d] = v;
        r2 += v * v;
      }
      if (r2 > 0.0f && C.intra_fene) {
        const float rinv = rsqrtf(r2);
        float spring, sc;
        fene_bond<float>(r2, r2 * rinv, fmaxf(si[0], si[1]), C.fene_r2max_f, C.fene_kappa_f, C.fene_kappa_push_f,
                         C.fene_ratio_f, C.fene_rss_f, C.cil, spring, sc);
        const float coef0 = -(C.motility_f[0] * sc + 2.0f * spring);
        const float coef1 = C.motility_f[1] * sc + 2.0f * spring;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          F[0][d] += coef0 * rij[d];
          F[1][d] += coef1 * rij[d];
        }
      } else if (r2 > 0.0f) {
        const float rinv = rsqrtf(r2);
        float rest = C.rest0_f;
        if (C.divide) {
          const int span = cy.y - cy.x;
          float frac = span > 0 ? __fdividef(static_cast<float>(ts - cy.x), static_cast<float>(span)) : 1.0f;
          frac = fminf(1.0f, fmaxf(0.0f, frac));
          rest = C.rest0_f + (C.rest1_f - C.rest0_f) * frac;
        }
        const float sp = C.kappa_f * (r2 * rinv - rest);
        const float coef0 = (sp - C.motility_f[0]) * rinv;
        const float coef1 = (C.motility_f[1] - sp) * rinv;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          F[0][d] += coef0 * rij[d];
          F[1][d] += coef1 * rij[d];
        }
      }
    }
    // ---- walls
    if (C.nwalls > 0) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float z = static_cast<float>(bi[j][D - 1]) * C.bwf[D - 1] + ui[j][D - 1];
        const float rad = 0.5f * si[j];
        for (int w = 0; w < C.nwalls; ++w) {
          const float dir = static_cast<float>(C.wall_dir[w]);
          const float delta = rad - dir * (z - C.wall_pos_f[w]);
          if (delta > 0.0f) F[j][D - 1] += dir * C.wall_E_f * delta * (delta * rsqrtf(delta));
        }
      }
    }
    // ---- passive noise
    if (a.noise_mode == 1) {
      uint32_t w[2][4];
      noise_words_cell<D>(g - C.cell_base, C.noise_per_cell, noise_index(ts, a.heun), C.rng_stream, a.seed_lo, a.seed_hi,
                              w[0], w[1]);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float amp = C.zeta_f[j] * C.amp_f;
#pragma unroll
        for (int h = 0; h < (D + 1) / 2; ++h) {
          const float u1 = static_cast<float>((w[j][2 * h] >> 8) + 1u) * 5.9604644775390625e-08f;
          const float u2 = static_cast<float>(w[j][2 * h + 1] >> 8) * 5.9604644775390625e-08f;
          const float m = fmaxf(-2.0f * __logf(u1), 0.0f);
          const float rad = m * rsqrtf(fmaxf(m, 1e-30f));  // sqrt(m), 0 when u1 == 1
          float sn, cs;
          __sincosf(6.2831853071795865f * u2, &sn, &cs);
          F[j][2 * h] += amp * rad * cs;
          if (2 * h + 1 < D) F[j][2 * h + 1] += amp * rad * sn;
        }
      }
    } else if (a.noise_mode == 2) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const size_t base = static_cast<size_t>(C.noise_per_cell ? g : 2 * g + j) * D;
#pragma unroll
        for (int d = 0; d < D; ++d) F[j][d] += C.zeta_f[j] * static_cast<float>(__ldg(a.noise + base + d));
      }
    }
  }
  // ---- pair forces from the Verlet lists: the whole warp
  pairs_finish<D, LAW, UNROLL, SEG>(a, C, sw0, R, F, sm, s_off);
  if (live) {
    double xin[2][D];
    float uref[2][D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      // this lane's own staged copies (complete: pairs_finish waited for them)
      const double2 xv = *reinterpret_cast<const double2 *>(sm.x + d * 64 + 2 * (tid & 31));
      xin[0][d] = xv.x;
      xin[1][d] = xv.y;
      if (tbits & 1u) F[0][d] += a.facc[d * SS + s0];
      if (tbits & 2u) F[1][d] += a.facc[d * SS + s0 + 1];
    }
    if (D == 2) {
      uref_unpack2(C.uq_inv, pr[0].z, uref[0]);
      uref_unpack2(C.uq_inv, pr[1].z, uref[1]);
    } else {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const float2 uv = *reinterpret_cast<const float2 *>(a.uref + d * SS + s0);
        uref[0][d] = uv.x;
        uref[1][d] = uv.y;
      }
    }
    // ---- checks, update (one FP64 add per axis, integer wrap tests), stores
    bool finite = true;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int d = 0; d < D; ++d) finite = finite && isfinite(F[j][d]);
    if (!finite) atomicOr(&a.cnt[c].err, kErrNan);
    if (a.frc) {
#pragma unroll
      for (int d = 0; d < D; ++d)
        *reinterpret_cast<double2 *>(a.frc + d * SS + s0) =
            make_double2(static_cast<double>(F[0][d]), static_cast<double>(F[1][d]));
    }
    if (tbits) {
#pragma unroll
      for (int d = 0; d < D; ++d) *reinterpret_cast<float2 *>(a.facc + d * SS + s0) = make_float2(0.0f, 0.0f);
    }
    if (a.integrate) {
      bool inside = true;
      float4 pn[2];
      double xo[2][D];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float temp = a.heun ? 0.5f * C.temp_f[j] : C.temp_f[j];
        // 2D: z carries the packed list reference to the next record
        pn[j] = make_float4(0.0f, 0.0f, D == 2 ? pr[j].z : 0.0f, pr[j].w);
        float dj2 = 0.0f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const float dxf = temp * F[j][d];
          double xn = xin[j][d] + f2d_exact(dxf);
          const long long xb = __double_as_longlong(xn);
          const long long lb = __double_as_longlong(C.box[d]);
          const bool lo = xb < 0, hi = xb >= lb;  // negative (incl. -0) / at or past L
          if (C.periodic[d]) {
            // the wrap, taken by the few warps with an element that crossed 0 or L (an FP64
            // add predicated into every thread would cost the FP64 pipe on all of them)
            if (__any_sync(__activemask(), lo || hi)) {
              if (lo) xn = (xb & 0x7fffffffffffffffll) ? xn + C.box[d] : 0.0;
              if (__double_as_longlong(xn) >= lb) xn -= C.box[d];
            }
          } else {
            inside = inside && !lo && !hi;
          }
          xo[j][d] = xn;
          const float un = ui[j][d] + dxf;
          pk_set(pn[j], d, un);
          const float dr = un - uref[j][d];
          dj2 += dr * dr;
          st2[j] += dxf * dxf;
        }
        d2 = fmaxf(d2, dj2);
      }
#pragma unroll
      for (int d = 0; d < D; ++d)
        *reinterpret_cast<double2 *>(a.x_out + d * SS + s0) = make_double2(xo[0][d], xo[1][d]);
      a.pk_next[s0] = pn[0];
      a.pk_next[s0 + 1] = pn[1];
      if (!inside) atomicOr(&a.cnt[c].err, kErrBox);
      if (D == 2) {
        // guard with the fixed-point rounding allowed for: trips no later than |u - uref| > skin/2
        const float h = fmaxf(sqrtf(s_half2) - (C.uq_inv[0] + C.uq_inv[1]), 0.0f);
        if (d2 > h * h) atomicOr(&a.skin[c].need, 1);
      } else if (d2 > s_half2) {
        atomicOr(&a.skin[c].need, 1);
      }
      if (a.vel) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
          double v[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const double vj = static_cast<double>(F[j][d] * C.mu_f[j]);
            v[j] = a.heun == 2 ? 0.5 * ((a.vel_prev ? a.vel_prev : a.vel)[d * SS + s0 + j] + vj) : vj;
          }
          *reinterpret_cast<double2 *>(a.vel + d * SS + s0) = make_double2(v[0], v[1]);
        }
      }
    }
  } else if (used && a.integrate) {
    // tombstones: the next records must keep w < 0 too, or the lists of others would see the
    // stale records of two steps ago in the other buffer
    a.pk_next[s0] = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
    a.pk_next[s0 + 1] = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
  }
  __syncwarp();  // every lane has read its touch word
  if (tword != 0u && (tid & 15) == 0) a.ftouch[s0 >> 5] = 0u;
  if (a.integrate) {
    // displacement statistics: warp reductions and shared atomics; the last warp of the block
    // to finish adds the block's values to the colony (no block barrier: warps with short
    // lists do not wait for the others)
    const unsigned dmax = __reduce_max_sync(0xffffffffu, __float_as_uint(d2));
    const float stp0 = sqrtf(st2[0]), stp1 = sqrtf(st2[1]);
    const unsigned smax = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(stp0, stp1)));
    float ssum = stp0 + stp1;
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) ssum += __shfl_xor_sync(0xffffffffu, ssum, q);
    if ((tid & 31) == 0) {
      atomicMax(&s_dmax, dmax);
      atomicMax(&s_smax, smax);
      atomicAdd(&s_ssum, ssum);
      __threadfence_block();
      if (atomicAdd(&s_warps_done, 1) == TILE / 32 - 1) {
        __threadfence_block();
        StatPart &P = a.spart[c * kStatSlots + (t & (kStatSlots - 1))];
        atomicMax(&P.dmax, atomicOr(&s_dmax, 0u));
        if (a.sched) {
          atomicMax(&P.smax, atomicOr(&s_smax, 0u));
          atomicAdd(&P.ssum, atomicAdd(&s_ssum, 0.0f));
        }
      }
    }
  }
}

// LOOP: the blocks take the tiles (over slot pairs) in turn, the grid of few cells in a large capacity;
// otherwise a tile each, which is 0.6 to 1.3 % of a leg faster where most blocks have one.
template <int D, int LAW, int UNROLL, int MINB, int TILE, bool LOOP>
__global__ void __launch_bounds__(TILE, MINB) k_force_cells(const ForceArgs a) {
  enter_step_kernel();
  if (!LOOP) {
    if (static_cast<int>(blockIdx.x) < a.tiles[a.B]) force_tile<D, LAW, UNROLL, MINB, TILE>(a, blockIdx.x);
  } else {
    for (int t = blockIdx.x; t < a.tiles[a.B]; t += gridDim.x) {
      force_tile<D, LAW, UNROLL, MINB, TILE>(a, t);
      __syncthreads();
    }
  }
}

template <int D, int LAW, int UNROLL, int MINB, int TILE, bool LOOP>
void launch_cells_t(const ForceArgs &a, int grid, cudaStream_t s) {
  constexpr int bytes = (TILE / 32) * pair_smem_warp<D, pair_seg<D, MINB, TILE>()>();
  static bool attr_set = false;  // per instantiation; the attribute is per function
  if (!attr_set) {
    cudaFuncSetAttribute(k_force_cells<D, LAW, UNROLL, MINB, TILE, LOOP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         bytes);
    attr_set = true;
  }
  launch_step(true, grid, TILE, bytes, s, k_force_cells<D, LAW, UNROLL, MINB, TILE, LOOP>, a);
}

// MINB is the CTAs per SM at 256 threads; 128-thread blocks keep its threads per SM (hence the
// register budget per thread), 512-thread blocks take at most as many threads per SM
template <int D, int LAW, int UNROLL, int MINB>
void launch_cells(const ForceArgs &a, int grid, int block, cudaStream_t s) {
  if (block == 128 && a.list_loop)
    launch_cells_t<D, LAW, UNROLL, 2 * MINB, 128, true>(a, grid, s);
  else if (block == 128)
    launch_cells_t<D, LAW, UNROLL, 2 * MINB, 128, false>(a, grid, s);
  else if (block == 512)
    launch_cells_t<D, LAW, UNROLL, (MINB / 2 > 0 ? MINB / 2 : 1), 512, false>(a, grid, s);
  else
    launch_cells_t<D, LAW, UNROLL, MINB, 256, false>(a, grid, s);
}

template <int D, int LAW>
void launch_list_dl(const ForceArgs &a, int grid, int variant, int block, cudaStream_t s) {
  // cell-major slots, one thread per cell, the warp's list entries flattened; variants
  // (chunks of 32 entries in flight per warp, CTAs per SM at 256 threads): 0 (4, 3), 1 (2, 3),
  // 2 (1, 3), 3 (1, 4), 4 (4, 4) in 2D and (2, 4) in 3D, which the default takes for many cells
  // (set_lane_bits in cil_api.cu); block: 128, 256 or 512 threads (cells per block). The reference's
  // soft-core well is compiled in the first variant only.
  if (LAW == CIL_FORCE_SC || variant == 0) {
    launch_cells<D, LAW, 4, 3>(a, grid, block, s);
  } else if constexpr (LAW != CIL_FORCE_SC) {
    if (variant == 4) {
      launch_cells<D, LAW, D == 2 ? 4 : 2, 4>(a, grid, block, s);
    } else if (variant == 1) {
      launch_cells<D, LAW, 2, 3>(a, grid, block, s);
    } else if (variant == 2) {
      launch_cells<D, LAW, 1, 3>(a, grid, block, s);
    } else {
      launch_cells<D, LAW, 1, 4>(a, grid, block, s);
    }
  }
}

template <int D>
void launch_list_d(const ForceArgs &a, int law, int grid, int variant, int block, cudaStream_t s) {
  switch (law) {
    case CIL_FORCE_LJ_WCA:
      launch_list_dl<D, CIL_FORCE_LJ_WCA>(a, grid, variant, block, s);
      break;
    case CIL_FORCE_SOFTCORE:
      launch_list_dl<D, CIL_FORCE_SOFTCORE>(a, grid, variant, block, s);
      break;
    case CIL_FORCE_SC:
      launch_list_dl<D, CIL_FORCE_SC>(a, grid, variant, block, s);
      break;
    default:
      launch_list_dl<D, CIL_FORCE_HERTZ>(a, grid, variant, block, s);
      break;
  }
}

template <int D, int LAW>
void launch_dl(const ForceArgs &a, int prec, int tiles, int lane_bits, cudaStream_t s) {
  if (prec == CIL_PREC_FP64) {
    constexpr int bytes = kF64Block / 32 * static_cast<int>(sizeof(F64Warp<D>));
    static_assert(bytes <= 48 * 1024, "within the default shared memory of a block");
    // a lane alone with its element has 4 candidates in flight; lanes that share one have one each
    if (lane_bits == 0)
      launch_step(true, 2 * tiles, kF64Block, bytes, s, k_force_fp64<D, LAW, 4>, a, lane_bits);
    else
      launch_step(true, tiles * (2 << lane_bits), kF64Block, bytes, s, k_force_fp64<D, LAW, 1>, a, lane_bits);
  } else {
    launch_step(true, tiles, kTile, 0, s, k_force_mixed<D, LAW>, a);
  }
}

template <int D>
void launch_d(const ForceArgs &a, int law, int prec, int tiles, int lane_bits, cudaStream_t s) {
  switch (law) {
    case CIL_FORCE_LJ_WCA:
      launch_dl<D, CIL_FORCE_LJ_WCA>(a, prec, tiles, lane_bits, s);
      break;
    case CIL_FORCE_SOFTCORE:
      launch_dl<D, CIL_FORCE_SOFTCORE>(a, prec, tiles, lane_bits, s);
      break;
    case CIL_FORCE_SC:
      launch_dl<D, CIL_FORCE_SC>(a, prec, tiles, lane_bits, s);
      break;
    default:
      launch_dl<D, CIL_FORCE_HERTZ>(a, prec, tiles, lane_bits, s);
      break;
  }
}

}  // namespace

// This file is compiled twice: with CIL_FORCE_DIM=3 it holds the 3D kernels alone, otherwise
// the 2D kernels and the dispatch (two translation units that build in parallel).
#if defined(CIL_FORCE_DIM) && CIL_FORCE_DIM == 3
void launch_force_list_3d(const ForceArgs &a, int law, int grid, int variant, int block, cudaStream_t s) {
  launch_list_d<3>(a, law, grid, variant, block, s);
}

void launch_force_3d(const ForceArgs &a, int law, int prec, int tiles, int lane_bits, cudaStream_t s) {
  launch_d<3>(a, law, prec, tiles, lane_bits, s);
}
#else
void launch_force_list_3d(const ForceArgs &a, int law, int grid, int variant, int block, cudaStream_t s);
void launch_force_3d(const ForceArgs &a, int law, int prec, int tiles, int lane_bits, cudaStream_t s);

void launch_force_list(const ForceArgs &a, int dim, int law, int grid, int variant, int block, cudaStream_t s) {
  if (dim == 2)
    launch_list_d<2>(a, law, grid, variant, block, s);
  else
    launch_force_list_3d(a, law, grid, variant, block, s);
}

void launch_force(const ForceArgs &a, int dim, int law, int prec, int tiles, int lane_bits,
                  cudaStream_t s) {
  if (dim == 2)
    launch_d<2>(a, law, prec, tiles, lane_bits, s);
  else
    launch_force_3d(a, law, prec, tiles, lane_bits, s);
}
#endif

}  // namespace cil
