// tile_element.cuh -- the residual / rate / stage / limiter kernel with four
// lanes per element and its contractions on the FP64 tensor cores (tile.cuh).
//
// The mathematics is the one-thread kernel's (element.cuh; src/spatial/
// assembly.py:52-162, src/spatial/limiter.py:103-243): the same formulas, the
// sums of the contractions in another order.  A warp does everything for its
// eight elements, with no block barrier before the reductions at the end:
//
//   copies   CTAs are persistent (one wave: 148 x the resident blocks), so the
//            table fragments are staged in shared memory once per CTA.  While a
//            warp works on one tile, the state and geometry rows of its next one
//            travel to shared memory (cp.async, no registers), the connectivity
//            to registers, and the step's starting state, needed last, follows.
//   volume   tile by tile: interpolation, Euler flux in registers, projection.
//   faces    slot by slot (a rolled loop, one copy of the flux code): the own
//            and the neighbour's edge nodes are the k-step of two mma's that
//            leave the own trace in the even and the neighbour's in the odd
//            accumulator column of the lane that evaluates that face point; the
//            weighted flux is the k-step of the lift.  The next slot's scattered
//            loads are in flight while this slot's fluxes are evaluated, the
//            neighbours' nodes on their way to shared memory (cp.async): as
//            ordinary loads into registers they spilled (a residual of 10^6
//            cubic triangles 541 -> 569 us, the 72-member sweep's 51 steps
//            25.2 -> 28.2 ms).  Both
//            elements of an edge form both traces from the same edge nodes, in
//            the same order, with the same table, owner's trace left, owner's
//            normal: bit-identical fluxes, so the scheme stays conservative.
//   mass     triangles: folded into the tables, 1 / det into the fluxes.
//            Quadrilaterals: M = Phi diag(w det) Phi^T has a square Phi (as many
//            volume points as nodes), so M^-1 is two constant contractions (one
//            folded) around a division by w det -- the per-element inverse mass
//            matrix (8 NP^2 bytes, 2 KB of the 3.6 KB a cubic quadrilateral's
//            stage would move) is not read.
//   limiter  on the new state where it is, in registers: cell average, Lebesgue
//            screen, probe scan (the same interpolation tables), minima over the
//            four lanes by shuffle, the bisection replayed on t*.
//
// What bounds it: FP64 latency and issue at 12 warps per SM (168 registers; four
// blocks at 128 spill and are slower at p >= 2: 436 against 380 us at 480 000
// cubic triangles when that was tried, before the lean reciprocals).  An SM sub-partition's FP64 unit does 16 multiply-adds a cycle
// either way, but one mma keeps it busy 16 cycles from one instruction (measured
// 32.8 TFLOP/s from four warps per SM, where multiply-adds reach 24), so the
// contractions no longer need warps to hide their latency nor instruction issue.
//
// Measured on a B200, HLLC stage 2 with the limiter quiet / limiting about half of
// the elements, against the one-thread kernel (k_element) and the block-of-four-
// warps kernel it replaces where that was in use (us per launch):
//   480 000 triangles      p = 1  176 / 207 (t1 257 / 286)   p = 2  260 / 385 (423 / 503)
//                          p = 3  325 / 530 (784 / 1000)
//   240 000 quadrilaterals p = 1  100 / 116 (202 / 222)      p = 2  196 / 264 (443 / 499)
//                          p = 3  262 / 369 (1240 / 1408)
// and inside a march, per stage: 140 triangles p = 1 10.9 -> 6.8, 2 240 triangles
// p = 2 14.4 -> 8.7, 4 480 quadrilaterals p = 3 44.2 -> 14.0.  The residual of 10^6
// cubic triangles 776 -> 540 us.
#pragma once
#include "flux.cuh"
#include "slope.cuh"
#include "tile.cuh"

#ifndef NZB_MINB_TILE
#define NZB_MINB_TILE 3
#endif

namespace nzb {

// The cell-average weights of this lane's nodes.
template <int K, int P, bool AFF>
__device__ __forceinline__ void tile_mean_weights(const TileGeo<K, AFF>& geo, const nzb_mesh& m, int64_t e, bool act,
                                                  const double* fr, double (&mw)[Tile<K, P>::NS]) {
  using T = Tile<K, P>;
  if constexpr (K == 0) {
#pragma unroll
    for (int c = 0; c < T::NS; ++c) mw[c] = fr[(T::MW + c) * 32];
  } else {
    double dm[T::NT][2];
#pragma unroll
    for (int t = 0; t < T::NT; ++t) dm[t][0] = dm[t][1] = 0.0;
#pragma unroll
    for (int v = 0; v < T::VS; ++v) {
      double a, b, c, d;
      const double det = geo.at(fr[(T::XI + v) * 32], fr[(T::ETA + v) * 32], a, b, c, d);
#pragma unroll
      for (int t = 0; t < T::NT; ++t) mma(dm[t], det, fr[(T::MW + v * T::NT + t) * 32]);
    }
    const double ra = lean_rcp(act ? __ldg(m.area + e) : 1.0);
#pragma unroll
    for (int c = 0; c < T::NS; ++c) mw[c] = dm[c >> 1][c & 1] * ra;
  }
}

// The element's average of the nodes u, on each of its four lanes: this lane's share, then the lanes'
// sum as one product with a matrix of ones.
template <int NS>
__device__ __forceinline__ void tile_mean(const double (&mw)[NS], const double (&u)[NS][4], double (&ub)[4]) {
  __syncwarp();
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    double a = 0.0, d[2] = {0.0, 0.0};
#pragma unroll
    for (int c = 0; c < NS; ++c) a = fma(mw[c], u[c][s], a);
    mma(d, a, 1.0);
    ub[s] = d[0];
  }
}

// The limiter on an element's nodes in tile layout, in place (limit_element's
// formulas).  Every lane of the warp calls it; act marks the element's lanes.
template <int K, int P, bool AFF>
__device__ __forceinline__ void tile_limit(double (&u)[Tile<K, P>::NS][4], const TileGeo<K, AFF>& geo, const nzb_mesh& m,
                                           const nzb_physics& ph, int64_t e, bool act, const double* fr,
                                           int& scaled, int& repaired) {
  using S = Shape<K, P>;
  using T = Tile<K, P>;
  const int lane = threadIdx.x & 31, l = lane & 3;
  const double g = ph.gamma;
  double mw[T::NS];
  tile_mean_weights<K, P, AFF>(geo, m, e, act, fr, mw);
  double ub[4];
  auto cell_mean = [&]() { tile_mean(mw, u, ub); };
  cell_mean();
  // last-resort repair of a non-physical cell average.  The test itself (rho below its floor or the
  // energy below e_min) is evaluated where the product form, with a margin for rounding, cannot rule
  // it out, which saves the division for every physical element.
  const double e_floor = ph.p_floor / (g - 1.0);
  {
    const double rho_new = ub[0] < ph.rho_floor ? ph.rho_floor : ub[0];
    const double er = ub[3] * rho_new, need = e_floor * rho_new + 0.5 * (ub[1] * ub[1] + ub[2] * ub[2]);
    const bool maybe = act && !(ub[0] >= ph.rho_floor && er - need > 1e-13 * er);
    if (__any_sync(0xffffffffu, maybe)) {
      const double e_min = e_floor + 0.5 * (ub[1] * ub[1] + ub[2] * ub[2]) / rho_new;
      const double rhoE_new = ub[3] < e_min ? e_min : ub[3];
      const bool rep = maybe && (ub[0] < ph.rho_floor || ub[3] < e_min);
      if (__any_sync(0xffffffffu, rep)) {
        if (rep) {
          const double d0 = rho_new - ub[0], d3 = rhoE_new - ub[3];
#pragma unroll
          for (int c = 0; c < T::NS; ++c) {
            if (4 * c + l < S::NP) {
              u[c][0] += d0;
              u[c][3] += d3;
            }
          }
          repaired = 1;
        }
        cell_mean();
      }
    }
  }
  double eps_r = ph.lim_fraction * ub[0];
  eps_r = eps_r < 0.5 * ph.rho_floor ? 0.5 * ph.rho_floor : eps_r;

  // sufficient screen: bound every probe through the Lebesgue constant.  p_lo >= eps_p is tested
  // multiplied out by rho_lo and rho_bar (both positive), without a division; the largest
  // deviations are compared across the lanes as floats rounded up, which keeps the bound a bound.
  bool probe = act;
  {
    double dev[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      double a = 0.0;
#pragma unroll
      for (int c = 0; c < T::NS; ++c) {
        const double d = fabs(u[c][s] - ub[s]);
        a = (4 * c + l < S::NP && d > a) ? d : a;
      }
      float f = __double2float_ru(a);
      f = fmaxf(f, __shfl_xor_sync(0xffffffffu, f, 1));
      dev[s] = (double)fmaxf(f, __shfl_xor_sync(0xffffffffu, f, 2));
    }
    const double lam = ph.lebesgue;
    const double rho_lo = ub[0] - lam * dev[0];
    const double m2 = ub[1] * ub[1] + ub[2] * ub[2];
    const double d2 = lam * lam * (dev[1] * dev[1] + dev[2] * dev[2]);
    const double m_hi2 = m2 + d2 + 2.0 * sqrt(m2 * d2);
    const double p_rho = (g - 1.0) * ((ub[3] - lam * dev[3]) * rho_lo - 0.5 * m_hi2);      // p_lo rho_lo
    const double pb_rho = (g - 1.0) * (ub[3] * ub[0] - 0.5 * m2);                            // pbar rho_bar
    const double lowest = fmax(ph.lim_fraction * pb_rho, 0.5 * ph.p_floor * ub[0]);          // eps_p rho_bar
    if (rho_lo >= eps_r && ub[0] > 0.0 && p_rho * ub[0] >= lowest * rho_lo) probe = false;
  }
  if (!__any_sync(0xffffffffu, probe)) return;
  const double pbar = (g - 1.0) * (ub[3] - 0.5 * (ub[1] * ub[1] + ub[2] * ub[2]) / ub[0]);
  double eps_p = ph.lim_fraction * pbar;
  eps_p = eps_p < 0.5 * ph.p_floor ? 0.5 * ph.p_floor : eps_p;

  // values at the two probe points this lane holds of a tile (volume tiles, then face tiles)
  auto probe_tile = [&](int tile, double (&w)[4][2]) {
#pragma unroll
    for (int s = 0; s < 4; ++s) w[s][0] = w[s][1] = 0.0;
    __syncwarp();
#pragma unroll
    for (int c = 0; c < T::NS; ++c) {
      const double b = fr[(T::PHI + tile * T::NS + c) * 32];
#pragma unroll
      for (int s = 0; s < 4; ++s) mma(w[s], u[c][s], b);
    }
  };
  auto probe_valid = [&](int tile, int j) -> bool {
    if (tile < T::VT) return 4 * (2 * tile + j) + l < S::NQV;
    const int fs = 2 * (tile - T::VT) + j;
    return P == 1 ? 2 * fs + (l >> 1) < S::NF : (fs < T::FS && l < S::NQF);
  };
  const double e1 = eps_p / (g - 1.0);
  const double cq = ub[3] * ub[0] - 0.5 * (ub[1] * ub[1] + ub[2] * ub[2]) - e1 * ub[0];
  double rmin = 1e300, pmin = 1e300, tstar = 1e300;
#pragma unroll 1
  for (int tile = 0; tile < T::VT + T::FT; ++tile) {
    double w[4][2];
    probe_tile(tile, w);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (!probe || !probe_valid(tile, j)) continue;
      const double v[4] = {w[0][j], w[1][j], w[2][j], w[3][j]};
      rmin = v[0] < rmin ? v[0] : rmin;
      const double pp = pressure_at(v, g);
      pmin = pp < pmin ? pp : pmin;
      // the root of rho (p - eps_p) along the segment from the average, where it can bind (probe_scan)
      if (cq > 0.0 && !(pp < eps_p) && v[0] > 0.0) continue;
      const double d0 = v[0] - ub[0], d1 = v[1] - ub[1], d2 = v[2] - ub[2], d3 = v[3] - ub[3];
      const double a = d3 * d0 - 0.5 * (d1 * d1 + d2 * d2);
      const double b = ub[3] * d0 + ub[0] * d3 - (ub[1] * d1 + ub[2] * d2) - e1 * d0;
      if (a >= 0.0 && b >= 0.0) continue;
      const double disc = b * b - 4.0 * a * cq;
      if (disc < 0.0) continue;
      const double q = -0.5 * (b + copysign(sqrt(disc), b));
      const double r1 = a != 0.0 ? q / a : 1e300, r2 = q != 0.0 ? cq / q : 1e300;
      const double p1 = r1 > 0.0 ? r1 : 1e300, p2 = r2 > 0.0 ? r2 : 1e300;
      const double t = p1 < p2 ? p1 : p2;
      tstar = t < tstar ? t : tstar;
    }
  }
  __syncwarp();
  rmin = quad_min(rmin);
  pmin = quad_min(pmin);
  tstar = quad_min(tstar);
  const bool lim = probe && (rmin < eps_r || pmin < eps_p);
  if (!__any_sync(0xffffffffu, lim)) return;
  double theta = 1.0;
  if (lim && rmin < eps_r) {
    const double gap = ub[0] - rmin;
    theta = (ub[0] - eps_r) / (gap > 0.0 ? gap : 1.0);
    theta = theta < 0.0 ? 0.0 : (theta > 1.0 ? 1.0 : theta);
  }
  // the reference's bisection replayed on t* (limit_element); a decision within 1e-7 theta of t* is
  // re-taken with the pointwise minimum pressure.  it = -1 is the test at theta itself.
  bool bis = lim;
  double lo = 0.0, hi = theta;
#pragma unroll 1
  for (int it = -1; it < ph.lim_steps; ++it) {
    const double t = it < 0 ? theta : 0.5 * (lo + hi);
    bool adm = t < tstar;
    const bool near = bis && !(fabs(t - tstar) > 1e-7 * theta);
    if (__any_sync(0xffffffffu, near)) {
      double pm = 1e300;
#pragma unroll 1
      for (int tile = 0; tile < T::VT + T::FT; ++tile) {
        double w[4][2];
        probe_tile(tile, w);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          double v[4];
#pragma unroll
          for (int s = 0; s < 4; ++s) v[s] = ub[s] + t * (w[s][j] - ub[s]);
          const double pp = pressure_at(v, g);
          if (probe_valid(tile, j)) pm = pp < pm ? pp : pm;
        }
      }
      pm = quad_min(pm);
      if (near) adm = pm >= eps_p;
    }
    if (it < 0) {
      bis = lim && !adm;
      if (!__any_sync(0xffffffffu, bis)) break;
    } else if (adm) {
      lo = t;
    } else {
      hi = t;
    }
  }
  if (bis) theta = lo;
  if (lim) {
#pragma unroll
    for (int c = 0; c < T::NS; ++c)
#pragma unroll
      for (int s = 0; s < 4; ++s) u[c][s] = ub[s] + theta * (u[c][s] - ub[s]);
    scaled = 1;
  }
}

// What the Superbee pass (k_tile_superbee) reads of a stage's new state: the cell averages and the
// domain's (an instance's) largest magnitude of each component -- by atomics on the bit patterns of
// non-negative doubles, exact and order-free, into lim_scale zeroed before the launch.
template <int K, int P, bool AFF>
__device__ __forceinline__ void tile_slope_means(const double (&u)[Tile<K, P>::NS][4], const TileGeo<K, AFF>& geo,
                                                 const nzb_mesh& m, int64_t e, int inst, bool act, const double* fr) {
  const int lane = threadIdx.x & 31, l = lane & 3;
  double mw[Tile<K, P>::NS], ub[4];
  tile_mean_weights<K, P, AFF>(geo, m, e, act, fr, mw);
  tile_mean(mw, u, ub);
  const double mine = l == 0 ? ub[0] : l == 1 ? ub[1] : l == 2 ? ub[2] : ub[3];
  if (act) m.lim_means[l * m.n_elem + e] = mine;
  double v = act ? fabs(mine) : 0.0;
  if (!(v == v)) v = 0.0;  // a NaN is dropped
  const int inst0 = __shfl_sync(0xffffffffu, inst, 0);
  const bool uniform = __all_sync(0xffffffffu, inst == inst0 || !act);
  if (uniform) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, v, o);
      v = w > v ? w : v;
    }
  }
  if ((uniform ? lane < 4 : act) && v > 0.0) {
    const int i = uniform ? inst0 : inst;
    atomicMax(reinterpret_cast<unsigned long long*>(m.lim_scale + (i < 0 ? 0 : 4 * i) + l),
              (unsigned long long)__double_as_longlong(v));
  }
}

// The Superbee factor, the scaling and the positivity limiter (slope.cuh's k_superbee) in tile layout:
// the face averages of the own trace are one contraction, face l's in lane l.  In place allowed.
// Measured on a B200: 2 240 quadratic triangles 15.8 us (averages, maxima and factor, one thread
// per element) -> 10.9 us and the averages in the stage kernel.
template <int K, int P, bool AFF>
__global__ void __launch_bounds__(TILE_WARPS * 32) k_tile_superbee(const nzb_mesh m, const nzb_physics ph, const double* V,
                                                                   double* out, unsigned long long* counters, uint8_t* flags) {
  using S = Shape<K, P>;
  using T = Tile<K, P>;
  constexpr int ROWS = TileGeo<K, AFF>::ROWS;
  __shared__ double geom[TILE_WARPS][ROWS * TILE_E];
  const int lane = threadIdx.x & 31, l = lane & 3, warp = threadIdx.x >> 5;
  const double* fr = (K == 0 ? g_tile_tri : g_tile_quad) + tile_offset<K>(P) + lane;
  const int64_t E = m.n_elem, plane = S::NP * E;
  const int64_t e0 = ((int64_t)blockIdx.x * TILE_WARPS + warp) * TILE_E, e = e0 + (lane >> 2);
  int scaled = 0, repaired = 0;
  chain_release();
  copy_rows(geom[warp], m.geo, ROWS, E, e0, E);
  copy_commit();
  int inst = -1, nb = -1;
  double share = 0.0;
  if (e < E) {
    inst = m.elem_inst ? __ldg(m.elem_inst + e) : -1;
    if (l < S::NF) nb = __ldg(m.face_nbr + l * E + e);
    share = __ldg(m.elem_share + e);
  }
  chain_wait();
  const bool act = e < E && (inst < 0 || __ldg(m.inst_status + inst) == 0);
  if (__any_sync(0xffffffffu, act)) {
    const int64_t off = l * E + e;
    double u[T::NS][4], ub[4], d[4][2];
#pragma unroll
    for (int c = 0; c < T::NS; ++c)
#pragma unroll
      for (int s = 0; s < 4; ++s) u[c][s] = act && 4 * c + l < S::NP ? V[off + (4 * c * E + s * plane)] : 0.0;
    double jump[4] = {0.0, 0.0, 0.0, 0.0}, sc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      ub[s] = act ? m.lim_means[s * E + e] : 0.0;
      if (act && nb >= 0) {
        jump[s] = m.lim_means[s * E + nb] - ub[s];
        sc[s] = m.lim_scale[(inst < 0 ? 0 : 4 * inst) + s];
      }
      d[s][0] = d[s][1] = 0.0;
    }
    TileGeo<K, AFF> geo;
    copy_wait<0>();
    geo.template load<P>(geom[warp] + (lane >> 2));
#pragma unroll
    for (int c = 0; c < T::NS; ++c) {
      const double b8 = __ldg(fr + (T::FM + c) * 32);
#pragma unroll
      for (int s = 0; s < 4; ++s) mma(d[s], u[c][s], b8);
    }
    double theta = 1.0;
    if (act && nb >= 0) {  // a boundary face is not limited against
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const double x = d[s][0] - ub[s], a = jump[s];
        if (fabs(x) <= 1e-12 || fabs(x) <= ph.tvb_constant * share * sc[s]) continue;
        double tf = superbee2(a, x) / x;
        tf = tf < 0.0 ? 0.0 : (tf > 1.0 ? 1.0 : tf);
        theta = tf < theta ? tf : theta;
      }
    }
    __syncwarp();
    theta = quad_min(theta);
    bool changed = false;
#pragma unroll
    for (int c = 0; c < T::NS; ++c)
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const double v = ub[s] + theta * (u[c][s] - ub[s]);
        if (4 * c + l < S::NP) {
          changed |= v != u[c][s];
          u[c][s] = v;
        }
      }
    const unsigned any = __ballot_sync(0xffffffffu, changed && act);
    tile_limit<K, P, AFF>(u, geo, m, ph, e, act, fr, scaled, repaired);
    if ((any >> (lane & 28)) & 15u) scaled = 1;
    if (act) {
#pragma unroll
      for (int c = 0; c < T::NS; ++c)
        if (4 * c + l < S::NP) {
#pragma unroll
          for (int s = 0; s < 4; ++s) out[off + (4 * c * E + s * plane)] = u[c][s];
        }
      if (flags && l == 0) flags[e] = (uint8_t)(scaled | (repaired << 1));
    }
  }
  if (counters) {
    const int ns = __syncthreads_count(l == 0 && scaled);
    const int nr = __syncthreads_count(l == 0 && repaired);
    if (threadIdx.x == 0) {
      if (ns) atomicAdd(counters + 0, (unsigned long long)ns);
      if (nr) atomicAdd(counters + 1, (unsigned long long)nr);
    }
  }
}

// What a lane reads for its point of a face slot: the neighbour's edge node of its
// k-step -- to its own places oth[32 s + lane] in shared memory -- and the edge's
// normal, |dX/dsigma| and length.
template <int K, int P>
struct FacePoint {
  int code, nb, k;  // of the face this lane's point lies on; k < 0: no face
  double nx, ny, jac, len;

  // ccode, cnb, ck: the connectivity of face l of the element (one face per lane)
  __device__ __forceinline__ void load(const nzb_mesh& m, const double* V, double* oth, int ccode, int cnb, int ck, int fs,
                                       int lane) {
    using S = Shape<K, P>;
    constexpr unsigned long long EN = packed_edge_nodes<K, P>();
    const int l = lane & 3;
    const int f = P == 1 ? 2 * fs + (l >> 1) : fs, j = P == 1 ? (l & 1) : l;
    const int src = (lane & 28) | (f & 3);
    code = __shfl_sync(0xffffffffu, ccode, src);
    nb = __shfl_sync(0xffffffffu, cnb, src);
    k = __shfl_sync(0xffffffffu, ck, src);
    const int64_t E = m.n_elem, plane = S::NP * E;
    nx = ny = jac = len = 0.0;
    if (f >= S::NF) k = -1;
    const bool other = k >= 0 && j < S::NE && nb >= 0;
    const int nn = (int)(EN >> (16 * ((code >> 1) & 7) + 4 * j)) & 15;
    const double* p = V + (other ? nn * E + nb : 0);
#pragma unroll
    for (int s = 0; s < 4; ++s) copy_one(oth + 32 * s + lane, p + s * plane, other);
    if (k < 0) return;
    const double* eg = m.edge_geo + 4 * (int64_t)k;
    nx = __ldg(eg);
    ny = __ldg(eg + 1);
    jac = __ldg(eg + 2);
    len = __ldg(eg + 3);
  }
};

// Shared memory of one block, in doubles: the staged fragments, then per warp two
// buffers of (state rows, geometry rows) -- one being worked on, one in flight --
// and the rows of the step's starting state (stages).
template <int K, int P, bool AFF, bool LIM>
struct TileSmem {
  using S = Shape<K, P>;
  static constexpr int FRAGS = Tile<K, P>::STAGED * 32;
  static constexpr int STATE = S::NP * 4 * TILE_E;
  static constexpr int BUF = STATE + TileGeo<K, AFF>::ROWS * TILE_E;
  static constexpr int OTHER = 4 * 32;  // the neighbours' nodes of one face slot
  static constexpr int WARP = 2 * BUF + (LIM ? STATE : 0) + OTHER;
  static constexpr int BYTES = (FRAGS + TILE_WARPS * WARP) * 8;
  // resident blocks per SM: what the shared memory allows (1 KB of it reserved per block), at most
  // three (168 registers a thread)
  static constexpr int FIT = (227 * 1024) / (BYTES + 1024);
  static constexpr int MINB = FIT < NZB_MINB_TILE ? FIT : NZB_MINB_TILE;
};

template <int K, int P, bool AFF, bool LIM>
__global__ void __launch_bounds__(TILE_WARPS * 32, (TileSmem<K, P, AFF, LIM>::MINB))
    k_tile(const nzb_mesh m, const nzb_physics ph, const Work w) {
  using S = Shape<K, P>;
  using T = Tile<K, P>;
  using L = TileSmem<K, P, AFF, LIM>;
  extern __shared__ __align__(16) double smem[];
  const int lane = threadIdx.x & 31, l = lane & 3, warp = threadIdx.x >> 5;
  const int64_t E = m.n_elem, plane = S::NP * E;
  const double g = ph.gamma;
  const bool rate = w.op != OP_RESIDUAL;
  const int fo = rate ? 1 : 0;
  const int first = rate ? T::COMMON : 0;
  stage_tiles<K, P>(smem, first, T::STAGED);
  const double* fr = smem + lane - first * 32;  // fragment n of this lane is fr[32 n]
  double* const wbuf = smem + L::FRAGS + warp * L::WARP;
  const double* const start = wbuf + 2 * L::BUF + (lane >> 2);  // this element's column of the starting state
  double* const oth = wbuf + L::WARP - L::OTHER;
  const int64_t blocks = m.fwd_blocks ? m.n_fwd_blocks : (E + TILE_EB - 1) / TILE_EB;
  const bool stage = LIM && w.op == OP_STAGE;

  // One tile ahead: its state and geometry rows on their way to shared memory, and in registers its
  // instance and (face l in lane l) its connectivity.
  int64_t blk = 0;
  int inst = -1, ccode = 0, cnb = -1, ck = -1;
  auto fetch = [&](int64_t at, double* buf, bool first_tile = false) {
    blk = listed_block(m.fwd_blocks, E, TILE_EB, at);
    const int64_t e0 = blk * TILE_EB + warp * TILE_E, e = e0 + (lane >> 2);
    copy_rows(buf + L::STATE, m.geo, TileGeo<K, AFF>::ROWS, E, e0, E);
    inst = ccode = 0;
    cnb = ck = -1;
    if (e < E) {
      inst = m.elem_inst ? __ldg(m.elem_inst + e) : -1;
      if (l < S::NF) {
        ccode = __ldg(m.face_code + l * E + e);
        cnb = __ldg(m.face_nbr + l * E + e);
        ck = __ldg(m.face_edge + l * E + e);
      }
    }
    if (first_tile) chain_wait();  // the states, below, are the previous kernel's
    copy_rows(buf, w.V, S::NP * 4, E, e0, E);
    copy_commit();
  };
  fetch(blockIdx.x, wbuf, true);
  __syncthreads();  // the staged fragments

  int cur = 0;
  for (int64_t b = blockIdx.x; b < blocks; b += gridDim.x) {
    const int64_t myblk = blk, e0 = myblk * TILE_EB + warp * TILE_E, e = e0 + (lane >> 2);
    const int myinst = inst, mycode = ccode, mynb = cnb;
    const bool act = e < E && (myinst < 0 || __ldg(m.inst_status + myinst) == 0);
    const int myk = act ? ck : -1;
    double* const buf = wbuf + cur * L::BUF;
    const double* const col = buf + (lane >> 2);  // this element's column: row r at col[8 r]
    const int64_t off = l * E + e;                // node 4c + l, component s: off + 4cE + s plane
    cur ^= 1;
    const bool more = b + gridDim.x < blocks;
    if (!more) chain_release();
    double nrm = 0.0;
    int scaled = 0, repaired = 0;

    // a warp whose elements are all retired (or past the end) only joins the block's reductions
    if (!__any_sync(0xffffffffu, act)) {
      copy_wait<0>();
      if (more) fetch(b + gridDim.x, wbuf + cur * L::BUF);
    } else {
      double u[T::NS][4];
      TileGeo<K, AFF> geo;
      if (LIM && w.op == OP_LIMIT) {
        copy_wait<0>();
        geo.template load<P>(col + L::STATE);
#pragma unroll
        for (int c = 0; c < T::NS; ++c)
#pragma unroll
          for (int s = 0; s < 4; ++s) u[c][s] = 4 * c + l < S::NP ? col[(s * S::NP + 4 * c + l) * 8] : 0.0;
        if (more) fetch(b + gridDim.x, wbuf + cur * L::BUF);
        if (ph.limiter == 1) tile_limit<K, P, AFF>(u, geo, m, ph, e, act, fr, scaled, repaired);
      } else {
        // the step's starting state is read last: its rows travel meanwhile
        const bool later = stage && w.stage > 1;
        FacePoint<K, P> fp;
        fp.load(m, w.V, oth, mycode, mynb, myk, 0, lane);
        if (later) copy_rows(wbuf + 2 * L::BUF, w.U0, S::NP * 4, E, e0, E);
        copy_commit();
        double scale_t = 0.0;  // the local step, or what it is formed from
        if (stage && act) scale_t = later ? w.dt[e] : __ldg(m.area + e);
        double acc[T::NT][4][2];
#pragma unroll
        for (int t = 0; t < T::NT; ++t)
#pragma unroll
          for (int s = 0; s < 4; ++s) acc[t][s][0] = acc[t][s][1] = 0.0;
        double rem[T::REM ? T::REM : 1][4];
#pragma unroll
        for (int r = 0; r < T::REM; ++r)
#pragma unroll
          for (int s = 0; s < 4; ++s) rem[r][s] = 0.0;
        const double* const frl = fr - lane + l;  // entry (k = l, n = 2 r) of fragment n is frl[32 n + 8 r]

        // ---- volume
        copy_wait<1>();
        geo.template load<P>(col + L::STATE);
#pragma unroll 1
        for (int vt = 0; vt < T::VT; ++vt) {
          double d[4][2];
#pragma unroll
          for (int s = 0; s < 4; ++s) d[s][0] = d[s][1] = 0.0;
#pragma unroll
          for (int c = 0; c < T::NS; ++c) {
            const double b8 = fr[(T::PHI + vt * T::NS + c) * 32];
#pragma unroll
            for (int s = 0; s < 4; ++s)
              mma(d[s], 4 * c + 3 < S::NP || 4 * c + l < S::NP ? col[(s * S::NP + 4 * c + l) * 8] : 0.0, b8);
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int v = 2 * vt + j;
            if (T::VS % 2 == 1 && v >= T::VS) continue;
            const double uq[4] = {d[0][j], d[1][j], d[2][j], d[3][j]};
            const Prim pr = lean_primitives(uq, g);
            const double F[4] = {pr.rho * pr.vx, pr.rho * pr.vx * pr.vx + pr.p, pr.rho * pr.vx * pr.vy, pr.rho * pr.vx * pr.H};
            const double G[4] = {pr.rho * pr.vy, pr.rho * pr.vx * pr.vy, pr.rho * pr.vy * pr.vy + pr.p, pr.rho * pr.vy * pr.H};
            // triangles: (xi_x F + xi_y G) det, det only for the residual (the rate divides it out
            // again); quadrilaterals: det (xi_x, xi_y) = (y_eta, -x_eta)
            double a00, a01, a10, a11, vs;
            if constexpr (K == 0) {
              a00 = geo.g[0];
              a01 = geo.g[1];
              a10 = geo.g[2];
              a11 = geo.g[3];
              vs = rate ? 1.0 : -geo.g[4];
            } else {
              double x_xi, x_eta, y_xi, y_eta;
              geo.at(fr[(T::XI + v) * 32], fr[(T::ETA + v) * 32], x_xi, x_eta, y_xi, y_eta);
              a00 = y_eta;
              a01 = -x_eta;
              a10 = -y_xi;
              a11 = x_xi;
              vs = -1.0;
            }
            double fx[4], fe[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              fx[s] = (a00 * F[s] + a01 * G[s]) * vs;
              fe[s] = (a10 * F[s] + a11 * G[s]) * vs;
            }
#pragma unroll
            for (int t = 0; t < T::MTS; ++t) {
              const double bx = fr[T::vx(fo, v, t, 0) * 32], be = fr[T::vx(fo, v, t, 1) * 32];
#pragma unroll
              for (int s = 0; s < 4; ++s) mma(acc[t][s], fx[s], bx);
#pragma unroll
              for (int s = 0; s < 4; ++s) mma(acc[t][s], fe[s], be);
            }
            if constexpr (T::REM > 0) {
              remainder<K, P>(rem, frl + T::vx(fo, v, T::NT - 1, 0) * 32, fx);
              remainder<K, P>(rem, frl + T::vx(fo, v, T::NT - 1, 1) * 32, fe);
            }
          }
        }

        // ---- faces
        // triangles' rates: the face term carries -1/det (the rate is -M^-1 R with M = det M_ref)
        const double fsc = (K == 0 && rate) ? -lean_rcp(geo.g[4]) : 1.0;
        double wave = 0.0;
#pragma unroll 1
        for (int fs = 0; fs < T::FS; ++fs) {
          // this slot's neighbour nodes have landed (the next tile's rows, asked for after the second slot's
          // nodes, may still be on their way)
          if (fs == 1 && more)
            copy_wait<1>();
          else
            copy_wait<0>();
          constexpr unsigned long long EN = packed_edge_nodes<K, P>();
          // the own trace in column 0, the neighbour's in column 1 of an accumulator of its own: in one they
          // would meet the other's zero columns, and an infinity times zero is a NaN
          double d[4][2], dn[4][2];
#pragma unroll
          for (int s = 0; s < 4; ++s) d[s][0] = d[s][1] = dn[s][0] = dn[s][1] = 0.0;
          {
            const int f = P == 1 ? 2 * fs + (l >> 1) : fs, j = P == 1 ? (l & 1) : l;
            const bool own = f < S::NF && j < S::NE;
            const double* p = col + (own ? (int)(EN >> (16 * f + 4 * j)) & 15 : 0) * 8;
            const double bo = fr[T::TRO * 32], bn = fr[T::TRN * 32];
#pragma unroll
            for (int s = 0; s < 4; ++s) mma(d[s], own ? p[s * S::NP * 8] : 0.0, bo);
#pragma unroll
            for (int s = 0; s < 4; ++s) mma(dn[s], oth[32 * s + lane], bn);
          }
          const int code = fp.code, nb = fp.nb;
          const bool valid = fp.k >= 0 && (P == 1 || l < S::NQF);
          const double nx = fp.nx, ny = fp.ny, jac = fp.jac, len = fp.len;
          // the next slot's scattered loads go out before this slot's fluxes
          if (fs + 1 < T::FS) {
            fp.load(m, w.V, oth, mycode, mynb, myk, fs + 1, lane);
            copy_commit();
          }
          if (fs == 0 && more) fetch(b + gridDim.x, wbuf + cur * L::BUF);
          double F[4] = {0.0, 0.0, 0.0, 0.0}, sp = 0.0;
          if (valid) {
            const bool side = code & 1;
            if (nb >= 0) {
              double L4[4], R4[4];
#pragma unroll
              for (int s = 0; s < 4; ++s) {
                L4[s] = side ? dn[s][1] : d[s][0];
                R4[s] = side ? d[s][0] : dn[s][1];
              }
              sp = lean_interface_flux(L4, R4, nx, ny, ph, F);
            } else {
              const double tc[4] = {d[0][0], d[1][0], d[2][0], d[3][0]};
              const double p_back = (myinst >= 0 && m.inst_p_back) ? __ldg(m.inst_p_back + myinst) : ph.p_back;
              sp = boundary_flux(code >> 4, tc, nx, ny, ph, p_back, F);
            }
            const double scale = jac * fr[T::WF * 32], coef = side ? -fsc : fsc;
#pragma unroll
            for (int s = 0; s < 4; ++s) F[s] = (F[s] * scale) * coef;
          }
          __syncwarp();
#pragma unroll
          for (int t = 0; t < T::MTS; ++t) {
            const double b8 = fr[T::lf(fo, fs, t) * 32];
#pragma unroll
            for (int s = 0; s < 4; ++s) mma(acc[t][s], F[s], b8);
          }
          if constexpr (T::REM > 0) remainder<K, P>(rem, frl + T::lf(fo, fs, T::NT - 1) * 32, F);
          // wave = sum over faces of the largest signal speed times the length; a NaN speed does
          // not count, as in the one-thread kernel
          double sm = sp > 0.0 ? sp : 0.0;
          if constexpr (P == 1) {
            const double o = __shfl_xor_sync(0xffffffffu, sm, 1);
            sm = (o > sm ? o : sm) * len;
            const double other = __shfl_xor_sync(0xffffffffu, sm, 2);
            wave += sm + other;
          } else {
            wave += quad_max(sm) * len;
          }
        }
        if (w.wave && act && l == 0) w.wave[e] = wave;
        remainder_sum<K, P>(acc, rem, l);

        // ---- quadrilaterals' rates: acc holds Phi^-1 R; -Phi^-T (acc / (w det))
        if (K == 1 && rate) {
          double y[T::NS][4];
#pragma unroll
          for (int c = 0; c < T::NS; ++c) {
            double x0, x1, x2, x3;
            const double det = geo.at(fr[(T::XI + c) * 32], fr[(T::ETA + c) * 32], x0, x1, x2, x3);
            const double wd = fr[(T::WV + c) * 32] * det;
            const double r = act && 4 * c + l < S::NP ? -lean_rcp(wd) : 0.0;
#pragma unroll
            for (int s = 0; s < 4; ++s) y[c][s] = acc[c >> 1][s][c & 1] * r;
          }
#pragma unroll
          for (int t = 0; t < T::NT; ++t)
#pragma unroll
            for (int s = 0; s < 4; ++s) acc[t][s][0] = acc[t][s][1] = 0.0;
#pragma unroll
          for (int r = 0; r < T::REM; ++r)
#pragma unroll
            for (int s = 0; s < 4; ++s) rem[r][s] = 0.0;
          __syncwarp();
#pragma unroll
          for (int c = 0; c < T::NS; ++c) {
#pragma unroll
            for (int t = 0; t < T::MTS; ++t) {
              const double b8 = fr[(T::MT + c * T::NT + t) * 32];
#pragma unroll
              for (int s = 0; s < 4; ++s) mma(acc[t][s], y[c][s], b8);
            }
            if constexpr (T::REM > 0) remainder<K, P>(rem, frl + (T::MT + c * T::NT + T::NT - 1) * 32, y[c]);
          }
          remainder_sum<K, P>(acc, rem, l);
        }

        if (!stage) {
#pragma unroll
          for (int c = 0; c < T::NS; ++c)
#pragma unroll
            for (int s = 0; s < 4; ++s) u[c][s] = acc[c >> 1][s][c & 1];
        } else {
          double dt = scale_t;
          if (!later) {
            const double d = wave < FLOOR ? FLOOR : wave;
            dt = w.dt_factor * 2.0 * scale_t * lean_rcp(d);
            if (act && l == 0) w.dt[e] = dt;
          }
          // the starting state's rows have landed (the next tile's may still be on their way)
          if (more)
            copy_wait<1>();
          else
            copy_wait<0>();
#pragma unroll
          for (int c = 0; c < T::NS; ++c) {
            const bool node = act && 4 * c + l < S::NP;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              const double r = acc[c >> 1][s][c & 1], v = node ? col[(s * S::NP + 4 * c + l) * 8] : 0.0;
              double un;
              if (!later) {
                const double rw = r * ph.norm_w[s];
                if (node) nrm = fma(rw, rw, nrm);
                un = v + dt * r;
              } else {
                const double u0 = node ? start[(s * S::NP + 4 * c + l) * 8] : 0.0;
                un = w.a * u0 + w.b * (v + dt * r);
              }
              u[c][s] = node ? un : 0.0;
            }
          }
          if (!later) {
            nrm = quad_sum(nrm);
            if (w.elem_norm && act && l == 0) w.elem_norm[e] = nrm;
          }
          if (ph.limiter == 1) tile_limit<K, P, AFF>(u, geo, m, ph, e, act, fr, scaled, repaired);
          if (ph.limiter == 2) tile_slope_means<K, P, AFF>(u, geo, m, e, myinst, act, fr);
        }
      }
      if (act) {
#pragma unroll
        for (int c = 0; c < T::NS; ++c)
          if (4 * c + l < S::NP) {
#pragma unroll
            for (int s = 0; s < 4; ++s) w.out[off + (4 * c * E + s * plane)] = u[c][s];
          }
        if (LIM && (w.op == OP_STAGE || w.op == OP_LIMIT) && w.flags && l == 0)
          w.flags[e] = (uint8_t)(scaled | (repaired << 1));
      }
      __syncwarp();  // this tile's rows have been read: the buffers may be filled again
    }
    // block-level reductions (every thread of the block reaches these)
    if (stage && w.norm_partial && w.stage == 1) {
      block_sum_store<TILE_WARPS>(l == 0 ? nrm : 0.0, w.norm_partial + myblk);
      __syncthreads();  // the sum's slots are free again
    }
    if (LIM && w.counters) {
      const int ns = __syncthreads_count(l == 0 && scaled);
      const int nr = __syncthreads_count(l == 0 && repaired);
      if (threadIdx.x == 0) {
        if (ns) atomicAdd(w.counters + 0, (unsigned long long)ns);
        if (nr) atomicAdd(w.counters + 1, (unsigned long long)nr);
      }
    }
  }
}

}  // namespace nzb
