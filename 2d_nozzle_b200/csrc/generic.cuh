// generic.cuh -- the DG step for any order and curved (Q = 2) elements, from
// the reference's per-element operators.
//
// The specialised kernels (element.cuh, tile_element.cuh) hold every table of an
// element type in the constant bank and rebuild the metric terms of straight
// elements at each point; they are instantiated for straight elements of
// order 0..3.  For higher orders (up to 21 basis functions and beyond) and for
// curved elements, whose metric terms vary point by point, this path reads
// the operators the reference itself builds (src/spatial/operators.py:209-
// 342): per element the weak-form gradients at the volume points, unfolded
// (grad_x, grad_y) and with the inverse mass folded in (grad_x_m, grad_y_m),
// the folded face basis (face_basis_m), per edge point the normal and
// |dX/dsigma|, and the reference tables in global memory.  Arrays are in the
// reference's layout; the state is (E, NP, 4).  The passes follow the
// reference's compiled path (src/backends/_numba_kernels.py):
//
//   k_gen_edge     eight lanes per edge, one per point (in turn past eight): both
//                  traces, the Riemann or boundary flux, fw = flux |dX/dsigma| w,
//                  the edge's largest signal speed;
//   k_gen_element  a warp per element, everything else of a residual, a rate, a
//                  stage or the limiter alone: the volume states and fluxes (a
//                  lane per point, through shared memory), the volume term and
//                  the gathered face terms, the wave-speed sum, the local step,
//                  the stage update a U0 + b (V + dt F) and the weighted norm's
//                  element sum, and the positivity limiter (mean repair, Lebesgue
//                  screen, probe values held in shared memory, 12-step pressure
//                  bisection).
//
// What bounds a stage: the operators are the element's own (7.8 KB read for a
// fourth-order triangle, 15 KB at p = 5), so they are read once, each by one warp, as
// FP64 mma A fragments: rows are nodes, a k-step four consecutive points of a
// row (32 contiguous bytes a row), the B operand the four components of the point
// fluxes (half its columns are unused, which costs nothing where loads decide).
// With a thread per element instead, each lane walked its own operators: 2 240
// elements were 18 blocks, 210 us for the element pass alone.  Measured on a B200,
// a whole stage (all passes, positivity limiter): 2 240 fourth-order triangles
// 310 -> 23 us, 4 480 curved quadratic quadrilaterals 165 -> 28 us.
// The flux, boundary and primitive formulas are physics.cuh's, shared with
// the specialised kernels.
#pragma once
#include <cstdint>

#include "element.cuh"
#include "flux.cuh"
#include "physics.cuh"
#include "slope.cuh"
#include "tile.cuh"

namespace nzb {

constexpr int GEN_NP_MAX = 36;
constexpr int GEN_WARPS = 4;  // elements (warps) of a block

enum { GEN_RESIDUAL = 0, GEN_RATE = 1, GEN_STAGE = 2, GEN_LIMIT = 3 };

struct GenWork {
  int op, stage, limit;    // limit: the positivity limiter ends the stage
  bool chained;            // this launch follows a kernel of the same call (tile.cuh)
  const double* V;         // state the rate is evaluated at (the limiter's state)
  const double* U0;        // step start state (a != 0)
  double* out;
  double* wave;            // (E, nullable)
  const double* fw;        // the edge pass's fluxes and speeds
  const double* smax;
  double* dt;
  double* elem_norm;       // stage 1: the element's weighted squares (nullable)
  unsigned long long* counters;
  double dt_factor, a, b;
};

// Shared doubles of one warp: the state, and the point fluxes or the limiter's probe values.
struct GenSmem {
  int np, nqv, nface, nqf;
  __host__ __device__ int points() const { return nqv + nface * nqf; }
  __host__ __device__ int scratch() const { return 8 * nqv > 4 * points() ? 8 * nqv : 4 * points(); }
  __host__ __device__ int warp() const { return 4 * np + scratch(); }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  return v;
}
__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w < v ? w : v;
  }
  return v;
}

__global__ void __launch_bounds__(128) k_gen_edge(const nzb_gen_mesh m, const nzb_physics ph, const double* U, double* fw,
                                                  double* smax) {
  chain_release();
  const int64_t n_edge = m.n_int + m.n_bnd;
  const int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  double best = 0.0;
  chain_wait();
  if (k < n_edge) {
    const int np = m.np, nqf = m.nqf, nf = m.nface;
    const bool interior = k < m.n_int;
    const int64_t le = m.edge_elem[2 * k], re = m.edge_elem[2 * k + 1];
    const int lf = m.edge_face[2 * k], rf = m.edge_face[2 * k + 1];
    const int tag = interior ? 0 : m.edge_tag[k - m.n_int];
    const double* Ul = U + le * np * 4;
    const double* Ur = U + (interior ? re : le) * np * 4;
    for (int q = threadIdx.x & 7; q < nqf; q += 8) {
      const double* bl = m.phi_face + (int64_t)lf * np * nqf + q;
      const double* br = m.phi_face + (int64_t)(nf + rf) * np * nqf + q;
      double UL[4] = {0.0, 0.0, 0.0, 0.0}, UR[4] = {0.0, 0.0, 0.0, 0.0}, F[4];
#pragma unroll 4
      for (int i = 0; i < np; ++i) {
        const double b = __ldg(bl + i * nqf);
#pragma unroll
        for (int s = 0; s < 4; ++s) UL[s] = fma(b, Ul[i * 4 + s], UL[s]);
      }
      if (interior) {
#pragma unroll 4
        for (int i = 0; i < np; ++i) {
          const double b = __ldg(br + i * nqf);
#pragma unroll
          for (int s = 0; s < 4; ++s) UR[s] = fma(b, Ur[i * 4 + s], UR[s]);
        }
      }
      const double nx = m.edge_normal[(k * nqf + q) * 2], ny = m.edge_normal[(k * nqf + q) * 2 + 1];
      const double sp = interior ? lean_interface_flux(UL, UR, nx, ny, ph, F) : boundary_flux(tag, UL, nx, ny, ph, ph.p_back, F);
      best = sp > best ? sp : best;
      const double scale = m.edge_jac[k * nqf + q] * m.w_face[q];
#pragma unroll
      for (int s = 0; s < 4; ++s) fw[(k * nqf + q) * 4 + s] = F[s] * scale;
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    const double v = __shfl_xor_sync(0xffffffffu, best, o);
    best = v > best ? v : best;
  }
  if (k < n_edge && (threadIdx.x & 7) == 0) smax[k] = best;
}

// The positivity limiter of one element in place (src/backends/_numba_kernels.py:927-1093;
// src/spatial/limiter.py:103-243), by its warp: su the (NP, 4) state, sp room for the probe values.
// Every decision is the same on every lane.
__device__ __forceinline__ void gen_limit_warp(const nzb_gen_mesh& m, const nzb_physics& ph, int64_t e, double* su,
                                               double* sp, int& scaled, int& repaired) {
  const int lane = threadIdx.x & 31;
  const int np = m.np, nqv = m.nqv, nqf = m.nqf, nf = m.nface;
  const double g = ph.gamma, g1 = g - 1.0, lam = ph.lebesgue;
  double ub[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = lane; i < np; i += 32) {
    const double w = __ldg(m.mean_weights + e * np + i);
#pragma unroll
    for (int s = 0; s < 4; ++s) ub[s] = fma(w, su[i * 4 + s], ub[s]);
  }
#pragma unroll
  for (int s = 0; s < 4; ++s) ub[s] = warp_sum(ub[s]);
  const double rho_new = ub[0] > ph.rho_floor ? ub[0] : ph.rho_floor;
  const double e_min = ph.p_floor / g1 + 0.5 * (ub[1] * ub[1] + ub[2] * ub[2]) / rho_new;
  const double rhoE_new = ub[3] > e_min ? ub[3] : e_min;
  const double d0 = rho_new - ub[0], d3 = rhoE_new - ub[3];
  if (d0 != 0.0 || d3 != 0.0) {
    for (int i = lane; i < np; i += 32) {
      su[i * 4] += d0;
      su[i * 4 + 3] += d3;
    }
    ub[0] = rho_new;
    ub[3] = rhoE_new;
    repaired = 1;
    __syncwarp();
  }
  const double pbar = g1 * (ub[3] - 0.5 * (ub[1] * ub[1] + ub[2] * ub[2]) / ub[0]);
  double eps_r = ph.lim_fraction * ub[0], eps_p = ph.lim_fraction * pbar;
  eps_r = eps_r < 0.5 * ph.rho_floor ? 0.5 * ph.rho_floor : eps_r;
  eps_p = eps_p < 0.5 * ph.p_floor ? 0.5 * ph.p_floor : eps_p;
  double dv[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = lane; i < np; i += 32)
#pragma unroll
    for (int s = 0; s < 4; ++s) dv[s] = fmax(dv[s], fabs(su[i * 4 + s] - ub[s]));
#pragma unroll
  for (int s = 0; s < 4; ++s) dv[s] = warp_max(dv[s]);
  const double rho_lo = ub[0] - lam * dv[0];
  if (rho_lo >= eps_r) {
    const double m_hi = sqrt(ub[1] * ub[1] + ub[2] * ub[2]) + lam * sqrt(dv[1] * dv[1] + dv[2] * dv[2]);
    if (g1 * (ub[3] - lam * dv[3] - 0.5 * m_hi * m_hi / rho_lo) >= eps_p) return;
  }
  // the probe values: the volume points, then the element's own trace at each face point; a lane
  // writes and reads its own points only
  const int npt = nqv + nf * nqf;
  for (int pt = lane; pt < npt; pt += 32) {
    const double* basis = m.phi_vol + pt;
    int stride = nqv;
    if (pt >= nqv) {
      const int f = (pt - nqv) / nqf, q = (pt - nqv) - f * nqf;
      basis = m.phi_face + ((int64_t)(m.face_side[e * nf + f] * nf + f) * np) * nqf + q;
      stride = nqf;
    }
    double u[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = 0; i < np; ++i) {
      const double b = __ldg(basis + i * stride);
#pragma unroll
      for (int s = 0; s < 4; ++s) u[s] = fma(b, su[i * 4 + s], u[s]);
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) sp[pt * 4 + s] = u[s];
  }
  // the smallest density and pressure of ubar + theta (u - ubar) over the points
  auto minima = [&](double theta, double& rmin, double& pmin) {
    double rm = 1e300, pm = 1e300;
    for (int pt = lane; pt < npt; pt += 32) {
      double u[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) u[s] = ub[s] + theta * (sp[pt * 4 + s] - ub[s]);
      rm = u[0] < rm ? u[0] : rm;
      const double r = u[0] > 1e-300 ? u[0] : 1e-300;
      const double pp = g1 * (u[3] - 0.5 * (u[1] * u[1] + u[2] * u[2]) / r);
      pm = pp < pm ? pp : pm;
    }
    rmin = warp_min(rm);
    pmin = warp_min(pm);
  };
  double rmin, pmin;
  minima(1.0, rmin, pmin);
  if (!(rmin < eps_r) && !(pmin < eps_p)) return;
  double theta = 1.0;
  if (rmin < eps_r) {
    const double gap = ub[0] - rmin;
    theta = gap <= 0.0 ? 0.0 : (ub[0] - eps_r) / gap;
    theta = theta < 0.0 ? 0.0 : (theta > 1.0 ? 1.0 : theta);
  }
  minima(theta, rmin, pmin);
  if (pmin < eps_p) {
    double lo = 0.0, hi = theta;
    for (int it = 0; it < ph.lim_steps; ++it) {
      const double mid = 0.5 * (lo + hi);
      minima(mid, rmin, pmin);
      if (pmin >= eps_p)
        lo = mid;
      else
        hi = mid;
    }
    theta = lo;
  }
  for (int i = lane; i < np; i += 32)
#pragma unroll
    for (int s = 0; s < 4; ++s) su[i * 4 + s] = ub[s] + theta * (su[i * 4 + s] - ub[s]);
  scaled = 1;
}

__device__ __forceinline__ void gen_count(unsigned long long* counters, int scaled, int repaired) {
  if (counters) {
    const bool first = (threadIdx.x & 31) == 0;
    const int ns = __syncthreads_count(first && scaled), nr = __syncthreads_count(first && repaired);
    if (threadIdx.x == 0) {
      if (ns) atomicAdd(counters + 0, (unsigned long long)ns);
      if (nr) atomicAdd(counters + 1, (unsigned long long)nr);
    }
  }
}

// MT: tiles of eight nodes.
template <int MT>
__global__ void __launch_bounds__(GEN_WARPS * 32) k_gen_element(const nzb_gen_mesh m, const nzb_physics ph, const GenWork w) {
  extern __shared__ double smem[];
  const int lane = threadIdx.x & 31, l = lane & 3, n = lane >> 2;
  const int np = m.np, nqv = m.nqv, nqf = m.nqf, nf = m.nface;
  const GenSmem L{np, nqv, nf, nqf};
  double* const su = smem + (threadIdx.x >> 5) * L.warp();
  double* const sp = su + 4 * np;
  const int64_t e = (int64_t)blockIdx.x * GEN_WARPS + (threadIdx.x >> 5);
  int scaled = 0, repaired = 0;
  chain_release();
  chain_wait();
  if (e < m.n_elem) {
    const int64_t base = e * np * 4;
    for (int k = lane; k < np * 4; k += 32) su[k] = w.V[base + k];
    __syncwarp();
    if (w.op != GEN_LIMIT) {
      const bool unfolded = w.op == GEN_RESIDUAL;
      const double g = ph.gamma;
      // face f's edge, sign and side in lane f
      int64_t ke = 0;
      double sg = 0.0, speed = 0.0;
      int sd = 0;
      if (lane < nf) {
        ke = m.face_edge[e * nf + lane];
        sg = m.face_sign[e * nf + lane];
        sd = m.face_side[e * nf + lane];
        speed = w.smax[ke] * m.edge_length[ke];
      }
      // ---- volume states and fluxes, a lane per point
      for (int q = lane; q < nqv; q += 32) {
        double u[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
        for (int i = 0; i < np; ++i) {
          const double b = __ldg(m.phi_vol + i * nqv + q);
#pragma unroll
          for (int s = 0; s < 4; ++s) u[s] = fma(b, su[i * 4 + s], u[s]);
        }
        const Prim pr = lean_primitives(u, g);
        double* F = sp + q * 8;
        F[0] = pr.rho * pr.vx;
        F[1] = pr.rho * pr.vx * pr.vx + pr.p;
        F[2] = pr.rho * pr.vx * pr.vy;
        F[3] = pr.rho * pr.vx * pr.H;
        F[4] = pr.rho * pr.vy;
        F[5] = pr.rho * pr.vx * pr.vy;
        F[6] = pr.rho * pr.vy * pr.vy + pr.p;
        F[7] = pr.rho * pr.vy * pr.H;
      }
      __syncwarp();
      // ---- acc[i][s] = sum_q (gx F + gy G) - sum_fq basis sign fw: A rows are nodes 8 mt + lane / 4,
      // a k-step four points, B columns the components (4..7 zero)
      double acc[MT][2];
#pragma unroll
      for (int t = 0; t < MT; ++t) acc[t][0] = acc[t][1] = 0.0;
      const double* gx = (unfolded ? m.grad_x : m.grad_x_m) + e * np * nqv;
      const double* gy = (unfolded ? m.grad_y : m.grad_y_m) + e * np * nqv;
#pragma unroll 2
      for (int q0 = 0; q0 < nqv; q0 += 4) {
        const int q = q0 + l;
        const bool col = n < 4 && q < nqv;
        const double bF = col ? sp[q * 8 + n] : 0.0, bG = col ? sp[q * 8 + 4 + n] : 0.0;
        double ax[MT], ay[MT];
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          const int i = 8 * t + n;
          const bool in = i < np && q < nqv;
          ax[t] = in ? __ldg(gx + i * nqv + q) : 0.0;
          ay[t] = in ? __ldg(gy + i * nqv + q) : 0.0;
        }
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          mma(acc[t], ax[t], bF);
          mma(acc[t], ay[t], bG);
        }
      }
      const int nfq = nf * nqf;
#pragma unroll 2
      for (int k0 = 0; k0 < nfq; k0 += 4) {
        const int kk = k0 + l, f = kk < nfq ? kk / nqf : 0, q = kk - f * nqf;
        const int64_t k = __shfl_sync(0xffffffffu, ke, f);
        const double sign = __shfl_sync(0xffffffffu, sg, f);
        const int side = __shfl_sync(0xffffffffu, sd, f);
        const double bw = n < 4 && kk < nfq ? -sign * w.fw[(k * nqf + q) * 4 + n] : 0.0;
        const double* basis = unfolded ? m.phi_face + ((int64_t)(side * nf + f) * np) * nqf + q
                                       : m.face_basis_m + ((e * nf + f) * np) * nqf + q;
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          const int i = 8 * t + n;
          mma(acc[t], i < np && kk < nfq ? __ldg(basis + i * nqf) : 0.0, bw);
        }
      }
      double wave = 0.0;
      for (int f = 0; f < nf; ++f) wave += __shfl_sync(0xffffffffu, speed, f);
      if (w.wave && lane == 0) w.wave[e] = wave;
      // node 8 t + lane / 4, components 2 l and 2 l + 1 (l < 2)
      if (w.op != GEN_STAGE) {
        __syncwarp();
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          const int i = 8 * t + n;
          if (l < 2 && i < np) {
            su[i * 4 + 2 * l] = unfolded ? -acc[t][0] : acc[t][0];
            su[i * 4 + 2 * l + 1] = unfolded ? -acc[t][1] : acc[t][1];
          }
        }
      } else {
        double d;
        if (w.stage == 1) {
          d = w.dt_factor * 2.0 * m.elem_area[e] / (wave < FLOOR ? FLOOR : wave);
          if (lane == 0) w.dt[e] = d;
        } else {
          d = w.dt[e];
        }
        double sq = 0.0;
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          const int i = 8 * t + n;
          if (l < 2 && i < np) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int k = i * 4 + 2 * l + c;
              const double f = acc[t][c], v = su[k];
              const double r = f * ph.norm_w[2 * l + c];
              sq = fma(r, r, sq);
              su[k] = w.a == 0.0 ? v + d * f : w.a * w.U0[base + k] + w.b * (v + d * f);
            }
          }
        }
        if (w.elem_norm) {
          sq = warp_sum(sq);
          if (lane == 0) w.elem_norm[e] = sq;
        }
      }
      __syncwarp();
    }
    if (w.op == GEN_LIMIT || (w.op == GEN_STAGE && w.limit)) {
      gen_limit_warp(m, ph, e, su, sp, scaled, repaired);
      __syncwarp();
    }
    for (int k = lane; k < np * 4; k += 32) w.out[base + k] = su[k];
  }
  if (w.op == GEN_LIMIT || w.op == GEN_STAGE) gen_count(w.counters, scaled, repaired);
}

// The Superbee TVB slope limiter (src/spatial/limiter.py:246-429) on the generic path, in the
// specialised kernels' three passes (slope.cuh): the cell averages ubar (E, 4); their maxima
// max_e |ubar_s| (one block; exact in any order); then per element the factor theta = the
// minimum over interior faces and components of clip(superbee(a, d) / d, 0, 1), with d the
// face-averaged own trace minus ubar and a the jump of cell averages across the face, a face
// quiet where |d| <= 1e-12 or |d| <= tvb (A_e / A_domain) max|ubar_s|; U <- ubar + theta (U -
// ubar); then the positivity limiter, as apply_limiter runs them.  An element counts as scaled
// when either limiter changed it.
__global__ void __launch_bounds__(128) k_gen_cell_means(const nzb_gen_mesh m, const double* __restrict__ U,
                                                        double* __restrict__ means) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.n_elem) return;
  const int np = m.np;
  double ub[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = 0; i < np; ++i) {
    const double w = m.mean_weights[e * np + i];
#pragma unroll
    for (int s = 0; s < 4; ++s) ub[s] = fma(w, U[(e * np + i) * 4 + s], ub[s]);
  }
#pragma unroll
  for (int s = 0; s < 4; ++s) means[e * 4 + s] = ub[s];
}

__global__ void __launch_bounds__(1024) k_gen_lim_scale(const double* __restrict__ means, int64_t E,
                                                        double* __restrict__ scale) {
  __shared__ double red[4][32];
  double mx[4] = {0.0, 0.0, 0.0, 0.0};
  for (int64_t e = threadIdx.x; e < E; e += blockDim.x)
#pragma unroll
    for (int s = 0; s < 4; ++s) mx[s] = fmax(mx[s], fabs(means[e * 4 + s]));
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    double v = mx[s];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) red[s][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double v = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) v = fmax(v, red[threadIdx.x][k]);
    scale[threadIdx.x] = v;
  }
}

__global__ void __launch_bounds__(GEN_WARPS * 32) k_gen_superbee(const nzb_gen_mesh m, const nzb_physics ph,
                                                                 double* __restrict__ U, const double* __restrict__ means,
                                                                 const double* __restrict__ scale,
                                                                 const double* __restrict__ share,
                                                                 unsigned long long* counters) {
  extern __shared__ double smem[];
  const int lane = threadIdx.x & 31;
  const int np = m.np, nf = m.nface, nqf = m.nqf;
  const GenSmem L{np, m.nqv, nf, nqf};
  double* const su = smem + (threadIdx.x >> 5) * L.warp();
  double* const sp = su + 4 * np;
  const int64_t e = (int64_t)blockIdx.x * GEN_WARPS + (threadIdx.x >> 5);
  int scaled = 0, repaired = 0;
  if (e < m.n_elem) {
    for (int k = lane; k < np * 4; k += 32) su[k] = U[e * np * 4 + k];
    __syncwarp();
    // the own traces at the face points, a lane per point
    for (int pt = lane; pt < nf * nqf; pt += 32) {
      const int f = pt / nqf, q = pt - f * nqf;
      const double* pf = m.phi_face + (int64_t)(m.face_side[e * nf + f] * nf + f) * np * nqf + q;
      double tr[4] = {0.0, 0.0, 0.0, 0.0};
      for (int i = 0; i < np; ++i) {
        const double c = __ldg(pf + i * nqf);
#pragma unroll
        for (int s = 0; s < 4; ++s) tr[s] = fma(c, su[i * 4 + s], tr[s]);
      }
#pragma unroll
      for (int s = 0; s < 4; ++s) sp[pt * 4 + s] = tr[s];
    }
    __syncwarp();
    // a lane per face and component
    double theta = 1.0;
    const int f = lane >> 2, s = lane & 3;
    if (f < nf) {
      const int64_t k = m.face_edge[e * nf + f];
      if (k < m.n_int) {  // a boundary face is not limited against
        const int64_t a0 = m.edge_elem[2 * k], a1 = m.edge_elem[2 * k + 1];
        const int64_t nb = a0 == e ? a1 : a0;
        double wsum = 0.0, tm = 0.0;
        for (int q = 0; q < nqf; ++q) {
          wsum += m.w_face[q];
          tm = fma(m.w_face[q], sp[(f * nqf + q) * 4 + s], tm);
        }
        const double ub = means[e * 4 + s];
        const double d = tm / wsum - ub;
        const double a = means[nb * 4 + s] - ub;
        const bool quiet = fabs(d) <= 1e-12 || fabs(d) <= ph.tvb_constant * share[e] * scale[s];
        if (!quiet) {
          double tf = superbee2(a, d) / d;
          tf = tf < 0.0 ? 0.0 : (tf > 1.0 ? 1.0 : tf);
          theta = tf < theta ? tf : theta;
        }
      }
    }
    theta = warp_min(theta);
    bool changed = false;
    for (int k = lane; k < np * 4; k += 32) {
      const double ub = means[e * 4 + (k & 3)];
      const double v = ub + theta * (su[k] - ub);
      changed |= v != su[k];
      su[k] = v;
    }
    changed = __any_sync(0xffffffffu, changed);
    __syncwarp();
    gen_limit_warp(m, ph, e, su, sp, scaled, repaired);
    __syncwarp();
    for (int k = lane; k < np * 4; k += 32) U[e * np * 4 + k] = su[k];
    scaled |= changed ? 1 : 0;
  }
  gen_count(counters, scaled, repaired);
}

// One stage's update per element: stage 1 forms the local step dt = c 2 A / max(wave, FLOOR) and the
// weighted squares of its rate (per-block partial sums); out = a U0 + b (V + dt F) (a = 0: V + dt F).
__global__ void __launch_bounds__(128) k_gen_update(const nzb_gen_mesh m, const nzb_physics ph, int stage,
                                                    double dt_factor, double a, double b, const double* __restrict__ V,
                                                    const double* __restrict__ U0, const double* __restrict__ F,
                                                    const double* __restrict__ wave, double* __restrict__ dt,
                                                    double* __restrict__ out, double* __restrict__ partial) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double sq = 0.0;
  if (e < m.n_elem) {
    const int n = m.np * 4;
    double d;
    if (stage == 1) {
      const double w = wave[e] < FLOOR ? FLOOR : wave[e];
      d = dt_factor * 2.0 * m.elem_area[e] / w;
      dt[e] = d;
    } else {
      d = dt[e];
    }
    for (int k = 0; k < n; ++k) {
      const int64_t o = e * n + k;
      const double f = F[o];
      if (stage == 1) {
        const double r = f * ph.norm_w[k & 3];
        sq = fma(r, r, sq);
      }
      out[o] = a == 0.0 ? V[o] + d * f : a * U0[o] + b * (V[o] + d * f);
    }
  }
  if (stage == 1 && partial) block_sum_store<4>(sq, partial + blockIdx.x);
}

}  // namespace nzb
