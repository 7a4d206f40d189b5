// adjoint_tile.cuh -- the state VJP (adjoint.cuh) in tile layout (tile.cuh): a warp
// owns eight elements, four lanes each, and the interpolations, projections, lift
// and inverse mass are FP64 mma's.
//
//   k_tile_jac  the linearised fluxes of a march: per element and face point the
//               4 x 4 Jacobian of (sign w |dX/dsigma| Fhat) with respect to the own
//               trace, by dual numbers, one face point per lane;
//   k_tile_vjp  the product and its epilogues (defect, rate, RK4 stage).  With
//               those Jacobians (JAC) a face point costs sixteen multiply-adds;
//               without, it is differentiated in place.
//
// Why the Jacobians are formed once per run of steps: an adjoint march applies the
// transposed linearisation about one frozen state 4 x check_interval times a run,
// and differentiating a Riemann flux in four dual directions is over a thousand
// FP64 instructions a face point, most of a product.  Reading sixteen numbers
// instead costs 128 B a point -- 1.15 KB per quadratic triangle and product, with
// everything else about twice that -- so the product becomes a memory-bound one.
// They are recomputed at the start of every run (nzb_adjoint_run), for the elements
// that march in it, so nothing outlives the states it was computed from.
//
// Layout: [tile][slot][4u + s][element of the tile, point of the slot], so a lane's
// sixteen loads are sixteen coalesced lines of its warp; while a warp works on one
// tile the Jacobian lines of its next are prefetched to L2, and the rows of U and
// lambda travel to shared memory.
//
// Measured on a B200 (us per RK4 stage, in a march): 2 240 quadratic triangles
// 23.5 -> 5.9, 143 360 of them (AUSM+-up) 223 -> 90, where a run of steps
// also forms the Jacobians once (163 us; a dual-number product in place takes 217).
#pragma once
#include "adjoint.cuh"
#include "flux.cuh"
#include "tile.cuh"

namespace nzb {

// Face points of a slot that the Jacobian array holds per element.
template <int K, int P>
struct TileJac {
  using S = Shape<K, P>;
  using T = Tile<K, P>;
  static constexpr int LPE = P == 1 ? 4 : S::NQF;
  static constexpr int ROW = TILE_E * LPE;           // doubles of one line
  static constexpr int TILE = T::FS * 16 * ROW;      // doubles of one tile
  static __host__ __device__ int64_t doubles(int64_t E) { return ((E + TILE_EB - 1) / TILE_EB) * TILE_WARPS * (int64_t)TILE; }
};

// The connectivity of this lane's point of face slot fs, from lane l holding face l's,
// and the edge's normal and |dX/dsigma|.
template <int K, int P>
struct AdjFace {
  int f, code, nb, k, own, oth;  // own, oth: this lane's k-step nodes, or -1
  __device__ __forceinline__ void set(int ccode, int cnb, int ck, int fs, int lane) {
    using S = Shape<K, P>;
    constexpr unsigned long long EN = packed_edge_nodes<K, P>();
    const int l = lane & 3, j = P == 1 ? (l & 1) : l;
    f = P == 1 ? 2 * fs + (l >> 1) : fs;
    const int src = (lane & 28) | (f & 3);
    code = __shfl_sync(0xffffffffu, ccode, src);
    nb = __shfl_sync(0xffffffffu, cnb, src);
    k = __shfl_sync(0xffffffffu, ck, src);
    if (f >= S::NF) k = -1;
    const bool node = k >= 0 && j < S::NE;
    own = node ? (int)(EN >> (16 * f + 4 * j)) & 15 : -1;
    oth = node && nb >= 0 ? (int)(EN >> (16 * ((code >> 1) & 7) + 4 * j)) & 15 : -1;
  }
};

// Jt[u][s] = sign w |dX/dsigma| dFhat_s / dU_u at one face point, U the own trace.
__device__ __forceinline__ void face_jacobian(const double (&tc)[4], const double (&tn)[4], int code, int nb, double nx,
                                              double ny, double scale, const nzb_physics& ph, double p_back,
                                              Dual<4> (&F)[4], double& coef) {
  Dual<4> own[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) own[s] = Dual<4>::seed(tc[s], s);
  const bool side = code & 1;
  if (nb >= 0) {
    if (side)
      interface_flux(tn, own, nx, ny, ph, F);
    else
      interface_flux(own, tn, nx, ny, ph, F);
  } else {
    boundary_flux(code >> 4, own, nx, ny, ph, p_back, F);
  }
  coef = side ? -scale : scale;
}

template <int K, int P>
__global__ void __launch_bounds__(TILE_WARPS * 32, 2)
    k_tile_jac(const nzb_mesh m, const nzb_physics ph, const double* __restrict__ U, double* __restrict__ jac) {
  using S = Shape<K, P>;
  using T = Tile<K, P>;
  using J = TileJac<K, P>;
  const int lane = threadIdx.x & 31, l = lane & 3;
  const int64_t E = m.n_elem, plane = S::NP * E;
  const double* fr = (K == 0 ? g_tile_tri : g_tile_quad) + tile_offset<K>(P) + lane;
  chain_release();
  chain_wait();
  const int64_t blk = listed_block(m.vjp_blocks, E, TILE_EB);
  const int64_t tile = blk * TILE_WARPS + (threadIdx.x >> 5), e = tile * TILE_E + (lane >> 2);
  int inst = -1, ccode = 0, cnb = -1, ck = -1;
  if (e < E) {
    inst = m.elem_inst ? __ldg(m.elem_inst + e) : -1;
    if (l < S::NF && (inst < 0 || __ldg(m.inst_status + inst) == 0)) {
      ccode = __ldg(m.face_code + l * E + e);
      cnb = __ldg(m.face_nbr + l * E + e);
      ck = __ldg(m.face_edge + l * E + e);
    }
  }
  const bool act = e < E && (inst < 0 || __ldg(m.inst_status + inst) == 0);
  if (!__any_sync(0xffffffffu, act)) return;
  const double p_back = (inst >= 0 && m.inst_p_back) ? __ldg(m.inst_p_back + inst) : ph.p_back;
  const double bo = __ldg(fr + T::A_TRO * 32), bn = __ldg(fr + T::A_TRN * 32), wq = __ldg(fr + T::A_WF * 32);
#pragma unroll 1
  for (int fs = 0; fs < T::FS; ++fs) {
    AdjFace<K, P> fp;
    fp.set(ccode, cnb, ck, fs, lane);
    double d[4][2];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      d[s][0] = d[s][1] = 0.0;
      const double a = fp.own >= 0 ? __ldg(U + fp.own * E + e + s * plane) : 0.0;
      const double b = fp.oth >= 0 ? __ldg(U + fp.oth * E + fp.nb + s * plane) : 0.0;
      mma(d[s], a, bo);
      mma(d[s], b, bn);
    }
    if (fp.k >= 0 && (P == 1 || l < S::NQF)) {
      const double* eg = m.edge_geo + 4 * (int64_t)fp.k;
      const double tc[4] = {d[0][0], d[1][0], d[2][0], d[3][0]}, tn[4] = {d[0][1], d[1][1], d[2][1], d[3][1]};
      Dual<4> F[4];
      double coef;
      face_jacobian(tc, tn, fp.code, fp.nb, __ldg(eg), __ldg(eg + 1), __ldg(eg + 2) * wq, ph, p_back, F, coef);
      double* dst = jac + tile * J::TILE + fs * 16 * J::ROW + (lane >> 2) * J::LPE + l;
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int s = 0; s < 4; ++s) dst[(4 * u + s) * J::ROW] = coef * F[s].d[u];
    }
    __syncwarp();
  }
}

// The volume point's product through the floored flux (a density or pressure floor active): rare, kept
// out of line so that its dual numbers cost the common path no registers.
static __device__ __noinline__ void floored_flux_vjp(const double* uq, double g, const double* cF, const double* cG, double* b) {
  Dual<4> Uq[4], F[4], G[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) Uq[s] = Dual<4>::seed(uq[s], s);
  euler_flux(Uq, g, F, G);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    double acc = 0.0;
#pragma unroll
    for (int s = 0; s < 4; ++s) acc = fma(cF[s], F[s].d[u], fma(cG[s], G[s].d[u], acc));
    b[u] = acc;
  }
}

// euler_flux_vjp with one reciprocal of the density; b = 0 and false where a floor is active.
__device__ __forceinline__ bool lean_flux_vjp(const double (&U)[4], double g, const double (&cF)[4], const double (&cG)[4],
                                              double (&b)[4]) {
  const double rho = U[0];
  b[0] = b[1] = b[2] = b[3] = 0.0;
  if (!(rho >= FLOOR)) return false;
  const double r = lean_rcp(rho);
  const double u = U[1] * r, v = U[2] * r;
  const double q2 = u * u + v * v;
  const double gm = g - 1.0;
  const double p = gm * (U[3] - 0.5 * rho * q2);
  if (!(p >= FLOOR)) return false;
  const double H = (U[3] + p) * r;
  const double phi = 0.5 * gm * q2;
  const double uv = u * v;
  b[0] = cF[1] * (phi - u * u) - cF[2] * uv + cF[3] * u * (phi - H) - cG[1] * uv + cG[2] * (phi - v * v) +
         cG[3] * v * (phi - H);
  b[1] = cF[0] + cF[1] * (3.0 - g) * u + cF[2] * v + cF[3] * (H - gm * u * u) + cG[1] * v - cG[2] * gm * u -
         cG[3] * gm * uv;
  b[2] = -cF[1] * gm * v + cF[2] * u - cF[3] * gm * uv + cG[0] + cG[1] * u + cG[2] * (3.0 - g) * v +
         cG[3] * (H - gm * v * v);
  b[3] = gm * (cF[1] + cG[2]) + g * (cF[3] * u + cG[3] * v);
  return true;
}

// Shared memory of one block, in doubles: the fragments, then per warp two buffers of
// state, lambda and geometry rows.  Resident blocks: three (168 registers) with stored
// Jacobians, two (255) where the dual-number flux is in the kernel.
template <int K, int P, bool AFF, bool JAC>
struct TileVjpSmem {
  using S = Shape<K, P>;
  using T = Tile<K, P>;
  static constexpr int FRAGS = (T::A_END - T::A_PHI) * 32;
  static constexpr int STATE = S::NP * 4 * TILE_E;
  static constexpr int BUF = 2 * STATE + TileGeo<K, AFF>::ROWS * TILE_E;
  static constexpr int WANT = JAC ? 3 : 2;
  static constexpr int BASE = (FRAGS + TILE_WARPS * 2 * BUF) * 8;
  static constexpr int EPI_BYTES = TILE_WARPS * 2 * STATE * 8;
  // the epilogue's dJ/dU and starting lambda travel to shared memory too where that costs no resident block
  static constexpr bool EPI = (227 * 1024) / (BASE + EPI_BYTES + 1024) >= WANT;
  static constexpr int WARP = 2 * BUF + (EPI ? 2 * STATE : 0);
  static constexpr int BYTES = BASE + (EPI ? EPI_BYTES : 0);
  static constexpr int FIT = (227 * 1024) / (BYTES + 1024);
  static constexpr int MINB = FIT < WANT ? FIT : WANT;
};

template <int K, int P, bool AFF, bool JAC>
__global__ void __launch_bounds__(TILE_WARPS * 32, (TileVjpSmem<K, P, AFF, JAC>::MINB))
    k_tile_vjp(const nzb_mesh m, const nzb_physics ph, const AdjWork w) {
  using S = Shape<K, P>;
  using T = Tile<K, P>;
  using J = TileJac<K, P>;
  using L = TileVjpSmem<K, P, AFF, JAC>;
  extern __shared__ __align__(16) double smem[];
  const int lane = threadIdx.x & 31, l = lane & 3, warp = threadIdx.x >> 5;
  const int64_t E = m.n_elem, plane = S::NP * E;
  const double g = ph.gamma;
  stage_tiles<K, P>(smem, T::A_PHI, T::A_END - T::A_PHI);
  const double* fr = smem + lane - T::A_PHI * 32;  // fragment n of this lane is fr[32 n]
  double* const wbuf = smem + L::FRAGS + warp * L::WARP;
  double* const ebuf = wbuf + 2 * L::BUF;  // dJ/dU, then the step's starting lambda (L::EPI)
  const int64_t blocks = m.vjp_blocks ? m.n_vjp_blocks : (E + TILE_EB - 1) / TILE_EB;

  // one tile ahead, as in the forward kernel
  int64_t blk = 0;
  int inst = -1, ccode = 0, cnb = -1, ck = -1;
  auto fetch = [&](int64_t at, double* buf, bool first_tile = false) {
    blk = listed_block(m.vjp_blocks, E, TILE_EB, at);
    const int64_t e0 = blk * TILE_EB + warp * TILE_E, e = e0 + (lane >> 2);
    copy_rows(buf + 2 * L::STATE, m.geo, TileGeo<K, AFF>::ROWS, E, e0, E);
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
    copy_rows(buf, w.U, S::NP * 4, E, e0, E);
    copy_rows(buf + L::STATE, w.lam, S::NP * 4, E, e0, E);
    copy_commit();
    // what is read straight from global memory later: the Jacobian lines and the epilogue's rows
    if (e0 < E) {
      if constexpr (JAC) {
        const double* p = w.jac + (e0 / TILE_E) * J::TILE;
        for (int k = lane * 16; k < J::TILE; k += 32 * 16) prefetch_line(p + k);
      }
      if (w.mode != ADJ_VJP) {
        for (int r = lane; r < S::NP * 4; r += 32) {
          const int64_t o = r * E + e0;
          prefetch_line(w.seed + o);
          if (w.mode == ADJ_RK4) {
            if (w.stage > 0) prefetch_line(w.lam0 + o);
            if (w.stage == 3) {
              prefetch_line(w.f0 + o);
              prefetch_line(w.f1 + o);
              prefetch_line(w.f2 + o);
            }
          }
        }
      }
    }
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
    const double* const ucol = buf + (lane >> 2);  // this element's columns: row r at [8 r]
    const double* const lcol = ucol + L::STATE;
    const int64_t off = l * E + e;  // node 4c + l, component s: off + 4cE + s plane
    cur ^= 1;
    const bool more = b + gridDim.x < blocks;
    if (!more) chain_release();
    double dsq = 0.0;
    copy_wait<0>();
    // read last: on its way meanwhile
    if (L::EPI && w.mode != ADJ_VJP) {
      copy_rows(ebuf, w.seed, S::NP * 4, E, e0, E);
      if (w.mode == ADJ_RK4) copy_rows(ebuf + L::STATE, w.lam0, S::NP * 4, E, e0, E);
      copy_commit();
    }
    if (more) fetch(b + gridDim.x, wbuf + cur * L::BUF);
    if (__any_sync(0xffffffffu, act)) {
      TileGeo<K, AFF> geo;
      geo.template load<P>(ucol + 2 * L::STATE);
      const double dte = w.mode == ADJ_RK4 && act ? __ldg(w.dt + e) : 0.0;
      const double* const ecol = ebuf + (lane >> 2);
      auto seed_at = [&](int c, int s) {
        return L::EPI ? ecol[(s * S::NP + 4 * c + l) * 8] : __ldg(w.seed + off + (4 * c * E + s * plane));
      };
      auto lam0_at = [&](int c, int s) {
        return L::EPI ? ecol[L::STATE + (s * S::NP + 4 * c + l) * 8] : w.lam0[off + (4 * c * E + s * plane)];
      };
      double acc[T::NT][4][2];
#pragma unroll
      for (int t = 0; t < T::NT; ++t)
#pragma unroll
        for (int s = 0; s < 4; ++s) acc[t][s][0] = acc[t][s][1] = 0.0;

      // ---- faces: J^T (lam_own - lam_neighbour); the neighbour's scattered nodes one slot ahead
      AdjFace<K, P> next;
      double lnb[4];
      auto neighbour = [&](int fs) {
        next.set(mycode, mynb, myk, fs, lane);
        const double* p = w.lam + (next.oth >= 0 ? next.oth * E + next.nb : 0);
#pragma unroll
        for (int s = 0; s < 4; ++s) lnb[s] = next.oth >= 0 ? p[s * plane] : 0.0;  // the chain's: an ordinary load (tile.cuh)
      };
      // the Jacobians are loaded as soon as the registers of the slot before are free
      double jt[JAC ? 16 : 1];
      auto jacobian = [&](int fs) {
        if constexpr (JAC) {
          const bool valid = next.k >= 0 && (P == 1 || l < S::NQF);
          const double* p = w.jac + (e0 / TILE_E) * J::TILE + fs * 16 * J::ROW + (lane >> 2) * J::LPE + l;
#pragma unroll
          for (int k = 0; k < 16; ++k) jt[k] = valid ? __ldg(p + k * J::ROW) : 0.0;
        }
      };
      neighbour(0);
      // ---- volume: phi_jq (J_F^T cF + J_G^T cG) at every volume point
#pragma unroll 1
      for (int vt = 0; vt < T::VT; ++vt) {
        double uq[4][2], lx[4][2], le[4][2];
#pragma unroll
        for (int s = 0; s < 4; ++s) uq[s][0] = uq[s][1] = lx[s][0] = lx[s][1] = le[s][0] = le[s][1] = 0.0;
#pragma unroll
        for (int c = 0; c < T::NS; ++c) {
          const double* f = fr + (T::A_PHI + (vt * T::NS + c) * 3) * 32;
          const bool node = 4 * c + 3 < S::NP || 4 * c + l < S::NP;
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const double us = node ? ucol[(s * S::NP + 4 * c + l) * 8] : 0.0;
            const double ls = node ? lcol[(s * S::NP + 4 * c + l) * 8] : 0.0;
            mma(uq[s], us, f[0]);
            mma(lx[s], ls, f[32]);
            mma(le[s], ls, f[64]);
          }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int v = 2 * vt + j;
          if (T::VS % 2 == 1 && v >= T::VS) continue;
          double a00, a01, a10, a11, vs;
          if constexpr (K == 0) {
            a00 = geo.g[0];
            a01 = geo.g[1];
            a10 = geo.g[2];
            a11 = geo.g[3];
            vs = -geo.g[4];
          } else {
            double x_xi, x_eta, y_xi, y_eta;
            geo.at(fr[(T::A_XI + v) * 32], fr[(T::A_ETA + v) * 32], x_xi, x_eta, y_xi, y_eta);
            a00 = y_eta;
            a01 = -x_eta;
            a10 = -y_xi;
            a11 = x_xi;
            vs = -1.0;
          }
          double cF[4], cG[4], q[4], b4[4];
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            q[s] = uq[s][j];
            cF[s] = vs * (a00 * lx[s][j] + a10 * le[s][j]);
            cG[s] = vs * (a01 * lx[s][j] + a11 * le[s][j]);
          }
          if (!lean_flux_vjp(q, g, cF, cG, b4) && act && 4 * v + l < S::NQV) {
            double x[16];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              x[s] = q[s];
              x[4 + s] = cF[s];
              x[8 + s] = cG[s];
            }
            floored_flux_vjp(x, g, x + 4, x + 8, x + 12);
#pragma unroll
            for (int s = 0; s < 4; ++s) b4[s] = x[12 + s];
          }
          __syncwarp();
#pragma unroll
          for (int t = 0; t < T::NT; ++t) {
            const double b8 = fr[(T::A_PT + v * T::NT + t) * 32];
#pragma unroll
            for (int u = 0; u < 4; ++u) mma(acc[t][u], b4[u], b8);
          }
        }
      }

      // ---- faces
      jacobian(0);
#pragma unroll 1
      for (int fs = 0; fs < T::FS; ++fs) {
        const AdjFace<K, P> fp = next;
        const bool valid = fp.k >= 0 && (P == 1 || l < S::NQF);
        const double bo = fr[T::A_TRO * 32], bn = fr[T::A_TRN * 32];
        double d[4][2];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          d[s][0] = d[s][1] = 0.0;
          mma(d[s], fp.own >= 0 ? lcol[(s * S::NP + fp.own) * 8] : 0.0, bo);
          mma(d[s], lnb[s], bn);
        }
        if (fs + 1 < T::FS) neighbour(fs + 1);
        double a[4] = {0.0, 0.0, 0.0, 0.0};
        if constexpr (JAC) {
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const double x = d[s][0] - d[s][1];
#pragma unroll
            for (int u = 0; u < 4; ++u) a[u] = fma(x, jt[4 * u + s], a[u]);
          }
          if (fs + 1 < T::FS) jacobian(fs + 1);
        } else {
          double t[4][2];
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            t[s][0] = t[s][1] = 0.0;
            const double o = fp.oth >= 0 ? __ldg(w.U + fp.oth * E + fp.nb + s * plane) : 0.0;
            mma(t[s], fp.own >= 0 ? ucol[(s * S::NP + fp.own) * 8] : 0.0, bo);
            mma(t[s], o, bn);
          }
          if (valid) {
            const double* eg = m.edge_geo + 4 * (int64_t)fp.k;
            const double p_back = (myinst >= 0 && m.inst_p_back) ? __ldg(m.inst_p_back + myinst) : ph.p_back;
            const double tc[4] = {t[0][0], t[1][0], t[2][0], t[3][0]}, tn[4] = {t[0][1], t[1][1], t[2][1], t[3][1]};
            Dual<4> F[4];
            double coef;
            face_jacobian(tc, tn, fp.code, fp.nb, __ldg(eg), __ldg(eg + 1), __ldg(eg + 2) * fr[T::A_WF * 32], ph, p_back, F,
                          coef);
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              const double x = coef * (d[s][0] - d[s][1]);
#pragma unroll
              for (int u = 0; u < 4; ++u) a[u] = fma(x, F[s].d[u], a[u]);
            }
          }
          __syncwarp();
        }
#pragma unroll
        for (int t = 0; t < T::NT; ++t) {
          const double b8 = fr[(T::A_LF + fs * T::NT + t) * 32];
#pragma unroll
          for (int u = 0; u < 4; ++u) mma(acc[t][u], a[u], b8);
        }
      }

      // ---- epilogue
      if (L::EPI && w.mode != ADJ_VJP) {
        if (more)
          copy_wait<1>();
        else
          copy_wait<0>();
      }
      if (w.mode == ADJ_VJP || w.mode == ADJ_DEFECT) {
#pragma unroll
        for (int c = 0; c < T::NS; ++c) {
          if (!act || 4 * c + l >= S::NP) continue;
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const int64_t o = off + (4 * c * E + s * plane);
            double v = acc[c >> 1][s][c & 1];
            if (w.mode == ADJ_DEFECT) {
              v -= seed_at(c, s);
              dsq = fma(v, v, dsq);
            }
            if (w.out) w.out[o] = v;
          }
        }
        if (w.mode == ADJ_DEFECT) {
          __syncwarp();
          dsq = quad_sum(dsq);
          if (w.elem_norm && act && l == 0) w.elem_norm[e] = dsq;
        }
      } else {
        // rate = -M^-1 (v - seed): triangles M_ref^-1 / det; quadrilaterals Phi^-T diag(1 / (w det)) Phi^-1
        double d[T::NS][4], r[T::NT][4][2];
#pragma unroll
        for (int c = 0; c < T::NS; ++c)
#pragma unroll
          for (int s = 0; s < 4; ++s)
            d[c][s] = act && 4 * c + l < S::NP
                          ? acc[c >> 1][s][c & 1] - seed_at(c, s)
                          : 0.0;
        double fsum[T::NS][4];  // last stage: f0 + 2 f1 + 2 f2, loaded ahead of the mass contractions
        if (w.mode == ADJ_RK4 && w.stage == 3) {
#pragma unroll
          for (int c = 0; c < T::NS; ++c)
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              const int64_t o = off + (4 * c * E + s * plane);
              fsum[c][s] = act && 4 * c + l < S::NP ? w.f0[o] + 2.0 * w.f1[o] + 2.0 * w.f2[o] : 0.0;
            }
        }
        auto apply = [&](int table) {
          __syncwarp();
#pragma unroll
          for (int t = 0; t < T::NT; ++t)
#pragma unroll
            for (int s = 0; s < 4; ++s) r[t][s][0] = r[t][s][1] = 0.0;
#pragma unroll
          for (int c = 0; c < T::NS; ++c)
#pragma unroll
            for (int t = 0; t < T::NT; ++t) {
              const double b8 = fr[(table + c * T::NT + t) * 32];
#pragma unroll
              for (int s = 0; s < 4; ++s) mma(r[t][s], d[c][s], b8);
            }
        };
        apply(T::A_MI);
        double scale = 1.0;
        if constexpr (K == 0) {
          scale = act ? -lean_rcp(geo.g[4]) : 0.0;
        } else {
#pragma unroll
          for (int c = 0; c < T::NS; ++c) {
            double x0, x1, x2, x3;
            const double det = geo.at(fr[(T::A_XI + c) * 32], fr[(T::A_ETA + c) * 32], x0, x1, x2, x3);
            const double z = act && 4 * c + l < S::NP ? -lean_rcp(fr[(T::A_WV + c) * 32] * det) : 0.0;
#pragma unroll
            for (int s = 0; s < 4; ++s) d[c][s] = r[c >> 1][s][c & 1] * z;
          }
          apply(T::A_MT);
        }
        if (act) {
#pragma unroll
          for (int c = 0; c < T::NS; ++c) {
            if (4 * c + l >= S::NP) continue;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              const int64_t o = off + (4 * c * E + s * plane);
              const double rr = r[c >> 1][s][c & 1] * scale;
              if (w.mode == ADJ_RATE) {
                w.out[o] = rr;
              } else if (w.stage == 0) {
                w.f0[o] = rr;
                w.out[o] = lam0_at(c, s) + 0.5 * dte * rr;
              } else if (w.stage == 1) {
                w.f1[o] = rr;
                w.out[o] = lam0_at(c, s) + 0.5 * dte * rr;
              } else if (w.stage == 2) {
                w.f2[o] = rr;
                w.out[o] = lam0_at(c, s) + dte * rr;
              } else {
                w.lam0[o] = lam0_at(c, s) + dte / 6.0 * (fsum[c][s] + rr);
              }
            }
          }
        }
      }
    }
    __syncwarp();  // this tile's rows have been read: the buffers may be filled again
    if (w.mode == ADJ_DEFECT && w.norm_partial) {
      block_sum_store<TILE_WARPS>(l == 0 ? dsq : 0.0, w.norm_partial + myblk);
      __syncthreads();  // the sum's slots are free again
    }
  }
}

}  // namespace nzb
