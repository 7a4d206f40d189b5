// tile.cuh -- element-tile layout and FP64 tensor-core (mma.m8n8k4) contractions.
//
// A warp owns a tile of eight elements: row lane/4 of every 8 x 4 operand and
// 8 x 8 accumulator fragment is one element, so an element is worked on by the
// four lanes of its row ("quad" lanes l = lane & 3).  Every dense contraction of
// the method -- interpolation to the points, the weak-form projection, the face
// lift, the inverse mass -- is  (8 elements x K) * (K x N table), with the data
// as the A operand and the reference tables as the B operand, one component of
// the state at a time.
//
// The index maps make one register layout serve everything.  A list of items
// (nodes, volume points, face points) is cut into slots of four, item 4c + l of
// slot c living in lane l.  A k-step of an A operand is exactly one slot.  An
// accumulator fragment holds columns 2l and 2l + 1 in lane l; the tables' columns
// are permuted so that column 2l + j of tile t is item 4 (2t + j) + l, i.e. the
// fragment's two registers are slots 2t and 2t + 1.  So the output of one
// contraction is the input of the next -- interpolated states go through the
// flux in registers and back into the tensor cores, new states into the
// limiter's interpolation -- with no shuffle, no shared memory and no barrier.
//
// The B fragments (lane holds B[k = lane & 3][n = lane >> 2]) are laid out in
// memory one 256-byte line per fragment, read through L1 where every warp of an
// SM finds them.
#pragma once
#include <cmath>
#include <vector>

#include "element.cuh"

namespace nzb {

constexpr int TILE_LANES = 4;    // lanes of an element
constexpr int TILE_E = 8;        // elements of a warp
constexpr int TILE_WARPS = 4;    // warps of a block
constexpr int TILE_EB = TILE_E * TILE_WARPS;  // elements of a block

// edge_node(f, j) for every face and j < 4, four bits each.
template <int K, int P>
__host__ __device__ constexpr unsigned long long packed_edge_nodes() {
  unsigned long long v = 0;
  for (int f = 0; f < n_faces(K); ++f)
    for (int j = 0; j <= P; ++j) v |= (unsigned long long)edge_node(K, P, f, j) << (16 * f + 4 * j);
  return v;
}

template <int K, int P>
struct Tile {
  using S = Shape<K, P>;
  static constexpr int NS = (S::NP + 3) / 4;   // node slots
  static constexpr int NT = (NS + 1) / 2;      // node tiles (two slots each)
  // Where the last node tile holds one or two nodes (of eight columns), they are summed by multiply-adds
  // in the lanes that hold the points, and over the lanes once at the end: REM nodes, MTS tiles by mma.
  static constexpr int REM = NS % 2 == 1 && NS > 1 && S::NP - 8 * (NT - 1) <= 2 ? S::NP - 8 * (NT - 1) : 0;
  static constexpr int MTS = REM ? NT - 1 : NT;
  static constexpr int VS = (S::NQV + 3) / 4;  // volume-point slots
  static constexpr int VT = (VS + 1) / 2;
  static constexpr int FPS = P == 1 ? 2 : 1;   // faces per face-point slot
  static constexpr int FS = (S::NF + FPS - 1) / FPS;
  static constexpr int FT = (FS + 1) / 2;
  // a face slot holds FPS faces' points and, as a k-step, their edge nodes
  static_assert(S::NE == S::NQF && S::NE * FPS <= 4, "a face slot holds its faces' points and edge nodes");

  // Fragment numbers (32 doubles each).  The point -> node tables come plain (residuals), before the
  // common part, and folded with the constant factor of the inverse mass (rates, stages), after it, so
  // what a kernel stages in shared memory is one range: [0, COMMON_END) or [COMMON, COMMON + COMMON_END).
  static constexpr int VXN = VS * NT * 2, LFN = FS * NT;  // fragments of one VX / LF table
  static constexpr int COMMON = VXN + LFN;
  static constexpr int PHI = COMMON;                // [VT][NS] nodes -> volume points
  static constexpr int PF = PHI + VT * NS;          // [FT][NS] nodes -> face points (the limiter's probes)
  static constexpr int TRO = PF + FT * NS;          // own edge nodes -> own trace, even columns
  static constexpr int TRN = TRO + 1;               // neighbour's edge nodes -> its trace, odd columns
  static constexpr int MT = TRN + 1;                // quads: [NS][NT] point values -> nodes (Phi^-T)
  static constexpr int MW = MT + (K == 1 ? NS * NT : 0);   // tri: [NS] lane values mw; quads: [VS][NT] points -> w_q phi_iq
  static constexpr int WV = MW + (K == 0 ? NS : VS * NT);  // [VS] lane values w_q (0 past the points)
  static constexpr int XI = WV + VS;                // quads: [VS] lane values xi_q
  static constexpr int ETA = XI + (K == 1 ? VS : 0);       // quads: [VS] lane values eta_q
  static constexpr int WF = ETA + (K == 1 ? VS : 0);       // lane value: the face point's weight
  static constexpr int COMMON_END = WF + 1;
  static constexpr int STAGED = COMMON_END;         // fragments staged by either range
  // The adjoint kernels' own range [A_PHI, COUNT) (adjoint_tile.cuh): the same tables as it reads them.
  static constexpr int A_PHI = COMMON_END + COMMON;  // [VT][NS][3] nodes -> phi, w dphi/dxi, w dphi/deta at the points
  static constexpr int A_TRO = A_PHI + 3 * VT * NS;  // traces, as TRO and TRN
  static constexpr int A_TRN = A_TRO + 1;
  static constexpr int A_PT = A_TRN + 1;             // [VS][NT] points -> nodes (phi)
  static constexpr int A_LF = A_PT + VS * NT;        // [FS][NT] face points -> nodes
  static constexpr int A_MI = A_LF + FS * NT;        // [NS][NT] tri: M_ref^-1; quads: nodes -> points, Phi^-1
  static constexpr int A_MT = A_MI + NS * NT;        // quads: [NS][NT], as MT
  static constexpr int A_WV = A_MT + (K == 1 ? NS * NT : 0);
  static constexpr int A_XI = A_WV + (K == 1 ? VS : 0);
  static constexpr int A_ETA = A_XI + (K == 1 ? VS : 0);
  static constexpr int A_WF = A_ETA + (K == 1 ? VS : 0);
  static constexpr int A_END = A_WF + 1;
  static constexpr int FM = A_END;                   // [NS] nodes -> the average over face l, in lane l's even column
  static constexpr int COUNT = FM + NS;
  // [VS][NT][2 xi, eta] points -> nodes and [FS][NT] face points -> nodes
  static constexpr int vx(int folded, int v, int t, int d) { return (folded ? COMMON_END : 0) + (v * NT + t) * 2 + d; }
  static constexpr int lf(int folded, int fs, int t) { return (folded ? COMMON_END : 0) + VXN + fs * NT + t; }
};

template <int K>
constexpr int tile_offset(int p) {
  return (p > 1 ? Tile<K, 1>::COUNT : 0) * 32 + (p > 2 ? Tile<K, 2>::COUNT : 0) * 32 + (p > 3 ? Tile<K, 3>::COUNT : 0) * 32;
}

// ---- host: the fragments of one (kind, order) from its table slot ---------------
// Folded tables (rates and stages) carry the part of the inverse mass that is the
// same for every element: triangles (M = det M_ref) all of M_ref^-1; quadrilaterals,
// whose volume rule has as many points as there are nodes, factor
// M = Phi diag(w det) Phi^T, so M^-1 = Phi^-T diag(1 / (w det)) Phi^-1: Phi^-1 is
// folded, the diagonal is applied per element and Phi^-T is the MT table.
template <int K, int P>
std::vector<double> tile_tables(const double* slot) {
  using S = Shape<K, P>;
  using T = Tile<K, P>;
  constexpr int NP = S::NP, NQV = S::NQV, NQF = S::NQF, NF = S::NF, NE = S::NE;
  const double *phi = slot + (S::O_PHI - S::BASE), *wxi = slot + (S::O_WXI - S::BASE), *weta = slot + (S::O_WETA - S::BASE);
  const double *minv = slot + (S::O_MINV - S::BASE), *wf = slot + (S::O_WF - S::BASE), *mw = slot + (S::O_MW - S::BASE);
  const double *wv = slot + (S::O_WV - S::BASE), *dgx = slot + (S::O_DGX - S::BASE), *dge = slot + (S::O_DGE - S::BASE);
  const double* pfe = slot + (S::O_PFE - S::BASE);
  // G: the folded constant matrix (M_ref^-1, or Phi^-1 by Gauss-Jordan with partial pivoting)
  std::vector<long double> G(NP * NP, 0.0L);
  if (K == 0) {
    for (int k = 0; k < NP * NP; ++k) G[k] = minv[k];
  } else {
    std::vector<long double> A(NP * NP);
    for (int i = 0; i < NP; ++i)
      for (int q = 0; q < NP; ++q) {
        A[i * NP + q] = q < NQV ? phi[i * NQV + q] : 0.0;
        G[i * NP + q] = i == q ? 1.0L : 0.0L;
      }
    for (int c = 0; c < NP; ++c) {
      int piv = c;
      for (int r = c + 1; r < NP; ++r)
        if (fabsl(A[r * NP + c]) > fabsl(A[piv * NP + c])) piv = r;
      for (int k = 0; k < NP; ++k) {
        std::swap(A[c * NP + k], A[piv * NP + k]);
        std::swap(G[c * NP + k], G[piv * NP + k]);
      }
      const long double d = A[c * NP + c];
      for (int k = 0; k < NP; ++k) {
        A[c * NP + k] /= d;
        G[c * NP + k] /= d;
      }
      for (int r = 0; r < NP; ++r) {
        const long double f = A[r * NP + c];
        if (r == c || f == 0.0L) continue;
        for (int k = 0; k < NP; ++k) {
          A[r * NP + k] -= f * A[c * NP + k];
          G[r * NP + k] -= f * G[c * NP + k];
        }
      }
    }
  }
  auto fold = [&](bool folded, int i, auto&& col) -> double {
    if (!folded) return (double)col(i);
    long double s = 0.0L;
    for (int m = 0; m < NP; ++m) s += G[i * NP + m] * (long double)col(m);
    return (double)s;
  };
  // the 1D basis of an edge's nodes at its points, walking the edge from its own
  // element: the tables' average over the faces and sides (they differ in the last bits)
  auto e1d = [&](int j, int q) -> double {
    long double s = 0.0L;
    for (int f = 0; f < NF; ++f)
      s += (long double)pfe[((0 * NF + f) * NE + j) * NQF + q] + (long double)pfe[((1 * NF + f) * NE + j) * NQF + NQF - 1 - q];
    return (double)(s / (2 * NF));
  };
  std::vector<double> out((size_t)T::COUNT * 32, 0.0);
  auto put = [&](int frag, auto&& value) {  // value(k, out slot parity, out lane)
    for (int lane = 0; lane < 32; ++lane) out[frag * 32 + lane] = value(lane & 3, (lane >> 2) & 1, lane >> 3);
  };
  auto put_lane = [&](int frag, auto&& value) {
    for (int lane = 0; lane < 32; ++lane) out[frag * 32 + lane] = value(lane & 3);
  };
  // (face, point) of lane l of face slot fs; face -1 where there is none
  auto face_of = [&](int fs, int l) { const int f = P == 1 ? 2 * fs + (l >> 1) : fs; return f < NF && (P == 1 || l < NE) ? f : -1; };
  auto pt_of = [&](int l) { return P == 1 ? (l & 1) : l; };
  for (int vt = 0; vt < T::VT; ++vt)
    for (int c = 0; c < T::NS; ++c)
      put(T::PHI + vt * T::NS + c, [&](int k, int j, int l) {
        const int i = 4 * c + k, q = 4 * (2 * vt + j) + l;
        return i < NP && q < NQV ? phi[i * NQV + q] : 0.0;
      });
  put(T::TRO, [&](int k, int j, int l) {
    return j == 0 && (P > 1 ? (k < NE && l < NQF) : (k >> 1) == (l >> 1)) ? e1d(pt_of(k), pt_of(l)) : 0.0;
  });
  put(T::TRN, [&](int k, int j, int l) {
    return j == 1 && (P > 1 ? (k < NE && l < NQF) : (k >> 1) == (l >> 1)) ? e1d(pt_of(k), NQF - 1 - pt_of(l)) : 0.0;
  });
  for (int ft = 0; ft < T::FT; ++ft)
    for (int c = 0; c < T::NS; ++c)
      put(T::PF + ft * T::NS + c, [&](int k, int j, int l) {
        const int i = 4 * c + k, fs = 2 * ft + j, f = fs < T::FS ? face_of(fs, l) : -1;
        const int e = i < NP && f >= 0 ? edge_pos(K, P, f, i) : -1;
        return e >= 0 ? pfe[(f * NE + e) * NQF + pt_of(l)] : 0.0;
      });
  for (int fo = 0; fo < 2; ++fo) {
    for (int v = 0; v < T::VS; ++v)
      for (int t = 0; t < T::NT; ++t)
        for (int d = 0; d < 2; ++d)
          put(T::vx(fo, v, t, d), [&](int k, int j, int l) {
            const int q = 4 * v + k, i = 4 * (2 * t + j) + l;
            if (i >= NP || q >= NQV) return 0.0;
            return fold(fo != 0, i, [&](int m) { return (d ? weta : wxi)[m * NQV + q]; });
          });
    for (int fs = 0; fs < T::FS; ++fs)
      for (int t = 0; t < T::NT; ++t)
        put(T::lf(fo, fs, t), [&](int k, int j, int l) {
          const int i = 4 * (2 * t + j) + l, f = face_of(fs, k);
          if (i >= NP || f < 0) return 0.0;
          return fold(fo != 0, i, [&](int m) {
            const int e = edge_pos(K, P, f, m);
            return e >= 0 ? pfe[(f * NE + e) * NQF + pt_of(k)] : 0.0;
          });
        });
  }
  for (int c = 0; K == 1 && c < T::NS; ++c)
    for (int t = 0; t < T::NT; ++t)
      put(T::MT + c * T::NT + t, [&](int k, int j, int l) {
        const int q = 4 * c + k, i = 4 * (2 * t + j) + l;
        return q < NP && i < NP ? (double)G[q * NP + i] : 0.0;
      });
  if (K == 0) {
    for (int c = 0; c < T::NS; ++c) put_lane(T::MW + c, [&](int l) { return 4 * c + l < NP ? mw[4 * c + l] : 0.0; });
  } else {
    for (int v = 0; v < T::VS; ++v)
      for (int t = 0; t < T::NT; ++t)
        put(T::MW + v * T::NT + t, [&](int k, int j, int l) {
          const int q = 4 * v + k, i = 4 * (2 * t + j) + l;
          return q < NQV && i < NP ? phi[i * NQV + q] * wv[q] : 0.0;
        });
    // bilinear shape functions on the unit square: d/dxi of vertex 3 is eta, d/deta of it xi
    for (int v = 0; v < T::VS; ++v) {
      put_lane(T::XI + v, [&](int l) { return 4 * v + l < NQV ? dge[3 * NQV + 4 * v + l] : 0.0; });
      put_lane(T::ETA + v, [&](int l) { return 4 * v + l < NQV ? dgx[3 * NQV + 4 * v + l] : 0.0; });
    }
  }
  for (int v = 0; v < T::VS; ++v) put_lane(T::WV + v, [&](int l) { return 4 * v + l < NQV ? wv[4 * v + l] : 0.0; });
  put_lane(T::WF, [&](int l) { return pt_of(l) < NQF ? wf[pt_of(l)] : 0.0; });

  // the adjoint range: new layouts of the interpolation, its transpose and the inverse mass, the rest copied
  for (int vt = 0; vt < T::VT; ++vt)
    for (int c = 0; c < T::NS; ++c)
      for (int d = 0; d < 3; ++d)
        put(T::A_PHI + (vt * T::NS + c) * 3 + d, [&](int k, int j, int l) {
          const int i = 4 * c + k, q = 4 * (2 * vt + j) + l;
          return i < NP && q < NQV ? (d == 0 ? phi : d == 1 ? wxi : weta)[i * NQV + q] : 0.0;
        });
  for (int v = 0; v < T::VS; ++v)
    for (int t = 0; t < T::NT; ++t)
      put(T::A_PT + v * T::NT + t, [&](int k, int j, int l) {
        const int q = 4 * v + k, i = 4 * (2 * t + j) + l;
        return q < NQV && i < NP ? phi[i * NQV + q] : 0.0;
      });
  for (int c = 0; c < T::NS; ++c)
    for (int t = 0; t < T::NT; ++t)
      put(T::A_MI + c * T::NT + t, [&](int k, int j, int l) {
        const int i = 4 * c + k, q = 4 * (2 * t + j) + l;
        return i < NP && q < NP ? (double)G[q * NP + i] : 0.0;
      });
  auto copy = [&](int to, int from, int n) {
    for (int k = 0; k < n * 32; ++k) out[to * 32 + k] = out[from * 32 + k];
  };
  copy(T::A_TRO, T::TRO, 2);
  copy(T::A_LF, T::lf(0, 0, 0), T::LFN);
  if (K == 1) {
    copy(T::A_MT, T::MT, T::NS * T::NT);
    copy(T::A_WV, T::WV, T::VS);
    copy(T::A_XI, T::XI, T::VS);
    copy(T::A_ETA, T::ETA, T::VS);
  }
  copy(T::A_WF, T::WF, 1);
  for (int c = 0; c < T::NS; ++c)
    put(T::FM + c, [&](int k, int j, int l) {
      const int i = 4 * c + k, e = j == 0 && i < NP && l < NF ? edge_pos(K, P, l, i) : -1;
      if (e < 0) return 0.0;
      long double s = 0.0L, w = 0.0L;
      for (int q = 0; q < NQF; ++q) {
        s += (long double)wf[q] * pfe[(l * NE + e) * NQF + q];
        w += wf[q];
      }
      return (double)(s / w);
    });
  return out;
}

// Whether a quadrilateral slot's vertex shape derivatives are those of the unit
// square with vertices (0,0), (1,0), (0,1), (1,1), as the tile kernels assume.
template <int P>
bool unit_square_tables(const double* slot) {
  using S = Shape<1, P>;
  const double *dgx = slot + (S::O_DGX - S::BASE), *dge = slot + (S::O_DGE - S::BASE);
  for (int q = 0; q < S::NQV; ++q) {
    const double eta = dgx[3 * S::NQV + q], xi = dge[3 * S::NQV + q];
    const double ex[4] = {-(1.0 - eta), 1.0 - eta, -eta, eta}, ee[4] = {-(1.0 - xi), -xi, 1.0 - xi, xi};
    for (int v = 0; v < 4; ++v)
      if (!(std::fabs(dgx[v * S::NQV + q] - ex[v]) < 1e-13 && std::fabs(dge[v * S::NQV + q] - ee[v]) < 1e-13)) return false;
  }
  return true;
}

// ---- device ----------------------------------------------------------------------
// One copy per translation unit, as c_tab (each unit that runs tile kernels uploads its own).
static __device__ __align__(16) double g_tile_tri[tile_offset<0>(MAX_ORDER + 1)];
static __device__ __align__(16) double g_tile_quad[tile_offset<1>(MAX_ORDER + 1)];

// Stage the fragments [first, first + n) of (K, P) in shared memory (the caller synchronises).
template <int K, int P>
__device__ __forceinline__ void stage_tiles(double* dst, int first, int n) {
  const double2* src = reinterpret_cast<const double2*>((K == 0 ? g_tile_tri : g_tile_quad) + tile_offset<K>(P) + first * 32);
  for (int k = threadIdx.x; k < n * 16; k += blockDim.x) reinterpret_cast<double2*>(dst)[k] = __ldg(src + k);
}

// Build and upload the fragments of one (kind, order) from its table slot into this unit's copy.
template <int K, int P>
static cudaError_t upload_tiles(const double* slot) {
  const std::vector<double> t = tile_tables<K, P>(slot);
  const size_t off = sizeof(double) * (size_t)tile_offset<K>(P);
  return K == 0 ? cudaMemcpyToSymbol(g_tile_tri, t.data(), sizeof(double) * t.size(), off)
                : cudaMemcpyToSymbol(g_tile_quad, t.data(), sizeof(double) * t.size(), off);
}

// D += A B: A 8 x 4 (row lane / 4, column lane % 4), B 4 x 8 (row lane % 4, column
// lane / 4), D 8 x 8 (row lane / 4, columns 2 (lane % 4) and the next).
__device__ __forceinline__ void mma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// The remaining nodes of a contraction (Tile::REM): this lane's share of node 8 MTS + r from its own item
// of the k-step is x times entry (k = l, column of that node) of the fragment, at row[8 r].
template <int K, int P, int N>
__device__ __forceinline__ void remainder(double (&rem)[N][4], const double* row, const double (&x)[4]) {
#pragma unroll
  for (int r = 0; r < Tile<K, P>::REM; ++r) {
    const double b = row[8 * r];
#pragma unroll
    for (int s = 0; s < 4; ++s) rem[r][s] = fma(b, x[s], rem[r][s]);
  }
}
// ... summed over the four lanes (a product with a matrix of ones) into the last tile's first slot.
template <int K, int P, int N>
__device__ __forceinline__ void remainder_sum(double (&acc)[Tile<K, P>::NT][4][2], const double (&rem)[N][4], int l) {
  using T = Tile<K, P>;
  if constexpr (T::REM > 0) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      double v = 0.0;
#pragma unroll
      for (int r = 0; r < T::REM; ++r) {
        double d[2] = {0.0, 0.0};
        mma(d, rem[r][s], 1.0);
        v = l == r ? d[0] : v;
      }
      acc[T::NT - 1][s][0] = v;
    }
  }
}

// Sum, maximum and minimum over an element's four lanes (every lane gets it; the
// same bits in each, since both operands of a step are the same pair).
__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ double quad_max(double v) {
  double o = __shfl_xor_sync(0xffffffffu, v, 1);
  v = o > v ? o : v;
  o = __shfl_xor_sync(0xffffffffu, v, 2);
  return o > v ? o : v;
}
__device__ __forceinline__ double quad_min(double v) {
  double o = __shfl_xor_sync(0xffffffffu, v, 1);
  v = o < v ? o : v;
  o = __shfl_xor_sync(0xffffffffu, v, 2);
  return o < v ? o : v;
}

// ---- launches that overlap their predecessor's tail --------------------------------
// A march is a chain of short dependent kernels.  Each but the first of a run is
// launched as a programmatic dependent of the one before it: its CTAs may start
// while that one drains (once all its CTAs have called chain_release), stage their
// tables and read the mesh's own arrays, and wait in chain_wait() before they touch
// anything a kernel of the chain writes.  chain_wait returns when the earlier kernel
// has completed and its writes are visible, and every kernel of a chain calls it, so
// that holds for all earlier ones; without such a launch both are no-ops.  The mesh's
// arrays are read before the wait, so a launch is chained only where the call itself
// put a kernel of the chain in front of it -- never right after work of the caller's
// (which may have written them, as nzb_geometry does).
// Whatever a kernel of the chain writes (states, lambda, the RK4 rates, edge fluxes, local steps) is read
// by ordinary loads after the wait: the read-only path (__ldg, or const __restrict__ on a kernel's
// parameter) holds for data that nothing writes while the kernel is resident, and the compiler may move
// such a load across the wait.  It is for the mesh, the tables and an adjoint's frozen state.
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_chained(bool chained, void (*kernel)(P...), unsigned blocks, unsigned threads, int smem, cudaStream_t st, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// ---- asynchronous copies: a tile's rows ------------------------------------------
// Copy `rows` rows of eight consecutive doubles (row r at src + r * stride + e0) into
// dst[8 r + 0..7], elements past E as zeros.  Eight bytes per lane: rows start at any
// element count's offset, so no wider alignment can be assumed.
__device__ __forceinline__ void copy_rows(double* dst, const double* __restrict__ src, int rows, int64_t stride, int64_t e0,
                                          int64_t E) {
  const int lane = threadIdx.x & 31;
  const int64_t e = e0 + (lane & 7);
  const int bytes = e < E ? 8 : 0;
  const double* p = src + (e < E ? e : 0) + (lane >> 3) * stride;
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst + lane);
#pragma unroll 4
  for (int r = 0; r < rows; r += 4) {
    if (r + (lane >> 3) < rows)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d + r * 64), "l"(p + r * stride), "r"(bytes) : "memory");
  }
}
// Copy one double of this lane (zero where !ok) to dst.
__device__ __forceinline__ void copy_one(double* dst, const double* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(ok ? 8 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Wait until at most N of this thread's committed groups are in flight, then for the warp's other lanes.
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
  __syncwarp();
}

// The metric terms of one element, the same in its four lanes, from its column of
// the staged geometry rows.  Triangles: the inverse Jacobian and det.
// Quadrilaterals: x(xi, eta) = x0 + ax xi + cx eta + bx xi eta (and y alike), so
// x_xi = ax + bx eta, x_eta = cx + bx xi.
template <int K, bool AFF>
struct TileGeo {
  static constexpr int ROWS = AFF ? 5 : 2 * n_faces(K);
  double g[K == 0 ? 5 : 6];

  template <int P>
  __device__ __forceinline__ void load(const double* col) {
    if constexpr (AFF) {
#pragma unroll
      for (int k = 0; k < 5; ++k) g[k] = col[8 * k];
    } else {
      constexpr int NV = n_faces(K);
      double x[NV], y[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        x[v] = col[8 * v];
        y[v] = col[8 * (NV + v)];
      }
      if constexpr (K == 1) {
        g[0] = x[1] - x[0];
        g[1] = x[2] - x[0];
        g[2] = (x[3] - x[2]) - g[0];
        g[3] = y[1] - y[0];
        g[4] = y[2] - y[0];
        g[5] = (y[3] - y[2]) - g[3];
      } else {  // a straight-sided triangle from its vertices: its metrics are constant
        double a, b, c, d;
        const double det = point_det<K, P>(x, y, 0, a, b, c, d);
        const double r = 1.0 / det;
        g[0] = d * r;
        g[1] = -b * r;
        g[2] = -c * r;
        g[3] = a * r;
        g[4] = det;
      }
    }
  }
  // quadrilaterals: the Jacobian at (xi, eta); returns det
  __device__ __forceinline__ double at(double xi, double eta, double& x_xi, double& x_eta, double& y_xi, double& y_eta) const {
    x_xi = fma(g[2], eta, g[0]);
    x_eta = fma(g[2], xi, g[1]);
    y_xi = fma(g[K == 0 ? 4 : 5], eta, g[3]);
    y_eta = fma(g[K == 0 ? 4 : 5], xi, g[4]);
    return x_xi * y_eta - x_eta * y_xi;
  }
};

}  // namespace nzb
