// forward_launch.cuh -- the launch of one residual, rate, stage or limiter pass
// for one (kind, order, geometry layout), shared by forward_tri.cu and
// forward_quad.cu (each translation unit instantiates it for its own kind).
//
// Variants (nzb_mesh.split, nzb_mesh.edge_pass):
//   split = 4      k_tile: four lanes per element, FP64 tensor cores
//                  (tile_element.cuh), p >= 1;
//   edge_pass = 1  k_edge (one thread per edge) then k_element with the
//                  fluxes lifted from the edge array;
//   otherwise      k_element: one thread per element, fluxes from both sides.
// With the Superbee limiter (limiter 2) the element kernel leaves the stage
// unlimited and three passes follow (cell means, their maximum -- per
// instance in a batch -- and the slope limiter with the positivity limiter);
// the tile kernel forms the means and maxima itself, so one follows it (2 240
// quadratic triangles, a stage: 24 -> 17 us), except under a block list.
#pragma once
#include <cuda_runtime.h>

#include <initializer_list>

#include "element.cuh"
#include "slope.cuh"
#include "tile_element.cuh"

namespace nzb {
namespace {

template <int K, int P, bool AFF>
cudaError_t tile_superbee(const nzb_mesh& m, const nzb_physics& ph, const double* V, double* out,
                          unsigned long long* counters, uint8_t* flags, bool chained, cudaStream_t st) {
  return launch_chained(chained, k_tile_superbee<K, P, AFF>, (unsigned)((m.n_elem + TILE_EB - 1) / TILE_EB), TILE_WARPS * 32, 0,
                        st, m, ph, V, out, counters, flags);
}

// The limiter on a state: averages, their maxima, then the factor, the scaling and the positivity limiter.
template <int K, int P, bool AFF>
cudaError_t superbee_passes(const nzb_mesh& m, const nzb_physics& ph, const double* V, double* out,
                            unsigned long long* counters, uint8_t* flags, cudaStream_t st) {
  const unsigned nb = (unsigned)((m.n_elem + 127) / 128);
  k_cell_means<K, P, AFF><<<nb, 128, 0, st>>>(m, V, m.lim_means);
  if (m.elem_inst)
    k_lim_scale_inst<<<nb, 128, 0, st>>>(m.lim_means, m.n_elem, m.elem_inst, m.lim_scale);
  else
    k_lim_scale<<<1, 1024, 0, st>>>(m.lim_means, m.n_elem, m.lim_scale);
  if constexpr (P > 0) {
    if (m.split == TILE_LANES) return tile_superbee<K, P, AFF>(m, ph, V, out, counters, flags, false, st);
  }
  k_superbee<K, P, AFF><<<nb, 128, 0, st>>>(m, ph, V, out, counters, flags);
  return cudaGetLastError();
}

// Persistent CTAs, as many as the GPU holds at once: the tables are staged once per
// CTA, and a warp prefetches its next tile while it works on one.
template <int K, int P, bool AFF, bool LIM>
cudaError_t launch_tile(const nzb_mesh& m, const nzb_physics& ph, const Work& w, int64_t blocks, cudaStream_t st) {
  using L = TileSmem<K, P, AFF, LIM>;
  constexpr int64_t most = 148 * L::MINB;
  // chained only within one wave: past it the dependents' waiting CTAs would hold slots
  return launch_chained(w.chained && blocks <= most, k_tile<K, P, AFF, LIM>, (unsigned)(blocks < most ? blocks : most), TILE_WARPS * 32, L::BYTES, st, m,
                        ph, w);
}

inline cudaError_t first_error(std::initializer_list<cudaError_t> all) {
  for (const cudaError_t e : all)
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

// The tile kernels' dynamic shared memory exceeds the default 48 KB limit at some
// orders: raise each instantiation's limit (once per device, at table upload).
template <int K, int P, bool AFF>
cudaError_t prepare_tile() {
  const cudaError_t e = cudaFuncSetAttribute(k_tile<K, P, AFF, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             TileSmem<K, P, AFF, true>::BYTES);
  return e != cudaSuccess ? e
                          : cudaFuncSetAttribute(k_tile<K, P, AFF, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 TileSmem<K, P, AFF, false>::BYTES);
}

template <int K, int P, bool AFF>
cudaError_t launch(const nzb_mesh& m, const nzb_physics& ph, const Work& w, cudaStream_t st) {
  const bool sb = ph.limiter == 2 && P > 0 && (w.op == OP_STAGE || w.op == OP_LIMIT);
  if (sb && w.op == OP_LIMIT) return superbee_passes<K, P, AFF>(m, ph, w.V, w.out, w.counters, w.flags, st);
  const bool lim = w.op == OP_STAGE || w.op == OP_LIMIT;
  bool done = false;
  if constexpr (P > 0) {
    if (m.split == TILE_LANES) {
      const int64_t blocks = m.fwd_blocks ? m.n_fwd_blocks : (m.n_elem + TILE_EB - 1) / TILE_EB;
      // Superbee: the stage kernel leaves the averages and, from zero, their maxima; one pass follows.
      // Under a block list it sees only the listed elements, so the averages keep their own passes.
      Work wt = w;
      const bool fused = sb && !m.fwd_blocks;
      if (sb) wt.chained = false;
      if (fused) {
        const cudaError_t e = cudaMemsetAsync(m.lim_scale, 0, sizeof(double) * 4 * (m.elem_inst ? m.n_inst : 1), st);
        if (e != cudaSuccess) return e;
      }
      if (blocks > 0) {  // an empty block list: nothing marches
        const cudaError_t e = lim ? launch_tile<K, P, AFF, true>(m, ph, wt, blocks, st)
                                  : launch_tile<K, P, AFF, false>(m, ph, wt, blocks, st);
        if (e != cudaSuccess) return e;
      }
      if (fused) return tile_superbee<K, P, AFF>(m, ph, w.out, w.out, w.counters, w.flags, true, st);
      done = true;
    }
  }
  if (!done) {
    constexpr int NT = Launch<K, P>::NT;
    const unsigned nb = (unsigned)(m.fwd_blocks ? m.n_fwd_blocks : (m.n_elem + NT - 1) / NT);
    const bool ep = m.edge_pass && w.op != OP_LIMIT;
    if (ep) {
      k_edge<K, P><<<(unsigned)((m.n_edge + 127) / 128), 128, 0, st>>>(m, ph, w.V);
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    if (nb == 0)
      ;  // an empty block list: nothing marches
    else if (lim && ep)
      k_element<K, P, AFF, true, true><<<nb, NT, 0, st>>>(m, ph, w);
    else if (lim)
      k_element<K, P, AFF, true, false><<<nb, NT, 0, st>>>(m, ph, w);
    else if (ep)
      k_element<K, P, AFF, false, true><<<nb, NT, 0, st>>>(m, ph, w);
    else
      k_element<K, P, AFF, false, false><<<nb, NT, 0, st>>>(m, ph, w);
  }
  if (sb) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return superbee_passes<K, P, AFF>(m, ph, w.out, w.out, w.counters, w.flags, st);
  }
  return cudaGetLastError();
}

}  // namespace
}  // namespace nzb
