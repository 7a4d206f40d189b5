// adjoint_launch.cuh -- the launches of the state VJP for one (kind, order, geometry
// layout), shared by adjoint_tri.cu and adjoint_quad.cu.
//
// Variants (nzb_mesh.vjp_split): 4 runs the tile kernels (adjoint_tile.cuh), with
// stored face Jacobians when the caller has them; otherwise one thread per element.
#pragma once
#include <cuda_runtime.h>

#include <initializer_list>

#include "adjoint_dispatch.cuh"
#include "adjoint_tile.cuh"

namespace nzb {
namespace {

template <int K, int P, bool AFF, bool JAC>
cudaError_t launch_tile_vjp(const nzb_mesh& m, const nzb_physics& ph, const AdjWork& w, int64_t blocks, cudaStream_t st) {
  using L = TileVjpSmem<K, P, AFF, JAC>;
  constexpr int64_t most = 148 * L::MINB;  // persistent CTAs: the resident ones of a B200
  // chained only within one wave: past it the dependents' waiting CTAs would hold slots
  return launch_chained(w.chained && blocks <= most, k_tile_vjp<K, P, AFF, JAC>, (unsigned)(blocks < most ? blocks : most), TILE_WARPS * 32, L::BYTES, st,
                        m, ph, w);
}

template <int K, int P, bool AFF>
cudaError_t launch_vjp(const nzb_mesh& m, const nzb_physics& ph, const AdjWork& w, cudaStream_t st) {
  if constexpr (P > 0) {
    if (m.vjp_split == TILE_LANES) {
      const int64_t blocks = m.vjp_blocks ? m.n_vjp_blocks : (m.n_elem + TILE_EB - 1) / TILE_EB;
      if (blocks == 0) return cudaSuccess;
      return w.jac ? launch_tile_vjp<K, P, AFF, true>(m, ph, w, blocks, st)
                   : launch_tile_vjp<K, P, AFF, false>(m, ph, w, blocks, st);
    }
  }
  const int64_t nb = m.vjp_blocks ? m.n_vjp_blocks : (m.n_elem + Launch<K, P>::NT - 1) / Launch<K, P>::NT;
  if (nb) k_vjp<K, P, AFF><<<(unsigned)nb, Launch<K, P>::NT, 0, st>>>(m, ph, w);
  return cudaGetLastError();
}

template <int K, int P>
cudaError_t launch_jac(const nzb_mesh& m, const nzb_physics& ph, const double* U, double* jac, cudaStream_t st) {
  const int64_t blocks = m.vjp_blocks ? m.n_vjp_blocks : (m.n_elem + TILE_EB - 1) / TILE_EB;
  if (blocks) k_tile_jac<K, P><<<(unsigned)blocks, TILE_WARPS * 32, 0, st>>>(m, ph, U, jac);
  return cudaGetLastError();
}

inline cudaError_t first_error(std::initializer_list<cudaError_t> all) {
  for (const cudaError_t e : all)
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

// The kernels' dynamic shared memory can exceed the default 48 KB: raise each
// instantiation's limit (once per device, at table upload).
template <int K, int P, bool AFF>
cudaError_t prepare_vjp() {
  return first_error({cudaFuncSetAttribute(k_tile_vjp<K, P, AFF, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           TileVjpSmem<K, P, AFF, true>::BYTES),
                      cudaFuncSetAttribute(k_tile_vjp<K, P, AFF, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           TileVjpSmem<K, P, AFF, false>::BYTES)});
}

}  // namespace
}  // namespace nzb
