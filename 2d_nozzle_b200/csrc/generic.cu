// generic.cu -- launchers of the any-order / curved-element kernels (generic.cuh).
#include "forward_dispatch.cuh"
#include "gen_geometry.cuh"
#include "gen_initial.cuh"
#include "gen_observe.cuh"
#include "generic.cuh"

namespace nzb {
namespace {

unsigned blocks(int64_t n) { return (unsigned)((n + 127) / 128); }
unsigned warp_blocks(int64_t n) { return (unsigned)((n + GEN_WARPS - 1) / GEN_WARPS); }

// Dynamic shared memory of a warp-per-element kernel, its limit raised past 48 KB where it needs more
// (more than 64 volume points).
template <class K>
cudaError_t warp_smem(K kernel, const nzb_gen_mesh& m, int* bytes) {
  *bytes = GEN_WARPS * GenSmem{m.np, m.nqv, m.nface, m.nqf}.warp() * (int)sizeof(double);
  return *bytes > 48 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, *bytes) : cudaSuccess;
}

template <int MT>
cudaError_t launch_element(const nzb_gen_mesh& m, const nzb_physics& ph, const GenWork& w, cudaStream_t st) {
  int bytes = 0;
  const cudaError_t e = warp_smem(k_gen_element<MT>, m, &bytes);
  if (e != cudaSuccess) return e;
  return launch_chained(w.chained, k_gen_element<MT>, warp_blocks(m.n_elem), GEN_WARPS * 32, bytes, st, m, ph, w);
}

cudaError_t element_pass(const nzb_gen_mesh& m, const nzb_physics& ph, const GenWork& w, cudaStream_t st) {
  switch ((m.np + 7) / 8) {
    case 1: return launch_element<1>(m, ph, w, st);
    case 2: return launch_element<2>(m, ph, w, st);
    case 3: return launch_element<3>(m, ph, w, st);
    case 4: return launch_element<4>(m, ph, w, st);
    case 5: return launch_element<5>(m, ph, w, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t edge_pass(const nzb_gen_mesh& m, const nzb_physics& ph, const double* U, double* fw, double* smax,
                      bool chained, cudaStream_t st) {
  return launch_chained(chained, k_gen_edge, blocks(8 * (m.n_int + m.n_bnd)), 128, 0, st, m, ph, U, fw, smax);
}

}  // namespace

cudaError_t gen_rate_launch(const nzb_gen_mesh& m, const nzb_physics& ph, int unfolded, const double* U, double* out,
                            double* wave, double* fw, double* smax, cudaStream_t st) {
  const cudaError_t e = edge_pass(m, ph, U, fw, smax, false, st);
  if (e != cudaSuccess) return e;
  GenWork w{};
  w.chained = true;
  w.op = unfolded ? GEN_RESIDUAL : GEN_RATE;
  w.V = U;
  w.out = out;
  w.wave = wave;
  w.fw = fw;
  w.smax = smax;
  return element_pass(m, ph, w, st);
}

cudaError_t gen_limit_launch(const nzb_gen_mesh& m, const nzb_physics& ph, double* U, unsigned long long* counters,
                             cudaStream_t st) {
  GenWork w{};
  w.op = GEN_LIMIT;
  w.V = U;
  w.out = U;
  w.counters = counters;
  return element_pass(m, ph, w, st);
}

// n steps: per stage the edge pass and the element pass, which ends with the update and the positivity
// limiter; the Superbee limiter's passes follow it where that is the limiter.
cudaError_t gen_run_launch(const nzb_gen_mesh& m, const nzb_physics& ph, const nzb_gen_run_args& r, int n_steps,
                           cudaStream_t st) {
  bool first = true;
  auto stage = [&](int k, const double* V, const double* U0, double* out, double a, double b) -> cudaError_t {
    cudaError_t e = edge_pass(m, ph, V, r.fw, r.smax, !first, st);
    if (e != cudaSuccess) return e;
    first = false;
    GenWork w{};
    w.chained = true;
    w.op = GEN_STAGE;
    w.stage = k;
    w.limit = ph.limiter == 1;
    w.V = V;
    w.U0 = U0;
    w.out = out;
    w.fw = r.fw;
    w.smax = r.smax;
    w.dt = r.dt;
    w.elem_norm = k == 1 ? r.elem_norm : nullptr;
    w.counters = w.limit ? r.counters : nullptr;
    w.dt_factor = r.dt_factor;
    w.a = a;
    w.b = b;
    e = element_pass(m, ph, w, st);
    if (e != cudaSuccess || ph.limiter != 2) return e;
    return gen_superbee_launch(m, ph, out, r.share, r.means, r.scale, r.counters, st);
  };
  for (int i = 0; i < n_steps; ++i) {
    cudaError_t e = cudaSuccess;
    if (!r.ssprk3) {
      e = stage(1, r.S0, nullptr, r.S0, 0.0, 1.0);  // an element writes only what it alone has read
    } else {
      e = stage(1, r.S0, nullptr, r.S2, 0.0, 1.0);
      if (e == cudaSuccess) e = stage(2, r.S2, r.S0, r.S1, 0.75, 0.25);
      if (e == cudaSuccess) e = stage(3, r.S1, r.S0, r.S0, 1.0 / 3.0, 2.0 / 3.0);
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t gen_update_launch(const nzb_gen_mesh& m, const nzb_physics& ph, const nzb_gen_update_args& a,
                              cudaStream_t st) {
  k_gen_update<<<blocks(m.n_elem), 128, 0, st>>>(m, ph, a.stage, a.dt_factor, a.a, a.b, a.V, a.U0, a.F, a.wave, a.dt,
                                                  a.out, a.partial);
  return cudaGetLastError();
}

cudaError_t gen_superbee_launch(const nzb_gen_mesh& m, const nzb_physics& ph, double* U, const double* share,
                                double* means, double* scale, unsigned long long* counters, cudaStream_t st) {
  k_gen_cell_means<<<blocks(m.n_elem), 128, 0, st>>>(m, U, means);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_gen_lim_scale<<<1, 1024, 0, st>>>(means, m.n_elem, scale);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  int bytes = 0;
  e = warp_smem(k_gen_superbee, m, &bytes);
  if (e != cudaSuccess) return e;
  k_gen_superbee<<<warp_blocks(m.n_elem), GEN_WARPS * 32, bytes, st>>>(m, ph, U, means, scale, share, counters);
  return cudaGetLastError();
}

cudaError_t gen_initial_launch(const nzb_gen_mesh& m, const nzb_physics& ph, const nzb_gen_initial_args& a,
                               cudaStream_t st) {
  const int bytes = GenInitSmem{m.np, m.nqv, a.ng}.total() * (int)sizeof(double);
  k_gen_initial_state<<<(unsigned)m.n_elem, 128, bytes, st>>>(m, ph, a);
  return cudaGetLastError();
}

cudaError_t gen_observables_launch(const nzb_gen_mesh& m, const nzb_physics& ph, const nzb_gen_obs_args& a,
                                   cudaStream_t st) {
  k_gen_observables<<<1, OBS_BT, 0, st>>>(m, ph, a);
  return cudaGetLastError();
}

cudaError_t gen_geometry_launch(const nzb_gen_mesh& m, const nzb_gen_geometry_args& a, cudaStream_t st) {
  const int bytes = GenGeoSmem{m.np, m.nqv, a.ng}.total() * (int)sizeof(double);
  if (bytes > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k_gen_elem_geometry, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
  }
  k_gen_elem_geometry<<<(unsigned)m.n_elem, 128, bytes, st>>>(m, a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (m.n_int + m.n_bnd > 0) k_gen_edge_geometry<<<blocks(m.n_int + m.n_bnd), 128, 0, st>>>(m, a);
  return cudaGetLastError();
}

}  // namespace nzb
