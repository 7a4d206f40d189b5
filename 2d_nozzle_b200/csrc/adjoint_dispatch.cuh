// adjoint_dispatch.cuh -- launchers of the adjoint kernels, one translation unit
// per element kind (adjoint_tri.cu, adjoint_quad.cu) so the dual-number kernels
// compile in parallel.  Each unit holds its own copy of the reference-element
// tables in constant memory; nzb_upload_tables fills every copy.
#pragma once
#include <cuda_runtime.h>

#include "adjoint.cuh"

#ifndef NZB_INTERNAL
#define NZB_INTERNAL __attribute__((visibility("hidden")))
#endif

namespace nzb {

NZB_INTERNAL cudaError_t vjp_launch_tri(const nzb_mesh& m, const nzb_physics& ph, const AdjWork& w, cudaStream_t st);
NZB_INTERNAL cudaError_t vjp_launch_quad(const nzb_mesh& m, const nzb_physics& ph, const AdjWork& w, cudaStream_t st);
NZB_INTERNAL cudaError_t vjp_coords_launch_tri(const nzb_mesh& m, const nzb_physics& ph, const CoordWork& w,
                                               cudaStream_t st);
NZB_INTERNAL cudaError_t vjp_coords_launch_quad(const nzb_mesh& m, const nzb_physics& ph, const CoordWork& w,
                                                cudaStream_t st);
// the face Jacobians of a linearisation (adjoint_tile.cuh) and the doubles they take (0: no such array)
NZB_INTERNAL cudaError_t vjp_jac_launch_tri(const nzb_mesh& m, const nzb_physics& ph, const double* U, double* jac,
                                            cudaStream_t st);
NZB_INTERNAL cudaError_t vjp_jac_launch_quad(const nzb_mesh& m, const nzb_physics& ph, const double* U, double* jac,
                                             cudaStream_t st);
NZB_INTERNAL int64_t vjp_jac_doubles_tri(int order, int64_t n_elem);
NZB_INTERNAL int64_t vjp_jac_doubles_quad(int order, int64_t n_elem);
// build and upload one order's tile fragments from its table slot (current device)
NZB_INTERNAL cudaError_t upload_tiles_vjp_tri(int order, const double* slot);
NZB_INTERNAL cudaError_t upload_tiles_vjp_quad(int order, const double* slot);
NZB_INTERNAL cudaError_t upload_tables_tri(const double* src, size_t count, size_t offset);
NZB_INTERNAL cudaError_t upload_tables_quad(const double* src, size_t count, size_t offset);

}  // namespace nzb
