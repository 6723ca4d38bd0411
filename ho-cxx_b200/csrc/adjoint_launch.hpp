// adjoint_launch.hpp -- launchers of the discrete-adjoint kernels (adjoint.cu).
#pragma once

#include <cuda_runtime.h>

#include "adjoint_chain.cuh"
#include "fr_launch.hpp"

namespace ho2d {

// ---- stage adjoint (one launch per body; the launches run in this order)
template <typename T>
cudaError_t launch_residual_adjoint(int K, const FrGeom<T>& g, const DevBases<T>& b, const StageAdjArgs<T>& a,
                                    cudaStream_t s);
template <typename T>
cudaError_t launch_velocity_adjoint(int K, const FrGeom<T>& g, const DevBases<T>& b, const StageAdjArgs<T>& a,
                                    cudaStream_t s);
// out = dir + transposed traces of the incoming slots sv (values) and sg (normal derivatives)
template <typename T>
cudaError_t launch_gather(int K, int N, const DevBases<T>& b, const T* dir, const T* sv, const T* sg, T* out,
                          cudaStream_t s);

// ---- vector helpers (FP64)
// out = a x + c y (out may alias x or y)
cudaError_t launch_axpby(size_t n, double* out, double a, const double* x, double c, const double* y, cudaStream_t s);
// y = x (FP32 -> FP64)
cudaError_t launch_copy_f2d(const float* x, double* y, size_t n, cudaStream_t s);
// out = x - J .* mu
cudaError_t launch_sub_scaled(size_t n, double* out, const double* x, const double* J, const double* mu,
                              cudaStream_t s);

}  // namespace ho2d
