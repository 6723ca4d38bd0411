// adjoint.cu -- kernels of the discrete adjoint of the FR stage (sm_100a).
//
//   k_residual_adjoint   reverse of residual_kernel (diffusion + advection type 1)
//   k_velocity_adjoint   reverse of velocity_kernel and update_diffusion_BC
//   k_gather             own part + transposed traces of the incoming slots
//
// The transposed Poisson solve runs on the forward solver's kernels (krylov.cu,
// rows_transpose.cuh). Element kernels here: K^2 threads per element, AShape<K>::EPB elements
// per CTA, every element's scratch in shared memory (adjoint_chain.cuh holds the bodies).
#include <cmath>

#include "adjoint_launch.hpp"
#include "fr_device.cuh"

namespace ho2d {

namespace {

#define HO2D_ADJ_DISPATCH_K(K, CALL)                      \
    switch (K) {                                          \
        case 1: { constexpr int KK = 1; CALL; } break;     \
        case 2: { constexpr int KK = 2; CALL; } break;     \
        case 3: { constexpr int KK = 3; CALL; } break;     \
        case 4: { constexpr int KK = 4; CALL; } break;     \
        case 5: { constexpr int KK = 5; CALL; } break;     \
        case 6: { constexpr int KK = 6; CALL; } break;     \
        case 7: { constexpr int KK = 7; CALL; } break;     \
        case 8: { constexpr int KK = 8; CALL; } break;     \
        default: return cudaErrorInvalidValue;            \
    }

template <int K>
unsigned agrid(int N) {
    return (unsigned)((N + AShape<K>::EPB - 1) / AShape<K>::EPB);
}

// ---------------------------------------------------------------- stage adjoint
template <int K, typename T>
__global__ void __launch_bounds__(AShape<K>::THREADS) k_residual_adjoint(FrGeom<T> g, DevBases<T> bp,
                                                                          StageAdjArgs<T> a) {
    using S = AShape<K>;
    __shared__ DevBases<T> b;
    __shared__ ResidualAdjScratch<K, T> sm[S::EPB];
    stage_bases(b, bp);
    __syncthreads();
    const int le = threadIdx.x / S::K2, ij = threadIdx.x % S::K2;
    const int el = blockIdx.x * S::EPB + le;
    const bool active = le < S::EPB && el < g.N;
    residual_adjoint_body<K, T>(ElemCtx<S::K2>{ij}, active, el, g, b, a, sm[active ? le : 0]);
}

template <int K, typename T>
__global__ void __launch_bounds__(AShape<K>::THREADS) k_velocity_adjoint(FrGeom<T> g, DevBases<T> bp,
                                                                          StageAdjArgs<T> a) {
    using S = AShape<K>;
    __shared__ DevBases<T> b;
    __shared__ VelocityAdjScratch<K, T> sm[S::EPB];
    stage_bases(b, bp);
    __syncthreads();
    const int le = threadIdx.x / S::K2, ij = threadIdx.x % S::K2;
    const int el = blockIdx.x * S::EPB + le;
    const bool active = le < S::EPB && el < g.N;
    velocity_adjoint_body<K, T>(ElemCtx<S::K2>{ij}, active, el, g, b, a, sm[active ? le : 0]);
}

// ---------------------------------------------------------------- psi gather
template <int K, typename T>
__global__ void __launch_bounds__(AShape<K>::THREADS) k_gather(int N, DevBases<T> bp, const T* __restrict__ dir,
                                                                const T* __restrict__ sv, const T* __restrict__ sg,
                                                                T* __restrict__ out) {
    using S = AShape<K>;
    __shared__ DevBases<T> b;
    __shared__ GatherScratch<K, T> sm[S::EPB];
    stage_bases(b, bp);
    __syncthreads();
    const int le = threadIdx.x / S::K2, ij = threadIdx.x % S::K2;
    const int el = blockIdx.x * S::EPB + le;
    const bool active = le < S::EPB && el < N;
    gather_body<K, T>(ElemCtx<S::K2>{ij}, active, el, b, dir, sv, sg, out, sm[active ? le : 0]);
}

// ---------------------------------------------------------------- vector helpers
__global__ void k_axpby(size_t n, double* out, double a, const double* x, double c, const double* y) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = a * x[i] + c * y[i];
}

__global__ void k_sub_scaled(size_t n, double* out, const double* x, const double* J, const double* mu) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = x[i] - J[i] * mu[i];
}

__global__ void k_copy_f2d(size_t n, const float* x, double* y) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) y[i] = double(x[i]);
}

unsigned vec_grid(size_t n) {
    const size_t b = (n + 255) / 256;
    return (unsigned)(b < 1 ? 1 : (b > 4 * 148 ? 4 * 148 : b));
}

}  // namespace

// ---------------------------------------------------------------- launchers
template <typename T>
cudaError_t launch_residual_adjoint(int K, const FrGeom<T>& g, const DevBases<T>& b, const StageAdjArgs<T>& a,
                                    cudaStream_t s) {
    HO2D_ADJ_DISPATCH_K(K, (k_residual_adjoint<KK, T><<<agrid<KK>(g.N), AShape<KK>::THREADS, 0, s>>>(g, b, a)));
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_velocity_adjoint(int K, const FrGeom<T>& g, const DevBases<T>& b, const StageAdjArgs<T>& a,
                                    cudaStream_t s) {
    HO2D_ADJ_DISPATCH_K(K, (k_velocity_adjoint<KK, T><<<agrid<KK>(g.N), AShape<KK>::THREADS, 0, s>>>(g, b, a)));
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_gather(int K, int N, const DevBases<T>& b, const T* dir, const T* sv, const T* sg, T* out,
                          cudaStream_t s) {
    HO2D_ADJ_DISPATCH_K(K, (k_gather<KK, T><<<agrid<KK>(N), AShape<KK>::THREADS, 0, s>>>(N, b, dir, sv, sg, out)));
    return cudaGetLastError();
}

cudaError_t launch_axpby(size_t n, double* out, double a, const double* x, double c, const double* y, cudaStream_t s) {
    k_axpby<<<vec_grid(n), 256, 0, s>>>(n, out, a, x, c, y);
    return cudaGetLastError();
}

cudaError_t launch_sub_scaled(size_t n, double* out, const double* x, const double* J, const double* mu,
                              cudaStream_t s) {
    k_sub_scaled<<<vec_grid(n), 256, 0, s>>>(n, out, x, J, mu);
    return cudaGetLastError();
}

cudaError_t launch_copy_f2d(const float* x, double* y, size_t n, cudaStream_t s) {
    k_copy_f2d<<<vec_grid(n), 256, 0, s>>>(n, x, y);
    return cudaGetLastError();
}

template cudaError_t launch_residual_adjoint<double>(int, const FrGeom<double>&, const DevBases<double>&,
                                                     const StageAdjArgs<double>&, cudaStream_t);
template cudaError_t launch_velocity_adjoint<double>(int, const FrGeom<double>&, const DevBases<double>&,
                                                     const StageAdjArgs<double>&, cudaStream_t);

template cudaError_t launch_gather<double>(int, int, const DevBases<double>&, const double*, const double*, const double*,
                                           double*, cudaStream_t);

}  // namespace ho2d
