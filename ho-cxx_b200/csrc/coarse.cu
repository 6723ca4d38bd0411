// coarse.cu -- the coarse part of the two-level Poisson preconditioner (sm_100a).
//
// Level 0 is the coarse space itself: one value per mesh vertex off the Dirichlet boundary,
// interpolated bilinearly in each element (order 1: one value per element). Its
// smoothed-aggregation hierarchy is built on the host (host_amg.cpp) down to a level of at
// most kDenseMax rows, whose inverse is precomputed. One V(1,1) cycle with SPAI-0 smoothing
// is linear in f, so every level's cycle is stored as three fixed row-padded operators,
//   f_next = M f,   u = S f + Q u_next,
// and a cycle is a chain of matrix-vector products with no intermediate residual or
// correction vectors:
//   restriction  f_0[v] = the element moments that meet in v   (k_vertex_rhs)
//   downs    f_{l+1} = M_l f_l              l = 0 .. d-1       (k_coarse_rows)
//   coarsest u_d = A_d^{-1} f_d                                (k_dense_gemv)
//   ups      u_l = S_l f_l + Q_l u_{l+1}    l = d-1 .. 0       (k_coarse_rows)
// The combination (krylov.cu, k_post_b) reads u_0 at each element's four corners.
//
// The moments (element_moments in rows.cuh) are kept by the kernels that write the
// residual vectors, so the cycle reads 4 values per element and runs beside the fine
// smoothing on a second stream. What bounds it is latency: four to six dependent launches
// over a few hundred KB to a few MB each, all L2-resident.
//
// Every kernel spans all SMs and sums in a fixed order (fixed lane-to-entry assignment
// and xor-shuffle trees), so results are bitwise reproducible.
#include <type_traits>

#include "device.cuh"
#include "fr_launch.hpp"

namespace ho2d {

namespace {

constexpr int kRowBatch = 2;  // rows a lane group works on at once
constexpr int kChunks = 4;    // row chunks of G entries loaded before any is used

// acc[r] += A_row[r] . x over the row chunks of one lane. All kRowBatch x kChunks loads
// of a step are issued before the first gather, so a lane keeps that many L2 requests in
// flight instead of waiting once per chunk.
template <typename T, typename X>
__device__ __forceinline__ void ell_accumulate(const DevEll<T>& A, const X& x, const int (&row)[kRowBatch],
                                               const bool (&ok)[kRowBatch], int G, int sub, T (&acc)[kRowBatch]) {
    const int w = A.w;
    const int nch = (w + G - 1) / G;
    for (int c0 = 0; c0 < nch; c0 += kChunks) {
        T v[kRowBatch][kChunks];
        int j[kRowBatch][kChunks];
#pragma unroll
        for (int r = 0; r < kRowBatch; ++r)
#pragma unroll
            for (int u = 0; u < kChunks; ++u) {
                const int k = (c0 + u) * G + sub;
                const bool in = ok[r] && k < w;
                const size_t e = in ? (size_t)row[r] * w + k : 0;
                v[r][u] = in ? A.val[e] : T(0);
                j[r][u] = in ? A.col[e] : 0;
            }
#pragma unroll
        for (int r = 0; r < kRowBatch; ++r)
#pragma unroll
            for (int u = 0; u < kChunks; ++u) acc[r] += v[r][u] * x[j[r][u]];
    }
}

// grid-wide down (f_next = M f) or up (u = S f + Q u_next): G lanes per row, the group's
// lanes combine their partial sums with an xor-shuffle tree.
template <typename T>
__global__ void __launch_bounds__(256) k_coarse_rows(DevEll<T> A, const T* __restrict__ xa, DevEll<T> B,
                                                      const T* __restrict__ xb,
                                                      int has_b, T* __restrict__ y, const KrylovScalars* sc) {
    const bool skip = sc->done;  // read early: the round trip overlaps the loads
    const int G = A.g;
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    const int group = gid / G, sub = gid % G, ngroups = (int)(gridDim.x * blockDim.x) / G;
    const int iters = (A.n + ngroups - 1) / ngroups;
    for (int it = 0; it < iters; it += kRowBatch) {
        T acc[kRowBatch];
        int row[kRowBatch];
        bool ok[kRowBatch];
#pragma unroll
        for (int r = 0; r < kRowBatch; ++r) {
            acc[r] = T(0);
            row[r] = group + (it + r) * ngroups;
            ok[r] = it + r < iters && row[r] < A.n;
        }
        ell_accumulate<T>(A, xa, row, ok, G, sub, acc);
        if (has_b) ell_accumulate<T>(B, xb, row, ok, G, sub, acc);
#pragma unroll
        for (int r = 0; r < kRowBatch; ++r) {
            T a = acc[r];
            for (int off = G >> 1; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
            if (sub == 0 && ok[r] && !skip) y[row[r]] = a;
        }
    }
}

// 16-byte vector of T
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
    using type = float4;
    static constexpr int N = 4;
    __device__ static float dot(const float4& a, const float4& b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
    // zero the components at and past `keep` (the tail of a vector that ends inside a piece)
    __device__ static void keep_first(float4& v, int keep) {
        if (keep < 4) v.w = 0.f;
        if (keep < 3) v.z = 0.f;
        if (keep < 2) v.y = 0.f;
    }
};
template <>
struct Vec16<double> {
    using type = double2;
    static constexpr int N = 2;
    __device__ static double dot(const double2& a, const double2& b) { return a.x * b.x + a.y * b.y; }
    __device__ static void keep_first(double2& v, int keep) {
        if (keep < 2) v.y = 0.0;
    }
};

constexpr int kGemvWarps = 8;  // rows (one warp each) per CTA
constexpr int kGemvUnroll = 8;

// u = W f for the dense coarsest inverse W (rows padded to w, a multiple of 4 entries):
// one warp per row, lanes stream the row in 16-byte pieces with kGemvUnroll loads in
// flight; f is read in the same pieces (its buffer is zero-padded past n).
template <typename T>
__global__ void __launch_bounds__(32 * kGemvWarps) k_dense_gemv(DevEll<T> W, const T* __restrict__ f,
                                                                 T* __restrict__ u, const KrylovScalars* sc) {
    using V = Vec16<T>;
    using VT = typename V::type;
    const bool skip = sc->done;
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * kGemvWarps + (threadIdx.x >> 5);
    if (row >= W.n) return;
    const int nvec = (W.n + V::N - 1) / V::N;
    const int tail = W.n - (nvec - 1) * V::N;  // entries of the last piece inside the vector
    const VT* wr = reinterpret_cast<const VT*>(W.val + (size_t)row * W.w);
    const VT* fv = reinterpret_cast<const VT*>(f);
    T acc = T(0);
    for (int c0 = lane; c0 < nvec; c0 += 32 * kGemvUnroll) {
        VT a[kGemvUnroll], b[kGemvUnroll];
#pragma unroll
        for (int q = 0; q < kGemvUnroll; ++q) {
            const int c = c0 + 32 * q;
            if (c < nvec) {
                a[q] = __ldg(wr + c);
                b[q] = __ldg(fv + c);
                // the padding of f is zero when written in this precision, but a buffer
                // shared by both precisions may hold the other one's bytes there
                if (c == nvec - 1) V::keep_first(b[q], tail);
            }
        }
#pragma unroll
        for (int q = 0; q < kGemvUnroll; ++q)
            if (c0 + 32 * q < nvec) acc += V::dot(a[q], b[q]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0 && !skip) u[row] = acc;
}

// u = W f for the dense coarsest inverse stored as BF16 (FP32 preconditioner): one warp per
// row, lanes stream the row in 16-byte pieces of 8 values with kGemvUnroll loads in flight;
// f is read as two float4 per piece (its buffer is zero-padded past n to a multiple of 8).
__global__ void __launch_bounds__(32 * kGemvWarps) k_dense_gemv16(DevEll<float> W, const float* __restrict__ f,
                                                                   float* __restrict__ u, const KrylovScalars* sc) {
    const bool skip = sc->done;
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * kGemvWarps + (threadIdx.x >> 5);
    if (row >= W.n) return;
    const int nvec = (W.n + 7) / 8;
    const int tail = W.n - (nvec - 1) * 8;  // values of the last piece inside the vector
    const uint4* wr = reinterpret_cast<const uint4*>(W.val16 + (size_t)row * W.w);
    const float4* fv = reinterpret_cast<const float4*>(f);
    float acc = 0.f;
    for (int c0 = lane; c0 < nvec; c0 += 32 * kGemvUnroll) {
        uint4 a[kGemvUnroll];
        float4 b0[kGemvUnroll], b1[kGemvUnroll];
#pragma unroll
        for (int q = 0; q < kGemvUnroll; ++q) {
            const int c = c0 + 32 * q;
            if (c < nvec) {
                a[q] = __ldg(wr + c);
                b0[q] = __ldg(fv + 2 * c);
                b1[q] = __ldg(fv + 2 * c + 1);
                if (c == nvec - 1) {  // a buffer shared by both precisions may hold other bytes there
                    Vec16<float>::keep_first(b0[q], tail);
                    Vec16<float>::keep_first(b1[q], tail - 4);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < kGemvUnroll; ++q) {
            if (c0 + 32 * q >= nvec) continue;
            const unsigned w4[4] = {a[q].x, a[q].y, a[q].z, a[q].w};
            const float fx[8] = {b0[q].x, b0[q].y, b0[q].z, b0[q].w, b1[q].x, b1[q].y, b1[q].z, b1[q].w};
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                acc += __uint_as_float(w4[h] << 16) * fx[2 * h];
                acc += __uint_as_float(w4[h] & 0xffff0000u) * fx[2 * h + 1];
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0 && !skip) u[row] = acc;
}

template <typename T>
void dense_gemv(const DevEll<T>& W, const T* f, T* u, const KrylovScalars* sc, cudaStream_t s) {
    const unsigned gd = (unsigned)((W.n + kGemvWarps - 1) / kGemvWarps);
    if constexpr (std::is_same<T, float>::value) {
        if (W.val16) {
            k_dense_gemv16<<<gd, 32 * kGemvWarps, 0, s>>>(W, f, u, sc);
            return;
        }
    }
    k_dense_gemv<T><<<gd, 32 * kGemvWarps, 0, s>>>(W, f, u, sc);
}

// the element moments that meet in level-0 unknown r, summed in the table's order
template <typename T>
__device__ __forceinline__ T vertex_sum(const int* __restrict__ v2e, int vw, const F0<T>& m, int r) {
    T acc = T(0);
    for (int k = 0; k < vw; ++k) {
        const int e = __ldg(v2e + (size_t)r * vw + k);
        if (e >= 0) acc += m[e];
    }
    return acc;
}

// f_0 from the element moments, one thread per unknown
template <typename T>
__global__ void __launch_bounds__(256) k_vertex_rhs(int n, const int* __restrict__ v2e, int vw, BicgVectors<T> v,
                                                     T* __restrict__ f, const KrylovScalars* sc, int mode) {
    const bool skip = sc->done;  // read early: the round trip overlaps the loads
    const F0<T> m = f0_of(v, sc, mode);
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const T a = vertex_sum<T>(v2e, vw, m, r);
    if (!skip) f[r] = a;
}

// u_0 = W f_0 when level 0 itself is the dense one (small meshes): every CTA forms f_0 in its
// shared memory (n values of T), then one warp per row. One launch instead of two: at 225
// unknowns the extra reads (a few KB per CTA, L2-resident) cost less than a launch.
template <typename T>
__global__ void __launch_bounds__(32 * kGemvWarps) k_dense_gemv_f0(DevEll<T> W, const int* __restrict__ v2e, int vw,
                                                                    BicgVectors<T> v, T* __restrict__ u,
                                                                    const KrylovScalars* sc, int mode) {
    extern __shared__ __align__(16) unsigned char f0_dyn[];
    T* f = reinterpret_cast<T*>(f0_dyn);
    const bool skip = sc->done;
    const F0<T> m = f0_of(v, sc, mode);
    for (int r = threadIdx.x; r < W.n; r += 32 * kGemvWarps) f[r] = vertex_sum<T>(v2e, vw, m, r);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * kGemvWarps + (threadIdx.x >> 5);
    if (row >= W.n) return;
    const T* wr = W.val + (size_t)row * W.w;
    T acc = T(0);
#pragma unroll 8
    for (int k = lane; k < W.n; k += 32) acc += __ldg(wr + k) * f[k];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0 && !skip) u[row] = acc;
}

// largest dense level 0 whose right-hand side every CTA forms for itself (the shared memory
// a launch gets without asking)
constexpr size_t kGemvF0Bytes = 48 * 1024;

template <typename T>
unsigned rows_grid(const DevEll<T>& A) {
    const long long lanes = (long long)A.n * A.g;
    const long long per_block = 256;
    long long blocks = (lanes + per_block * kRowBatch - 1) / (per_block * kRowBatch);
    return (unsigned)(blocks < 1 ? 1 : blocks);
}

}  // namespace

template <typename T>
static bool gemv_forms_f0(const Precond<T>& pc) {
    return pc.nlev == 1 && (size_t)pc.dense.n * sizeof(T) <= kGemvF0Bytes;
}

template <typename T>
cudaError_t coarse_cycle(const Precond<T>& pc, const BicgVectors<T>& v, const KrylovScalars* sc, int mode,
                         cudaStream_t s) {
    if (gemv_forms_f0(pc)) {
        const unsigned gd = (unsigned)((pc.dense.n + kGemvWarps - 1) / kGemvWarps);
        k_dense_gemv_f0<T><<<gd, 32 * kGemvWarps, pc.dense.n * sizeof(T), s>>>(pc.dense, pc.v2e, pc.vw, v, pc.lev[0].u, sc,
                                                                               mode);
        return cudaGetLastError();
    }
    const int n0 = pc.lev[0].n, d = pc.nlev - 1;
    k_vertex_rhs<T><<<(unsigned)((n0 + 255) / 256), 256, 0, s>>>(n0, pc.v2e, pc.vw, v, pc.lev[0].f, sc, mode);
    for (int l = 0; l < d; ++l) {
        const CoarseLevel<T>& L = pc.lev[l];
        k_coarse_rows<T><<<rows_grid(L.M), 256, 0, s>>>(L.M, L.f, DevEll<T>(), nullptr, 0, pc.lev[l + 1].f, sc);
    }
    dense_gemv<T>(pc.dense, pc.lev[d].f, pc.lev[d].u, sc, s);
    for (int l = d - 1; l >= 0; --l) {
        const CoarseLevel<T>& L = pc.lev[l];
        k_coarse_rows<T><<<rows_grid(L.S), 256, 0, s>>>(L.S, L.f, L.Q, pc.lev[l + 1].u, 1, L.u, sc);
    }
    return cudaGetLastError();
}

template <typename T>
int coarse_launches(const Precond<T>& pc) {
    if (pc.nlev <= 0) return 0;
    return gemv_forms_f0(pc) ? 1 : 2 * pc.nlev;
}

// Algorithmic bytes of one coarse cycle as coarse_cycle launches it: the element moments (p's
// and s's are combinations of up to three vectors) and the restriction table, every
// row-padded operator's values and column indices, the dense inverse, each level's
// right-hand side read and result written.
template <typename T>
double coarse_cycle_bytes(const Precond<T>& pc) {
    if (pc.nlev <= 0) return 0.0;
    const int d = pc.nlev - 1;
    auto ell = [](const DevEll<T>& A) { return (double)A.n * A.w * (sizeof(T) + (A.col ? 4 : 0)); };
    const double dsz = pc.dense.val16 ? 2.0 : (double)sizeof(T);
    const int n0 = pc.lev[0].n;
    double b = (double)n0 * pc.vw * (4.0 + 3.0 * sizeof(T)) + (double)n0 * sizeof(T);
    b += (double)pc.dense.n * pc.dense.w * dsz + 2.0 * pc.dense.n * sizeof(T);
    for (int l = 0; l < d; ++l) {
        b += ell(pc.lev[l].M) + (double)(pc.lev[l].n + pc.lev[l + 1].n) * sizeof(T);
        b += ell(pc.lev[l].S) + ell(pc.lev[l].Q) + (double)(2 * pc.lev[l].n + pc.lev[l + 1].n) * sizeof(T);
    }
    return b;
}

#define HO2D_INSTANTIATE_COARSE(T)                                                                   \
    template cudaError_t coarse_cycle<T>(const Precond<T>&, const BicgVectors<T>&, const KrylovScalars*, int,  \
                                         cudaStream_t);                                                      \
    template int coarse_launches<T>(const Precond<T>&);                                              \
    template double coarse_cycle_bytes<T>(const Precond<T>&);

HO2D_INSTANTIATE_COARSE(double)
HO2D_INSTANTIATE_COARSE(float)

}  // namespace ho2d
