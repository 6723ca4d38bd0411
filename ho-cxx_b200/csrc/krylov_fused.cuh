// krylov_fused.cuh -- a whole BiCGSTAB solve of a small mesh as one kernel (sm_100a).
//
// On a small mesh an iteration of the captured solve (krylov.cu) is a chain of nine to
// fifteen dependent launches that each work for a microsecond or two: launch gaps and the
// tails of the grid reductions are the solve. Here one resident grid (cooperative launch)
// keeps the chain inside a kernel, with a grid barrier where a launch boundary was. The
// phases are those kernels' bodies on the same element tiles, in the same order:
//   fine smoothing + restriction | coarse levels | z and its traces | operator | update
// What bounds it is latency: a barrier (about 1.3 us) and one or two L2 round trips a phase,
// 9 phases an iteration with a dense level 0, 13 with one level below it. An iteration on the
// 16 x 16 cavity at K = 4 takes 32 us, 43 as launches.
// A dot product is one partial sum per CTA; after the barrier every CTA adds all of them in
// the same order, so the scalars are the same bits everywhere and need no broadcast. The
// operator's, the update's and the smoothing's partial sums have buffers of their own
// (2 x grid doubles each): a CTA that is ahead never writes where another still reads.
//
// Memory. What the kernel itself writes is read with ld.cg (L2): another CTA may have written
// it, and L1 is not coherent. The static data (metrics, tables, factors) keep the read-only
// path. Every CTA has at most one tile; its smoother element data are copied into shared
// memory once and stay there for the whole solve.
//
// A barrier's wait is bounded: when it runs out, the CTA records it (dev_error, which the host
// reports) and returns, and so does every other CTA.
#pragma once

#include <algorithm>

#include "fr_launch.hpp"
#include "rows_transpose.cuh"
#include "smoother.cuh"

namespace ho2d {

namespace {

// The line between this kernel and the captured loop of launches, both measured on uniform
// cavities (ms for 16 solves, loop / one kernel). It pays while every SM has at most one tile:
// K = 4 FP64 8 tiles 12.9 / 9.4, 113 tiles 16.4 / 14.6, 145 tiles 17.1 / 15.2, 200 tiles
// 17.4 / 17.6; K = 3 FP64 123 tiles 14.4 / 13.6, 149 tiles 14.4 / 15.0; K = 5 mixed 141 tiles
// 25.1 / 23.1. At low order the coarse levels outgrow the tiles: K = 2 mixed 4,096 vertices
// 10.1 / 9.6, 7,921 vertices (127 tiles) 10.2 / 10.8.
constexpr int kFusedMaxCoarse = 6144;
// Smallest grid: CTAs without an element tile still work on the coarse levels. 20 solves on the
// 16 x 16 cavity, K = 4: 66 ms with 8 CTAs, 47.8 with 32, 43.9 with 64, 44.7 with 100, 46.6 with
// 148; coupled step on 24 x 96 elements 21.0, 20.8, 19.7, 18.7, 18.9 ms.
constexpr int kFusedMinGrid = 96;
constexpr int kSmemPerCta = 227 * 1024;

constexpr unsigned kBarrierPolls = 1u << 22;  // about a second of L2 round trips

// ---- loads of data that this kernel writes
template <typename T>
__device__ __forceinline__ T ldm(const T* p) {
    return __ldcg(p);
}

template <int K, typename T>
__device__ __forceinline__ void ldm_row(const T* p, T (&v)[K]) {
    if constexpr (sizeof(T) == 4 && K % 4 == 0) {
#pragma unroll
        for (int i = 0; i < K; i += 4) {
            const float4 q = __ldcg(reinterpret_cast<const float4*>(p + i));
            v[i] = q.x;
            v[i + 1] = q.y;
            v[i + 2] = q.z;
            v[i + 3] = q.w;
        }
    } else if constexpr (sizeof(T) == 4 && K % 2 == 0) {
#pragma unroll
        for (int i = 0; i < K; i += 2) {
            const float2 q = __ldcg(reinterpret_cast<const float2*>(p + i));
            v[i] = q.x;
            v[i + 1] = q.y;
        }
    } else if constexpr (sizeof(T) == 8 && K % 2 == 0) {
#pragma unroll
        for (int i = 0; i < K; i += 2) {
            const double2 q = __ldcg(reinterpret_cast<const double2*>(p + i));
            v[i] = q.x;
            v[i + 1] = q.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < K; ++i) v[i] = __ldcg(p + i);
    }
}

template <typename T>
__device__ __forceinline__ void ldm4(const T* p, T (&v)[4]) {
    ldm_row<4, T>(p, v);
}

// Grid barrier: bar[0] counts arrivals, and barrier number `epoch` of the solve is passed once
// it reaches base + epoch x grid. (A count that only grows needs one release and one acquire
// a barrier; resetting it and publishing a generation cost two more L2 round trips, 3 us in
// all against 1.3.) False: the wait ran out here or in another CTA.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned target, int* dev_error, bool& s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned n = 0, c;
        bool ok = true;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(bar) : "memory");
            if ((int)(c - target) >= 0) break;
            if (++n > kBarrierPolls) {
                atomicExch(dev_error, 1);
                ok = false;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok;
}

// out[j] = the sum over the CTAs of partials[j][.], the same in every CTA and thread.
template <int NV, int NT>
__device__ __forceinline__ void sum_partials(const double* partials, double (&out)[NV], double (&red)[NV][NT / 32]) {
    const int G = (int)gridDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        double x = 0.0;
        for (int i = threadIdx.x; i < G; i += NT) x += __ldcg(&partials[j * G + i]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
        if (lane == 0) red[j][warp] = x;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) x += red[j][w];
        out[j] = x;
    }
    __syncthreads();
}

// This CTA's partial sums (published by the barrier that follows).
template <int NV, int NT>
__device__ __forceinline__ void store_partials(const double (&v)[NV], double* partials, double (&red)[NV][NT / 32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        double x = v[j];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
        if (lane == 0) red[j][warp] = x;
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) x += red[threadIdx.x][w];
        partials[threadIdx.x * gridDim.x + blockIdx.x] = x;
    }
    __syncthreads();
}

// rows of y = A xa (+ B xb) over the whole grid, G lanes per row; x is written in this kernel
template <typename T>
__device__ __forceinline__ T ell_row(const DevEll<T>& A, const T* x, int row, int sub, int G) {
    T acc = T(0);
#pragma unroll 4
    for (int k = sub; k < A.w; k += G) {
        const size_t e = (size_t)row * A.w + k;
        acc += __ldg(A.val + e) * ldm(x + __ldg(A.col + e));
    }
    return acc;
}

template <typename T>
__device__ __forceinline__ void coarse_rows(const DevEll<T>& A, const T* xa, const DevEll<T>* B, const T* xb, T* y) {
    const int G = A.g, nthreads = gridDim.x * blockDim.x, gid = blockIdx.x * blockDim.x + threadIdx.x;
    const int sub = gid % G, ngroups = nthreads / G, iters = (A.n + ngroups - 1) / ngroups;
    for (int it = 0; it < iters; ++it) {
        const int row = gid / G + it * ngroups;
        const bool ok = row < A.n;
        T a = ok ? ell_row(A, xa, row, sub, G) : T(0);
        if (B && ok) a += ell_row(*B, xb, row, sub, G);
        for (int off = G >> 1; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
        if (sub == 0 && ok) y[row] = a;
    }
}

// u = W f for the dense coarsest inverse: one warp per row
template <typename T>
__device__ __forceinline__ void dense_rows(const DevEll<T>& W, const T* f, T* u) {
    const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < W.n; row += nw) {
        T acc = T(0);
        if (W.val16) {
            const unsigned short* wr = W.val16 + (size_t)row * W.w;
#pragma unroll 8
            for (int k = lane; k < W.n; k += 32) acc += T(__uint_as_float((unsigned)__ldg(wr + k) << 16)) * ldm(f + k);
        } else {
            const T* wr = W.val + (size_t)row * W.w;
#pragma unroll 16
            for (int k = lane; k < W.n; k += 32) acc += __ldg(wr + k) * ldm(f + k);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
        if (lane == 0) u[row] = acc;
    }
}

// Bytes of shared memory that hold one CTA's smoother element data for the whole solve.
template <int K, typename T, int BS>
constexpr int resident_bytes() {
    return Rows<K>::EPC * PostRows<K, T, BS>::ELEM;
}

// The solve. BS: the smoother's element data (smoother.cuh); TR: the transposed operator (v.b
// is the right-hand side and x starts at zero). CTA b works on element tile b alone, whose
// smoother data stay in its shared memory (fused_launch: at least as many CTAs as tiles).
template <int K, typename T, int BS, bool TR>
__global__ void __launch_bounds__(Rows<K>::THREADS, sizeof(T) == 4 ? 3 : 1)
    k_fused_solve(const __grid_constant__ MfOp<T> op, const __grid_constant__ BicgVectors<T> v,
                  const __grid_constant__ Precond<T> pc, ReduceScratch rs, unsigned* bar, int max_iter) {
    using R = Rows<K>;
    using PS = PostRows<K, T, BS>;
    using DT = typename PS::DT;
    constexpr int K2 = R::K2, NT = R::THREADS;
    extern __shared__ __align__(16) unsigned char res_dyn[];
    __shared__ RowScratch<K, T> sm[R::WARPS];
    __shared__ double red[2][NT / 32];
    __shared__ bool s_ok;
    KrylovScalars* sc = rs.sc;
    const int N = op.g.N, ntiles = (N + R::EPC - 1) / R::EPC, tile = blockIdx.x;  // at most one tile a CTA
    const int d = pc.nlev - 1;  // -1: no coarse level
    const double tol = __ldcg(&sc->tol);
    const unsigned char* el_data = BS == 2 ? reinterpret_cast<const unsigned char*>(op.kron_f)
                                 : BS == 1 ? reinterpret_cast<const unsigned char*>(op.dinv_bf16)
                                           : reinterpret_cast<const unsigned char*>(op.dinv);
    {
        const int e0 = blockIdx.x * R::EPC, ne = max(0, min(R::EPC, N - e0));
        const uint4* src = reinterpret_cast<const uint4*>(el_data + (size_t)e0 * PS::ELEM);
        uint4* dst = reinterpret_cast<uint4*>(res_dyn);
#pragma unroll 4
        for (int i = threadIdx.x; i < ne * (PS::ELEM / 16); i += NT) dst[i] = __ldg(src + i);
        __syncthreads();
    }
    double rho = 0.0, rho_old = 1.0, alpha = 1.0, omega = 1.0, rnorm2 = 0.0, bnorm2 = 0.0, eps2 = 0.0;
    int it = 0, s_exit = 0, breakdown = 0, zero_rhs = 0;
    bool done = false;
    // bar[1]: the count at the end of the previous solve, written by its CTA 0
    unsigned target = __ldcg(bar + 1);
    auto sync = [&]() { return grid_barrier(bar, target += gridDim.x, &sc->dev_error, s_ok); };

    // traces of x, the initial residual's operand
    if constexpr (!TR) {
        if (tile < ntiles) {
            const RowIdx<K> ix(N, tile);
            T row[K];
            int dst[4];
            if (ix.active) {
                ldm_row<K, T>(v.x + (size_t)ix.el * K2 + ix.t * K, row);
                load4i(op.g.scat + ((size_t)ix.el * K + ix.t) * 4, dst);
            }
            row_emit_traces<K, T>(op.b, sm[ix.warp].tr[0][ix.lw], row, dst, v.xtv, v.xtg, ix.t, ix.active);
            __syncwarp();
        }
        if (!sync()) return;
    }

    // mode 2: the initial residual; 0: v = A ph; 1: t = A sh
    for (int mode = 2;;) {
        double part[2] = {0.0, 0.0};
        if (tile < ntiles) {
            const RowIdx<K> ix(N, tile);
            const size_t p = (size_t)ix.el * K2 + ix.t * K;
            T y[K], q[K];
            if constexpr (TR) {
                if (ix.active) ldm_row<K, T>(mode == 2 ? v.b + p : (mode == 0 ? v.rhat : v.s) + p, q);
                if (mode != 2) {
                    // the gather over the own part that the z phase left in v or t
                    T tv[4] = {T(0), T(0), T(0), T(0)}, tg[4] = {T(0), T(0), T(0), T(0)};
                    if (ix.active) {
                        const size_t q4 = ((size_t)ix.el * K + ix.t) * 4;
                        ldm4<T>(v.tv + q4, tv);
                        ldm4<T>(v.tg + q4, tg);
                        ldm_row<K, T>((mode == 0 ? v.v : v.t) + p, y);
                    }
                    transpose_traces<K, T>(op.b, tv, tg, sm[ix.warp].tr[0][ix.lw], ix, y);
                } else {
#pragma unroll
                    for (int i = 0; i < K; ++i) y[i] = T(0);
                }
            } else {
                const T* x = mode == 2 ? v.x : (mode == 0 ? v.ph : v.sh);
                const T *tv = mode == 2 ? v.xtv : v.tv, *tg = mode == 2 ? v.xtg : v.tg;
                ApplyIn<K, T> in;
                row_apply_static<K, T>(op.g, ix, in);
                if (ix.active) {
                    const size_t q4 = ((size_t)ix.el * K + ix.t) * 4;
                    ldm_row<K, T>(x + p, in.xr);
#pragma unroll
                    for (int j = 0; j < K; ++j) in.xc[j] = ldm(x + (size_t)ix.el * K2 + j * K + ix.t);
                    ldm4<T>(tv + q4, in.ntv);
                    ldm4<T>(tg + q4, in.ntg);
                } else {
#pragma unroll
                    for (int i = 0; i < K; ++i) in.xr[i] = in.xc[i] = T(0);
#pragma unroll
                    for (int f = 0; f < 4; ++f) in.ntv[f] = in.ntg[f] = T(0);
                }
                row_apply_core<K, T>(op, in, sm[ix.warp], ix, y);
                if (ix.active) ldm_row<K, T>(mode == 2 ? v.b + p : (mode == 0 ? v.rhat : v.s) + p, q);
            }
            if (ix.active) {
                if (mode == 2) {
                    T zero[K];
#pragma unroll
                    for (int i = 0; i < K; ++i) {
                        y[i] = q[i] - y[i];  // r
                        zero[i] = T(0);
                        part[0] += double(y[i]) * double(y[i]);
                        part[1] += double(q[i]) * double(q[i]);
                    }
                    store_row<K, T>(v.r + p, y);
                    store_row<K, T>(v.rhat + p, y);
                    if (TR) store_row<K, T>(v.x + p, zero);
                } else {
                    store_row<K, T>((mode == 0 ? v.v : v.t) + p, y);
#pragma unroll
                    for (int i = 0; i < K; ++i) {
                        part[0] += double(y[i]) * double(q[i]);
                        part[1] += double(y[i]) * double(y[i]);
                    }
                }
            }
            if (mode != 1) element_moments<K, T>(v.h, y, sm[ix.warp].com[ix.lw], ix, mode == 2 ? v.er : v.ev);
        }
        store_partials<2, NT>(part, rs.partials, red);
        if (!sync()) return;
        double out[2];
        sum_partials<2, NT>(rs.partials, out, red);
        if (mode == 2) {
            rnorm2 = rho = out[0];
            bnorm2 = out[1];
            eps2 = tol * tol * out[1];
            zero_rhs = out[1] == 0.0;
            done = zero_rhs || out[0] <= eps2 || (TR && !isfinite(out[0]));
            mode = 0;
        } else if (mode == 0) {
            if (out[0] == 0.0 || rho == 0.0 || (TR && !isfinite(out[0]))) {
                breakdown = 1;
                done = true;
            } else {
                alpha = rho / out[0];
            }
            mode = 1;
        } else {
            omega = out[1] > 0.0 ? out[0] / out[1] : 0.0;
            mode = 3;
        }
        if (done) break;
    update:
        if (mode == 3) {  // x, r and the end of the iteration
            double up[2] = {0.0, 0.0};
            if (tile < ntiles) {
                const RowIdx<K> ix(N, tile);
                const size_t p = (size_t)ix.el * K2 + ix.t * K;
                T r[K];
                if (ix.active) {
                    T x[K], ph[K];
                    ldm_row<K, T>(v.x + p, x);
                    ldm_row<K, T>(v.ph + p, ph);
                    if (s_exit) {
#pragma unroll
                        for (int i = 0; i < K; ++i) x[i] = x[i] + T(alpha) * ph[i];
                    } else {
                        T sh[K], sv[K], tv[K], rh[K];
                        ldm_row<K, T>(v.sh + p, sh);
                        ldm_row<K, T>(v.s + p, sv);
                        ldm_row<K, T>(v.t + p, tv);
                        ldm_row<K, T>(v.rhat + p, rh);
#pragma unroll
                        for (int i = 0; i < K; ++i) {
                            x[i] = x[i] + (T(alpha) * ph[i] + T(omega) * sh[i]);
                            r[i] = sv[i] - T(omega) * tv[i];
                            up[0] += double(r[i]) * double(r[i]);
                            up[1] += double(rh[i]) * double(r[i]);
                        }
                        store_row<K, T>(v.r + p, r);
                    }
                    store_row<K, T>(v.x + p, x);
                }
                if (!s_exit) element_moments<K, T>(v.h, r, sm[ix.warp].com[ix.lw], ix, v.er);
            }
            it += 1;
            if (s_exit) break;  // rnorm2 is already ||s||^2
            store_partials<2, NT>(up, rs.partials + 2 * gridDim.x, red);
            if (!sync()) return;
            sum_partials<2, NT>(rs.partials + 2 * gridDim.x, out, red);
            rnorm2 = out[0];
            rho_old = rho;
            rho = out[1];
            if (out[0] <= eps2 || it >= max_iter || omega == 0.0) done = true;
            if (sizeof(T) == 4 && !(out[0] <= 1e12 * bnorm2)) done = true;
            if (!isfinite(out[0])) done = true;
            if (done) break;
            mode = 0;
        }
        // fine smoothing of p (mode 0) or s (mode 1), and the restriction beside it
        F0<T> f0;
        f0.a = v.er;
        f0.b = f0.c = v.er;
        f0.cb = f0.cc = T(0);
        const double beta = (rho / rho_old) * (alpha / omega);
        if (mode == 1) {
            f0.b = v.ev;
            f0.cb = T(-alpha);
        } else if (it > 0) {
            f0.b = v.ep[it & 1];
            f0.c = v.ev;
            f0.cb = T(beta);
            f0.cc = T(-beta * omega);
        }
        auto moment = [&](int e) { return ldm(f0.a + e) + f0.cb * ldm(f0.b + e) + f0.cc * ldm(f0.c + e); };
        double sp[2] = {0.0, 0.0};
        if (tile < ntiles) {
            const RowIdx<K> ix(N, tile);
            const int t = ix.t, el = ix.el;
            const size_t p = (size_t)el * K2 + t * K;
            T f[K];
            if (ix.active) {
                T rr[K];
                ldm_row<K, T>(v.r + p, rr);
                if (mode == 0 && it == 0) {
#pragma unroll
                    for (int i = 0; i < K; ++i) f[i] = rr[i];
                } else {
                    T vv[K];
                    ldm_row<K, T>(v.v + p, vv);
                    if (mode == 0) {
                        T pp[K];
                        ldm_row<K, T>(v.p + p, pp);
#pragma unroll
                        for (int i = 0; i < K; ++i) f[i] = rr[i] + T(beta) * (pp[i] - T(omega) * vv[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < K; ++i) f[i] = rr[i] - T(alpha) * vv[i];
                    }
                }
                store_row<K, T>((mode == 0 ? v.p : v.s) + p, f);
#pragma unroll
                for (int i = 0; i < K; ++i) {
                    sm[ix.warp].tr[0][ix.lw][t][i] = f[i];
                    sp[0] += double(f[i]) * double(f[i]);
                }
                if (mode == 0 && d >= 0)
                    for (int c = t; c < 4; c += K) v.ep[(it + 1) & 1][el * 4 + c] = moment(el * 4 + c);
            }
            __syncwarp();
            const unsigned char* data = res_dyn + (size_t)(ix.warp * R::EPW + ix.lw) * PS::ELEM;
            int kx = -1;
            if constexpr (BS == 2) {
                if (ix.active) kx = __ldg(op.kron_x + el);
            }
            T acc[K];
            smoother_rows<K, T, BS>(op, reinterpret_cast<const DT*>(data), reinterpret_cast<const T*>(data), kx,
                                    &sm[ix.warp].tr[0][ix.lw][0][0], sm[ix.warp].tr[1][ix.lw], t, ix.active, acc);
            if (ix.active) store_row<K, T>(v.zf + p, acc);
            __syncwarp();  // the scratch is rewritten by the next phase
        }
        if (d >= 0) {
            T* f = pc.lev[0].f;
            const int n0 = pc.lev[0].n;
            for (int r = blockIdx.x * NT + threadIdx.x; r < n0; r += gridDim.x * NT) {
                T acc = T(0);
                for (int k = 0; k < pc.vw; ++k) {
                    const int e = __ldg(pc.v2e + (size_t)r * pc.vw + k);
                    if (e >= 0) acc += moment(e);
                }
                f[r] = acc;
            }
        }
        if (mode == 1) store_partials<2, NT>(sp, rs.partials + 4 * gridDim.x, red);
        if (!sync()) return;
        if (mode == 1) {
            sum_partials<2, NT>(rs.partials + 4 * gridDim.x, out, red);
            if (out[0] <= eps2) {
                s_exit = 1;
                rnorm2 = out[0];
                mode = 3;
                goto update;
            }
        }
        // coarse levels
        for (int l = 0; l < d; ++l) {
            coarse_rows<T>(pc.lev[l].M, pc.lev[l].f, nullptr, nullptr, pc.lev[l + 1].f);
            if (!sync()) return;
        }
        if (d >= 0) {
            dense_rows<T>(pc.dense, pc.lev[d].f, pc.lev[d].u);
            if (!sync()) return;
        }
        for (int l = d - 1; l >= 0; --l) {
            coarse_rows<T>(pc.lev[l].S, pc.lev[l].f, &pc.lev[l].Q, pc.lev[l + 1].u, pc.lev[l].u);
            if (!sync()) return;
        }
        // z = P u0 + w zf, its traces (or its own part of A^T z)
        if (tile < ntiles) {
            const RowIdx<K> ix(N, tile);
            const int t = ix.t;
            const size_t p = (size_t)ix.el * K2 + t * K;
            T z[K];
            int dst[4];
#pragma unroll
            for (int i = 0; i < K; ++i) z[i] = T(0);
            if (ix.active) {
                T f[K], l = T(0), r = T(0);
                ldm_row<K, T>(v.zf + p, f);
                load4i(op.g.scat + ((size_t)ix.el * K + t) * 4, dst);
                if (d >= 0) {
                    int c[4];
                    load4i(pc.conn + (size_t)ix.el * 4, c);
                    T u[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) u[k] = c[k] >= 0 ? ldm(pc.lev[0].u + c[k]) : T(0);
                    const T y0 = v.h.hp[t * 2 + 0], y1 = v.h.hp[t * 2 + 1];
                    l = u[0] * y0 + u[3] * y1;
                    r = u[1] * y0 + u[2] * y1;
                }
#pragma unroll
                for (int i = 0; i < K; ++i)
                    z[i] = (l * v.h.hp[i * 2 + 0] + r * v.h.hp[i * 2 + 1]) + T(pc.omega) * f[i];
                store_row<K, T>((mode == 0 ? v.ph : v.sh) + p, z);
            }
            if constexpr (TR) {
                T own[K];
                row_transpose_own<K, T>(op, z, sm[ix.warp], ix, v.tv, v.tg, own);
                if (ix.active) store_row<K, T>((mode == 0 ? v.v : v.t) + p, own);
            } else {
                row_emit_traces<K, T>(op.b, sm[ix.warp].tr[0][ix.lw], z, dst, v.tv, v.tg, t, ix.active);
                __syncwarp();
            }
        }
        if (!sync()) return;
    }
    // a zero right-hand side has a zero solution
    if (zero_rhs)
        for (size_t i = (size_t)blockIdx.x * NT + threadIdx.x; i < (size_t)N * K2; i += (size_t)gridDim.x * NT)
            v.x[i] = T(0);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        bar[1] = target;
        sc->rho = rho;
        sc->rho_old = rho_old;
        sc->alpha = alpha;
        sc->omega = omega;
        sc->rnorm2 = rnorm2;
        sc->bnorm2 = bnorm2;
        sc->eps2 = eps2;
        sc->it = it;
        sc->breakdown = breakdown;
        sc->s_exit = s_exit;
        sc->zero_rhs = zero_rhs;
        sc->done = 1;
    }
}

// Launches the solve when the mesh fits: a tile for each CTA of the resident grid.
template <int K, typename T, int BS, bool TR>
cudaError_t fused_launch(const MfOp<T>& op, const BicgVectors<T>& v, const FusedScratch& fs, int max_iter,
                         const Precond<T>& pc, KrylovScalars* sc, cudaStream_t s, bool* fits) {
    *fits = false;
    constexpr int dyn = resident_bytes<K, T, BS>();
    if constexpr (dyn + (int)sizeof(RowScratch<K, T>) * Rows<K>::WARPS + 1024 <= kSmemPerCta) {
        auto kern = k_fused_solve<K, T, BS, TR>;
        cudaError_t e;
        int dev = 0, sms = 0, nb = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn)) != cudaSuccess) return e;
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, Rows<K>::THREADS, dyn)) != cudaSuccess)
            return e;
        const int tiles = (op.g.N + Rows<K>::EPC - 1) / Rows<K>::EPC, cap = std::min(nb * sms, kFusedMaxGrid);
        if (cap < kFusedMinGrid || tiles > std::min(cap, sms) || (pc.nlev > 0 && pc.lev[0].n > kFusedMaxCoarse))
            return cudaSuccess;
        *fits = true;
        cudaLaunchConfig_t cfg = {};
        // at least a warp for every row of the dense level, and kFusedMinGrid for the others
        const int rows = pc.nlev > 0 ? (pc.dense.n + Rows<K>::WARPS - 1) / Rows<K>::WARPS : 0;
        cfg.gridDim = dim3((unsigned)std::min(cap, std::max(std::max(tiles, rows), kFusedMinGrid)));
        cfg.blockDim = dim3(Rows<K>::THREADS);
        cfg.dynamicSmemBytes = dyn;
        cfg.stream = s;
        cudaLaunchAttribute at = {};
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        const ReduceScratch rs{fs.partials, nullptr, sc};
        return cudaLaunchKernelEx(&cfg, kern, op, v, pc, rs, fs.bar, max_iter);
    }
    return cudaSuccess;
}

#define HO2D_FUSED_SWITCH(K, CALL)                         \
    switch (K) {                                           \
        case 2: { constexpr int KK = 2; return CALL; }     \
        case 3: { constexpr int KK = 3; return CALL; }     \
        case 4: { constexpr int KK = 4; return CALL; }     \
        case 5: { constexpr int KK = 5; return CALL; }     \
        case 6: { constexpr int KK = 6; return CALL; }     \
        default: *fits = false; return cudaSuccess;        \
    }

}  // namespace
}  // namespace ho2d
