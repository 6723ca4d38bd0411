// krylov.cu -- matrix-free FR Poisson operator and preconditioned BiCGSTAB (sm_100a).
//
// Operator. The reference assembles the FR Laplacian into a CSR matrix with up to
// 5 K^4 entries per element (src/HO_2D.cpp:1533-1804, 3011-3062) and hands it to AMGCL.
// That matrix is exactly the method-2 FR Laplacian of calc_RHS_diffusion applied with
// homogeneous Poisson boundary values, so here A x is evaluated matrix-free from face
// traces (row_apply in rows.cuh): per DOF it reads x, 3 metric coefficients and a share
// of the face data instead of 5 K^2 matrix entries. Every kernel that produces
// a vector the operator is applied to next also writes that vector's face traces, so
// one operator application is one launch.
//
// Solver. Right-preconditioned BiCGSTAB (van der Vorst 1992) replacing AMGCL's BiCGSTAB
// (src/HO_2D.hpp:53-54, src/HO_2D.cpp:1960). Preconditioner, two-level and additive:
//   z = P A1^{-1} R f + w D^{-1} f,
// P = continuous bilinear interpolation from the mesh vertices, R = its transpose times the
// quadrature weights, A1 = the bilinear finite-element Laplacian on the vertices
// (host_amg.cpp), A1^{-1} approximated by one smoothed-aggregation V-cycle, D = the
// K^2 x K^2 diagonal blocks of A. (Two-level methods for discontinuous schemes with this
// coarse space: Dobrev, Lazarov, Vassilevski, Zikatanov 2006.) The vertices carry the
// element's linear modes, which element-wise constants leave to the smoother, and because
// P u has no jumps the sum needs no A P u: the smoothing and the coarse cycle are
// independent, and the combination reads four values per element.
// With HO2D_PRECOND=bj the preconditioner is z = w D^{-1} f (block-Jacobi).
// Scalars stay on the device; every vector update fuses the dot products the next step
// needs, reduced deterministically (per-CTA partials summed in a fixed order by the last
// CTA to finish); a `done` flag turns the rest of an enqueued batch into no-ops, so the
// host only polls for convergence every few iterations.
#include <type_traits>

#include "device.cuh"
#include "fr_device.cuh"
#include "fr_launch.hpp"
#include "kron_apply.cuh"
#include "rows.cuh"
#include "smoother.cuh"
#include "rows_transpose.cuh"
#include "apply_stage.cuh"
#include "bulk_copy.cuh"

namespace ho2d {

namespace {

// Deterministic grid-wide sum of NV values per thread, in two levels so no CTA reads more
// than a few hundred partials: every CTA stores its sums; the last CTA to finish within
// each group of kReduceGroup consecutive CTAs adds the group's sums (fixed order) and
// stores the group total; the last group to finish adds the group totals (fixed order)
// and gets `out`, returning true in that CTA only. Counters: counter[0] for the groups,
// counter[1 + g] for group g; every one is back to zero when the kernel ends. partials
// holds NV x (gridDim.x + the number of groups) doubles. Collective (all threads).
constexpr int kReduceGroup = 64;

template <int NV>
__device__ __forceinline__ bool grid_reduce(const double (&v)[NV], double* partials, unsigned* counter,
                                            double (&out)[NV]) {
    __shared__ double red[NV][32];
    __shared__ double fin[NV];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int G = (int)gridDim.x, ng = (G + kReduceGroup - 1) / kReduceGroup;
    const int grp = (int)blockIdx.x / kReduceGroup;
    const int g0 = grp * kReduceGroup, gs = min(kReduceGroup, G - g0);
    double* gpart = partials + (size_t)NV * G;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        double x = v[j];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
        if (lane == 0) red[j][warp] = x;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            double x = lane < nw ? red[j][lane] : 0.0;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
            if (lane == 0) partials[j * G + blockIdx.x] = x;
        }
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(&counter[1 + grp], 1u) == (unsigned)gs - 1);
    __syncthreads();
    if (!s_last) return false;
    // the group's total: warp 0 adds its <= 64 CTA sums (lanes l and l + 32, then a tree)
    __threadfence();
    if (warp == 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            double x = lane < gs ? __ldcg(&partials[j * G + g0 + lane]) : 0.0;
            if (lane + 32 < gs) x += __ldcg(&partials[j * G + g0 + lane + 32]);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
            if (lane == 0) gpart[j * ng + grp] = x;
        }
        if (lane == 0) counter[1 + grp] = 0u;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(&counter[0], 1u) == (unsigned)ng - 1);
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        double x = 0.0;
#pragma unroll 4
        for (int i = threadIdx.x; i < ng; i += blockDim.x) x += __ldcg(&gpart[j * ng + i]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
        if (lane == 0) red[j][warp] = x;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            double x = lane < nw ? red[j][lane] : 0.0;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
            if (lane == 0) fin[j] = x;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NV; ++j) out[j] = fin[j];
    if (threadIdx.x == 0) counter[0] = 0u;
    return true;
}

}  // namespace

// ---------------------------------------------------------------- fine-level kernels
// The operator kernels run row-parallel (rows.cuh): K threads per element, Rows<K>::EPC
// elements per CTA.
template <int K>
static __host__ __device__ constexpr unsigned rgrid_of(int N) {
    return (unsigned)((N + Rows<K>::EPC - 1) / Rows<K>::EPC);
}

// Resident CTAs an SM that the operator kernels' registers are cut down to. In the iteration
// (k_mf_v, k_mf_t) FP32 takes four (128 registers). FP64 takes three (168) up to order 7: without a
// limit the compiler takes 162 to 252, and two CTAs are left to hide the loads; at orders 6 and 7
// three spill 140 to 230 bytes and still win. Order 8 would spill 320 and 410 bytes and keeps its
// 238 registers. us per launch of k_mf_v / k_mf_t in FP64 with two CTAs and with three: K = 3 on
// 400 x 400 elements 61.8 / 46.7 and 49.1 / 36.4, K = 4 (340^2) 67.9 / 53.3 and 55.8 / 42.7, K = 5
// (320^2) 80.4 / 65.2 and 63.8 / 51.4, K = 6 (256^2) 67.0 / 57.3 and 63.3 / 49.5, K = 7 (224^2)
// 70.0 / 60.0 and 66.0 / 59.5, K = 8 (200^2) 69.4 / 65.8 and 73.3 / 75.9. (Four CTAs spill
// everywhere: K = 6 on 256 x 512 elements 146 against 116.)
template <int K, typename T>
constexpr int kOperatorCtas = sizeof(T) == 4 ? 4 : (K <= 7 ? 3 : 1);
// The residuals (k_mf_init, k_mf_residual): three in FP64 at orders 6 and 7 (k_mf_init with two and with
// three, the same meshes: 66.5 and 60.2 us, 71.0 and 67.3), elsewhere the compiler's own choice (0),
// which stops at 168 registers up to order 5 and at 128 at order 2, where any stated minimum takes
// 160 (500^2 elements: 42.3 us, 47.2 with it), and does not spill at order 8 (72.1, 81.7 with three).
template <int K, typename T>
constexpr int kResidualCtas = sizeof(T) == 8 && (K == 6 || K == 7) ? 3 : 0;

// CTAs of one full wave of each reducing row kernel (resident CTAs per SM x SMs), per K and
// precision ([K][0] FP64, [K][1] FP32): those kernels loop over element tiles, so one wave
// covers any mesh and each CTA reduces once. Set by krylov_configure.
struct WaveSizes {
    unsigned init = 0, v = 0, t = 0, xr = 0, res = 0, v_st = 0, t_st = 0, tr = 0;
};
static WaveSizes g_wave[9][2];

template <int K, typename T>
static unsigned wave_of(unsigned WaveSizes::*which, int N) {
    const unsigned w = g_wave[K][std::is_same<T, float>::value ? 1 : 0].*which;
    const unsigned nt = rgrid_of<K>(N);
    return w == 0 || w > nt ? nt : w;
}

// incoming face traces of x (the operand of an operator application that no Krylov
// kernel produced: the initial guess, a refinement iterate, a caller's vector)
template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS) k_trace_in(MfOp<T> op, const T* __restrict__ x, T* __restrict__ tv,
                                                                T* __restrict__ tg) {
    asm volatile("griddepcontrol.launch_dependents;");  // (k_mf_apply, where it follows)
    __shared__ T buf[Rows<K>::WARPS][Rows<K>::EPW][K][K];
    const RowIdx<K> ix(op.g.N, blockIdx.x);
    T row[K];
    int dst[4];
    if (ix.active) {
        load_row<K, T>(x + (size_t)ix.el * K * K + ix.t * K, row);
        load4i(op.g.scat + ((size_t)ix.el * K + ix.t) * 4, dst);
    }
    row_emit_traces<K, T>(op.b, buf[ix.warp][ix.lw], row, dst, tv, tg, ix.t, ix.active);
}

// r = b - A x (x's traces in xtv/xtg), rhat = r; ||r||^2, ||b||^2; element moments of r. Like
// every reducing row kernel it runs as one wave of CTAs, each taking element tiles
// blockIdx.x, blockIdx.x + gridDim.x, ... and reducing once.
template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS, kResidualCtas<K, T>) k_mf_init(MfOp<T> op, BicgVectors<T> v, ReduceScratch rs) {
    __shared__ RowScratch<K, T> sm[Rows<K>::WARPS];
    const int ntiles = (int)rgrid_of<K>(op.g.N);
    double part[2] = {0.0, 0.0};
    auto tile_body = [&](int tile) {
        const RowIdx<K> ix(op.g.N, tile);
        T y[K], r[K];
        row_apply<K, T>(op, v.x, v.xtv, v.xtg, sm[ix.warp], ix, y);
        if (ix.active) {
            const size_t p = (size_t)ix.el * K * K + ix.t * K;
            T bb[K];
            load_row<K, T>(v.b + p, bb);
#pragma unroll
            for (int i = 0; i < K; ++i) {
                r[i] = bb[i] - y[i];
                part[0] += double(r[i]) * double(r[i]);
                part[1] += double(bb[i]) * double(bb[i]);
            }
            store_row<K, T>(v.r + p, r);
            store_row<K, T>(v.rhat + p, r);
        }
        element_moments<K, T>(v.h, r, sm[ix.warp].com[ix.lw], ix, v.er);
    };
    // FP32: one wave of CTAs over the tiles; FP64 keeps one tile per CTA (the loop would
    // push the operator past the register file)
    if constexpr (sizeof(T) == 4) {
#pragma unroll 1
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) tile_body(tile);
    } else {
        if ((int)blockIdx.x < ntiles) tile_body(blockIdx.x);
    }
    double out[2];
    if (grid_reduce<2>(part, rs.partials, rs.counter, out) && threadIdx.x == 0) {
        KrylovScalars* sc = rs.sc;
        sc->rnorm2 = out[0];
        sc->bnorm2 = out[1];
        sc->eps2 = sc->tol * sc->tol * out[1];
        sc->rho = out[0];
        sc->rho_old = sc->alpha = sc->omega = 1.0;
        sc->beta = 0.0;
        sc->it = 0;
        sc->breakdown = 0;
        sc->s_exit = 0;
        sc->zero_rhs = out[1] == 0.0;
        sc->done = (out[1] == 0.0) || (out[0] <= sc->eps2);
    }
}

template <typename T>
__global__ void k_zero_if(T* x, size_t n, const KrylovScalars* sc) {
    if (!sc->zero_rhs) return;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = T(0);
}


// The warp's smoother element data: one bulk copy of its EPW inverse blocks (or factor
// sets) into its slice of the dynamic shared memory when PostRows::kStage, issued by lane 0
// on barrier bar; blk/fk point at this element's data (staged or global).
template <int K, typename T, int BS>
struct SmootherData {
    const typename PostRows<K, T, BS>::DT* blk = nullptr;
    const T* fk = nullptr;
    int kx = -1;
    int wn = 0;
    __device__ __forceinline__ void start(const MfOp<T>& op, const RowIdx<K>& ix, unsigned char* dyn, uint64_t* bar,
                                          bool issue) {
        using PS = PostRows<K, T, BS>;
        using DT = typename PS::DT;
        constexpr int EPW = Rows<K>::EPW;
        const DT* dsrc;
        if constexpr (BS == 1) dsrc = op.dinv_bf16;
        else dsrc = op.dinv;
        const int wel0 = (blockIdx.x * Rows<K>::WARPS + ix.warp) * EPW;
        wn = min(EPW, op.g.N - wel0);
        blk = dsrc + (size_t)(ix.active ? ix.el : 0) * PS::STRIDE;
        fk = BS == 2 ? op.kron_f + (size_t)(ix.active ? ix.el : 0) * PS::KFS : nullptr;
        if constexpr (BS == 2) {
            if (ix.active) kx = op.kron_x[ix.el];
        }
        if constexpr (PS::kStage) {
            unsigned char* stage = dyn + (size_t)ix.warp * PS::SPAN;
            if (issue && wn > 0 && ix.lane == 0) {
                const unsigned char* src = BS == 2 ? reinterpret_cast<const unsigned char*>(op.kron_f)
                                                   : reinterpret_cast<const unsigned char*>(dsrc);
                mbar_init(bar);
                const unsigned bytes = (unsigned)(wn * PS::ELEM);
                mbar_arrive_expect(bar, bytes);
                bulk_load(stage, src + (size_t)wel0 * PS::ELEM, bytes, bar);
            }
            if constexpr (BS == 2) fk = reinterpret_cast<const T*>(stage + (size_t)ix.lw * PS::ELEM);
            else blk = reinterpret_cast<const DT*>(stage + (size_t)ix.lw * PS::ELEM);
        }
    }
    // wait for the copy; a wait that runs out is recorded for the host, the copy gets a
    // second bounded wait, and the kernel runs on so its reductions stay consistent
    __device__ __forceinline__ void wait(uint64_t* bar, KrylovScalars* sc, int lane) {
        if constexpr (PostRows<K, T, BS>::kStage) {
            if (wn > 0 && !mbar_wait_bounded(bar, 0, kBulkWaitPolls)) {
                if (lane == 0) atomicExch(&sc->dev_error, 1);
                mbar_wait_bounded(bar, 0, kBulkWaitPolls);
            }
        }
    }
};

// Fine part of one preconditioner application, with the BiCGSTAB vector update that
// produces its operand:
//   mode 0:  p = r + beta (p - omega v)  (p = r on the first iteration),  f = p
//   mode 1:  s = r - alpha v, ||s||^2 (s_exit test),                      f = s
// then zf = M f with the smoother's element inverse M (exact FP32/FP64 block, BF16 block or
// Kronecker-sum factors). It needs nothing of the coarse cycle, which runs beside it on a
// second stream; k_post_b combines the two. Mode 0 also stores the element moments of the new
// p for the next iteration. Row-parallel (rows.cuh): thread t of an element owns row t. The
// warp's element data are requested first, by one bulk copy into shared memory
// (PostRows::kStage), so the copy overlaps the vector loads.
template <int K, typename T, int BS = 0>
__global__ void __launch_bounds__(Rows<K>::THREADS) k_post_a(MfOp<T> op, BicgVectors<T> v, int has_coarse,
                                                              ReduceScratch rs, int mode) {
    using R = Rows<K>;
    constexpr int K2 = R::K2, EPW = R::EPW;
    KrylovScalars* sc = rs.sc;
    const int done = sc->done;  // uniform; read early so the round trip overlaps the loads
    extern __shared__ __align__(128) unsigned char post_dyn[];
    __shared__ __align__(8) uint64_t bar[R::WARPS];
    __shared__ __align__(16) T sr[R::WARPS][EPW][K2];
    __shared__ T zb[R::WARPS][EPW][K][K];
    const RowIdx<K> ix(op.g.N, blockIdx.x);
    const int t = ix.t, lw = ix.lw, el = ix.el;
    const bool act = ix.active;
    SmootherData<K, T, BS> sd;
    sd.start(op, ix, post_dyn, &bar[ix.warp], !done);
    const size_t p = (size_t)el * K2 + t * K;
    T rr[K], vv[K], pp[K];
    if (act) {
        load_row<K, T>(v.r + p, rr);
        load_row<K, T>(v.v + p, vv);
        if (mode == 0) load_row<K, T>(v.p + p, pp);
    }
    if (mode == 0 && has_coarse && act) {
        const F0<T> f0 = f0_of(v, sc, mode);
        for (int c = t; c < 4; c += K) v.ep[(sc->it + 1) & 1][el * 4 + c] = f0[el * 4 + c];
    }
    // the operand: p or s
    T f[K];
    if (mode == 0) {
        if (sc->it == 0) {
#pragma unroll
            for (int i = 0; i < K; ++i) f[i] = rr[i];
        } else {
            const double beta = (sc->rho / sc->rho_old) * (sc->alpha / sc->omega);
            const T om = T(sc->omega);
#pragma unroll
            for (int i = 0; i < K; ++i) f[i] = rr[i] + T(beta) * (pp[i] - om * vv[i]);
        }
    } else {
        const T al = T(sc->alpha);
#pragma unroll
        for (int i = 0; i < K; ++i) f[i] = rr[i] - al * vv[i];
    }
    if (done) return;  // uniform over the grid: no copy was issued
    if (act) {
        store_row<K, T>((mode == 0 ? v.p : v.s) + p, f);
#pragma unroll
        for (int i = 0; i < K; ++i) sr[ix.warp][lw][t * K + i] = f[i];
    }
    __syncwarp();
    sd.wait(&bar[ix.warp], sc, ix.lane);
    T acc[K];
    smoother_rows<K, T, BS>(op, sd.blk, sd.fk, sd.kx, sr[ix.warp][lw], zb[ix.warp][lw], t, act, acc);
    if (act) store_row<K, T>(v.zf + p, acc);
    if (mode == 1) {
        double part[1] = {0.0};
        if (act) {
#pragma unroll
            for (int i = 0; i < K; ++i) part[0] += double(f[i]) * double(f[i]);
        }
        double out[1];
        if (grid_reduce<1>(part, rs.partials, rs.counter, out) && threadIdx.x == 0) {
            sc->snorm2 = out[0];
            sc->s_exit = out[0] <= sc->eps2;
        }
    }
}

// The preconditioner application's result z = P u0 + w zf, row t of an element: the coarse
// function is bilinear in the element, so the thread interpolates its four corner values to
// the row's two ends and runs along the row between them. conn == nullptr: no coarse level.
template <int K, typename T>
__device__ __forceinline__ void combine_row(const HatBases<T>& h, const int* __restrict__ conn,
                                            const T* __restrict__ u0, const T* __restrict__ zf, T w, int el, int t,
                                            T (&z)[K]) {
    T f[K];
    load_row<K, T>(zf, f);
    T l = T(0), r = T(0);
    if (conn) {
        int c[4];
        load4i(conn + (size_t)el * 4, c);
        T u[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) u[q] = c[q] >= 0 ? u0[c[q]] : T(0);
        const T y0 = h.hp[t * 2 + 0], y1 = h.hp[t * 2 + 1];
        l = u[0] * y0 + u[3] * y1;
        r = u[1] * y0 + u[2] * y1;
    }
#pragma unroll
    for (int i = 0; i < K; ++i) z[i] = (l * h.hp[i * 2 + 0] + r * h.hp[i * 2 + 1]) + w * f[i];
}

// z of the preconditioner application and its face traces. Bound by HBM: zf read, z and the
// two trace buffers written; the four corner values are L2 reads shared by an element's
// threads.
template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS) k_post_b(MfOp<T> op, BicgVectors<T> v,
                                                              const int* __restrict__ conn,
                                                              const T* __restrict__ u0, double w,
                                                              const KrylovScalars* sc, int mode) {
    using R = Rows<K>;
    if (sc->done) return;  // uniform
    __shared__ T zb[R::WARPS][R::EPW][K][K];
    const RowIdx<K> ix(op.g.N, blockIdx.x);
    const size_t p = (size_t)ix.el * R::K2 + ix.t * K;
    T zz[K];
    int dst[4];
    if (ix.active) {
        load4i(op.g.scat + ((size_t)ix.el * K + ix.t) * 4, dst);
        combine_row<K, T>(v.h, conn, u0, v.zf + p, T(w), ix.el, ix.t, zz);
        store_row<K, T>((mode == 0 ? v.ph : v.sh) + p, zz);
    }
    row_emit_traces<K, T>(op.b, zb[ix.warp][ix.lw], zz, dst, v.tv, v.tg, ix.t, ix.active);
}

// The FP32 operator's tile loop with its inputs staged in shared memory (apply_stage.cuh):
// the copies of a warp's next tile are issued as soon as the lanes have read the current
// one, so they run under the current tile's arithmetic. body(ix, y, sec_row) finishes
// each tile. A copy whose wait runs out is recorded for the host (dev_error) and gets a
// second bounded wait; after that the warp issues no more copies and runs on, so the
// grid reduction stays consistent.
template <int K, typename Body>
__device__ __forceinline__ void staged_apply_loop(const MfOp<float>& op, const float* x, const float* tvin,
                                                  const float* tgin, const float* sec, RowScratch<K, float>* sm,
                                                  KrylovScalars* sc, Body body) {
    using S = ApplyStage<K>;
    using R = Rows<K>;
    extern __shared__ __align__(128) unsigned char apply_dyn[];
    __shared__ __align__(8) uint64_t bar[R::WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int N = op.g.N, ntiles = (int)rgrid_of<K>(N);
    float* st = reinterpret_cast<float*>(apply_dyn + (size_t)warp * S::WARP_BYTES);
    auto count = [&](int tile) {
        return tile < ntiles ? max(0, min(R::EPW, N - stage_first<K>(tile, warp))) : 0;
    };
    if (lane == 0) mbar_init(&bar[warp]);
    __syncwarp();
    if (lane == 0 && count(blockIdx.x) > 0)
        stage_issue<K>(st, &bar[warp], op.g, x, tvin, tgin, sec, stage_first<K>(blockIdx.x, warp), count(blockIdx.x));
    unsigned phase = 0;
    bool ok = true;
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const RowIdx<K> ix(N, tile);
        if (ok && count(tile) > 0) {
            if (!mbar_wait_bounded(&bar[warp], phase & 1u, kBulkWaitPolls)) {
                if (lane == 0) atomicExch(&sc->dev_error, 1);
                ok = mbar_wait_bounded(&bar[warp], phase & 1u, kBulkWaitPolls);
            }
            ++phase;
        }
        ApplyIn<K, float> in;
        float sr[K];
        stage_read<K>(st, op.g, x, sec, stage_first<K>(tile, warp), ix, in, sr);
        __syncwarp();  // every lane has read the slice
        const int next = tile + (int)gridDim.x;
        if (lane == 0 && ok && count(next) > 0) {
            stage_release();
            stage_issue<K>(st, &bar[warp], op.g, x, tvin, tgin, sec, stage_first<K>(next, warp), count(next));
        }
        float y[K];
        row_apply_core<K, float>(op, in, sm[warp], ix, y);
        body(ix, y, sr);
    }
}

// v = A ph; alpha = rho / (rhat, v); element moments of v. ST: the FP32 loop with staged
// inputs (dynamic shared memory ApplyStage<K>::CTA_BYTES).
// (registers: kOperatorCtas)
template <int K, typename T, bool ST = false>
__global__ void __launch_bounds__(Rows<K>::THREADS, kOperatorCtas<K, T>)
    k_mf_v(MfOp<T> op, BicgVectors<T> v, ReduceScratch rs) {
    KrylovScalars* sc = rs.sc;
    // the flag is uniform over the grid (only this kernel's last CTA writes it, after every
    // CTA has read it)
    if (sc->done) return;
    __shared__ RowScratch<K, T> sm[Rows<K>::WARPS];
    const int ntiles = (int)rgrid_of<K>(op.g.N);
    double part[1] = {0.0};
    auto finish = [&](const RowIdx<K>& ix, const T (&y)[K], const T (&rh)[K]) {
        if (ix.active) {
            const size_t p = (size_t)ix.el * K * K + ix.t * K;
            store_row<K, T>(v.v + p, y);
#pragma unroll
            for (int i = 0; i < K; ++i) part[0] += double(rh[i]) * double(y[i]);
        }
        element_moments<K, T>(v.h, y, sm[ix.warp].com[ix.lw], ix, v.ev);
    };
    auto tile_body = [&](int tile) {
        const RowIdx<K> ix(op.g.N, tile);
        T y[K];
        row_apply<K, T>(op, v.ph, v.tv, v.tg, sm[ix.warp], ix, y);
        T rh[K];
        if (ix.active) load_row<K, T>(v.rhat + (size_t)ix.el * K * K + ix.t * K, rh);
        finish(ix, y, rh);
    };
    if constexpr (ST && sizeof(T) == 4) {
        staged_apply_loop<K>(op, v.ph, v.tv, v.tg, v.rhat, sm, sc, finish);
    } else if constexpr (sizeof(T) == 4) {
        // FP32: one wave of CTAs over the tiles; FP64 keeps one tile per CTA (the loop
        // would push the operator past the register file)
#pragma unroll 1
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            if (tile + (int)gridDim.x < ntiles)
                prefetch_apply_rows<K, T>(op.g, v.ph, v.tv, v.tg, v.rhat, tile + gridDim.x);
            tile_body(tile);
        }
    } else {
        if ((int)blockIdx.x < ntiles) tile_body(blockIdx.x);
    }
    double out[1];
    if (grid_reduce<1>(part, rs.partials, rs.counter, out) && threadIdx.x == 0) {
        if (out[0] == 0.0 || sc->rho == 0.0) {
            sc->breakdown = 1;
            sc->done = 1;
        } else {
            sc->alpha = sc->rho / out[0];
        }
    }
}

// t = A sh; omega = (t, s) / (t, t). ST as in k_mf_v.
template <int K, typename T, bool ST = false>
__global__ void __launch_bounds__(Rows<K>::THREADS, kOperatorCtas<K, T>)
    k_mf_t(MfOp<T> op, BicgVectors<T> v, ReduceScratch rs) {
    KrylovScalars* sc = rs.sc;
    if (sc->done || sc->s_exit) return;  // uniform
    __shared__ RowScratch<K, T> sm[Rows<K>::WARPS];
    const int ntiles = (int)rgrid_of<K>(op.g.N);
    double part[2] = {0.0, 0.0};
    auto finish = [&](const RowIdx<K>& ix, const T (&y)[K], const T (&sv)[K]) {
        if (ix.active) {
            const size_t p = (size_t)ix.el * K * K + ix.t * K;
            store_row<K, T>(v.t + p, y);
#pragma unroll
            for (int i = 0; i < K; ++i) {
                part[0] += double(y[i]) * double(sv[i]);
                part[1] += double(y[i]) * double(y[i]);
            }
        }
    };
    auto tile_body = [&](int tile) {
        const RowIdx<K> ix(op.g.N, tile);
        T y[K];
        row_apply<K, T>(op, v.sh, v.tv, v.tg, sm[ix.warp], ix, y);
        T sv[K];
        if (ix.active) load_row<K, T>(v.s + (size_t)ix.el * K * K + ix.t * K, sv);
        finish(ix, y, sv);
    };
    if constexpr (ST && sizeof(T) == 4) {
        staged_apply_loop<K>(op, v.sh, v.tv, v.tg, v.s, sm, sc, finish);
    } else if constexpr (sizeof(T) == 4) {
        // FP32: one wave of CTAs over the tiles; FP64 keeps one tile per CTA (the loop
        // would push the operator past the register file)
#pragma unroll 1
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            if (tile + (int)gridDim.x < ntiles)
                prefetch_apply_rows<K, T>(op.g, v.sh, v.tv, v.tg, v.s, tile + gridDim.x);
            tile_body(tile);
        }
    } else {
        if ((int)blockIdx.x < ntiles) tile_body(blockIdx.x);
    }
    double out[2];
    if (grid_reduce<2>(part, rs.partials, rs.counter, out) && threadIdx.x == 0)
        sc->omega = out[1] > 0.0 ? out[0] / out[1] : 0.0;
}

// x += alpha ph + omega sh; r = s - omega t; ||r||^2, (rhat, r); element moments of r;
// convergence test. After an s-exit (||s|| already below tolerance) only x += alpha ph.
// The last CTA to finish ends the iteration: it updates the scalars, sets `done`, and
// inside a captured solve sets the condition of the graph's while node (iterate while
// not done). Every CTA reads `done` and `s_exit` before any CTA arrives at the counter,
// so the last CTA may change them. Every body execution either increments `it` (capped at
// max_iter) or finds `done` set and clears the condition, so the device loop always ends.
// Each thread updates element rows.
template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS) k_xr_update(int N, BicgVectors<T> v, ReduceScratch rs, int max_iter,
                                                                 cudaGraphConditionalHandle h, int has_handle) {
    __shared__ T mom[Rows<K>::WARPS][Rows<K>::EPW][4][K];
    KrylovScalars* sc = rs.sc;
    if (sc->done) {  // the solve ended earlier in this body (breakdown)
        if (has_handle && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(h, 0u);
        return;
    }
    const T alpha = T(sc->alpha);
    const bool s_exit = sc->s_exit;
    const double omega = sc->omega;
    const int ntiles = (int)rgrid_of<K>(N);
    double part[2] = {0.0, 0.0};
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const RowIdx<K> ix(N, tile);
        const size_t p = (size_t)ix.el * K * K + ix.t * K;
        T r[K];
        if (ix.active) {
            T x[K], ph[K];
            load_row<K, T>(v.x + p, x);
            load_row<K, T>(v.ph + p, ph);
            if (s_exit) {
#pragma unroll
                for (int i = 0; i < K; ++i) x[i] = x[i] + alpha * ph[i];
                store_row<K, T>(v.x + p, x);
            } else {
                T sh[K], sv[K], tv[K], rh[K];
                load_row<K, T>(v.sh + p, sh);
                load_row<K, T>(v.s + p, sv);
                load_row<K, T>(v.t + p, tv);
                load_row<K, T>(v.rhat + p, rh);
#pragma unroll
                for (int i = 0; i < K; ++i) {
                    x[i] = x[i] + (alpha * ph[i] + T(omega) * sh[i]);
                    r[i] = sv[i] - T(omega) * tv[i];
                    part[0] += double(r[i]) * double(r[i]);
                    part[1] += double(rh[i]) * double(r[i]);
                }
                store_row<K, T>(v.x + p, x);
                store_row<K, T>(v.r + p, r);
            }
        }
        if (!s_exit) element_moments<K, T>(v.h, r, mom[ix.warp][ix.lw], ix, v.er);
    }
    double out[2];
    if (grid_reduce<2>(part, rs.partials, rs.counter, out) && threadIdx.x == 0) {
        sc->it += 1;
        if (s_exit) {
            sc->rnorm2 = sc->snorm2;
            sc->done = 1;
        } else {
            sc->rnorm2 = out[0];
            sc->rho_old = sc->rho;
            sc->rho = out[1];
            if (out[0] <= sc->eps2 || sc->it >= max_iter || omega == 0.0) sc->done = 1;
            // an FP32 solve whose residual has grown a millionfold is lost (krylov_usable
            // then drops its result)
            if (sizeof(T) == 4 && !(out[0] <= 1e12 * sc->bnorm2)) sc->done = 1;
            if (!isfinite(out[0])) sc->done = 1;
        }
        if (has_handle) cudaGraphSetConditional(h, sc->done ? 0u : 1u);
    }
}

__global__ void k_set_loop(const KrylovScalars* sc, cudaGraphConditionalHandle h) {
    cudaGraphSetConditional(h, sc->done ? 0u : 1u);
}

// r = b - A x (FP64 refinement residual); ||r||^2 -> rnorm2, ||b||^2 -> bnorm2
template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS, kResidualCtas<K, T>) k_mf_residual(MfOp<T> op, const double* __restrict__ b,
                                                                   const T* __restrict__ x, const T* __restrict__ xtv,
                                                                   const T* __restrict__ xtg, double* __restrict__ r,
                                                                   ReduceScratch rs) {
    __shared__ RowScratch<K, T> sm[Rows<K>::WARPS];
    const int ntiles = (int)rgrid_of<K>(op.g.N);
    double part[2] = {0.0, 0.0};
    auto tile_body = [&](int tile) {
        const RowIdx<K> ix(op.g.N, tile);
        T y[K];
        row_apply<K, T>(op, x, xtv, xtg, sm[ix.warp], ix, y);
        if (ix.active) {
            const size_t p = (size_t)ix.el * K * K + ix.t * K;
            double bb[K], rr[K];
            load_row<K, double>(b + p, bb);
#pragma unroll
            for (int i = 0; i < K; ++i) {
                rr[i] = bb[i] - double(y[i]);
                part[0] += rr[i] * rr[i];
                part[1] += bb[i] * bb[i];
            }
            store_row<K, double>(r + p, rr);
        }
    };
    // FP32: one wave of CTAs over the tiles; FP64 keeps one tile per CTA (the loop would
    // push the operator past the register file)
    if constexpr (sizeof(T) == 4) {
#pragma unroll 1
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) tile_body(tile);
    } else {
        if ((int)blockIdx.x < ntiles) tile_body(blockIdx.x);
    }
    double out[2];
    if (grid_reduce<2>(part, rs.partials, rs.counter, out) && threadIdx.x == 0) {
        rs.sc->rnorm2 = out[0];
        rs.sc->bnorm2 = out[1];
    }
}

// y = A x (operator only). The traces come from k_trace_in, launched right before it as its
// programmatic primary (mf_apply_op): everything else is loaded while that kernel still runs,
// and the traces (read through L2, since they are being written) after it has ended. A call
// on 9,216 elements at K = 5 is bound by the two launches and the host's synchronisation.
// Registers: the compiler's own choice (K = 2 on 500^2 elements 28.0 us, with a minimum of three CTAs
// an SM 30.2; K = 6 on 256^2 41.3 and 48.9; K = 8 on 200^2 53.1 and 62.8). Without the wait, all loads
// together, it took 22.7, 38.8 and 47.9 us by itself, but the call, whose two launches overlap, is 4
// to 13% shorter as it is (medians of 2,500 calls at 14 sizes, 12^2 elements to the fixed scratch's
// limit).
template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS)
    k_mf_apply(MfOp<T> op, const T* __restrict__ x, const T* xtv, const T* xtg, T* __restrict__ y) {
    __shared__ RowScratch<K, T> sm[Rows<K>::WARPS];
    const RowIdx<K> ix(op.g.N, blockIdx.x);
    const size_t p = (size_t)ix.el * K * K + ix.t * K, q4 = ((size_t)ix.el * K + ix.t) * 4;
    ApplyIn<K, T> in;
    row_apply_static<K, T>(op.g, ix, in);
#pragma unroll
    for (int i = 0; i < K; ++i) in.xr[i] = in.xc[i] = T(0);
    if (ix.active) {
        load_row<K, T>(x + p, in.xr);
        load_col<K, T>(x + (size_t)ix.el * K * K + ix.t, in.xc);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");  // returns at once without a primary
#pragma unroll
    for (int f = 0; f < 4; ++f) in.ntv[f] = in.ntg[f] = T(0);
    if (ix.active) {
        load4_cg<T>(xtv + q4, in.ntv);
        load4_cg<T>(xtg + q4, in.ntg);
    }
    T yy[K];
    row_apply_core<K, T>(op, in, sm[ix.warp], ix, yy);
    if (ix.active) store_row<K, T>(y + p, yy);
}

// ---------------------------------------------------------------- transposed solve
// BiCGSTAB on A^T mu = b (the discrete adjoint) on the same iteration: the smoother's element
// inverses and the hats are the transposed ones (op.dinv, v.h), the coarse hierarchy is the
// forward one (its operator is symmetric), and an operator application is k_tr_own, which
// also forms the preconditioned vector z = P u0 + w zf, then the gather with its dot products.

// x = 0, r = rhat = b; ||b||^2; element moments of r
template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS) k_tr_init(int N, BicgVectors<T> v, ReduceScratch rs) {
    __shared__ T mom[Rows<K>::WARPS][Rows<K>::EPW][4][K];
    const int ntiles = (int)rgrid_of<K>(N);
    double part[1] = {0.0};
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const RowIdx<K> ix(N, tile);
        T r[K];
        if (ix.active) {
            const size_t p = (size_t)ix.el * K * K + ix.t * K;
            T z[K];
            load_row<K, T>(v.b + p, r);
#pragma unroll
            for (int i = 0; i < K; ++i) {
                z[i] = T(0);
                part[0] += double(r[i]) * double(r[i]);
            }
            store_row<K, T>(v.x + p, z);
            store_row<K, T>(v.r + p, r);
            store_row<K, T>(v.rhat + p, r);
        }
        element_moments<K, T>(v.h, r, mom[ix.warp][ix.lw], ix, v.er);
    }
    double out[1];
    if (grid_reduce<1>(part, rs.partials, rs.counter, out) && threadIdx.x == 0) {
        KrylovScalars* sc = rs.sc;
        sc->rnorm2 = sc->bnorm2 = sc->rho = out[0];
        sc->eps2 = sc->tol * sc->tol * out[0];
        sc->rho_old = sc->alpha = sc->omega = 1.0;
        sc->beta = 0.0;
        sc->it = 0;
        sc->breakdown = 0;
        sc->s_exit = 0;
        sc->zero_rhs = out[0] == 0.0;
        sc->done = out[0] == 0.0 || !isfinite(out[0]);
    }
}

// z = P u0 + w zf into ph or sh, its own part of A^T z into v or t, and the neighbours' slots.
// Combining here saves the pass over z that a separate operator launch would read: per point
// zf read, z and the own part written, three metric coefficients; per face point four
// coefficients and two slots.
template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS, sizeof(T) == 4 ? 4 : 3)
    k_tr_own(MfOp<T> op, BicgVectors<T> v, const int* __restrict__ conn, const T* __restrict__ u0, double w,
             const KrylovScalars* sc, int mode) {
    if (sc->done) return;  // uniform
    __shared__ RowScratch<K, T> sm[Rows<K>::WARPS];
    const RowIdx<K> ix(op.g.N, blockIdx.x);
    const size_t p = (size_t)ix.el * K * K + ix.t * K;
    T z[K], own[K];
#pragma unroll
    for (int i = 0; i < K; ++i) z[i] = T(0);
    if (ix.active) {
        combine_row<K, T>(v.h, conn, u0, v.zf + p, T(w), ix.el, ix.t, z);
        store_row<K, T>((mode == 0 ? v.ph : v.sh) + p, z);
    }
    row_transpose_own<K, T>(op, z, sm[ix.warp], ix, v.tv, v.tg, own);
    if (ix.active) store_row<K, T>((mode == 0 ? v.v : v.t) + p, own);
}

// The gather of v = A^T ph (mode 0: alpha, element moments of v) or t = A^T sh (mode 1: omega),
// in place over the own part. One wave of CTAs over the element tiles.
template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS) k_tr_gather(MfOp<T> op, BicgVectors<T> v, ReduceScratch rs,
                                                                 int mode) {
    KrylovScalars* sc = rs.sc;
    if (sc->done || (mode == 1 && sc->s_exit)) return;  // uniform, as in k_mf_v and k_mf_t
    __shared__ T buf[Rows<K>::WARPS][Rows<K>::EPW][K][K];
    __shared__ T mom[Rows<K>::WARPS][Rows<K>::EPW][4][K];
    const int ntiles = (int)rgrid_of<K>(op.g.N);
    T* y_out = mode == 0 ? v.v : v.t;
    const T* second = mode == 0 ? v.rhat : v.s;
    double part[2] = {0.0, 0.0};
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const RowIdx<K> ix(op.g.N, tile);
        const size_t p = (size_t)ix.el * K * K + ix.t * K;
        T y[K], q[K];
        if (ix.active) load_row<K, T>(second + p, q);
        row_transpose_gather<K, T>(op.b, y_out, v.tv, v.tg, buf[ix.warp][ix.lw], ix, y);
        if (ix.active) {
            store_row<K, T>(y_out + p, y);
#pragma unroll
            for (int i = 0; i < K; ++i) {
                part[0] += double(y[i]) * double(q[i]);
                part[1] += double(y[i]) * double(y[i]);
            }
        }
        if (mode == 0) element_moments<K, T>(v.h, y, mom[ix.warp][ix.lw], ix, v.ev);
    }
    double out[2];
    if (grid_reduce<2>(part, rs.partials, rs.counter, out) && threadIdx.x == 0) {
        if (mode == 1) {
            sc->omega = out[1] > 0.0 ? out[0] / out[1] : 0.0;
        } else if (out[0] == 0.0 || sc->rho == 0.0 || !isfinite(out[0])) {
            sc->breakdown = 1;
            sc->done = 1;
        } else {
            sc->alpha = sc->rho / out[0];
        }
    }
}

// y = A^T x as the two operator launches alone: own part and slots, then the gather, and with
// b given r = b - y, ||r||^2 -> rnorm2, ||b||^2 -> bnorm2 (y may then be null).
template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS) k_tr_apply_own(MfOp<T> op, const T* __restrict__ x,
                                                                    T* __restrict__ own_out, T* __restrict__ sv,
                                                                    T* __restrict__ sg) {
    __shared__ RowScratch<K, T> sm[Rows<K>::WARPS];
    const RowIdx<K> ix(op.g.N, blockIdx.x);
    const size_t p = (size_t)ix.el * K * K + ix.t * K;
    T z[K], own[K];
#pragma unroll
    for (int i = 0; i < K; ++i) z[i] = T(0);
    if (ix.active) load_row<K, T>(x + p, z);
    row_transpose_own<K, T>(op, z, sm[ix.warp], ix, sv, sg, own);
    if (ix.active) store_row<K, T>(own_out + p, own);
}

template <int K, typename T>
__global__ void __launch_bounds__(Rows<K>::THREADS) k_tr_apply_gather(MfOp<T> op, const T* own,
                                                                       const T* __restrict__ sv,
                                                                       const T* __restrict__ sg, T* y_out,
                                                                       const T* __restrict__ b, T* __restrict__ r_out,
                                                                       ReduceScratch rs) {
    __shared__ T buf[Rows<K>::WARPS][Rows<K>::EPW][K][K];
    const int ntiles = (int)rgrid_of<K>(op.g.N);
    double part[2] = {0.0, 0.0};
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const RowIdx<K> ix(op.g.N, tile);
        const size_t p = (size_t)ix.el * K * K + ix.t * K;
        T y[K];
        row_transpose_gather<K, T>(op.b, own, sv, sg, buf[ix.warp][ix.lw], ix, y);
        if (!ix.active) continue;
        if (!b) {
            store_row<K, T>(y_out + p, y);
            continue;
        }
        T bb[K], r[K];
        load_row<K, T>(b + p, bb);
#pragma unroll
        for (int i = 0; i < K; ++i) {
            r[i] = bb[i] - y[i];
            part[0] += double(r[i]) * double(r[i]);
            part[1] += double(bb[i]) * double(bb[i]);
        }
        store_row<K, T>(r_out + p, r);
    }
    if (!b) return;
    double out[2];
    if (grid_reduce<2>(part, rs.partials, rs.counter, out) && threadIdx.x == 0) {
        rs.sc->rnorm2 = out[0];
        rs.sc->bnorm2 = out[1];
    }
}

// The inverse blocks of the transposed operator: D^-T stored as D^-1 is (transposed), so the
// smoother reads both in the same order. One warp-row per block row; the reads of a warp are
// contiguous, the writes strided inside one element's few KB.
template <typename T>
__global__ void k_transpose_blocks(int N, int K2, int stride, const T* __restrict__ a, T* __restrict__ at) {
    const size_t n = (size_t)N * K2 * K2, step = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
        const size_t el = i / ((size_t)K2 * K2);
        const int q = (int)(i - el * K2 * K2), r = q / K2, c = q - r * K2;
        at[el * stride + (size_t)c * K2 + r] = a[el * stride + q];
    }
}

// ---------------------------------------------------------------- FP64 refinement on the device
// The mixed-precision solve as one graph: FP64 residual, then while the refinement
// continues { FP32 right-hand side, inner BiCGSTAB (its own while node), psi += x,
// FP64 residual }. k_refine_ctl decides after every FP64 residual, with the rule the
// host loop uses: stop on a non-finite or zero residual norm, at the target, at the sweep
// cap, or when the last sweep did not halve the residual (stalled: the host finishes the
// solve in FP64); otherwise ask the inner solve for max(inner_tol, aim / current) relative
// reduction (at most 0.5), so the last sweep does not overshoot.
__global__ void k_refine_begin(KrylovScalars* sc) {
    sc->sweeps = 0;
    sc->iters_total = 0;
    sc->zero_psi = 0;
    sc->finite = 1;
    sc->stalled = 0;
}

__global__ void k_refine_ctl(KrylovScalars* sc, cudaGraphConditionalHandle h) {
    const double bn = sc->bnorm2, rn = sc->rnorm2;
    const bool fin = isfinite(bn) && isfinite(rn);
    double res = bn > 0.0 ? sqrt(rn / bn) : 0.0;
    bool stop = !fin;
    if (fin && bn == 0.0) {
        sc->zero_psi = 1;
        res = 0.0;
        stop = true;
    }
    if (!stop && (rn <= sc->tol_outer * sc->tol_outer * bn || sc->sweeps >= sc->max_sweeps)) stop = true;
    // a sweep that did not halve the residual: iterative refinement with an FP32 inner solve
    // needs cond(A) * eps_32 < 1, which this operator no longer meets
    if (!stop && sc->sweeps > 0 && !(res <= 0.5 * sc->res)) {
        stop = true;
        sc->stalled = 1;
    }
    sc->res = res;
    sc->finite = fin;
    if (!stop) {
        const double need = sc->aim_outer / res;
        sc->tol = fmin(0.5, fmax(sc->inner_tol, need));
        sc->sweeps += 1;
    }
    cudaGraphSetConditional(h, stop ? 0u : 1u);
}

// right-hand side of the inner solve (the FP64 residual rounded to FP32) and its zero
// initial guess
__global__ void k_refine_prep(const double* __restrict__ r, float* __restrict__ b, float* __restrict__ x, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        b[i] = (float)r[i];
        x[i] = 0.f;
    }
}

// psi += x; the inner iterations are added to the solve's total. An inner solve that broke
// down adds nothing: the residual stays, which the decision after it takes for a stall, and
// the FP64 solve goes on from psi.
__global__ void k_refine_axpy(const float* __restrict__ e, double* __restrict__ x, size_t n, KrylovScalars* sc) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && krylov_usable(*sc)) x[i] += (double)e[i];
    if (i == 0) sc->iters_total += sc->it;
}

// a zero right-hand side gives psi = 0
__global__ void k_refine_finish(double* __restrict__ x, size_t n, const KrylovScalars* sc) {
    if (!sc->zero_psi) return;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = 0.0;
}

__global__ void k_d2f(const double* a, float* b, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = (float)a[i];
}
__global__ void k_axpy_f2d(const float* e, double* x, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += (double)e[i];
}

// ---------------------------------------------------------------- launchers
#ifndef HO2D_KSWITCH  // (a build of a few orders only, to look at their registers, defines its own)
#define HO2D_KSWITCH(K, CALL)                              \
    switch (K) {                                           \
        case 1: { constexpr int KK = 1; CALL; } break;      \
        case 2: { constexpr int KK = 2; CALL; } break;      \
        case 3: { constexpr int KK = 3; CALL; } break;      \
        case 4: { constexpr int KK = 4; CALL; } break;      \
        case 5: { constexpr int KK = 5; CALL; } break;      \
        case 6: { constexpr int KK = 6; CALL; } break;      \
        case 7: { constexpr int KK = 7; CALL; } break;      \
        case 8: { constexpr int KK = 8; CALL; } break;      \
        default: return cudaErrorInvalidValue;             \
    }
#endif


int krylov_max_blocks(int K, int N) {
    const int k2 = K * K;
    const int epb = (256 / k2) > 32 ? 32 : ((256 / k2) > 0 ? 256 / k2 : 1);
    return (N + epb - 1) / epb;
}

template <typename T>
cudaError_t krylov_init(const MfOp<T>& op, const BicgVectors<T>& v, const ReduceScratch& rs,
                        cudaStream_t s) {
    const int N = op.g.N;
    if (op.transposed) {
        HO2D_KSWITCH(op.K, (k_tr_init<KK, T><<<wave_of<KK, T>(&WaveSizes::tr, N), Rows<KK>::THREADS, 0, s>>>(N, v, rs)));
        return cudaGetLastError();
    }
    HO2D_KSWITCH(op.K, (k_trace_in<KK, T><<<rgrid_of<KK>(N), Rows<KK>::THREADS, 0, s>>>(op, v.x, v.xtv, v.xtg)));
    HO2D_KSWITCH(op.K, (k_mf_init<KK, T><<<wave_of<KK, T>(&WaveSizes::init, N), Rows<KK>::THREADS, 0, s>>>(op, v, rs)));
    const size_t n = (size_t)N * op.K * op.K;
    k_zero_if<T><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(v.x, n, rs.sc);
    return cudaGetLastError();
}

// One BiCGSTAB iteration: [coarse cycle on P^T p] -> p update + smoothing (ph) -> v = A ph
// -> [coarse cycle on P^T s] -> s update + smoothing (sh) -> t = A sh -> x, r update and
// loop control.
// A preconditioner application is its coarse cycle (on the side stream when op.side is
// set) beside the fine smoothing part k_post_a, then the combination k_post_b. With ev
// (10 events) everything runs in order on s with the boundaries recorded: ev[0] coarse
// ev[1] fine part ev[2] combination ev[3] operator ev[4] coarse ev[5] fine part ev[6]
// combination ev[7] operator ev[8] update ev[9]. TR: the transposed solve's iteration.
template <int K, typename T, bool TR = false>
static void iteration_impl(const MfOp<T>& op, const BicgVectors<T>& v, const ReduceScratch& rs, int max_iter,
                           const Precond<T>& pc, cudaGraphConditionalHandle h, int has_handle, cudaStream_t s,
                           cudaEvent_t* ev = nullptr) {
    auto mark = [&](int i) {
        if (ev) cudaEventRecord(ev[i], s);
    };
    const int N = op.g.N;
    const int mg = pc.nlev > 0;
    const unsigned gp = rgrid_of<K>(N);
    constexpr int tp = Rows<K>::THREADS;
    auto post_a = [&](int mode) {
        if constexpr (TR) {
            if (op.dinv_in_place) {
                k_post_a<K, T, 3><<<gp, tp, PostRows<K, T, 3>::SMEM, s>>>(op, v, mg, rs, mode);
                return;
            }
        }
        if constexpr (!TR) {
            if (op.kron_f) {
                k_post_a<K, T, 2><<<gp, tp, PostRows<K, T, 2>::SMEM, s>>>(op, v, mg, rs, mode);
                return;
            }
        }
        if constexpr (std::is_same<T, float>::value && !TR) {
            if (op.dinv_bf16) {
                k_post_a<K, T, 1><<<gp, tp, PostRows<K, T, 1>::SMEM, s>>>(op, v, mg, rs, mode);
                return;
            }
        }
        k_post_a<K, T, 0><<<gp, tp, PostRows<K, T, 0>::SMEM, s>>>(op, v, mg, rs, mode);
    };
    // one preconditioner application: the coarse cycle beside the fine part (on the side
    // stream, joined before the combination), or after it without a side stream
    auto precond = [&](int mode, int m0) {
        const bool fork = mg && op.side && !ev;  // a profiled iteration runs everything in order
        mark(m0);
        if (fork) {
            cudaEventRecord(op.ev_fork, s);
            cudaStreamWaitEvent(op.side, op.ev_fork, 0);
            coarse_cycle<T>(pc, v, rs.sc, mode, op.side);
            cudaEventRecord(op.ev_join, op.side);
        } else if (mg) {
            coarse_cycle<T>(pc, v, rs.sc, mode, s);
        }
        mark(m0 + 1);
        post_a(mode);
        if (fork) cudaStreamWaitEvent(s, op.ev_join, 0);
        mark(m0 + 2);
        if constexpr (TR) k_tr_own<K, T><<<gp, tp, 0, s>>>(op, v, mg ? pc.conn : nullptr, pc.lev[0].u, pc.omega, rs.sc, mode);
        else k_post_b<K, T><<<gp, tp, 0, s>>>(op, v, mg ? pc.conn : nullptr, pc.lev[0].u, pc.omega, rs.sc, mode);
    };
    const unsigned gwv = wave_of<K, T>(&WaveSizes::v, N), gwt = wave_of<K, T>(&WaveSizes::t, N),
                   gwx = wave_of<K, T>(&WaveSizes::xr, N);
    // the FP32 operator with its inputs staged by bulk copies, or read through L2 prefetches
    auto apply_v = [&]() {
        if constexpr (TR) {
            k_tr_gather<K, T><<<wave_of<K, T>(&WaveSizes::tr, N), tp, 0, s>>>(op, v, rs, 0);
            return;
        }
        if constexpr (std::is_same<T, float>::value) {
            if (op.staged) {
                k_mf_v<K, T, true><<<wave_of<K, T>(&WaveSizes::v_st, N), Rows<K>::THREADS, ApplyStage<K>::CTA_BYTES,
                                     s>>>(op, v, rs);
                return;
            }
        }
        k_mf_v<K, T><<<gwv, Rows<K>::THREADS, 0, s>>>(op, v, rs);
    };
    auto apply_t = [&]() {
        if constexpr (TR) {
            k_tr_gather<K, T><<<wave_of<K, T>(&WaveSizes::tr, N), tp, 0, s>>>(op, v, rs, 1);
            return;
        }
        if constexpr (std::is_same<T, float>::value) {
            if (op.staged) {
                k_mf_t<K, T, true><<<wave_of<K, T>(&WaveSizes::t_st, N), Rows<K>::THREADS, ApplyStage<K>::CTA_BYTES,
                                     s>>>(op, v, rs);
                return;
            }
        }
        k_mf_t<K, T><<<gwt, Rows<K>::THREADS, 0, s>>>(op, v, rs);
    };
    precond(0, 0);
    mark(3);
    apply_v();
    precond(1, 4);
    mark(7);
    apply_t();
    mark(8);
    k_xr_update<K, T><<<gwx, Rows<K>::THREADS, 0, s>>>(N, v, rs, max_iter, h, has_handle);
    mark(9);
}

template <int K, typename T>
static cudaError_t configure_waves() {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    WaveSizes& ws = g_wave[K][std::is_same<T, float>::value ? 1 : 0];
    auto w = [&](auto kern, unsigned& out, int dyn = 0) {
        int nb = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, Rows<K>::THREADS, dyn);
        out = (unsigned)(nb > 0 ? nb : 1) * (unsigned)sms;
    };
    w(k_xr_update<K, T>, ws.xr);
    w(k_tr_gather<K, T>, ws.tr);
    if constexpr (sizeof(T) == 4) {  // the FP64 operator kernels take one tile per CTA
        w(k_mf_init<K, T>, ws.init);
        w(k_mf_v<K, T>, ws.v);
        w(k_mf_t<K, T>, ws.t);
        w(k_mf_v<K, T, true>, ws.v_st, ApplyStage<K>::CTA_BYTES);
        w(k_mf_t<K, T, true>, ws.t_st, ApplyStage<K>::CTA_BYTES);
        w(k_mf_residual<K, T>, ws.res);
    }
    return e;
}

// Dynamic shared memory of the smoothing kernels that stage their blocks (above the
// 48 KB a launch gets without asking); once per device before the first launch or capture.
template <int K>
static cudaError_t configure_post() {
    cudaError_t e = cudaSuccess;
    auto one = [&](auto kern, int bytes) {
        if (e == cudaSuccess && bytes > 0)
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    one(k_post_a<K, double, 0>, PostRows<K, double, 0>::SMEM);
    one(k_post_a<K, double, 2>, PostRows<K, double, 2>::SMEM);
    one(k_post_a<K, double, 3>, PostRows<K, double, 3>::SMEM);
    one(k_post_a<K, float, 3>, PostRows<K, float, 3>::SMEM);
    one(k_post_a<K, float, 0>, PostRows<K, float, 0>::SMEM);
    one(k_post_a<K, float, 1>, PostRows<K, float, 1>::SMEM);
    one(k_post_a<K, float, 2>, PostRows<K, float, 2>::SMEM);
    return e;
}

cudaError_t krylov_configure(int K) {
    cudaError_t e = cudaSuccess;
    HO2D_KSWITCH(K, (e = configure_post<KK>()));
    if (e == cudaSuccess) HO2D_KSWITCH(K, (e = configure_waves<KK, double>()));
    if (e == cudaSuccess) HO2D_KSWITCH(K, (e = configure_waves<KK, float>()));
    return e;
}

template <typename T>
int krylov_launches_per_iteration(const Precond<T>& pc) {
    return 7 + 2 * coarse_launches(pc);
}

template <typename T>
cudaError_t krylov_iteration(const MfOp<T>& op, const BicgVectors<T>& v, const ReduceScratch& rs, int max_iter,
                             const Precond<T>& pc, cudaStream_t s) {
    if (op.transposed) {
        HO2D_KSWITCH(op.K, (iteration_impl<KK, T, true>(op, v, rs, max_iter, pc, cudaGraphConditionalHandle(), 0, s)));
        return cudaGetLastError();
    }
    HO2D_KSWITCH(op.K, (iteration_impl<KK, T>(op, v, rs, max_iter, pc, cudaGraphConditionalHandle(), 0, s)));
    return cudaGetLastError();
}

template <typename T>
cudaError_t krylov_iteration_timed(const MfOp<T>& op, const BicgVectors<T>& v, const ReduceScratch& rs, int max_iter,
                                   const Precond<T>& pc, cudaEvent_t* ev, cudaStream_t s) {
    HO2D_KSWITCH(op.K, (iteration_impl<KK, T>(op, v, rs, max_iter, pc, cudaGraphConditionalHandle(), 0, s, ev)));
    return cudaGetLastError();
}

// the instances of the one-kernel solve (krylov_fused_*.cu)
#define HO2D_FUSED_DECL(NAME, T)                                                                               \
    cudaError_t NAME(const MfOp<T>&, const BicgVectors<T>&, const FusedScratch&, int, const Precond<T>&,        \
                     KrylovScalars*, cudaStream_t, bool*)
HO2D_FUSED_DECL(fused_f64, double);
HO2D_FUSED_DECL(fused_tr64, double);
HO2D_FUSED_DECL(fused_f32_exact, float);
HO2D_FUSED_DECL(fused_f32_bf16, float);
HO2D_FUSED_DECL(fused_f32_kron, float);
HO2D_FUSED_DECL(fused_tr32, float);

template <typename T>
cudaError_t krylov_fused(const MfOp<T>& op, const BicgVectors<T>& v, const FusedScratch& fs, int max_iter,
                         const Precond<T>& pc, KrylovScalars* sc, cudaStream_t s, bool* fits) {
    if (op.dinv_in_place) {
        *fits = false;
        return cudaSuccess;
    }
    if constexpr (std::is_same<T, float>::value) {
        if (op.transposed) return fused_tr32(op, v, fs, max_iter, pc, sc, s, fits);
        if (op.kron_f) return fused_f32_kron(op, v, fs, max_iter, pc, sc, s, fits);
        if (op.dinv_bf16) return fused_f32_bf16(op, v, fs, max_iter, pc, sc, s, fits);
        return fused_f32_exact(op, v, fs, max_iter, pc, sc, s, fits);
    } else {
        if (op.transposed) return fused_tr64(op, v, fs, max_iter, pc, sc, s, fits);
        // factors come with at least 48 MB of blocks (kKronMinBytes, setup_device.cu), more tiles than
        // the one-kernel solve takes at any order
        if (op.kron_f) {
            *fits = false;
            return cudaSuccess;
        }
        return fused_f64(op, v, fs, max_iter, pc, sc, s, fits);
    }
}

// Captures a whole solve into `*graph_out`: initial residual, then a while node whose body
// is one BiCGSTAB iteration; the loop condition lives on the device, so a solve is one
// graph launch with no host round trip. A small mesh's solve is one kernel (krylov_fused).
template <typename T>
cudaError_t krylov_capture_solve(const MfOp<T>& op, const BicgVectors<T>& v, const ReduceScratch& rs,
                                 int max_iter, const Precond<T>& pc, cudaStream_t s, cudaGraph_t* graph_out,
                                 bool* one_kernel) {
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaGraphCreate(&g, 0);
    if (e != cudaSuccess) return e;
    if ((e = cudaStreamBeginCaptureToGraph(s, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
        cudaSuccess)
        return e;
    bool& fused = *one_kernel;
    if ((e = krylov_fused<T>(op, v, {rs.fused_partials, rs.fused_bar}, max_iter, pc, rs.sc, s, &fused)) != cudaSuccess)
        return e;
    if (fused) {
        if ((e = cudaStreamEndCapture(s, &g)) != cudaSuccess) return e;
        *graph_out = g;
        return cudaGetLastError();
    }
    cudaGraphConditionalHandle h;
    if ((e = cudaGraphConditionalHandleCreate(&h, g, 0, 0)) != cudaSuccess) return e;
    krylov_init<T>(op, v, rs, s);
    k_set_loop<<<1, 1, 0, s>>>(rs.sc, h);
    cudaStreamCaptureStatus st;
    const cudaGraphNode_t* deps = nullptr;
    size_t ndeps = 0;
    cudaGraph_t cg = nullptr;
    if ((e = cudaStreamGetCaptureInfo(s, &st, nullptr, &cg, &deps, &ndeps)) != cudaSuccess) return e;
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t cnode;
    if ((e = cudaGraphAddNode(&cnode, cg, deps, ndeps, &cp)) != cudaSuccess) return e;
    if ((e = cudaStreamUpdateCaptureDependencies(s, &cnode, 1, cudaStreamSetCaptureDependencies)) != cudaSuccess)
        return e;
    if ((e = cudaStreamEndCapture(s, &g)) != cudaSuccess) return e;
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    if ((e = cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
        cudaSuccess)
        return e;
    if (op.transposed) HO2D_KSWITCH(op.K, (iteration_impl<KK, T, true>(op, v, rs, max_iter, pc, h, 1, s)))
    else HO2D_KSWITCH(op.K, (iteration_impl<KK, T>(op, v, rs, max_iter, pc, h, 1, s)));
    if ((e = cudaStreamEndCapture(s, &body)) != cudaSuccess) return e;
    *graph_out = g;
    return cudaGetLastError();
}

// Captures a whole mixed-precision solve (FP64 refinement around the FP32 BiCGSTAB) into
// `*graph_out`: the refinement loop and each sweep's BiCGSTAB loop are nested while nodes
// whose conditions are set on the device, so a solve is one graph launch and no host
// round trip. psi64 is updated in place; rhs, the FP64 residual r64 and the FP64 traces
// (xtv64, xtg64) are the refinement's vectors; v32 holds the inner solve's (v32.b is the
// inner right-hand side, v32.x its solution).
cudaError_t krylov_capture_refined_solve(const MfOp<double>& A64, const MfOp<float>& A32,
                                         const BicgVectors<float>& v32, const ReduceScratch& rs, int max_iter,
                                         const Precond<float>& pc, double* psi64, const double* rhs, double* r64,
                                         double* xtv64, double* xtg64, cudaStream_t s, cudaGraph_t* graph_out,
                                         bool* one_kernel) {
    const size_t n = (size_t)A64.g.N * A64.K * A64.K;
    const unsigned gn = (unsigned)((n + 255) / 256);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaGraphCreate(&g, 0);
    if (e != cudaSuccess) return e;
    cudaGraphConditionalHandle ho, hi = 0;
    if ((e = cudaGraphConditionalHandleCreate(&ho, g, 0, 0)) != cudaSuccess) return e;
    // adds a while node on handle h after the capture's current dependencies and returns
    // its body graph; the stream's capture continues after the node
    auto add_while = [&](cudaGraphConditionalHandle h, cudaGraph_t* body) -> cudaError_t {
        cudaStreamCaptureStatus st;
        const cudaGraphNode_t* deps = nullptr;
        size_t ndeps = 0;
        cudaGraph_t cg = nullptr;
        cudaError_t err = cudaStreamGetCaptureInfo(s, &st, nullptr, &cg, &deps, &ndeps);
        if (err != cudaSuccess) return err;
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t node;
        if ((err = cudaGraphAddNode(&node, cg, deps, ndeps, &cp)) != cudaSuccess) return err;
        if ((err = cudaStreamUpdateCaptureDependencies(s, &node, 1, cudaStreamSetCaptureDependencies)) != cudaSuccess)
            return err;
        *body = cp.conditional.phGraph_out[0];
        return cudaSuccess;
    };
    // top level: reset, FP64 residual, decision, the refinement loop, zero-rhs fix-up
    if ((e = cudaStreamBeginCaptureToGraph(s, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
        cudaSuccess)
        return e;
    k_refine_begin<<<1, 1, 0, s>>>(rs.sc);
    mf_residual<double>(A64, rhs, psi64, xtv64, xtg64, r64, rs, s);
    k_refine_ctl<<<1, 1, 0, s>>>(rs.sc, ho);
    cudaGraph_t outer = nullptr;
    if ((e = add_while(ho, &outer)) != cudaSuccess) return e;
    k_refine_finish<<<gn, 256, 0, s>>>(psi64, n, rs.sc);
    if ((e = cudaStreamEndCapture(s, &g)) != cudaSuccess) return e;
    // one refinement sweep
    if ((e = cudaStreamBeginCaptureToGraph(s, outer, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
        cudaSuccess)
        return e;
    k_refine_prep<<<gn, 256, 0, s>>>(r64, const_cast<float*>(v32.b), v32.x, n);
    bool& fused = *one_kernel;
    if ((e = krylov_fused<float>(A32, v32, {rs.fused_partials, rs.fused_bar}, max_iter, pc, rs.sc, s, &fused)) !=
        cudaSuccess)
        return e;
    cudaGraph_t inner = nullptr;
    if (!fused) {
        krylov_init<float>(A32, v32, rs, s);
        if ((e = cudaGraphConditionalHandleCreate(&hi, g, 0, 0)) != cudaSuccess) return e;
        k_set_loop<<<1, 1, 0, s>>>(rs.sc, hi);
        if ((e = add_while(hi, &inner)) != cudaSuccess) return e;
    }
    k_refine_axpy<<<gn, 256, 0, s>>>(v32.x, psi64, n, rs.sc);
    mf_residual<double>(A64, rhs, psi64, xtv64, xtg64, r64, rs, s);
    k_refine_ctl<<<1, 1, 0, s>>>(rs.sc, ho);
    if ((e = cudaStreamEndCapture(s, &outer)) != cudaSuccess) return e;
    if (fused) {
        *graph_out = g;
        return cudaGetLastError();
    }
    // one BiCGSTAB iteration
    if ((e = cudaStreamBeginCaptureToGraph(s, inner, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
        cudaSuccess)
        return e;
    HO2D_KSWITCH(A32.K, (iteration_impl<KK, float>(A32, v32, rs, max_iter, pc, hi, 1, s)));
    if ((e = cudaStreamEndCapture(s, &inner)) != cudaSuccess) return e;
    *graph_out = g;
    return cudaGetLastError();
}

// kernel launches of one captured refined solve: begin, residual, decision and fix-up, then
// per sweep right-hand side, initial residual (3), loop set-up, update, residual and
// decision, plus the inner iterations (with the one-kernel inner solve: right-hand side, solve,
// update, residual (2) and decision)
int krylov_refined_launches(int sweeps, int inner_iters, const Precond<float>& pc, bool one_kernel) {
    if (one_kernel) return 5 + sweeps * 6;
    return 5 + sweeps * 9 + inner_iters * krylov_launches_per_iteration(pc);
}

template <typename T>
cudaError_t mf_residual(const MfOp<T>& op, const double* b, const T* x, T* xtv, T* xtg, double* r,
                        const ReduceScratch& rs, cudaStream_t s) {
    HO2D_KSWITCH(op.K, (k_trace_in<KK, T><<<rgrid_of<KK>(op.g.N), Rows<KK>::THREADS, 0, s>>>(op, x, xtv, xtg)));
    HO2D_KSWITCH(op.K, (k_mf_residual<KK, T><<<wave_of<KK, T>(&WaveSizes::res, op.g.N), Rows<KK>::THREADS, 0, s>>>(op, b, x, xtv, xtg, r,
                                                                                                  rs)));
    return cudaGetLastError();
}

template <typename T>
cudaError_t mf_apply_op(const MfOp<T>& op, const T* x, T* xtv, T* xtg, T* y, cudaStream_t s) {
    HO2D_KSWITCH(op.K, (k_trace_in<KK, T><<<rgrid_of<KK>(op.g.N), Rows<KK>::THREADS, 0, s>>>(op, x, xtv, xtg)));
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    HO2D_KSWITCH(op.K, (cfg.gridDim = dim3(rgrid_of<KK>(op.g.N)), cfg.blockDim = dim3(Rows<KK>::THREADS),
                        e = cudaLaunchKernelEx(&cfg, k_mf_apply<KK, T>, op, x, (const T*)xtv, (const T*)xtg, y)));
    return e;
}

template <typename T>
cudaError_t mf_apply_only(const MfOp<T>& op, const T* x, const T* xtv, const T* xtg, T* y, int reps, cudaStream_t s) {
    for (int r = 0; r < reps; ++r)
        HO2D_KSWITCH(op.K, (k_mf_apply<KK, T><<<rgrid_of<KK>(op.g.N), Rows<KK>::THREADS, 0, s>>>(op, x, xtv, xtg, y)));
    return cudaGetLastError();
}

template <typename T>
cudaError_t mf_apply_transpose(const MfOp<T>& op, const T* x, T* own, T* sv, T* sg, T* y, const T* b, T* r,
                               const ReduceScratch& rs, cudaStream_t s) {
    HO2D_KSWITCH(op.K, (k_tr_apply_own<KK, T><<<rgrid_of<KK>(op.g.N), Rows<KK>::THREADS, 0, s>>>(op, x, own, sv, sg)));
    HO2D_KSWITCH(op.K, (k_tr_apply_gather<KK, T><<<wave_of<KK, T>(&WaveSizes::tr, op.g.N), Rows<KK>::THREADS, 0, s>>>(
                           op, own, sv, sg, y, b, r, rs)));
    return cudaGetLastError();
}

template <typename T>
cudaError_t transpose_blocks(int N, int K, const T* a, T* at, cudaStream_t s) {
    k_transpose_blocks<T><<<8 * 148, 256, 0, s>>>(N, K * K, padded_count(K * K * K * K, (int)sizeof(T)), a, at);
    return cudaGetLastError();
}

cudaError_t launch_copy_d2f(const double* a, float* b, size_t n, cudaStream_t s) {
    if (n) k_d2f<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a, b, n);
    return cudaGetLastError();
}
cudaError_t launch_axpy_f2d(const float* e, double* x, size_t n, cudaStream_t s) {
    if (n) k_axpy_f2d<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(e, x, n);
    return cudaGetLastError();
}

#define HO2D_INSTANTIATE_KRYLOV(T)                                                                                \
    template cudaError_t krylov_init<T>(const MfOp<T>&, const BicgVectors<T>&, const ReduceScratch&,             \
                                        cudaStream_t);                                                            \
    template cudaError_t krylov_iteration<T>(const MfOp<T>&, const BicgVectors<T>&, const ReduceScratch&, int,    \
                                             const Precond<T>&, cudaStream_t);                                    \
    template int krylov_launches_per_iteration<T>(const Precond<T>&);                                             \
    template cudaError_t krylov_iteration_timed<T>(const MfOp<T>&, const BicgVectors<T>&, const ReduceScratch&,   \
                                                   int, const Precond<T>&, cudaEvent_t*, cudaStream_t);           \
    template cudaError_t krylov_capture_solve<T>(const MfOp<T>&, const BicgVectors<T>&, const ReduceScratch&,     \
                                                 int, const Precond<T>&, cudaStream_t, cudaGraph_t*, bool*);      \
    template cudaError_t mf_residual<T>(const MfOp<T>&, const double*, const T*, T*, T*, double*,                 \
                                        const ReduceScratch&, cudaStream_t);                                      \
    template cudaError_t mf_apply_op<T>(const MfOp<T>&, const T*, T*, T*, T*, cudaStream_t);                      \
    template cudaError_t mf_apply_only<T>(const MfOp<T>&, const T*, const T*, const T*, T*, int, cudaStream_t);   \
    template cudaError_t transpose_blocks<T>(int, int, const T*, T*, cudaStream_t);                               \
    template cudaError_t krylov_fused<T>(const MfOp<T>&, const BicgVectors<T>&, const FusedScratch&, int,          \
                                         const Precond<T>&, KrylovScalars*, cudaStream_t, bool*);

template cudaError_t mf_apply_transpose<double>(const MfOp<double>&, const double*, double*, double*, double*, double*,
                                                const double*, double*, const ReduceScratch&, cudaStream_t);
HO2D_INSTANTIATE_KRYLOV(double)
HO2D_INSTANTIATE_KRYLOV(float)

}  // namespace ho2d
