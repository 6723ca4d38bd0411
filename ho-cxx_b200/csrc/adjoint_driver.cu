// adjoint_driver.cu -- the discrete adjoint of the time loop: checkpointed forward sweep,
// recomputation of one segment at a time, the reverse sweep over the RK stages, and the
// transposed Poisson solve.
//
// No counterpart in the reference. The forward map of a step is the stage sequence of
// solve_advection_diffusion (src/HO_2D.cpp:1465-1531) with the stages of
// Euler_time_integrate (1806-1839). Its adjoint here is the transpose of the discrete
// map (adjoint_chain.cuh for the stage kernels, BiCGSTAB on A^T for the Poisson solve),
// exact up to the Poisson tolerance of the forward recomputation and of the transposed
// solve.
//
// Memory: one FP64 vorticity per checkpoint (every ckpt_every steps) and, during the
// backward sweep, the stage inputs and streamfunctions of one segment
// (ckpt_every x stages x 2 FP64 fields); the trajectory is never stored whole.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "adjoint_launch.hpp"
#include "solver_state.hpp"

namespace ho2d {

namespace {

// Explicit schemes of solve_advection_diffusion as Butcher tableaux: stage inputs
// w_s = omega + sum_r a[s][r] k_r at time t + c[s] dt, and omega' = omega + sum_s b[s] k_s.
struct Tableau {
    int ns = 1;
    double c[4] = {0, 0, 0, 0};
    double b[4] = {1, 0, 0, 0};
    double a[4][4] = {};
};

Tableau tableau(int ti_type) {
    Tableau t;
    if (ti_type == 4) {
        t.ns = 4;
        const double c[4] = {0.0, 0.5, 0.5, 1.0}, b[4] = {1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0};
        for (int s = 0; s < 4; ++s) {
            t.c[s] = c[s];
            t.b[s] = b[s];
        }
        t.a[1][0] = 0.5;
        t.a[2][1] = 0.5;
        t.a[3][2] = 1.0;
    } else if (ti_type == 2) {
        t.ns = 2;
        t.c[1] = 1.0;
        t.b[0] = t.b[1] = 0.5;
        t.a[1][0] = 1.0;
    }
    return t;
}

}  // namespace

int Solver::adjoint_steps() const { return adj_ ? adj_->nsteps : -1; }

// Buffers of the adjoint, allocated once per setup.
Error Solver::adjoint_prepare() {
    if (!setup_done_) return {1, "call ho2d_setup first"};
    if (!adj_) adj_.reset(new AdjointState);
    AdjointState& a = *adj_;
    if (a.ready) return {0, ""};
    DeviceState& d = *d_;
    HO2D_CUDA(cudaSetDevice(d.device), "cudaSetDevice");
    if (krylov32_) HO2D_TRY(upload_precision_arrays());
    const int N = mesh_.n_el, K = in_.knod, K2 = K * K, neb = std::max(1, mesh_.n_eb);
    const size_t nv = (size_t)N * K2, nf = (size_t)N * 4 * K;
    const std::vector<double> zv(nv, 0.0), zf(nf, 0.0), zb((size_t)neb * K, 0.0);
    for (auto& b : a.kv) HO2D_CUDA(upload(b, zv), "alloc adjoint Krylov");
    for (DeviceBuffer* b : {&a.res64, &a.x32, &a.b32, &a.lam_k, &a.lw_out, &a.lw_dir, &a.lux, &a.luy, &a.lw_stage,
                            &a.lpsi_dir, &a.lpsi, &a.mu, &a.lam, &a.wT, &a.psiT})
        HO2D_CUDA(upload(*b, zv), "alloc adjoint fields");
    for (auto& b : a.mus) HO2D_CUDA(upload(b, zv), "alloc adjoint fields");
    for (DeviceBuffer* b : {&a.sv, &a.sg, &a.swv, &a.swg, &a.sU, &a.spv, &a.spg})
        HO2D_CUDA(upload(*b, zf), "alloc adjoint slots");
    for (DeviceBuffer* b : {&a.lbc_d, &a.lbc_nv, &a.lpv}) HO2D_CUDA(upload(*b, zb), "alloc adjoint boundary");
    HO2D_CUDA(cudaDeviceSynchronize(), "adjoint setup");
    a.ready = true;
    return {0, ""};
}

// The transposed copy of the inverse blocks `dinv` in precision gi (0 FP64, 1 FP32), made once. It is
// as large as the blocks, the largest array of a solver by far (5.0 GB in FP64 on 512 x 512
// elements at K = 7), so it is made only where that leaves as much memory free; elsewhere the smoother
// reads the blocks in place (HO2D_ADJOINT_COPY=0 asks for that). A gradient on 64 x 64 elements at
// K = 5 (4 steps) takes 80 ms with the copy and 82 without, on 96 x 96 at K = 7 (2 steps) 127 and 170.
template <typename T>
Error Solver::adjoint_blocks(const T* dinv, int gi) {
    AdjointState& a = *adj_;
    if (a.dinvT[gi].get() || a.in_place[gi]) return {0, ""};
    DeviceState& d = *d_;
    const int N = mesh_.n_el, K = in_.knod;
    const size_t bytes = ((size_t)N * padded_count(K * K * K * K, (int)sizeof(T)) + 1) * sizeof(T);
    const char* e = std::getenv("HO2D_ADJOINT_COPY");
    size_t room = 0, total = 0;
    HO2D_CUDA(cudaMemGetInfo(&room, &total), "cudaMemGetInfo");
    a.in_place[gi] = (e && std::string(e) == "0") || room < 2 * bytes;
    if (!a.in_place[gi] && a.dinvT[gi].alloc(bytes) != cudaSuccess) {
        cudaGetLastError();
        a.in_place[gi] = true;
    }
    if (a.in_place[gi]) return {0, ""};
    HO2D_CUDA(cudaMemsetAsync(a.dinvT[gi].get(), 0, bytes, d.stream), "memset");
    HO2D_CUDA(transpose_blocks<T>(N, K, dinv, a.dinvT[gi].as<T>(), d.stream), "transposed blocks");
    launches_ += 1;
    return {0, ""};
}

// An allocation of the adjoint's time loop; the transposed copies give way to it.
Error Solver::adjoint_alloc(DeviceBuffer& b, size_t bytes, const char* what) {
    AdjointState& a = *adj_;
    cudaError_t e = b.alloc(bytes);
    if (e == cudaErrorMemoryAllocation && (a.dinvT[0].get() || a.dinvT[1].get())) {
        cudaGetLastError();
        for (int gi = 0; gi < 2; ++gi) {
            if (!a.dinvT[gi].get()) continue;
            a.graph[gi].reset();
            a.dinvT[gi].reset();
            a.in_place[gi] = true;
        }
        e = b.alloc(bytes);
    }
    HO2D_CUDA(e, what);
    return {0, ""};
}

// BiCGSTAB on A^T x = b in precision T to relative tolerance tol; x starts at zero. The
// forward solver's iteration (krylov.cu) on the transposed operator: D^-T for D^-1, and the
// coarse space's interpolation and restriction exchanged.
template <typename T>
Error Solver::kt_run(T* x, const T* b, bool f32, double tol, int& iters) {
    DeviceState& d = *d_;
    AdjointState& a = *adj_;
    const int K = in_.knod, gi = f32 ? 1 : 0;
    MfOp<T> op = make_op<T>(d, mesh_, K, f32);
    HO2D_TRY(adjoint_blocks<T>(op.dinv, gi));
    op.transposed = 1;
    op.dinv_in_place = a.in_place[gi] ? 1 : 0;
    if (!op.dinv_in_place) op.dinv = a.dinvT[gi].as<T>();
    op.dinv_bf16 = nullptr;
    op.kron_f = op.kron_exact = nullptr;
    op.kron_x = nullptr;
    op.staged = 0;
    BicgVectors<T> v = krylov_vectors<T>(d, x, b);
    std::swap(v.h.hp, v.h.hr);
    T** kv[8] = {&v.r, &v.rhat, &v.p, &v.v, &v.s, &v.t, &v.ph, &v.sh};
    for (int i = 0; i < 8; ++i) *kv[i] = a.kv[i].as<T>();
    v.tv = a.sv.as<T>();
    v.tg = a.sg.as<T>();
    const Precond<T>& pc = *reinterpret_cast<const Precond<T>*>(f32 ? (const void*)&d.pc32 : (const void*)&d.pc64);
    const ReduceScratch rs = reduce_scratch(d);
    // the boundary entries of the slots must read as zero in precision T; the FP64 and FP32
    // solves share these buffers
    HO2D_CUDA(cudaMemsetAsync(a.sv.get(), 0, a.sv.bytes(), d.stream), "memset");
    HO2D_CUDA(cudaMemsetAsync(a.sg.get(), 0, a.sg.bytes(), d.stream), "memset");
    d.h_sc->tol = tol;  // the stream is idle: the last read of h_sc was synchronised
    HO2D_CUDA(cudaMemcpyAsync(&rs.sc->tol, &d.h_sc->tol, sizeof(double), cudaMemcpyHostToDevice, d.stream), "tol");
    auto poll = [&]() -> Error {
        HO2D_CUDA(cudaMemcpyAsync(d.h_sc, rs.sc, sizeof(KrylovScalars), cudaMemcpyDeviceToHost, d.stream), "poll");
        HO2D_CUDA(cudaStreamSynchronize(d.stream), "poll");
        if (d.h_sc->dev_error) return {5, kWaitRanOut};
        return {0, ""};
    };
    if (use_graphs_) {
        // one launch of the captured solve (init and a device-side while loop); the graph
        // bakes in the operands, so it is recaptured when they change
        SolveGraph& sg = a.graph[gi];
        if (!sg.exec || sg.max_iter != max_iter_ || a.graph_x[gi] != (const void*)x || a.graph_b[gi] != (const void*)b) {
            sg.reset();
            HO2D_CUDA(krylov_capture_solve<T>(op, v, rs, max_iter_, pc, d.stream, &sg.graph, &sg.one_kernel), "graph capture");
            HO2D_CUDA(cudaGraphInstantiate(&sg.exec, sg.graph, cudaGraphInstantiateFlagUseNodePriority),
                      "graph instantiate");
            sg.max_iter = max_iter_;
            a.graph_x[gi] = x;
            a.graph_b[gi] = b;
        }
        HO2D_CUDA(cudaGraphLaunch(sg.exec, d.stream), "graph launch");
        HO2D_TRY(poll());
        iters = d.h_sc->it;
        launches_ += sg.one_kernel ? 1 : 2 + (int64_t)iters * krylov_launches_per_iteration(pc);
        return {0, ""};
    }
    HO2D_CUDA(krylov_init<T>(op, v, rs, d.stream), "transposed init");
    launches_ += 1;
    // batches of iterations between polls of the done flag; an iteration enqueued after
    // the solve finished returns at once in every kernel
    int chunk = std::max(1, adj_prev_iters_ - 1);
    for (;;) {
        for (int c = 0; c < chunk; ++c) {
            HO2D_CUDA(krylov_iteration<T>(op, v, rs, max_iter_, pc, d.stream), "transposed iteration");
            launches_ += krylov_launches_per_iteration(pc);
        }
        HO2D_TRY(poll());
        if (d.h_sc->done) break;
        chunk = 2;
    }
    iters = d.h_sc->it;
    return {0, ""};
}

// mu = A^-T rhs (FP64 vectors): FP64 BiCGSTAB, or with a mixed-precision Krylov mode FP32
// BiCGSTAB inside FP64 iterative refinement on the FP64 transposed residual.
Error Solver::transposed_solve(const double* rhs, double* mu) {
    const NvtxRange nvtx_range("ho2d.poisson_transpose");
    DeviceState& d = *d_;
    AdjointState& a = *adj_;
    const int N = mesh_.n_el, K = in_.knod;
    const size_t nv = (size_t)N * K * K;
    const ReduceScratch rs = reduce_scratch(d);
    bool finite = true;
    const RefineGoal goal = refine_goal(true);
    last_adj_iters_ = 0;
    int sweeps = 0;
    if (!krylov32_) {
        int it = 0;
        HO2D_TRY(kt_run<double>(mu, rhs, false, transposed_target(), it));
        last_adj_iters_ = it;
        const double bn = d.h_sc->bnorm2, rn = d.h_sc->rnorm2;
        finite = std::isfinite(bn) && std::isfinite(rn);
        last_adj_res_ = bn > 0 ? std::sqrt(rn / bn) : 0.0;
    } else {
        const MfOp<double> op = make_op<double>(d, mesh_, K, false);
        HO2D_CUDA(cudaMemsetAsync(mu, 0, nv * 8, d.stream), "memset");
        double prev = 0.0;
        bool lost = false;
        for (;; ++sweeps) {
            HO2D_CUDA(cudaMemsetAsync(a.sv.get(), 0, a.sv.bytes(), d.stream), "memset");  // shared with FP32
            HO2D_CUDA(cudaMemsetAsync(a.sg.get(), 0, a.sg.bytes(), d.stream), "memset");
            HO2D_CUDA(mf_apply_transpose<double>(op, mu, a.kv[0].as<double>(), a.sv.as<double>(), a.sg.as<double>(), nullptr,
                                                 rhs, a.res64.as<double>(), rs, d.stream),
                      "transposed residual");
            launches_ += 2;
            HO2D_CUDA(cudaMemcpyAsync(d.h_sc, rs.sc, sizeof(KrylovScalars), cudaMemcpyDeviceToHost, d.stream), "poll");
            HO2D_CUDA(cudaStreamSynchronize(d.stream), "poll");
            const double bn = d.h_sc->bnorm2, rn = d.h_sc->rnorm2;
            finite = std::isfinite(bn) && std::isfinite(rn);
            last_adj_res_ = bn > 0 ? std::sqrt(rn / bn) : 0.0;
            if (!finite || bn == 0.0) break;
            if (rn <= goal.accept * goal.accept * bn || sweeps >= 30) break;
            // a sweep that did not halve the residual (the forward refinement's rule) or an FP32
            // solve that broke down: the FP64 solve of the remaining residual finishes
            if (lost || (sweeps > 0 && !(last_adj_res_ <= 0.5 * prev))) {
                if (last_adj_res_ <= tol_) break;  // above what it aimed at, but within the tolerance
                int it = 0;
                HO2D_TRY(kt_run<double>(a.x32.as<double>(), a.res64.as<double>(), false,
                                        std::min(0.5, transposed_target() / last_adj_res_), it));
                last_adj_iters_ += it;
                last_adj_res_ *= std::sqrt(d.h_sc->rnorm2 / d.h_sc->bnorm2);
                finite = std::isfinite(last_adj_res_);
                HO2D_CUDA(launch_axpby(nv, mu, 1.0, mu, 1.0, a.x32.as<double>(), d.stream), "axpy");
                launches_ += 1;
                break;
            }
            prev = last_adj_res_;
            HO2D_CUDA(launch_copy_d2f(a.res64.as<double>(), a.b32.as<float>(), nv, d.stream), "d2f");
            const double need = goal.aim / last_adj_res_;
            const double itol = std::min(0.5, std::max(inner_tol_, need));
            int it = 0;
            HO2D_TRY(kt_run<float>(a.x32.as<float>(), a.b32.as<float>(), true, itol, it));
            last_adj_iters_ += it;
            lost = !krylov_usable(*d.h_sc);
            if (lost) continue;
            HO2D_CUDA(launch_axpy_f2d(a.x32.as<float>(), mu, nv, d.stream), "axpy");
            launches_ += 2;
        }
    }
    adj_prev_iters_ = std::max(1, krylov32_ ? last_adj_iters_ / std::max(1, sweeps) : last_adj_iters_);
    if (!finite) return {7, "non-finite values in the transposed Poisson solve"};
    return {0, ""};
}

// Adjoint of one stage at the stage input in d.w_stage with its streamfunction in
// d.psi64 (both set by the caller, time_ at the step's start): lam of k in a.lam_k ->
// lam of the stage input in out; lam of BC_parl_vel accumulates in a.lpv.
Error Solver::stage_adjoint_dev(double coeff, double* out) {
    DeviceState& d = *d_;
    AdjointState& a = *adj_;
    const int N = mesh_.n_el, K = in_.knod;
    const size_t nv = (size_t)N * K * K;
    HO2D_TRY(stage_t<double>(coeff, 0, false, false));  // the stage's fields from its psi
    const FrGeom<double> g = geom_of<double>(d, mesh_, false);
    StageAdjArgs<double> sa;
    sa.w = d.w_stage.as<double>();
    sa.u = d.u.as<double>();
    sa.v = d.v.as<double>();
    sa.w_tv = d.w_tv.as<double>();
    sa.U_t = d.U_t.as<double>();
    sa.bc_w = d.bc_w.as<double>();
    sa.bc_nv = d.bc_nv.as<double>();
    sa.lam_k = a.lam_k.as<double>();
    sa.lw_dir = a.lw_dir.as<double>();
    sa.lux = a.lux.as<double>();
    sa.luy = a.luy.as<double>();
    sa.slot_wv = a.swv.as<double>();
    sa.slot_wg = a.swg.as<double>();
    sa.slot_U = a.sU.as<double>();
    sa.lbc_d = a.lbc_d.as<double>();
    sa.lbc_nv = a.lbc_nv.as<double>();
    sa.lw_stage = a.lw_stage.as<double>();
    sa.lpsi_dir = a.lpsi_dir.as<double>();
    sa.slot_pv = a.spv.as<double>();
    sa.slot_pg = a.spg.as<double>();
    sa.lpv = a.lpv.as<double>();
    sa.dt = in_.dt;
    sa.re_inv = in_.reyn_inv;
    sa.adv_type = in_.adv_type;
    HO2D_CUDA(launch_residual_adjoint<double>(K, g, d.b64, sa, d.stream), "residual adjoint");
    HO2D_CUDA(launch_velocity_adjoint<double>(K, g, d.b64, sa, d.stream), "velocity adjoint");
    HO2D_CUDA(launch_gather<double>(K, N, d.b64, a.lpsi_dir.as<double>(), a.spv.as<double>(), a.spg.as<double>(),
                                    a.lpsi.as<double>(), d.stream),
              "psi gather");
    launches_ += 3;
    // psi = A^-1 (-J omega - boundary terms): lam of omega -= J A^-T lam of psi
    HO2D_TRY(transposed_solve(a.lpsi.as<double>(), a.mu.as<double>()));
    HO2D_CUDA(launch_sub_scaled(nv, out, a.lw_stage.as<double>(), d.m64[4].as<double>(), a.mu.as<double>(), d.stream),
              "combine");
    launches_ += 1;
    return {0, ""};
}

// Advection types 1 and 2 (residual_adjoint_continuous for type 2); both are checked on the
// host and on the GPU against complex-step derivatives of the oracle. Every precision: with
// the FP32 stage (HO2D_MIXED) the forward sweep and the segment recomputation follow the
// mixed trajectory, and each stage is linearised in FP64 at its states.
static Error adjoint_supported(const Input& in) {
    if (in.adv_type != 1 && in.adv_type != 2) return {4, "the adjoint covers advection types 1 and 2"};
    if (in.problem_type == 11) return {4, "the adjoint does not cover hybrid runs (problem type 11)"};
    return {0, ""};
}

Error Solver::stage_adjoint(double coeff, const double* lam_k, double* lam_w, double* lam_pv) {
    HO2D_TRY(adjoint_supported(in_));
    HO2D_TRY(adjoint_prepare());
    DeviceState& d = *d_;
    AdjointState& a = *adj_;
    const size_t nv = (size_t)mesh_.n_el * in_.knod * in_.knod, nb = (size_t)mesh_.n_eb * in_.knod;
    if (stage32_) {  // the FP32 stage input kept, and widened in place for the FP64 stage
        if (a.w32_save.bytes() < nv * 4) HO2D_TRY(adjoint_alloc(a.w32_save, nv * 4, "alloc"));
        HO2D_CUDA(cudaMemcpyAsync(a.w32_save.get(), d.w_stage.get(), nv * 4, cudaMemcpyDeviceToDevice, d.stream),
                  "copy");
        HO2D_CUDA(launch_copy_f2d(a.w32_save.as<float>(), d.w_stage.as<double>(), nv, d.stream), "f2d");
    }
    HO2D_TRY(stage_t<double>(coeff, 0, false, true));  // the stage at the current state: psi of this input
    HO2D_CUDA(cudaMemcpyAsync(a.lam_k.get(), lam_k, nv * 8, cudaMemcpyHostToDevice, d.stream), "copy");
    HO2D_CUDA(cudaMemsetAsync(a.lpv.get(), 0, a.lpv.bytes(), d.stream), "memset");
    HO2D_TRY(stage_adjoint_dev(coeff, a.lw_out.as<double>()));
    HO2D_CUDA(cudaMemcpyAsync(lam_w, a.lw_out.get(), nv * 8, cudaMemcpyDeviceToHost, d.stream), "copy");
    if (lam_pv && nb) HO2D_CUDA(cudaMemcpyAsync(lam_pv, a.lpv.get(), nb * 8, cudaMemcpyDeviceToHost, d.stream), "copy");
    if (stage32_)  // the FP32 stage input back
        HO2D_CUDA(cudaMemcpyAsync(d.w_stage.get(), a.w32_save.get(), nv * 4, cudaMemcpyDeviceToDevice, d.stream),
                  "copy");
    HO2D_CUDA(cudaStreamSynchronize(d.stream), "stage adjoint");
    return {0, ""};
}

Error Solver::apply_poisson_transpose(const double* x, double* y) {
    HO2D_TRY(adjoint_prepare());
    DeviceState& d = *d_;
    AdjointState& a = *adj_;
    const size_t nv = (size_t)mesh_.n_el * in_.knod * in_.knod;
    HO2D_CUDA(cudaMemcpyAsync(a.lpsi.get(), x, nv * 8, cudaMemcpyHostToDevice, d.stream), "copy");
    HO2D_CUDA(cudaMemsetAsync(a.sv.get(), 0, a.sv.bytes(), d.stream), "memset");  // shared with FP32
    HO2D_CUDA(cudaMemsetAsync(a.sg.get(), 0, a.sg.bytes(), d.stream), "memset");
    const ReduceScratch rs = reduce_scratch(d);
    HO2D_CUDA(mf_apply_transpose<double>(make_op<double>(d, mesh_, in_.knod, false), a.lpsi.as<double>(),
                                         a.mu.as<double>(), a.sv.as<double>(), a.sg.as<double>(), a.mu.as<double>(),
                                         nullptr, nullptr, rs, d.stream),
              "transposed operator");
    launches_ += 2;
    HO2D_CUDA(cudaMemcpyAsync(y, a.mu.get(), nv * 8, cudaMemcpyDeviceToHost, d.stream), "copy");
    HO2D_CUDA(cudaStreamSynchronize(d.stream), "apply transpose");
    return {0, ""};
}

// One stored FP64 field of the time loop (checkpoint, segment stage input or psi), kept in
// FP64 or, with FP32 state storage, rounded to FP32.
Error Solver::store_state(void* dst, const double* src) {
    DeviceState& d = *d_;
    const size_t nv = (size_t)mesh_.n_el * in_.knod * in_.knod;
    if (adj_->state_bytes == 4) HO2D_CUDA(launch_copy_d2f(src, static_cast<float*>(dst), nv, d.stream), "store state");
    else HO2D_CUDA(cudaMemcpyAsync(dst, src, nv * 8, cudaMemcpyDeviceToDevice, d.stream), "store state");
    return {0, ""};
}

Error Solver::load_state(double* dst, const void* src) {
    DeviceState& d = *d_;
    const size_t nv = (size_t)mesh_.n_el * in_.knod * in_.knod;
    if (adj_->state_bytes == 4) HO2D_CUDA(launch_copy_f2d(static_cast<const float*>(src), dst, nv, d.stream), "load state");
    else HO2D_CUDA(cudaMemcpyAsync(dst, src, nv * 8, cudaMemcpyDeviceToDevice, d.stream), "load state");
    return {0, ""};
}

// The stage input d.w_stage from omega, in the stage precision (FP32 under HO2D_MIXED).
static cudaError_t stage_input_from(const DeviceState& d, bool stage32, const double* w, size_t nv) {
    if (stage32) return launch_copy_d2f(w, d.w_stage.as<float>(), nv, d.stream);
    return cudaMemcpyAsync(d.w_stage.get(), w, nv * 8, cudaMemcpyDeviceToDevice, d.stream);
}

Error Solver::adjoint_forward(int nsteps, int ckpt_every) {
    const NvtxRange nvtx_range("ho2d.adjoint_forward");
    HO2D_TRY(adjoint_supported(in_));
    if (nsteps < 0 || ckpt_every < 1) return {1, "adjoint_forward needs nsteps >= 0 and ckpt_every >= 1"};
    HO2D_TRY(adjoint_prepare());
    DeviceState& d = *d_;
    AdjointState& a = *adj_;
    const size_t nv = (size_t)mesh_.n_el * in_.knod * in_.knod;
    const int nck = (nsteps + ckpt_every - 1) / ckpt_every;
    const size_t wb = adj_state32_ ? 4 : 8;  // bytes per stored value
    if (a.state_bytes != wb) {
        a.ckpt.clear();
        a.seg_w.reset();
        a.seg_psi.reset();
        a.state_bytes = wb;
    }
    while ((int)a.ckpt.size() < nck) {
        std::unique_ptr<DeviceBuffer> b(new DeviceBuffer);
        HO2D_TRY(adjoint_alloc(*b, nv * wb, "alloc checkpoint"));
        a.ckpt.push_back(std::move(b));
    }
    a.nsteps = -1;  // valid again once the sweep completes
    a.t0 = time_;
    a.every = ckpt_every;
    // the stage input of a step is omega itself
    HO2D_CUDA(stage_input_from(d, stage32_, d.omega.as<double>(), nv), "copy");
    for (int n = 0; n < nsteps; ++n) {
        if (n % ckpt_every == 0) HO2D_TRY(store_state(a.ckpt[n / ckpt_every]->get(), d.omega.as<double>()));
        HO2D_TRY(step(1));
    }
    HO2D_CUDA(cudaMemcpyAsync(a.wT.get(), d.omega.get(), nv * 8, cudaMemcpyDeviceToDevice, d.stream), "copy");
    HO2D_CUDA(cudaMemcpyAsync(a.psiT.get(), d.psi64.get(), nv * 8, cudaMemcpyDeviceToDevice, d.stream), "copy");
    HO2D_CUDA(cudaStreamSynchronize(d.stream), "adjoint forward");
    a.nsteps = nsteps;
    return {0, ""};
}

Error Solver::adjoint_backward(const double* dJ_dw, double* grad_w0, double* grad_pv) {
    const NvtxRange nvtx_range("ho2d.adjoint_backward");
    HO2D_TRY(adjoint_supported(in_));
    if (!adj_ || adj_->nsteps < 0) return {1, "ho2d_adjoint_backward needs a completed ho2d_adjoint_forward"};
    HO2D_TRY(adjoint_prepare());
    DeviceState& d = *d_;
    AdjointState& a = *adj_;
    HO2D_CUDA(cudaSetDevice(d.device), "cudaSetDevice");
    const size_t nv = (size_t)mesh_.n_el * in_.knod * in_.knod, nb = (size_t)mesh_.n_eb * in_.knod;
    const Tableau tb = tableau(in_.ti_type);
    const int ns = tb.ns, every = a.every, nsteps = a.nsteps;
    const size_t wb = a.state_bytes;
    const size_t seg_bytes = (size_t)every * ns * nv * wb;
    if (a.seg_w.bytes() < seg_bytes) {
        HO2D_TRY(adjoint_alloc(a.seg_w, seg_bytes, "alloc segment"));
        HO2D_TRY(adjoint_alloc(a.seg_psi, seg_bytes, "alloc segment"));
    }
    char* seg_w = static_cast<char*>(a.seg_w.get());
    char* seg_psi = static_cast<char*>(a.seg_psi.get());
    double* lam = a.lam.as<double>();
    double* lk = a.lam_k.as<double>();
    auto copy = [&](void* dst, const void* src) -> Error {
        HO2D_CUDA(cudaMemcpyAsync(dst, src, nv * 8, cudaMemcpyDeviceToDevice, d.stream), "copy");
        return {0, ""};
    };
    HO2D_CUDA(cudaMemcpyAsync(lam, dJ_dw, nv * 8, cudaMemcpyHostToDevice, d.stream), "copy");
    HO2D_CUDA(cudaMemsetAsync(a.lpv.get(), 0, a.lpv.bytes(), d.stream), "memset");
    const int nseg = (nsteps + every - 1) / every;
    for (int seg = nseg - 1; seg >= 0; --seg) {
        const int n0 = seg * every, n1 = std::min(nsteps, n0 + every);
        // recompute the segment from its checkpoint, keeping every stage input and psi; the
        // stages are the FP64 ones the adjoint linearises (under HO2D_MIXED the checkpoints
        // come from the FP32-stage trajectory and each segment is recomputed in FP64 from them)
        HO2D_TRY(load_state(d.omega.as<double>(), a.ckpt[seg]->get()));
        HO2D_TRY(copy(d.w_stage.get(), d.omega.get()));
        for (int n = n0; n < n1; ++n) {
            time_ = a.t0 + n * in_.dt;
            for (int s = 0; s < ns; ++s) {
                const size_t off = ((size_t)(n - n0) * ns + s) * nv * wb;
                HO2D_TRY(store_state(seg_w + off, d.w_stage.as<double>()));
                HO2D_TRY(stage_t<double>(tb.c[s], s, true));
                HO2D_TRY(store_state(seg_psi + off, d.psi64.as<double>()));
            }
        }
        // reverse sweep: lam_k_s = b_s lam + sum_{r > s} a_rs mu_r, lam += sum_s mu_s
        for (int n = n1 - 1; n >= n0; --n) {
            for (int s = ns - 1; s >= 0; --s) {
                const size_t off = ((size_t)(n - n0) * ns + s) * nv * wb;
                HO2D_CUDA(launch_axpby(nv, lk, tb.b[s], lam, 0.0, lam, d.stream), "lam_k");
                for (int r = s + 1; r < ns; ++r)
                    if (tb.a[r][s] != 0.0) HO2D_CUDA(launch_axpby(nv, lk, 1.0, lk, tb.a[r][s], a.mus[r].as<double>(), d.stream), "lam_k");
                HO2D_TRY(load_state(d.w_stage.as<double>(), seg_w + off));
                HO2D_TRY(load_state(d.psi64.as<double>(), seg_psi + off));
                time_ = a.t0 + n * in_.dt;
                HO2D_TRY(stage_adjoint_dev(tb.c[s], a.mus[s].as<double>()));
            }
            for (int s = 0; s < ns; ++s) HO2D_CUDA(launch_axpby(nv, lam, 1.0, lam, 1.0, a.mus[s].as<double>(), d.stream), "lam");
            launches_ += 2 * ns + 1;
        }
    }
    HO2D_CUDA(cudaMemcpyAsync(grad_w0, lam, nv * 8, cudaMemcpyDeviceToHost, d.stream), "copy");
    if (grad_pv && nb) HO2D_CUDA(cudaMemcpyAsync(grad_pv, a.lpv.get(), nb * 8, cudaMemcpyDeviceToHost, d.stream), "copy");
    // back to the state at T
    HO2D_TRY(copy(d.omega.get(), a.wT.get()));
    HO2D_CUDA(stage_input_from(d, stage32_, a.wT.as<double>(), nv), "copy");
    HO2D_TRY(copy(d.psi64.get(), a.psiT.get()));
    time_ = a.t0 + nsteps * in_.dt;
    HO2D_CUDA(cudaStreamSynchronize(d.stream), "adjoint backward");
    return {0, ""};
}

template Error Solver::kt_run<double>(double*, const double*, bool, double, int&);
template Error Solver::kt_run<float>(float*, const float*, bool, double, int&);

}  // namespace ho2d
