// rows_harness.cpp -- the row-parallel Poisson operator and its transpose (rows.cuh,
// rows_transpose.cuh) run on the host, for CPU tests: each warp is 32 threads, __syncwarp a
// barrier between them, so the device source itself runs, phase by phase. Element geometry and
// bases come from the test in the device layout (PoisGeom, DevBases). Never part of the library.
#include <cuda_runtime.h>

#include <barrier>
#include <cstring>
#include <thread>
#include <vector>

namespace {
struct Warp {
    std::barrier<> bar{32};
    int votes[32];
};
thread_local Warp* t_warp = nullptr;
thread_local struct { unsigned x; } t_idx;
}  // namespace

template <typename T>
T __ldg(const T* p) { return *p; }
template <typename T>
T __ldcg(const T* p) { return *p; }
inline void __syncwarp() { t_warp->bar.arrive_and_wait(); }
inline int __any_sync(unsigned, int v) {
    t_warp->votes[t_idx.x & 31] = v;
    __syncwarp();
    int any = 0;
    for (int i = 0; i < 32; ++i) any |= t_warp->votes[i];
    __syncwarp();
    return any;
}
#define threadIdx t_idx

#include "rows_transpose.cuh"

using namespace ho2d;

namespace {

// body(ix, sm) on every lane of every warp of the mesh
template <int K, typename F>
void for_warps(int N, F body) {
    using R = Rows<K>;
    for (int w = 0; w < (N + R::EPW - 1) / R::EPW; ++w) {
        Warp warp;
        RowScratch<K, double> sm;
        std::vector<std::thread> lanes;
        for (int l = 0; l < 32; ++l)
            lanes.emplace_back([&, l] {
                t_warp = &warp;
                t_idx.x = (unsigned)((w % R::WARPS) * 32 + l);
                body(RowIdx<K>(N, w / R::WARPS), sm);
            });
        for (auto& t : lanes) t.join();
    }
}

template <int K>
int apply_k(const MfOp<double>& op, const double* x, double* y, double* s1, double* s2, int transposed) {
    const int N = op.g.N;
    if (!transposed) {
        for_warps<K>(N, [&](const RowIdx<K>& ix, RowScratch<K, double>& sm) {
            double row[K];
            int dst[4];
            if (ix.active) {
                load_row<K, double>(x + (size_t)ix.el * K * K + ix.t * K, row);
                load4i(op.g.scat + ((size_t)ix.el * K + ix.t) * 4, dst);
            }
            row_emit_traces<K, double>(op.b, sm.tr[0][ix.lw], row, dst, s1, s2, ix.t, ix.active);
        });
        for_warps<K>(N, [&](const RowIdx<K>& ix, RowScratch<K, double>& sm) {
            ApplyIn<K, double> in;
            row_apply_load<K, double>(op.g, x, s1, s2, ix, in);
            double r[K];
            row_apply_core<K, double>(op, in, sm, ix, r);
            if (ix.active) store_row<K, double>(y + (size_t)ix.el * K * K + ix.t * K, r);
        });
        return 0;
    }
    std::vector<double> own((size_t)N * K * K);
    for_warps<K>(N, [&](const RowIdx<K>& ix, RowScratch<K, double>& sm) {
        double z[K], o[K];
        for (int i = 0; i < K; ++i) z[i] = 0.0;
        if (ix.active) load_row<K, double>(x + (size_t)ix.el * K * K + ix.t * K, z);
        row_transpose_own<K, double>(op, z, sm, ix, s1, s2, o);
        if (ix.active) store_row<K, double>(own.data() + (size_t)ix.el * K * K + ix.t * K, o);
    });
    for_warps<K>(N, [&](const RowIdx<K>& ix, RowScratch<K, double>& sm) {
        double r[K];
        row_transpose_gather<K, double>(op.b, own.data(), s1, s2, sm.tr[0][ix.lw], ix, r);
        if (ix.active) store_row<K, double>(y + (size_t)ix.el * K * K + ix.t * K, r);
    });
    return 0;
}

}  // namespace

// y = A x, or A^T x with transposed. g: G11, G12, G22 [N][K][K]; f: fa, fb, nfa, nfb [N][K][4];
// scat [N][K][4], code [N][4], minv [N_eb][K][K]; bases as DevBases<double>.
extern "C" int poisson_rows_host(int K, int N, const double* const* g, const double* const* f, const double* minv,
                                 const int* code, const int* scat, const double* bases, const double* x, double* y,
                                 int transposed) {
    MfOp<double> op;
    op.K = K;
    op.g.N = N;
    op.g.G11 = g[0];
    op.g.G12 = g[1];
    op.g.G22 = g[2];
    op.g.fa = f[0];
    op.g.fb = f[1];
    op.g.nfa = f[2];
    op.g.nfb = f[3];
    op.g.minv = minv;
    op.g.code = code;
    op.g.scat = scat;
    std::memcpy(&op.b, bases, sizeof op.b);
    // the incoming slots, 16-byte aligned as the device's; boundary entries stay zero
    std::vector<double> s1((size_t)N * 4 * K, 0.0), s2((size_t)N * 4 * K, 0.0);
    switch (K) {
        case 2: return apply_k<2>(op, x, y, s1.data(), s2.data(), transposed);
        case 3: return apply_k<3>(op, x, y, s1.data(), s2.data(), transposed);
        case 4: return apply_k<4>(op, x, y, s1.data(), s2.data(), transposed);
        case 5: return apply_k<5>(op, x, y, s1.data(), s2.data(), transposed);
        case 6: return apply_k<6>(op, x, y, s1.data(), s2.data(), transposed);
        case 7: return apply_k<7>(op, x, y, s1.data(), s2.data(), transposed);
        case 8: return apply_k<8>(op, x, y, s1.data(), s2.data(), transposed);
        default: return 1;
    }
}
