// host_amg.hpp -- coarse space of the Poisson preconditioner and its smoothed-aggregation
// hierarchy (host setup).
#pragma once

#include <vector>

#include "host.hpp"

namespace ho2d {

// The coarsest level is inverted densely once it has at most this many rows; the device
// applies the inverse as one grid-wide matrix-vector product (4096^2 FP32 values = 64 MB).
// Level 0 is inverted densely only below kDenseMaxFirst rows: beyond that one coarsening
// step is cheaper than a large dense level 0 (16 FP64 solves at K = 5, one kernel each: 900
// rows dense 19.3 ms, 1,521 rows with a second level 16.7 ms).
constexpr int kDenseMax = 4096;
constexpr int kDenseMaxFirst = 512;

struct Csr {
    int n = 0, m = 0;
    std::vector<int> ptr, col;
    std::vector<double> val;
};

struct AmgLevel {
    Csr A, P, R;            // P, R empty on the coarsest level
    std::vector<double> m;  // SPAI-0 smoother weights
    // The V(1,1) cycle of this level with pre-smoothing from zero, u' = m .* f, and
    // post-smoothing u = u'' + m .* (f - A u''), u'' = u' + P u_c, as three fixed operators:
    //   f_c = M f,  u = S f + Q u_c   with
    //   M = R (I - A diag(m)),  S = 2 diag(m) - diag(m) A diag(m),  Q = (I - diag(m) A) P.
    Csr M, S, Q;  // empty on the coarsest level
};

// Row-padded (ELL) copy of a sparse matrix: every row holds exactly w entries (w a
// multiple of 4), padding entries have column 0 and value 0, so a row is read without a
// row pointer and every row starts on a 16-byte boundary.
struct Ell {
    int n = 0, m = 0, w = 0;
    std::vector<int> col;     // [n][w]
    std::vector<double> val;  // [n][w]
};
Ell to_ell(const Csr& A);

// Whether the FP32 preconditioner holds the coarsest inverse in BF16 (half the bytes of the
// largest coarse read; the preconditioner's precision changes only the iteration count): where
// it is a level below level 0, on meshes of more than kDense16Elements elements. Smaller ones
// keep FP32: their coarsest level has a few hundred rows and is read from L2.
constexpr int kDense16Elements = 1024;
inline bool dense_in_bf16(int n_el, int levels) { return levels > 1 && n_el > kDense16Elements; }

struct CoarseHierarchy {
    std::vector<AmgLevel> levels;  // levels[0] is the coarse space's own operator
    int n_dense = 0;
    std::vector<double> dense_inv;  // row-major inverse of the coarsest operator
};

// The coarse space: a value at every mesh vertex off the Dirichlet boundary, interpolated
// bilinearly in each element's reference square. conn[4 el + c]: the unknown at corner c
// ((-,-), (+,-), (+,+), (-,+)) or -1; v2e: per unknown the vw-wide list of the corners
// (4 el + c, ascending; -1 pads) that meet in it; hp, hr [K][2]: the 1-D hats at the solution
// points and the hats times K quadrature weights (HatBases, fr_launch.hpp). Unknowns are
// numbered in the order the elements meet them, so they are as local as the elements.
// At order 1 an element has one value and the space is the elements themselves (P = identity).
struct CoarseSpace {
    int n = 0, vw = 0;
    std::vector<int> conn, v2e;
    std::vector<double> hp, hr;
};
CoarseSpace coarse_space(const Mesh& m, const Bases& B, const BoundaryConditions& bc);
// The bilinear finite-element Laplacian on that space, integrated with the solution points'
// quadrature: -K^2 sum_q w_q grad phi_a . G grad phi_b over the contravariant coefficients
// g[0..2] = G11, G12, G22 ([N][K][K]). On affine elements this is R A P of the FR operator to
// rounding, because continuous functions have no jumps to lift; elsewhere it differs from it
// by about 1% and is preferred for its 9-point rows (R A P has 21) and its symmetry, which
// lets the transposed problem use the same hierarchy.
Csr coarse_operator(const CoarseSpace& s, const Bases& B, const std::vector<double>* g);

// A1 = P^T A P for P = element indicator: the sum of each K^2 x K^2 block.
Csr p0_coarse_operator(const PoissonOperator& op, int N);
// Coarsens A1 until a level has at most dense_max rows (level 0 itself: at most
// dense_max_first rows) and inverts that level densely.
// invert_dense = false leaves H.dense_inv empty (the caller inverts the last level).
Error build_coarse_hierarchy(const Csr& A1, CoarseHierarchy& H, int dense_max = kDenseMax,
                             int dense_max_first = kDenseMaxFirst, bool invert_dense = true);

}  // namespace ho2d
