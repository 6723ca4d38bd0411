// coarse_harness.cpp -- host build of the coarse space of the Poisson preconditioner
// (coarse_space and coarse_operator in ho-cxx_b200/csrc/host_amg.cpp) for CPU tests.
#include <algorithm>
#include <string>
#include <vector>

#include "host.hpp"
#include "host_amg.hpp"

// The case's coarse space and operator: dims = {unknowns, vw, nonzeros}; the arrays are
// written when given.
extern "C" int coarse_case(const char* path, long* dims, int* conn, int* v2e, double* hp, double* hr, int* ptr, int* col,
                           double* val) {
    using namespace ho2d;
    Input in;
    Mesh m;
    Bases B;
    Metrics M;
    BoundaryConditions bc;
    Error e = read_input(path, in);
    if (e.code) return e.code;
    e = read_msh(in.base_dir + "/" + in.mesh_file, in.occ, m);
    if (e.code) return e.code;
    e = make_bases(in.knod, m.lnod, B);
    if (e.code) return e.code;
    make_metrics(m, B, M);
    e = setup_bcs(in, m, B, bc);
    if (e.code) return e.code;
    std::vector<double> g[3];
    for (size_t p = 0; p < M.J.size(); ++p) {
        g[0].push_back((M.xeta[p] * M.xeta[p] + M.yeta[p] * M.yeta[p]) / M.J[p]);
        g[1].push_back(-(M.xxi[p] * M.xeta[p] + M.yxi[p] * M.yeta[p]) / M.J[p]);
        g[2].push_back((M.xxi[p] * M.xxi[p] + M.yxi[p] * M.yxi[p]) / M.J[p]);
    }
    const CoarseSpace s = coarse_space(m, B, bc);
    const Csr A = B.K > 1 && s.n ? coarse_operator(s, B, g) : Csr();
    dims[0] = s.n;
    dims[1] = s.vw;
    dims[2] = (long)A.col.size();
    if (!conn) return 0;
    std::copy(s.conn.begin(), s.conn.end(), conn);
    std::copy(s.v2e.begin(), s.v2e.end(), v2e);
    std::copy(s.hp.begin(), s.hp.end(), hp);
    std::copy(s.hr.begin(), s.hr.end(), hr);
    std::copy(A.ptr.begin(), A.ptr.end(), ptr);
    std::copy(A.col.begin(), A.col.end(), col);
    std::copy(A.val.begin(), A.val.end(), val);
    return 0;
}
