"""Storage of the coarsest inverse in the FP32 preconditioner (host build, no GPU): BF16 only on
meshes of more than 1,024 elements whose hierarchy has a level below level 0. Level 0 is inverted
directly up to 512 unknowns, so cavities of 24 to 32 elements a side have two levels and still
keep FP32.
"""

import ctypes
import os
import shutil
import subprocess

import pytest

from ho2d import meshgen

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "ho-cxx_b200", "csrc")

HARNESS = """
#include "host.hpp"
#include "host_amg.hpp"
using namespace ho2d;
extern "C" int dense_storage(const char* path, int* levels, int* bf16) {
    Input in; Mesh m; Bases B; Metrics M; BoundaryConditions bc; CoarseHierarchy H;
    Error e = read_input(path, in);
    if (!e.code) e = read_msh(in.base_dir + "/" + in.mesh_file, in.occ, m);
    if (!e.code) e = make_bases(in.knod, m.lnod, B);
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
    e = build_coarse_hierarchy(coarse_operator(coarse_space(m, B, bc), B, g), H, kDenseMax, kDenseMaxFirst, false);
    *levels = (int)H.levels.size();
    *bf16 = dense_in_bf16(m.n_el, *levels);
    return e.code;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("dense_harness")
    (d / "h.cpp").write_text(HARNESS)
    srcs = [str(d / "h.cpp")] + [os.path.join(CSRC, f) for f in ("host_io.cpp", "host_setup.cpp", "host_hybrid.cpp",
                                                                "host_amg.cpp", "host_kron.cpp")]
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, *srcs, "-o", str(d / "l.so")], check=True,
                   capture_output=True, text=True)
    return ctypes.CDLL(str(d / "l.so"))


@pytest.mark.parametrize("n,two_levels,bf16", [(16, False, False), (23, False, False), (24, True, False),
                                               (32, True, False), (33, True, True)])
def test_small_meshes_keep_the_inverse_in_fp32(lib, tmp_path, n, two_levels, bf16):
    inp = meshgen.make_case("cavity%d" % n, str(tmp_path), knod=2, steps=1)
    levels, b = ctypes.c_int(), ctypes.c_int()
    assert lib.dense_storage(inp.encode(), ctypes.byref(levels), ctypes.byref(b)) == 0
    assert (levels.value > 1, bool(b.value)) == (two_levels, bf16)
