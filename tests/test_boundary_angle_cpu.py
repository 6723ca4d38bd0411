"""Re-entrant corners of the domain (largest_boundary_angle, host build, no GPU), on whose presence the FP64
solve's stopping residual depends: the backward-facing step has one, walls, round bodies and quadratic
elements' straight walls have none.
"""

import ctypes
import math
import os
import shutil
import subprocess

import pytest

from turned import turned_cavity

from ho2d import meshgen

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "ho-cxx_b200", "csrc")

HARNESS = """
#include "host.hpp"
using namespace ho2d;
extern "C" int boundary_angle(const char* path, double* angle, int* corner) {
    Input in; Mesh m;
    Error e = read_input(path, in);
    if (!e.code) e = read_msh(in.base_dir + "/" + in.mesh_file, in.occ, m);
    *angle = largest_boundary_angle(m);
    *corner = *angle > kCornerAngle;
    return e.code;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("angle_harness")
    (d / "h.cpp").write_text(HARNESS)
    srcs = [str(d / "h.cpp")] + [os.path.join(CSRC, f) for f in ("host_io.cpp", "host_setup.cpp", "host_hybrid.cpp",
                                                                "host_amg.cpp", "host_kron.cpp")]
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, *srcs, "-o", str(d / "l.so")], check=True,
                   capture_output=True, text=True)
    return ctypes.CDLL(str(d / "l.so"))


@pytest.mark.parametrize("mesh,degrees,corner", [("cavity4", 180, False), ("cavityj5", 180, False), ("turned5", 180, False),
                                                 ("cavityq3", 180, False), ("bfs2", 270, True), ("cyl4x8", 225, False),
                                                 ("cyl3x4", 270, True), ("cyl5x40", 189, False)])
def test_largest_boundary_angle(lib, tmp_path, mesh, degrees, corner):
    if mesh.startswith("turned"):
        inp = turned_cavity(str(tmp_path), 5, 3)
    else:
        inp = meshgen.make_case(mesh, str(tmp_path), knod=3, steps=1)
    a, c = ctypes.c_double(), ctypes.c_int()
    assert lib.boundary_angle(inp.encode(), ctypes.byref(a), ctypes.byref(c)) == 0
    assert abs(math.degrees(a.value) - degrees) < 1e-6 and bool(c.value) == corner
