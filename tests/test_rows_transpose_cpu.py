"""The row-parallel Poisson operator and its transpose (rows.cuh, rows_transpose.cuh: the source
that the solver's kernels are compiled from) on the host (tests/rows_harness.cpp, a thread per
lane) against the oracle's assembled matrix and its transpose, at every order, on meshes with
Dirichlet and Neumann faces and with faces met in both directions.

Tolerance: both sums have about 10 K^2 terms of size up to max|A| max|x|: 1e-12 of the norm.
"""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import REPO
from turned import reversed_faces, turned_cavity

from ho2d import meshgen

import ho2d_oracle as O

CSRC = os.path.join(REPO, "ho-cxx_b200", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    inc = "/usr/local/cuda/include"
    if shutil.which("g++") is None or not os.path.isfile(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("g++ or cuda_runtime.h not available")
    out = str(tmp_path_factory.mktemp("rows_harness") / "l.so")
    subprocess.run(["g++", "-O1", "-std=c++20", "-shared", "-fPIC", "-pthread", "-w", "-I", inc, "-I", CSRC,
                    os.path.join(REPO, "tests", "rows_harness.cpp"), "-o", out], check=True, capture_output=True, text=True)
    return ctypes.CDLL(out)


def geometry(c):
    """The oracle case in the device layout of PoisGeom: face arrays [N][K][4]."""
    K, N, M, B = c.K, c.N, c.M, c.B
    xx, xe, yx, ye, J = (M[k].reshape(N, K, K) for k in ("xxi", "xeta", "yxi", "yeta", "J"))
    g = [(xe * xe + ye * ye) / J, -(xx * xe + yx * ye) / J, (xx * xx + yx * yx) / J]
    fa, fb = (M[k].reshape(N, 4, K) / M["fJ"].reshape(N, 4, K) for k in ("fA", "fB"))
    nfa, nfb = np.zeros_like(fa), np.zeros_like(fb)
    code, scat = np.full((N, 4), -1, np.int32), np.full((N, K, 4), -1, np.int32)
    minv = np.zeros((max(1, c.neb), K, K))
    rev = reversed_faces(c)
    for el in range(N):
        for f in range(4):
            nb, nf = c.f_nbr[el, f], c.f_nijp[el, f]
            if nb >= 0:
                code[el, f] = nf + 4 * rev[el, f]
                for k in range(K):
                    kn = K - 1 - k if rev[el, f] else k
                    nfa[el, f, k], nfb[el, f, k] = fa[nb, nf, kn], fb[nb, nf, kn]
                    scat[nb, kn, nf] = (el * K + k) * 4 + f
                continue
            e = c.f_bidx[el, f]
            if c.sw_p[e] == O.DIRICHLET:
                continue
            code[el, f] = -2 - e  # rows k of the common-value system: -fb_k l_c'(x_k) + fa_k g' delta_kc
            A = -fb[el, f][:, None] * B.D.reshape(K, K).T + np.diag(fa[el, f] * B.gp[f & 1])
            minv[e] = np.linalg.inv(A)
    bases = np.zeros(64 + 16 * 4 + 2)
    bases[:K * K] = B.D.ravel()
    for off, arr in ((64, B.sbb), (80, B.sbgb), (96, B.R), (112, B.gR)):
        bases[off:off + 2 * K] = arr.ravel()
    bases[128:130] = B.gp
    faces = [np.ascontiguousarray(a.transpose(0, 2, 1)) for a in (fa, fb, nfa, nfb)]
    return [np.ascontiguousarray(a) for a in g], faces, minv, code, scat, bases


def pointers(arrays):
    return (ctypes.c_void_p * len(arrays))(*[a.ctypes.data for a in arrays])


CASES = [("turned%d" % n, k) for n, k in ((5, 2), (4, 3), (5, 4), (4, 5), (3, 6), (3, 7), (3, 8))] + \
    [("cyl4x9", 4), ("bfs2", 3), ("cavityq3", 4), ("cavityj7", 5)]


@pytest.mark.parametrize("mesh,knod", CASES)
def test_operator_and_transpose_match_the_assembled_matrix(lib, tmp_path, mesh, knod):
    if mesh.startswith("turned"):
        inp = turned_cavity(str(tmp_path), int(mesh[6:]), knod)
    else:
        inp = meshgen.make_case(mesh, str(tmp_path), knod=knod, steps=1)
    c = O.Case(inp)
    if mesh.startswith("turned"):
        n_rev = reversed_faces(c).sum()
        assert 0 < n_rev < (c.f_nbr >= 0).sum()
    g, f, minv, code, scat, bases = geometry(c)
    x = np.random.Generator(np.random.PCG64(7)).standard_normal(c.N * c.K * c.K)
    y = np.zeros_like(x)
    for transposed, A in ((0, c.A), (1, c.A.T)):
        assert lib.poisson_rows_host(c.K, c.N, pointers(g), pointers(f), *[ctypes.c_void_p(a.ctypes.data) for a in
                                     (minv, code, scat, bases, x, y)], transposed) == 0
        ref = A @ x
        assert np.linalg.norm(y - ref) <= 1e-12 * np.linalg.norm(ref), (transposed, np.linalg.norm(y - ref))
