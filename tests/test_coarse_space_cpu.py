"""The coarse space of the Poisson preconditioner (host build, no GPU): its tables against the
mesh, and its finite-element operator against R A P of the oracle's assembled Poisson matrix.

On elements whose sides are straight the two operators are the same: continuous functions
have no jumps, and the solution points' quadrature integrates both exactly. Tolerance: A's
entries are sums of about 4 K products of size up to max|A|, and R A P adds 25 K^4 of them,
so rounding stays below 1e-11 of the largest entry for K <= 8.
"""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from ho2d import meshgen

import ho2d_oracle as O

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "ho-cxx_b200", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("coarse_harness") / "libcoarse_harness.so")
    srcs = [os.path.join(REPO, "tests", "coarse_harness.cpp")] + [
        os.path.join(CSRC, f) for f in ("host_io.cpp", "host_setup.cpp", "host_hybrid.cpp", "host_amg.cpp", "host_kron.cpp")]
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, *srcs, "-o", out], check=True,
                   capture_output=True, text=True)
    return ctypes.CDLL(out)


def coarse(lib, inp, N, K):
    dims = (ctypes.c_long * 3)()
    null = ctypes.c_void_p()
    assert lib.coarse_case(inp.encode(), dims, null, null, null, null, null, null, null) == 0
    n, vw, nnz = dims
    a = dict(conn=np.zeros((N, 4), np.int32), v2e=np.zeros((n, vw), np.int32), hp=np.zeros((K, 2)), hr=np.zeros((K, 2)),
             ptr=np.zeros(n + 1, np.int32), col=np.zeros(nnz, np.int32), val=np.zeros(nnz))
    assert lib.coarse_case(inp.encode(), dims, *[x.ctypes.data_as(ctypes.c_void_p) for x in a.values()]) == 0
    return n, a


def hats(a, hx):
    """[K2][4] tensor hats, corners (-,-), (+,-), (+,+), (-,+), points [j][i]."""
    return np.stack([np.outer(hx[:, y], hx[:, x]).ravel() for x, y in ((0, 0), (1, 0), (1, 1), (0, 1))], 1)


def interpolation(a, n, N, K, hx):
    K2 = K * K
    rows = np.repeat(np.arange(N * K2).reshape(N, K2, 1), 4, 2)
    cols = np.repeat(a["conn"][:, None, :], K2, 1)
    vals = np.repeat(hats(a, hx)[None], N, 0)
    keep = cols >= 0
    return sp.csr_matrix((vals[keep], (rows[keep], cols[keep])), shape=(N * K2, n))


@pytest.mark.parametrize("mesh,knod", [("cavityj5", 2), ("cavityj6", 3), ("cavityj4", 5), ("cavityj3", 8), ("cyl4x8", 4),
                                       ("cavity2", 3)])
def test_tables_and_operator(lib, tmp_path, mesh, knod):
    inp = meshgen.make_case(mesh, str(tmp_path), knod=knod, steps=1)
    c = O.Case(inp)
    N, K = c.N, c.K
    n, a = coarse(lib, inp, N, K)
    conn, v2e = a["conn"], a["v2e"]
    # the tables: a corner has an unknown exactly when its node is on no Dirichlet edge, the
    # same one in every element it belongs to; v2e lists each unknown's corners once
    nodes = np.array([q[:4] for q in c.mesh.elem_nodes])
    fixed = {v for e in range(c.neb) if c.sw_p[e] == O.DIRICHLET for v in c.mesh.edge_nodes[e][:2]}
    of_node = {}
    for el in range(N):
        for q in range(4):
            assert (conn[el, q] < 0) == (nodes[el, q] in fixed)
            assert of_node.setdefault(nodes[el, q], conn[el, q]) == conn[el, q]
    assert sorted(v for v in of_node.values() if v >= 0) == list(range(n))
    for v in range(n):
        lst = v2e[v][v2e[v] >= 0]
        assert list(lst) == sorted(np.flatnonzero(conn.ravel() == v))
    # hats: a partition of unity; hr = hp times K times the normalised quadrature weight
    x, w = np.polynomial.legendre.leggauss(K)
    np.testing.assert_allclose(a["hp"], np.stack([(1 - x) / 2, (1 + x) / 2], 1), rtol=0, atol=1e-14)
    np.testing.assert_allclose(a["hr"], a["hp"] * (K * w / 2)[:, None], rtol=0, atol=1e-14)
    # operator
    F = sp.csr_matrix((a["val"], a["col"], a["ptr"]), shape=(n, n))
    assert abs(F - F.T).max() <= 1e-13 * abs(F).max()
    P, R = interpolation(a, n, N, K, a["hp"]), interpolation(a, n, N, K, a["hr"]).T
    G = sp.csr_matrix(R @ c.A @ P)
    # (cyl4x8: Neumann outlet; its lift of the boundary flux is not in F)
    tol = 1e-11 if mesh.startswith("cavity") else 0.05
    assert abs(F - G).max() <= tol * abs(G).max()


def test_order_one_is_the_element_space(lib, tmp_path):
    inp = meshgen.make_case("cavityj5", str(tmp_path), knod=1, steps=1)
    n, a = coarse(lib, inp, 25, 1)
    assert n == 25 and list(a["conn"][:, 0]) == list(range(25)) and (a["conn"][:, 1:] == -1).all()
    assert list(a["v2e"].ravel()) == [4 * e for e in range(25)]


def test_all_vertices_fixed_leaves_an_empty_space(lib, tmp_path):
    inp = meshgen.make_case("cavity1", str(tmp_path), knod=3, steps=1)
    n, a = coarse(lib, inp, 1, 3)
    assert n == 0 and (a["conn"] == -1).all()
