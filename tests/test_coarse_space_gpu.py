"""Poisson solves with the vertex coarse space on the GPU against the oracle's direct solve, at
the sizes where its tables and kernels have their edges: no unknown (one element), a single
one, every order, an element space (order 1), a Neumann outlet, a vertex with other than four
elements, and a dense level 0 too large for one CTA's shared memory (HO2D_DENSE_MAX).
"""

import numpy as np
import pytest

from ho2d import FP64, HO_2D, MIXED_KRYLOV, meshgen

import ho2d_oracle as O

pytestmark = pytest.mark.gpu


def solve(inp, precision, w0):
    s = HO_2D()
    s.read_input_file(inp)
    s.set_precision(precision)
    s.set_poisson_tolerance(1e-13, 2000)
    s.setup()
    s.set_vorticity(w0)
    s.Euler_time_integrate(0.0)
    psi = s.get_streamfunction()
    s.close()
    return psi


@pytest.mark.parametrize("precision", [FP64, MIXED_KRYLOV])
@pytest.mark.parametrize("mesh,knod,dense", [("cavity1", 3, None), ("cavity2", 3, None), ("cavityj3", 1, None),
                                             ("cavityj7", 2, None), ("cavityj33", 3, None), ("cavityj9", 4, None),
                                             ("cavityj8", 5, None), ("cavityj7", 6, None), ("cavityj5", 7, None),
                                             ("cavityj5", 8, None), ("cyl6x12", 4, None), ("cyl5x9", 1, None),
                                             ("cavityq5", 4, None), ("cavityj85", 2, "8000"), ("cavityj40", 3, "20")])
def test_streamfunction_matches_oracle(tmp_path, monkeypatch, mesh, knod, dense, precision):
    if dense:
        monkeypatch.setenv("HO2D_DENSE_MAX", dense)
    inp = meshgen.make_case(mesh, str(tmp_path), knod=knod, steps=1)
    c = O.Case(inp)
    w0 = np.random.Generator(np.random.PCG64(7)).standard_normal((c.N, c.K, c.K))
    c.omega = w0.copy()
    c.update_bcs(0.0)
    c.solve_poisson(w0)
    psi = solve(inp, precision, w0)
    # residual 1e-13 times the conditioning (below 1e4 at these sizes), as the parity tests
    assert np.abs(psi - c.psi).max() <= 1e-9 * np.abs(c.psi).max()


# both sides of the line between the one-kernel solve and the loop of launches (148 tiles of 32
# elements at K = 4): the same solve as host-driven launches (HO2D_GRAPHS=0) agrees, with the
# last tile full, one element short and one element over
@pytest.mark.parametrize("precision", [FP64, MIXED_KRYLOV])
@pytest.mark.parametrize("nr,nt", [(4, 8), (3, 11), (5, 13), (37, 128), (34, 139), (61, 78)])
def test_one_kernel_solve_and_launches(tmp_path, monkeypatch, nr, nt, precision):
    inp = meshgen.make_case("cyl%dx%d" % (nr, nt), str(tmp_path), knod=4, steps=1)
    w0 = np.random.Generator(np.random.PCG64(9)).standard_normal((nr * nt, 4, 4))
    psi = solve(inp, precision, w0)
    monkeypatch.setenv("HO2D_GRAPHS", "0")
    ref = solve(inp, precision, w0)
    # both at residual 1e-13; the conditioning of a stretched O-grid of this size is below 1e5
    assert np.abs(psi - ref).max() <= 2e-8 * np.abs(ref).max()
