"""The transposed solve as launches (k_tr_init, k_tr_own, k_tr_gather and k_post_a on the transposed
blocks, in the captured loop and driven from the host), which every mesh of more than 148
element tiles and every order above 6 runs, and the transposed operator on faces met in both
directions.
"""

import numpy as np
import pytest

from turned import reversed_faces, turned_cavity

from ho2d import FP64, HO_2D, MIXED_KRYLOV, meshgen

import ho2d_cs as CS
import ho2d_oracle as O

pytestmark = pytest.mark.gpu


def solver(inp, precision=FP64, tol=1e-13):
    s = HO_2D()
    s.read_input_file(inp)
    s.set_precision(precision)
    s.set_poisson_tolerance(tol, 2000)
    s.setup()
    return s


@pytest.mark.parametrize("knod", range(2, 9))
def test_operator_and_transpose_on_turned_elements(tmp_path, knod):
    """Sums of about 10 K^2 terms: 1e-12 of the norm, as in the CPU test of the same source."""
    inp = turned_cavity(str(tmp_path), 5, knod)
    c = O.Case(inp)
    assert 0 < reversed_faces(c).sum()
    s = solver(inp)
    x = np.random.Generator(np.random.PCG64(3)).standard_normal(c.N * c.K * c.K)
    for y, ref in ((s.apply_poisson(x), c.A @ x), (s.apply_poisson_transpose(x), c.A.T @ x)):
        assert np.linalg.norm(np.ravel(y) - ref) <= 1e-12 * np.linalg.norm(ref)
    s.close()


# graphs "1": one kernel up to order 6, the captured loop at 7 and 8; "0": launches from the host
@pytest.mark.parametrize("graphs", ["1", "0"])
@pytest.mark.parametrize("precision", [FP64, MIXED_KRYLOV])
@pytest.mark.parametrize("knod", range(2, 9))
def test_stage_adjoint_dot_product(tmp_path, monkeypatch, knod, precision, graphs):
    """<lam_k, J v> = <J^T lam_k, v> with J v the complex-step derivative of the oracle's stage, on
    turned elements. The bound is that of the other dot-product tests: the Poisson tolerance
    times the conditioning."""
    monkeypatch.setenv("HO2D_GRAPHS", graphs)
    inp = turned_cavity(str(tmp_path), 5, knod)
    c = O.Case(inp)
    s = solver(inp, precision)
    rng = np.random.Generator(np.random.PCG64(11))
    shape = (c.N, c.K, c.K)
    w, lam_k = rng.standard_normal(shape), rng.standard_normal(shape)
    s.set_vorticity(w)
    gw, gpv = s.stage_adjoint(0.5, lam_k)
    dw, dpv = rng.standard_normal(shape), rng.standard_normal((c.neb, c.K))
    _, dk = CS.stage_jvp(c, w, dw, dpv, 0.5)
    lhs, rhs = float(np.vdot(lam_k, dk)), float(np.vdot(gw, dw) + np.vdot(gpv, dpv))
    assert abs(lhs - rhs) <= 1e-9 * np.linalg.norm(lam_k) * np.linalg.norm(dk), (lhs, rhs)
    s.close()


# both sides of the line between the one kernel and the loop of launches (148 tiles of 32 elements at
# K = 4), the last tile full, one element short and one over: the same gradient from the captured solve and from
# launches driven by the host. (64 x 64 at K = 5 and 30 x 40 at K = 7: loops only.)
@pytest.mark.parametrize("precision", [FP64, MIXED_KRYLOV])
@pytest.mark.parametrize("mesh,knod", [("cyl37x128", 4), ("cyl34x139", 4), ("cyl61x78", 4), ("cavityj64", 5), ("cyl30x40", 7)])
def test_captured_and_host_driven_solves_agree(tmp_path, monkeypatch, mesh, knod, precision):
    inp = meshgen.make_case(mesh, str(tmp_path), knod=knod, steps=1)
    out = []
    for graphs in ("1", "0"):
        monkeypatch.setenv("HO2D_GRAPHS", graphs)
        s = solver(inp, precision)
        rng = np.random.Generator(np.random.PCG64(9))
        shape = (s.N_el, s.Knod, s.Knod)
        s.set_vorticity(rng.standard_normal(shape))
        out.append(s.stage_adjoint(0.0, rng.standard_normal(shape))[0])
        assert s.adjoint_stats()[1] <= 1e-13
        s.close()
    # both at residual 1e-13; the conditioning of a stretched O-grid of this size is below 1e5
    assert np.abs(out[0] - out[1]).max() <= 2e-8 * np.abs(out[1]).max()
