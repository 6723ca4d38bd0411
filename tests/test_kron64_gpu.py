"""FP64 solves with Kronecker-sum factors as the smoother (by default from 48 MB of inverse blocks
on; HO2D_KRON64_MIN moves the line) on strongly jittered cavities, where some elements keep their
exact block and others of the same warp do not: against the oracle's direct solve, and in iterations
against the exact blocks.
"""

import numpy as np
import pytest

from ho2d import FP64, HO_2D, meshgen

import ho2d_oracle as O

pytestmark = pytest.mark.gpu


def solve(inp, w0):
    s = HO_2D()
    s.read_input_file(inp)
    s.set_precision(FP64)
    s.set_poisson_tolerance(1e-13, 2000)
    s.setup()
    s.set_vorticity(w0)
    s.Euler_time_integrate(0.0)
    psi, iters = s.get_streamfunction(), s.poisson_stats()[0]
    k2 = s.Knod ** 2
    data = s.profile_krylov(1)["smoother"][1] / s.N_el - (4.5 * k2 + 8) * 8  # an element, beside vectors and moments
    s.close()
    return psi, iters, data


@pytest.mark.parametrize("graphs", ["1", "0"])
@pytest.mark.parametrize("knod", range(3, 9))
def test_solve_with_factors(tmp_path, monkeypatch, knod, graphs):
    monkeypatch.setenv("HO2D_GRAPHS", graphs)
    n, k2 = 11, knod * knod
    inp = meshgen.make_case("cavityj%d" % n, str(tmp_path), knod=knod, steps=1, jitter=0.3)
    c = O.Case(inp)
    w0 = np.random.Generator(np.random.PCG64(7)).standard_normal((c.N, c.K, c.K))
    c.omega = w0.copy()
    c.update_bcs(0.0)
    c.solve_poisson(w0)
    _, it_blocks, data = solve(inp, w0)
    assert data == 8 * k2 * k2
    monkeypatch.setenv("HO2D_KRON64_MIN", "0")
    psi, iters, data = solve(inp, w0)
    kept = (data - 8 * (4 * k2 + 2 * knod)) / (8 * k2 * k2) * n * n  # elements with their exact block
    assert abs(kept - round(kept)) < 1e-6 and 0 < round(kept) < n * n, kept
    # residual 1e-13 times the conditioning (below 1e4 at these sizes), as the parity tests
    assert np.abs(psi - c.psi).max() <= 1e-9 * np.abs(c.psi).max()
    assert iters <= 1.5 * it_blocks + 2, (iters, it_blocks)
