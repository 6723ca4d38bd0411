"""The residual that Poisson solves end with, on the GPU. The FP64 solve, the refinement of
HO2D_MIXED_KRYLOV and the adjoint's transposed solves aim at a tenth of the tolerance (the
reason stands at Solver::solve_target); at 1e-9 nothing stalls, so every solve has to get there.
HO2D_MIXED stops at the tolerance.
"""

import numpy as np
import pytest

from ho2d import FP64, HO_2D, MIXED, MIXED_KRYLOV, meshgen

pytestmark = pytest.mark.gpu

TOL = 1e-9


@pytest.mark.parametrize("graphs", ["1", "0"])
@pytest.mark.parametrize("mesh,knod", [("cyl6x13", 4), ("cavityj72", 5)])  # one kernel a solve; launches
@pytest.mark.parametrize("precision,bound", [(FP64, 0.1), (MIXED_KRYLOV, 0.1), (MIXED, 1.0)])
def test_solves_end_below_their_target(tmp_path, monkeypatch, precision, bound, mesh, knod, graphs):
    monkeypatch.setenv("HO2D_GRAPHS", graphs)
    s = HO_2D()
    s.read_input_file(meshgen.make_case(mesh, str(tmp_path), knod=knod, steps=1))
    s.set_precision(precision)
    s.set_poisson_tolerance(TOL, 500)
    s.setup()
    rng = np.random.Generator(np.random.PCG64(1))
    shape = (s.N_el, s.Knod, s.Knod)
    forward, transposed = [], []
    for _ in range(6):
        s.set_vorticity(rng.standard_normal(shape))
        s.Euler_time_integrate(0.0)
        forward.append(s.poisson_stats()[1])
        s.stage_adjoint(0.0, rng.standard_normal(shape))
        transposed.append(s.adjoint_stats()[1])
    s.close()
    assert max(forward) <= bound * TOL, forward
    assert max(transposed) <= 0.1 * TOL, transposed
