"""The residual that Poisson solves end with, on the GPU: in FP64 a tenth of the tolerance, the
adjoint's transposed solves included, in the refinement of HO2D_MIXED_KRYLOV and of the transposed
solves 0.3 of it (the reason stands at Solver::solve_target). HO2D_MIXED stops at the tolerance.
At 1e-9 nothing stalls, so every solve has to get there.
"""

import numpy as np
import pytest

from ho2d import FP64, HO_2D, MIXED, MIXED_KRYLOV, meshgen

pytestmark = pytest.mark.gpu

TOL = 1e-9


@pytest.mark.parametrize("graphs", ["1", "0"])
@pytest.mark.parametrize("mesh,knod", [("cyl6x13", 4), ("cavityj72", 5)])  # one kernel a solve; launches
@pytest.mark.parametrize("precision,bound,bound_transposed", [(FP64, 0.1, 0.1), (MIXED_KRYLOV, 0.3, 0.3), (MIXED, 1.0, 0.3)])
def test_solves_end_below_their_target(tmp_path, monkeypatch, precision, bound, bound_transposed, mesh, knod, graphs):
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
    assert max(transposed) <= bound_transposed * TOL, transposed
