"""The residual that Poisson solves end with, on the GPU: in FP64 0.3 of the tolerance, with a
re-entrant corner a tenth (there the adjoint's transposed solves too), in the refinement of
HO2D_MIXED_KRYLOV and of the transposed solves 0.3 of it (the reasons stand at Solver::fp64_target).
HO2D_MIXED stops at the tolerance. At 1e-9 nothing stalls, so every solve has to get there.
"""

import numpy as np
import pytest

from ho2d import FP64, HO_2D, MIXED, MIXED_KRYLOV, meshgen

pytestmark = pytest.mark.gpu

TOL = 1e-9


@pytest.mark.parametrize("graphs", ["1", "0"])
@pytest.mark.parametrize("mesh,knod,corner", [("cyl6x13", 4, False), ("bfs3", 4, True), ("cavityj72", 5, False),
                                              ("bfs9", 5, True)])  # one kernel a solve; launches
@pytest.mark.parametrize("precision", [FP64, MIXED_KRYLOV, MIXED])
def test_solves_end_below_their_target(tmp_path, monkeypatch, precision, mesh, knod, corner, graphs):
    bound = {FP64: 0.1 if corner else 0.3, MIXED_KRYLOV: 0.3, MIXED: 1.0}[precision]
    bound_transposed = (0.1 if corner else 1.0) if precision == FP64 else 0.3
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
