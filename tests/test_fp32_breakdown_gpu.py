"""An FP32 inner solve that breaks down: the FP64 solve finishes. Fields scaled by 2^140 have FP64
norms but leave FP32's range, so the right-hand side of the first inner solve is infinite and its
result unusable; scaled back, the answer is that of the unscaled field. (The operators are linear
and the scale is a power of two; the paths differ, so the bound is the residual, 1e-13, times the
conditioning, below 1e4 at these sizes.) Forward refinement in its captured and its host-driven
form, and the transposed one.
"""

import numpy as np
import pytest

from ho2d import HO_2D, MIXED_KRYLOV, meshgen

pytestmark = pytest.mark.gpu

SCALE = 140


@pytest.mark.parametrize("graphs", ["1", "0"])
@pytest.mark.parametrize("mesh,knod", [("cavityj9", 4), ("cavityj72", 5), ("cyl9x17", 7)])
def test_fp64_finishes_what_fp32_cannot(tmp_path, monkeypatch, mesh, knod, graphs):
    monkeypatch.setenv("HO2D_GRAPHS", graphs)
    s = HO_2D()
    s.read_input_file(meshgen.make_case(mesh, str(tmp_path), knod=knod, steps=1))
    s.set_precision(MIXED_KRYLOV)
    s.set_poisson_tolerance(1e-12, 500)
    s.setup()
    rng = np.random.Generator(np.random.PCG64(7))
    shape = (s.N_el, s.Knod, s.Knod)
    w, lam = rng.standard_normal(shape), rng.standard_normal(shape)

    def streamfunction(scale):
        s.set_time(0.0)
        s.set_vorticity(np.ldexp(w, scale))
        s.Euler_time_integrate(0.0)
        assert s.poisson_stats()[1] <= 1e-12
        return np.ldexp(s.get_streamfunction(), -scale)

    psi = streamfunction(0)
    grad = s.stage_adjoint(0.0, lam)[0]
    finishes = s.fp64_finishes()
    scaled = np.ldexp(s.stage_adjoint(0.0, np.ldexp(lam, SCALE))[0], -SCALE)
    assert s.adjoint_stats()[1] <= 1e-12
    assert np.abs(scaled - grad).max() <= 1e-9 * np.abs(grad).max()
    if not mesh.startswith("cyl"):  # (an inflow does not scale with the vorticity)
        scaled = streamfunction(SCALE)
        assert s.fp64_finishes() == finishes + 1
        assert np.abs(scaled - psi).max() <= 1e-9 * np.abs(psi).max()
    s.close()
