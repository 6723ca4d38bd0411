"""Algorithmic bytes that ho2d_profile_krylov reports, in values an element: what the iteration's
kernels read and write, the four element moments of r, v and p among them.
"""

import numpy as np
import pytest

from ho2d import FP64, HO_2D, MIXED_KRYLOV, meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,width", [(FP64, 8), (MIXED_KRYLOV, 4)])
@pytest.mark.parametrize("knod", [3, 6])
def test_bytes_count_the_moments(tmp_path, knod, precision, width):
    s = HO_2D()
    s.read_input_file(meshgen.make_case("cavityj9", str(tmp_path), knod=knod, steps=1))
    s.set_precision(precision)
    s.set_smoother(0)
    s.setup()
    s.set_vorticity(np.random.Generator(np.random.PCG64(3)).standard_normal((81, knod, knod)))
    s.Euler_time_integrate(0.0)
    values = {k: v[1] / 81 / width for k, v in s.profile_krylov(1).items()}
    s.close()
    k2 = knod * knod
    # block, r and v, p in half the launches, the new p or s and M f; moments of r, v, p and the new p in half
    assert values["smoother"] == pytest.approx(k2 * k2 + 4.5 * k2 + 0.5 * 16)
    # operand, 3 metric coefficients, second vector, result; 6 values a face point, 4 codes; moments of v in half
    assert values["operator"] == pytest.approx(6 * k2 + 24 * knod + 16 / width + 0.5 * 4)
    assert values["xr_update"] == pytest.approx(8 * k2 + 4)
