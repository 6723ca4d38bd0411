"""The Kronecker-sum fit of the device setup: the same decisions as the host's fit, element by
element, and a setup that the fit does not dominate. The FP64 smoother takes factors from 48 MB
of inverse blocks on, at K = 8 between 38^2 (45 MB) and 40^2 elements (50 MB); by one thread an
element the fit's defect alone took 0.6 s there, several times the rest of the setup.
"""

import time

import numpy as np
import pytest

from ho2d import FP64, HO_2D, MIXED_KRYLOV, capi, meshgen

pytestmark = pytest.mark.gpu


def solver(inp, precision, smoother=-1, device=True):
    s = HO_2D()
    s.read_input_file(inp)
    s.set_precision(precision)
    s.set_smoother(smoother)
    s.set_device_setup(device)
    return s


@pytest.mark.parametrize("knod", range(2, 9))
def test_device_fit_keeps_the_same_blocks_as_the_host_fit(tmp_path, knod):
    inp = meshgen.make_case("cavityj17", str(tmp_path), knod=knod, steps=1, jitter=0.3)
    kept = []
    for device in (True, False):
        s = solver(inp, MIXED_KRYLOV, capi.SMOOTHER_KRON, device)
        s.setup()
        kept.append(s.smoother())
        s.close()
    assert kept[0] == kept[1]
    assert 0 < kept[0][1] < 17 * 17


def test_fit_does_not_dominate_the_setup(tmp_path):
    times = []
    for n in (38, 40):
        inp = meshgen.make_case("cavityj%d" % n, str(tmp_path / str(n)), knod=8, steps=1)
        best = 1e9
        for _ in range(4):
            s = solver(inp, FP64)
            t = time.perf_counter()
            s.setup()
            best = min(best, time.perf_counter() - t)
            s.close()
        times.append(best)
    assert times[1] <= 2.0 * times[0], times


def test_order_2_keeps_blocks(tmp_path):
    """At order 2 the factors are more values than the block (20 and 16): the FP64 smoother reads
    blocks also on a mesh with more than 48 MB of them."""
    n = 632
    s = solver(meshgen.make_case("cavityj%d" % n, str(tmp_path), knod=2, steps=1), FP64)
    s.setup()
    s.set_vorticity(np.random.Generator(np.random.PCG64(3)).standard_normal((n * n, 2, 2)))
    s.Euler_time_integrate(0.0)
    data = s.profile_krylov(2)["smoother"][1] / (n * n) - (4.5 * 4 + 8) * 8  # an element, beside vectors and moments
    s.close()
    assert data == 16 * 8, data
