"""The Kronecker-sum fit of the device setup: the same decisions as the host's fit, element by
element, and a setup that the fit does not dominate. The FP64 smoother takes factors from 48 MB
of inverse blocks on, at K = 8 between 38^2 (45 MB) and 40^2 elements (50 MB); by one thread an
element the fit's defect alone took 0.6 s there, several times the rest of the setup.
"""

import time

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
