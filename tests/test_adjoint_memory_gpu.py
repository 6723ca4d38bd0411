"""The adjoint's transposed solves without a transposed copy of the inverse blocks, which a mesh that
nearly fills the GPU has no room for (HO2D_ADJOINT_COPY=0 asks for it): the same bits, launch for
launch, and no memory of the blocks' size.
"""

import numpy as np
import pytest

from ho2d import FP64, HO_2D, MIXED_KRYLOV, meshgen

pytestmark = pytest.mark.gpu


def gradient(inp, precision):
    torch = pytest.importorskip("torch")
    s = HO_2D()
    s.read_input_file(inp)
    s.set_precision(precision)
    s.set_poisson_tolerance(1e-10, 500)
    s.setup()
    shape = (s.N_el, s.Knod, s.Knod)
    rng = np.random.Generator(np.random.PCG64(5))
    s.set_vorticity(rng.standard_normal(shape))
    before = torch.cuda.mem_get_info()[0]
    out = s.stage_adjoint(0.0, rng.standard_normal(shape))
    used = before - torch.cuda.mem_get_info()[0]
    stats = s.adjoint_stats()
    s.close()
    return out, stats, used


@pytest.mark.parametrize("precision", [FP64, MIXED_KRYLOV])
@pytest.mark.parametrize("mesh,knod", [("cyl5x9", 1), ("cavityj9", 2), ("cyl5x9", 3), ("cavityj11", 4), ("cyl4x8", 5),
                                       ("cavityj7", 6), ("cavityj5", 7), ("cavityj5", 8)])
def test_blocks_in_place_give_the_same_gradient(tmp_path, monkeypatch, mesh, knod, precision):
    monkeypatch.setenv("HO2D_GRAPHS", "0")  # the same launches on both sides
    inp = meshgen.make_case(mesh, str(tmp_path), knod=knod, steps=1)
    with_copy = gradient(inp, precision)
    monkeypatch.setenv("HO2D_ADJOINT_COPY", "0")
    in_place = gradient(inp, precision)
    assert with_copy[1] == in_place[1]
    for a, b in zip(with_copy[0], in_place[0]):
        assert np.array_equal(a, b)


def test_blocks_in_place_take_no_memory(tmp_path, monkeypatch):
    inp = meshgen.make_case("cavityj64", str(tmp_path), knod=7, steps=1)
    blocks = 64 * 64 * 7 ** 4 * 8
    gradient(inp, FP64)  # (the context's own allocations)
    with_copy = gradient(inp, FP64)
    monkeypatch.setenv("HO2D_ADJOINT_COPY", "0")
    in_place = gradient(inp, FP64)
    assert with_copy[2] - in_place[2] >= 0.9 * blocks, (with_copy[2], in_place[2], blocks)
    for a, b in zip(with_copy[0], in_place[0]):  # captured loops of launches on both sides
        assert np.array_equal(a, b)
