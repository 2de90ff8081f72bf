"""GPU: the lane kernels of simplices and the wave where a block takes several tiles (meshes
just above two full blocks per SM, whose groups leave partly filled last blocks), alone and
in a batch, and the FP32 form bit for bit.

FP64: against the row kernel (variant 1), 1e-12 of the largest coefficient, stage vectors as
in the lane tests.  FP32: the lane kernels keep the operations and their order of the kernel
that is chosen automatically without them, so every result is equal to its: the tile kernel's
(variant 2) for the wave where that is the choice, the row kernel's elsewhere."""
import numpy as np
import pytest

import hpgem_b200
from hpgem_b200 import _native

from lane_helpers import kernel_class

pytestmark = pytest.mark.gpu

FP64, FP32 = _native.PRECISION_FP64, _native.PRECISION_FP32


def solver(cells, tri, order, physics, precision, variant=0, tableau="RK4_4"):
    d = len(cells)
    if physics == "advection":
        s = hpgem_b200.Advection(d, order, [0.7, -0.4, 0.5][:d], tableau=tableau, precision=precision)
    else:
        s = hpgem_b200.AcousticWave(d, order, c_inv=0.8, tableau=tableau, precision=precision,
                                    flux="upwind" if physics == "wave_upwind" else "central")
    s.readMesh(hpgem_b200.structured_description(cells, [0.0] * d, [1.0] * d, tri, True))
    if variant == 0:
        assert kernel_class(s) == "lane tables"
    s.handle.set_kernel_variant(variant)
    s.handle.set_state(0, np.random.default_rng(order).standard_normal(s.handle.vector_length))
    return s


def results(s, cells, order):
    s.handle.time_derivative(0, 1)
    k = s.handle.get_state(1)
    s.handle.step(0.0, 0.01 / max(cells) / (2 * order + 1) ** 2, 9)
    return s.handle.get_state(0), s.handle.get_state(2), k


# (cells, simplices, order, physics): four and two tiles a block, of one, two and four warps each
LARGE = [([140, 138], True, 3, "advection"), ([20, 20, 20], True, 3, "advection"), ([16, 16, 16], True, 4, "advection"),
         ([140, 138], True, 2, "wave"), ([140, 138], True, 4, "wave_upwind"), ([20, 20, 20], True, 2, "wave_upwind"),
         ([16, 16, 16], True, 3, "wave"), ([140, 138], False, 3, "wave"), ([34, 34, 34], False, 1, "wave_upwind")]


@pytest.mark.parametrize("cells,tri,order,physics", LARGE)
def test_several_tiles_a_block(cells, tri, order, physics):
    a, b = [results(solver(cells, tri, order, physics, FP64, v), cells, order) for v in (0, 1)]
    tol = 1e-12 if order <= 3 else 1e-10
    for x, y, t in zip(a, b, (1e-12, tol, tol)):
        assert np.abs(x - y).max() < t * np.abs(y).max()


@pytest.mark.parametrize("precision", [FP64, FP32])
@pytest.mark.parametrize("cells,tri,order,physics", [LARGE[0], LARGE[3], LARGE[5], LARGE[6]])
def test_several_tiles_a_block_in_a_batch(cells, tri, order, physics, precision):
    dt = 0.01 / max(cells) / (2 * order + 1) ** 2
    small = [24, 20] if len(cells) == 2 else [14, 18, 12]  # (one tile a block, in the same class)
    members = [solver(c, tri, order, physics, precision) for c in (cells, small)]
    batch = hpgem_b200.Batch(2)
    for s in members:
        batch.add(s, dt, 5)
    assert batch.num_classes == 1
    batch.step(5)
    batch.synchronize()
    batch.close()
    for c, s in zip((cells, small), members):
        alone = solver(c, tri, order, physics, precision)
        alone.handle.step(0.0, dt, 5)
        want = alone.handle.get_state(0)
        assert np.abs(s.handle.get_state(0) - want).max() < 1e-12 * np.abs(want).max()


# ... and the kernel variant of the automatic choice without the lane kernels
EQUAL = [([24, 24], True, p, "wave", 2) for p in (1, 2, 3, 4, 5)] + \
        [([24, 24], True, 3, "wave_upwind", 2), ([9, 7], False, 2, "wave", 2), ([8, 9], False, 4, "wave", 1),
         ([5, 4, 3], False, 1, "wave_upwind", 2), ([4, 3, 5], False, 2, "wave", 1), ([8, 8, 8], True, 1, "wave", 2),
         ([14, 10, 12], True, 2, "wave_upwind", 2), ([14, 18, 12], True, 3, "wave", 2), ([14, 18, 12], True, 3, "wave_upwind", 2),
         ([140, 138], True, 2, "wave", 1), ([140, 138], True, 4, "wave", 2), ([20, 20, 20], True, 2, "wave", 2),
         ([34, 34, 34], False, 1, "wave", 2)] + \
        [([34, 30], True, p, "advection", 1) for p in (1, 2, 3, 4)] + [([8, 8, 8], True, p, "advection", 1) for p in (1, 2, 3)] + \
        [([140, 138], True, 4, "advection", 1), ([20, 20, 20], True, 2, "advection", 1)]


@pytest.mark.parametrize("tableau", ["RK4_4", "RK3TVD"])
@pytest.mark.parametrize("cells,tri,order,physics,variant", EQUAL)
def test_fp32_equals_the_general_choice(cells, tri, order, physics, variant, tableau):
    a, b = [results(solver(cells, tri, order, physics, FP32, v, tableau), cells, order) for v in (0, variant)]
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("cells,order", [([8, 4], 1), ([11, 3], 2), ([67, 71], 4), ([5, 6], 5), ([11, 9, 13], 2)])
def test_fp32_sum_factorised_lanes_equal_the_one_shot_kernel(cells, order):
    res = []
    for variant in (0, 1):
        d = len(cells)
        s = hpgem_b200.Advection(d, order, [0.7, -0.4, 0.5][:d], tableau="RK4_4", precision=FP32)
        s.readMesh(hpgem_b200.structured_description(cells, [0.0] * d, [1.0] * d, False, True))
        if variant == 0:
            assert kernel_class(s) == "sum-factorised lanes"
        s.handle.set_kernel_variant(variant)
        s.handle.set_state(0, np.random.default_rng(order).standard_normal(s.handle.vector_length))
        res.append(results(s, cells, order))
    for x, y in zip(*res):
        assert np.array_equal(x, y)
