"""GPU: the one-element-per-thread kernels (tiled layout, the automatic choice on
structured meshes) against the general kernels they replace there (kernel variant 1), at
element counts around a tile of 32, along-axis and mixed-sign velocities, tableaux with
zero, one and several vectors in a stage input, and after a change of the variant between
steps.

Both kernels evaluate the same operator from the same 64-bit geometry; the lane kernels
fold it into fewer matrices first, so they differ by rounding only: 1e-12 of the largest
coefficient as in the parity tests, in the FP32 form 2e-6 (a few FP32 roundings, 6e-8
each, per step and stage over the steps taken here, damped by dt)."""
import numpy as np
import pytest

import hpgem_b200
from hpgem_b200 import _native

pytestmark = pytest.mark.gpu

RTOL = {_native.PRECISION_FP64: 1e-12, _native.PRECISION_FP32: 2e-6}


def rel_err(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def solver(cells, order, a, tableau, precision):
    s = hpgem_b200.Advection(len(cells), order, a, tableau=tableau, precision=precision)
    d = len(cells)
    return s.readMesh(hpgem_b200.structured_description(cells, [0.0] * d, [1.0] * d, False, True))


# (cells, velocity): one tile not quite full, exactly full, one element more; several blocks; 3D
QUADS = [([5, 6], [0.7, -0.4]), ([8, 4], [-0.3, 0.9]), ([11, 3], [1.0, 0.0]), ([67, 71], [0.0, -1.0])]
HEXES = [([3, 3, 3], [0.5, -0.6, 0.7]), ([4, 4, 2], [-1.0, 0.0, 0.3]), ([11, 9, 13], [0.2, 0.3, 0.9])]


@pytest.mark.parametrize("precision", [_native.PRECISION_FP64, _native.PRECISION_FP32])
@pytest.mark.parametrize("tableau", ["ForwardEuler", "RK4_4", "DormandPrince"])
@pytest.mark.parametrize("cells,a,order", [(c, a, p) for c, a in QUADS for p in (1, 2, 3, 4, 5)] +
                         [(c, a, p) for c, a in HEXES for p in (1, 2)])
def test_tensor_lane_matches_the_one_shot_kernel(cells, a, order, tableau, precision):
    res = {}
    for variant in (0, 1):
        s = solver(cells, order, a, tableau, precision)
        s.handle.set_kernel_variant(variant)
        assert s.handle.kernel_kind == "tensor"
        u0 = np.random.default_rng(order).standard_normal(s.handle.vector_length)
        s.handle.set_state(0, u0)
        assert np.array_equal(s.handle.get_state(0), u0)
        h = 1.0 / max(cells)
        s.handle.step(0.0, 0.02 * h / (2 * order + 1) ** 2, 3)
        stages = 7 if tableau == "DormandPrince" else 4 if tableau == "RK4_4" else 1
        res[variant] = [s.handle.get_state(v) for v in range(stages + 1)]
    assert rel_err(res[0][0], res[1][0]) < RTOL[precision]
    for k0, k1 in zip(res[0][1:], res[1][1:]):  # the stage vectors are k / dt larger: their own rounding
        assert rel_err(k0, k1) < (1e-12 if precision == _native.PRECISION_FP64 else 5e-6)


@pytest.mark.parametrize("precision", [_native.PRECISION_FP64, _native.PRECISION_FP32])
def test_variant_change_keeps_every_vector(precision):
    s = solver([13, 9], 3, [0.8, -0.5], "RK4_4", precision)
    h = s.handle
    h.set_state(0, np.random.default_rng(3).standard_normal(h.vector_length))
    h.step(0.0, 1e-4, 2)
    before = [h.get_state(v) for v in range(5)]
    for variant in (1, 2, 0):
        h.set_kernel_variant(variant)
        for v in range(5):
            assert np.array_equal(h.get_state(v), before[v])
    h.step(0.0, 1e-4, 1)
    mixed = h.get_state(0)
    t = solver([13, 9], 3, [0.8, -0.5], "RK4_4", precision)
    t.handle.set_state(0, before[0])
    t.handle.step(0.0, 1e-4, 1)
    assert np.array_equal(mixed, t.handle.get_state(0))


# Simplices and the wave: (cells, triangular, order, physics).  Meshes whose groups fill
# whole tiles, leave the last tile partly filled, and (sides 2 mod 4) have odd groups along
# the periodic wrap; every basis size of the two kernels.
WAVES = [([24, 24], True, p) for p in (1, 2, 3, 4, 5)] + [([26, 22], True, 2), ([6, 6], False, 1), ([4, 4], True, 2), ([2, 2, 2], True, 2), ([4, 4, 4], True, 4),
         ([9, 7], False, 2), ([12, 11], False, 3), ([8, 9], False, 4), ([7, 8], False, 5),
         ([8, 8, 8], True, 1), ([8, 8, 8], True, 2), ([14, 10, 12], True, 2), ([8, 8, 8], True, 3),
         ([8, 8, 8], True, 4), ([5, 4, 3], False, 1), ([4, 3, 5], False, 2)]
ADVECTIONS = [([24, 24], True, p) for p in (1, 2, 3, 4, 5)] + [([34, 30], True, 3), ([6, 4], True, 3), ([10, 10], True, 5), ([4, 4, 4], True, 2)] + \
             [([8, 8, 8], True, p) for p in (1, 2, 3, 4, 5)]


def any_solver(cells, tri, order, physics, tableau, precision):
    d = len(cells)
    if physics == "advection":
        s = hpgem_b200.Advection(d, order, [0.7, -0.4, 0.5][:d], tableau=tableau, precision=precision)
    else:
        s = hpgem_b200.AcousticWave(d, order, c_inv=0.8, tableau=tableau, precision=precision,
                                    flux="upwind" if physics == "wave_upwind" else "central")
    return s.readMesh(hpgem_b200.structured_description(cells, [0.0] * d, [1.0] * d, tri, True))


def stage_tolerance(order, dim, precision):
    """Of the stage vectors: their operators carry the mass inverse, so both kernels'
    results have its condition number times the round-off (1e7 for tetrahedra at p = 5)."""
    if precision == _native.PRECISION_FP64:
        return 1e-12 if order <= 3 else 1e-10
    return 5e-6 if order <= 2 else 1e-4


@pytest.mark.parametrize("precision", [_native.PRECISION_FP64, _native.PRECISION_FP32])
@pytest.mark.parametrize("tableau", ["RK4_4", "RK3TVD"])
@pytest.mark.parametrize("cells,tri,order,physics",
                         [c + ("wave",) for c in WAVES] + [c + ("wave_upwind",) for c in WAVES] +
                         [c + ("advection",) for c in ADVECTIONS])
def test_lane_kernels_match_the_general_kernels(cells, tri, order, physics, tableau, precision):
    if precision == _native.PRECISION_FP32 and not tri and (len(cells), order) in ((2, 3), (3, 2), (2, 4), (2, 5)):
        pytest.skip("the row kernel's block does not launch for these FP32 shapes")
    res = {}
    for variant in (0, 1):
        s = any_solver(cells, tri, order, physics, tableau, precision)
        s.handle.set_kernel_variant(variant)
        u0 = np.random.default_rng(order).standard_normal(s.handle.vector_length)
        s.handle.set_state(0, u0)
        assert np.array_equal(s.handle.get_state(0), u0)
        s.handle.time_derivative(0, 1)
        k = s.handle.get_state(1)
        s.handle.step(0.0, 0.01 / max(cells) / (2 * order + 1) ** 2, 3)
        res[variant] = (s.handle.get_state(0), s.handle.get_state(2), k)
    tol = stage_tolerance(order, len(cells), precision)
    assert rel_err(res[0][0], res[1][0]) < RTOL[precision]
    assert rel_err(res[0][1], res[1][1]) < tol
    assert rel_err(res[0][2], res[1][2]) < tol


def test_lane_members_of_a_batch_match_alone():
    """A batch takes the members of lane handles as classes of their own; partly filled
    chunks, several members of one class, both physics, the FP32 form beside FP64."""
    specs = [([24, 24], True, 3, "advection", 0), ([34, 30], True, 3, "advection", 0), ([24, 24], True, 5, "advection", 1),
             ([8, 8, 8], True, 2, "wave", 0), ([14, 10, 12], True, 2, "wave", 0), ([8, 8, 8], True, 3, "wave_upwind", 1),
             ([67, 71], False, 2, "advection", 1), ([11, 3], False, 2, "advection", 1)]
    batch = hpgem_b200.Batch(16)
    runs = []
    for i, (cells, tri, order, physics, precision) in enumerate(specs):
        s = any_solver(cells, tri, order, physics, "RK4_4", precision)
        u0 = np.random.default_rng(i).standard_normal(s.handle.vector_length)
        s.handle.set_state(0, u0)
        runs.append((s, u0, batch.add(s, 1e-5 * (1 + i), 3 + i % 3)))
    batch.step(6)
    batch.synchronize()
    for i, (spec, (s, u0, slot)) in enumerate(zip(specs, runs)):
        assert batch.remaining(slot) == 0
        t = any_solver(*spec[:4], "RK4_4", spec[4])
        t.handle.set_state(0, u0)
        t.handle.step(0.0, 1e-5 * (1 + i), 3 + i % 3)
        assert rel_err(s.handle.get_state(0), t.handle.get_state(0)) < 1e-12
    batch.close()
