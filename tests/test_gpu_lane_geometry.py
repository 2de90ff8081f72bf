"""GPU: the lane kernels on meshes from files whose cells are not all equal, flat cells
among them, against the general kernels (variant 1), which read every element's own
geometry.

The state varies along the long axis of the cells only, so the right-hand side is what that
axis gives, about 2 pi.  Rounding there: 1.1e-16 of the largest terms, which are those of
the short axis and cancel: 2 / h of that axis times the operators' row sums (below 100 for
the orders here).  A cell that stepped with another one's geometry would be off by their
difference, many times that.
"""
import numpy as np
import pytest

import hpgem_b200
from hpgem_b200 import _native

from lane_helpers import kernel_class, write_mesh_file

pytestmark = pytest.mark.gpu


def moved(n, length, by):
    """Node positions of n cells, every second inner node moved by `by` cells."""
    x = np.linspace(0.0, length, n + 1)
    x[1:-1:2] += by * length / n
    return x


def solver(path, dim, order, physics):
    if physics == "advection":
        s = hpgem_b200.Advection(dim, order, [0.7, -0.4, 0.5][:dim], tableau="RK4_4")
    else:
        s = hpgem_b200.AcousticWave(dim, order, c_inv=0.8, tableau="RK4_4", flux="upwind")
    return s.readMeshFile(path)


# (cells, long axis, aspect ratio, by, triangles, order, physics, kernel class)
CASES = [([16, 16, 4], 0, 1e5, 4e-9, False, 2, "advection", "sum-factorised"),
         ([16, 16, 4], 0, 1e5, 0.0, False, 2, "advection", "sum-factorised lanes"),
         ([64, 4], 0, 1e5, 2e-9, True, 2, "advection", "lane tables"),
         ([64, 4], 0, 1e5, 2e-9, True, 2, "wave_upwind", "lane tables"),
         ([64, 4], 0, 1e5, 2e-9, False, 3, "wave_upwind", "lane tables"),
         ([32, 32], 0, 1.0, 0.2, False, 2, "advection", "sum-factorised"),
         ([32, 32], 0, 1.0, 0.2, True, 3, "advection", "lane tables"),
         ([32, 32], 1, 1.0, 0.2, True, 3, "wave_upwind", "lane tables")]


@pytest.mark.parametrize("cells,long_axis,aspect,by,triangles,order,physics,kind", CASES)
def test_every_cell_steps_with_its_own_geometry(tmp_path, cells, long_axis, aspect, by, triangles, order, physics, kind):
    dim = len(cells)
    if dim == 3 and aspect > 1:  # flat: one short axis
        lengths = [1.0, 1.0, 1.0 / aspect]
    else:
        lengths = [1.0 if c == long_axis else 1.0 / aspect for c in range(dim)]
    axes = [moved(n, lengths[c], by if c == long_axis else 0.0) for c, n in enumerate(cells)]
    path = write_mesh_file(tmp_path / "mesh.hpgem", axes, triangles)
    short = max(2 * n / length for n, length in zip(cells, lengths))  # 2 / h
    tol = max(1e-12, 1.1e-16 * 100 * short / (2 * np.pi))
    res = []
    for variant in (0, 1):
        s = solver(path, dim, order, physics)
        if variant == 0:
            assert kernel_class(s) == kind
        s.handle.set_kernel_variant(variant)
        x = s.quadraturePoints().reshape(-1, dim)[:, long_axis]
        V = 1 if physics == "advection" else dim + 1
        values = np.stack([np.sin(2 * np.pi * x + 0.3 * v) for v in range(V)], axis=1)
        s.handle.project(values, 0)
        s.handle.time_derivative(0, 1)
        k = s.handle.get_state(1)
        s.handle.step(0.0, 1e-3 / max(cells) / aspect, 5)
        res.append((k, s.handle.get_state(0)))
    assert np.abs(res[0][0] - res[1][0]).max() / np.abs(res[1][0]).max() < tol
    assert np.abs(res[0][1] - res[1][1]).max() / np.abs(res[1][1]).max() < 1e-12
