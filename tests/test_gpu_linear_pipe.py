"""GPU: the pipelined stored-matrix tiles against the oracle and against the staged tiles
they replace where a stage's input is one vector, at row counts around a pass of 64 (and a
chunk of 32) columns, odd row counts (8-byte copies), partly filled tiles, the FP32 form,
a tableau whose stages read several vectors, and a caller's vector that starts at an odd
double.  Tolerances as in the linear parity tests."""
import ctypes

import numpy as np
import pytest
import torch

import hpgem_b200
from hpgem_b200 import _native
from oracle.dg import ADVECTION, WAVE, Problem
from oracle.linear import LinearOracle, assemble
from oracle.mesh import mesh_from_description

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float(np.abs(np.asarray(a).reshape(-1) - np.asarray(b).reshape(-1)).max() / np.abs(b).max())


def make(cells, tri, order, physics, tableau="RK4_4", precision=_native.PRECISION_FP64):
    d = len(cells)
    desc = hpgem_b200.structured_description(cells, [0.0] * d, [1.0] * d, tri, True)
    s = hpgem_b200.HpgemAPILinear(d, order, physics, advection=[0.7, -0.4, 0.5][:d], tableau=tableau,
                                  precision=precision).readMesh(desc)
    mesh = mesh_from_description(desc)
    prob = Problem(mesh, order, WAVE, cinv=1.0) if physics == "wave" else Problem(mesh, order, ADVECTION,
                                                                                  a=[0.7, -0.4, 0.5][:d])
    return s, prob, LinearOracle(*assemble(prob))


# rows per element: 25 (odd, narrow), 27, 36, 64 (one pass), 125 (two passes, odd), 40 and 45
CASES = [([9, 8], False, 4, "advection"), ([5, 4, 4], False, 2, "advection"), ([8, 9], False, 5, "advection"),
         ([5, 4, 4], False, 3, "advection"), ([4, 4, 3], False, 4, "advection"), ([8, 8, 8], True, 2, "wave"),
         ([16, 16], True, 4, "wave")]


@pytest.mark.parametrize("tableau", ["RK4_4", "RK3TVD"])
@pytest.mark.parametrize("cells,tri,order,physics", CASES)
def test_pipelined_tiles_match_the_oracle(cells, tri, order, physics, tableau):
    s, prob, oracle = make(cells, tri, order, physics, tableau)
    assert s.handle.kernel_kind == "linear"
    u0 = np.random.default_rng(order).standard_normal(prob.n_dof)
    M = np.einsum("q,qi,qj->ij", prob.rule.weights, prob.phi, prob.phi)
    tol = max(1e-12, 4.0 * np.linalg.cond(M) * np.finfo(float).eps)
    s.handle.set_state(0, u0)
    s.handle.time_derivative(0, 1)
    assert rel_err(s.handle.get_state(1), oracle.time_derivative(u0)) < tol
    dt = 0.01 / max(cells) / (2 * order + 1) ** 2
    s.handle.step(0.0, dt, 10)
    t, _, _ = make(cells, tri, order, physics, tableau)
    t.handle.set_state(0, u0)
    for _ in range(10):
        t.handle.step(0.0, dt, 1)
    assert np.array_equal(s.handle.get_state(0), t.handle.get_state(0))  # graph runs and single steps
    if tableau == "RK4_4":
        assert rel_err(s.handle.get_state(0), oracle.step(u0, dt, 10)) < 1e-12 + tol * dt


def test_callers_vector_at_an_odd_double():
    s, prob, oracle = make([5, 4, 4], False, 3, "advection")
    u0 = np.random.default_rng(1).standard_normal(prob.n_dof)
    out = []
    for shift in (0, 1):
        u = torch.zeros(prob.n_dof + 2, dtype=torch.float64, device="cuda")
        k = torch.zeros_like(u)
        u[shift:shift + prob.n_dof] = torch.from_numpy(u0).cuda()
        torch.cuda.synchronize()
        _native.check(_native.load().hgg_time_derivative_static(s.handle._raw, ctypes.c_void_p(u[shift:].data_ptr()),
                                                                ctypes.c_void_p(k[shift:].data_ptr())), s.handle._raw)
        out.append(k[shift:shift + prob.n_dof].cpu().numpy())
    assert np.array_equal(out[0], out[1])


def test_fp32_folded_triangles_many_and_few_tiles():
    """Folded triangles at p = 5 in the FP32 form: few tiles take the pipelined kernel, many
    the staged one, both the same products in the same order; a batch takes the pipelined."""
    for cells in ([32, 32], [128, 128]):
        d = hpgem_b200.structured_description(cells, [0.0] * 2, [1.0] * 2, True, True)
        a = hpgem_b200.Advection(2, 5, [0.7, -0.4], tableau="RK4_4", precision=_native.PRECISION_FP32).readMesh(d)
        b = hpgem_b200.Advection(2, 5, [0.7, -0.4], tableau="RK4_4", precision=_native.PRECISION_FP32).readMesh(d)
        assert a.handle.kernel_kind == "linear"
        u0 = np.random.default_rng(2).standard_normal(a.handle.vector_length)
        for s in (a, b):
            s.handle.set_state(0, u0)
        a.handle.step(0.0, 1e-5, 3)
        batch = hpgem_b200.Batch(2)
        batch.add(b, 1e-5, 3)
        batch.step(3)
        batch.synchronize()
        assert np.array_equal(a.handle.get_state(0), b.handle.get_state(0))
        batch.close()
