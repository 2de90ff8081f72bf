"""GPU: chained stages (a stage resident while the previous one still writes) against the
same stages started one after the other has ended: the same kernels on the same inputs, so
the results are equal bit for bit.  Many steps on meshes of 1, 2 and 32 tiles of 32
elements, where several stages share an SM and the overlap is largest, and on one mesh of
several waves; every chained kernel, both precisions, tableaux that read one and several
stage vectors."""
import numpy as np
import pytest

import hpgem_b200
from hpgem_b200 import _native

pytestmark = pytest.mark.gpu

# (cells, simplices, order, physics): 1, 2 and about 32 tiles of each kernel, then many
CASES = [([8, 4], False, 2, "advection"), ([8, 8], False, 4, "advection"), ([32, 32], False, 2, "advection"),
         ([4, 4, 2], False, 1, "advection"), ([150, 210], False, 3, "advection"),
         ([4, 4, 2], False, 3, "advection"), ([4, 4, 4], False, 3, "advection"), ([10, 10, 10], False, 3, "advection"),
         ([28, 28, 28], False, 3, "advection"),
         ([8, 4], True, 3, "advection"), ([24, 20], True, 2, "advection"), ([4, 4, 4], True, 2, "advection"),
         ([12, 12, 12], True, 2, "advection"),
         ([8, 4], True, 2, "wave"), ([24, 20], True, 3, "wave_upwind"), ([4, 4, 4], True, 2, "wave"),
         ([8, 9], False, 3, "wave"), ([12, 12, 12], True, 2, "wave_upwind")]


def solver(cells, tri, order, physics, tableau, precision):
    d = len(cells)
    if physics == "advection":
        s = hpgem_b200.Advection(d, order, [0.7, -0.4, 0.5][:d], tableau=tableau, precision=precision)
    else:
        s = hpgem_b200.AcousticWave(d, order, c_inv=0.8, tableau=tableau, precision=precision,
                                    flux="upwind" if physics == "wave_upwind" else "central")
    return s.readMesh(hpgem_b200.structured_description(cells, [0.0] * d, [1.0] * d, tri, True))


@pytest.mark.parametrize("precision", [_native.PRECISION_FP64, _native.PRECISION_FP32])
@pytest.mark.parametrize("tableau", ["RK4_4", "DormandPrince"])
@pytest.mark.parametrize("cells,tri,order,physics", CASES)
def test_chained_stages_match_stages_run_one_by_one(cells, tri, order, physics, tableau, precision):
    lib = _native.load()
    u0 = None
    res = []
    for overlap in (1, 0):
        h = solver(cells, tri, order, physics, tableau, precision).handle
        _native.check(lib.hgg_test_set_overlap(h._raw, overlap), h._raw)
        if u0 is None:
            u0 = np.random.default_rng(5).standard_normal(h.vector_length)
        h.set_state(0, u0)
        h.step(0.0, 0.02 / max(cells) / (2 * order + 1) ** 2, 203)  # graphs of eight steps and single ones
        res.append([h.get_state(v) for v in (0, 1, 2)])
    assert np.isfinite(res[0][0]).all()
    for chained, serial in zip(*res):
        assert np.array_equal(chained, serial)
