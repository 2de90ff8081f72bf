"""GPU: device memory of a handle (the bytes its creation takes from the device's pool).
Beside the solution's two buffers, the stage vectors and one conversion vector, a handle
keeps stage inputs formed ahead only where its kernels read them."""
import numpy as np
import pytest

import hpgem_b200
from hpgem_b200 import _native

from lane_helpers import kernel_class

pytestmark = pytest.mark.gpu


def used_bytes():
    from cuda.bindings import driver
    err, pool = driver.cuDeviceGetMemPool(0)
    assert err == driver.CUresult.CUDA_SUCCESS
    err, value = driver.cuMemPoolGetAttribute(pool, driver.CUmemPool_attribute.CU_MEMPOOL_ATTR_USED_MEM_CURRENT)
    assert err == driver.CUresult.CUDA_SUCCESS
    return int(value)


def description(cells, tri):
    d = len(cells)
    return hpgem_b200.structured_description(cells, [0.0] * d, [1.0] * d, tri, True)


# (make, vectors of doubles: 2 of the solution, the stages', conversion, inputs formed ahead)
CASES = {
    "folded triangles on the lane kernels": (
        lambda: hpgem_b200.Advection(2, 4, [0.7, -0.4], tableau="RK4_4").readMesh(description([160, 160], True)), 2 + 4 + 1),
    "folded triangles in the FP32 form": (
        lambda: hpgem_b200.Advection(2, 5, [0.7, -0.4], tableau="RK4_4", precision=_native.PRECISION_FP32).readMesh(
            description([160, 160], True)), 2 + 2 + 1 + 2),
    "stored matrices, chain tableau": (
        lambda: hpgem_b200.HpgemAPILinear(3, 3, "advection", advection=[0.7, -0.4, 0.5], tableau="RK4_4").readMesh(
            description([20, 20, 20], False)), 2 + 4 + 2),
    "stored matrices, several vectors in a stage": (
        lambda: hpgem_b200.HpgemAPILinear(3, 3, "advection", advection=[0.7, -0.4, 0.5], tableau="RK3TVD").readMesh(
            description([20, 20, 20], False)), 2 + 3),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_vectors_of_a_handle(name):
    make, vectors = CASES[name]
    warm = make()  # (the process's first handle takes its own)
    warm.handle.close()
    before = used_bytes()
    s = make()
    n = s.handle.vector_length
    used = used_bytes() - before
    # indices, geometry and tables: below 160 bytes an element and 2 MB
    assert used <= 8 * n * vectors * 1.02 + 160 * s.n_elements + (2 << 20), (used / (8.0 * n), vectors)


def test_variant_change_of_folded_triangles():
    """Off the lane layout the stored-matrix tiles get their inputs, and step as before."""
    res = []
    for variant in (0, 1):
        s = hpgem_b200.Advection(2, 4, [0.7, -0.4], tableau="RK4_4").readMesh(description([40, 40], True))
        s.handle.set_kernel_variant(variant)
        s.handle.set_state(0, np.random.default_rng(1).standard_normal(s.handle.vector_length))
        s.handle.step(0.0, 1e-5, 5)
        res.append(s.handle.get_state(0))
    assert np.abs(res[0] - res[1]).max() < 1e-12 * np.abs(res[1]).max()


class limited_pool:
    """The device's memory pool replaced by one of at most `size` bytes."""

    def __init__(self, size):
        from cuda.bindings import driver
        self.driver, self.size = driver, size

    def check(self, result):
        assert result[0] == self.driver.CUresult.CUDA_SUCCESS, result
        return result[1] if len(result) > 1 else None

    def __enter__(self):
        d = self.driver
        self.before = self.check(d.cuDeviceGetMemPool(0))
        props = d.CUmemPoolProps()
        props.allocType = d.CUmemAllocationType.CU_MEM_ALLOCATION_TYPE_PINNED
        props.location.type = d.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE
        props.location.id = 0
        props.maxSize = self.size
        self.pool = self.check(d.cuMemPoolCreate(props))
        self.check(d.cuDeviceSetMemPool(0, self.pool))

    def __exit__(self, *args):
        self.check(self.driver.cuDeviceSetMemPool(0, self.before))
        self.check(self.driver.cuMemPoolDestroy(self.pool))


def test_problem_that_fits_without_the_lane_kernels_only():
    """720 000 triangles at p = 3, RK4: six vectors of 58 MB and 100 bytes an element fit
    448 MB, the lane kernels' conversion vector beside them does not."""
    make = lambda: hpgem_b200.Advection(2, 3, [0.7, -0.4], tableau="RK4_4").readMesh(description([600, 600], True))
    roomy = make()
    u0 = np.random.default_rng(2).standard_normal(roomy.handle.vector_length)
    roomy.handle.set_state(0, u0)
    roomy.handle.step(0.0, 1e-6, 2)
    assert kernel_class(roomy) == "lane tables"
    with limited_pool(448 << 20):
        s = make()
        s.handle.set_state(0, u0)
        s.handle.step(0.0, 1e-6, 2)
        got = s.handle.get_state(0)
        s.handle.close()
    want = roomy.handle.get_state(0)
    assert np.abs(got - want).max() < 1e-12 * np.abs(want).max()


def test_stored_matrices_without_room_for_inputs_formed_ahead():
    """32^3 hexahedra at p = 3, RK4: six vectors of 16.8 MB, not eight, in 128 MB; the staged
    tiles then form the same products in the same order."""
    make = lambda: hpgem_b200.HpgemAPILinear(3, 3, "advection", advection=[0.7, -0.4, 0.5], tableau="RK4_4").readMesh(
        description([32, 32, 32], False))
    roomy = make()
    u0 = np.random.default_rng(2).standard_normal(roomy.handle.vector_length)
    roomy.handle.set_state(0, u0)
    roomy.handle.step(0.0, 1e-5, 2)
    with limited_pool(128 << 20):
        s = make()
        s.handle.set_state(0, u0)
        s.handle.step(0.0, 1e-5, 2)
        got = s.handle.get_state(0)
        s.handle.close()
    assert np.array_equal(got, roomy.handle.get_state(0))
