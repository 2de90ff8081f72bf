"""GPU: the kernel variant of a handle that is a member of a batch.  The batch steps the
member with the kernel it took it in with, whatever the variant is set to meanwhile, and the
handle's own steps after it has left use the variant that was set.  Both organisations
evaluate the same operator: 1e-12 of the largest coefficient, as in the lane tests."""
import numpy as np
import pytest

import hpgem_b200

from lane_helpers import kernel_class, write_mesh_file

pytestmark = pytest.mark.gpu


def make(cells, tri, order, physics):
    d = len(cells)
    if physics == "advection":
        s = hpgem_b200.Advection(d, order, [0.7, -0.4, 0.5][:d], tableau="RK4_4")
    else:
        s = hpgem_b200.AcousticWave(d, order, c_inv=0.8, tableau="RK4_4", flux="upwind")
    s.readMesh(hpgem_b200.structured_description(cells, [0.0] * d, [1.0] * d, tri, True))
    s.handle.set_state(0, np.random.default_rng(3).standard_normal(s.handle.vector_length))
    return s


@pytest.mark.parametrize("cells,tri,order,physics", [([13, 9], False, 3, "advection"), ([24, 20], True, 3, "advection"),
                                                     ([24, 20], True, 4, "advection"), ([8, 8, 8], True, 2, "wave")])
@pytest.mark.parametrize("variants", [(0, 1), (0, 2), (1, 0)])
def test_variant_set_on_a_member(cells, tri, order, physics, variants):
    dt = 0.01 / max(cells) / (2 * order + 1) ** 2
    ref = make(cells, tri, order, physics)
    ref.handle.step(0.0, dt, 12)
    want = ref.handle.get_state(0)
    s = make(cells, tri, order, physics)
    s.handle.set_kernel_variant(variants[0])
    batch = hpgem_b200.Batch(2)
    slot = batch.add(s, dt, 9)
    batch.step(3)
    s.handle.set_kernel_variant(variants[1])  # (the steps may still run)
    batch.step(3)
    batch.synchronize()
    s.handle.set_kernel_variant(variants[0])
    s.handle.set_kernel_variant(variants[1])
    batch.step(3)
    batch.synchronize()
    assert batch.remaining(slot) == 0
    batch.remove(slot)
    batch.close()
    assert (kernel_class(s) in ("lane tables", "sum-factorised lanes")) == (variants[1] == 0)
    s.handle.step(0.0, dt, 3)
    got = s.handle.get_state(0)
    assert np.abs(got - want).max() / np.abs(want).max() < 1e-12


def test_batch_closed_with_a_member():
    s = make([24, 20], True, 3, "advection")
    batch = hpgem_b200.Batch(1)
    batch.add(s, 1e-5, 2)
    batch.step(2)
    batch.synchronize()
    s.handle.set_kernel_variant(1)
    batch.close()
    s.handle.step(0.0, 1e-5, 2)
    ref = make([24, 20], True, 3, "advection")
    ref.handle.step(0.0, 1e-5, 4)
    assert np.abs(s.handle.get_state(0) - ref.handle.get_state(0)).max() < 1e-12 * np.abs(ref.handle.get_state(0)).max()


def test_source_set_on_a_stored_matrix_member():
    """A batch steps its members without source terms (it takes no handle that has one), also
    a member that is given one later."""
    d = hpgem_b200.structured_description([5, 4, 6], [0.0] * 3, [1.0] * 3, False, True)
    solvers = [hpgem_b200.HpgemAPILinear(3, 2, "advection", advection=[0.7, -0.4, 0.5], tableau="RK4_4").readMesh(d)
               for _ in range(2)]
    u0 = np.random.default_rng(4).standard_normal(solvers[0].handle.vector_length)
    for s in solvers:
        s.handle.set_state(0, u0)
    batch = hpgem_b200.Batch(1)
    slot = batch.add(solvers[0], 1e-4, 3)
    solvers[0].setSourceTerm(lambda x, t: np.ones(len(x)))
    batch.step(3)
    batch.synchronize()
    batch.remove(slot)
    batch.close()
    solvers[1].handle.step(0.0, 1e-4, 3)
    want = solvers[1].handle.get_state(0)
    assert np.abs(solvers[0].handle.get_state(0) - want).max() < 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("cells,order,physics,alone", [([8, 8], 3, "advection", 2), ([6, 6], 1, "wave", 4), ([4, 4], 4, "advection", 9)])
def test_batches_step_many_sparse_tiles_with_the_general_kernels(tmp_path, cells, order, physics, alone):
    """A small mesh whose triangles all differ has a tile for each of them: the lane kernel is
    the faster for as many such meshes as run at once (two tiles per SM: `alone` of these),
    the others of a batch take the general kernels.  Their vectors go back when they leave."""
    path = write_mesh_file(tmp_path / "mesh.hpgem", [np.linspace(0.0, 1.0, n + 1) for n in cells], True, 0.1)
    solvers = []
    for i in range(alone + 3):
        if physics == "advection":
            s = hpgem_b200.Advection(2, order, [0.7, -0.4], tableau="RK4_4").readMeshFile(path)
        else:
            s = hpgem_b200.AcousticWave(2, order, c_inv=0.8, tableau="RK4_4", flux="upwind").readMeshFile(path)
        s.handle.set_state(0, np.random.default_rng(6).standard_normal(s.handle.vector_length))
        solvers.append(s)
    ref = solvers.pop()
    dt = 0.01 / max(cells) / (2 * order + 1) ** 2
    batch = hpgem_b200.Batch(len(solvers) + 1)
    slots = [batch.add(s, dt, 5) for s in solvers]
    members = {c["kind"]: c["members"] for c in batch.class_info()}
    assert members.pop("lane tables") == alone and list(members.values()) == [2]
    batch.step(5)
    batch.synchronize()
    halves = [s.handle.get_state(0) for s in solvers]
    for slot in slots:
        batch.remove(slot)
    again = batch.add(solvers[-1], dt, 4)  # there is room among the tiles again
    assert [c["kind"] for c in batch.class_info()] == ["lane tables"]
    assert np.array_equal(solvers[-1].handle.get_state(0), halves[-1])
    batch.step(4)
    batch.synchronize()
    batch.remove(again)
    batch.close()
    ref.handle.step(0.0, dt, 9)
    want = ref.handle.get_state(0)
    for s in solvers[:-1]:
        s.handle.step(0.0, dt, 4)
    for s in solvers:
        assert np.abs(s.handle.get_state(0) - want).max() < 1e-12 * np.abs(want).max()


def test_sparse_member_of_two_batches(tmp_path):
    """The second batch takes the layout the first one steps the member with, and the room
    among the tiles is what it was when it has left."""
    path = write_mesh_file(tmp_path / "mesh.hpgem", [np.linspace(0.0, 1.0, 9)] * 2, True, 0.1)
    solvers = [hpgem_b200.Advection(2, 3, [0.7, -0.4], tableau="RK4_4").readMeshFile(path) for _ in range(4)]
    first, second = hpgem_b200.Batch(4), hpgem_b200.Batch(4)
    kept = first.add(solvers[0], 1e-5, 0)
    slots = [second.add(s, 1e-5, 0) for s in (solvers[1], solvers[2], solvers[0])]  # two of them fill the tiles
    for _ in range(3):
        second.remove(slots.pop())
    assert second.num_classes == 0
    second.add(solvers[1], 1e-5, 0)
    second.add(solvers[2], 1e-5, 0)
    second.add(solvers[3], 1e-5, 0)
    members = {c["kind"]: c["members"] for c in second.class_info()}
    assert members.pop("lane tables") == 2 and list(members.values()) == [1]
    first.remove(kept)
    first.close()
    second.close()
