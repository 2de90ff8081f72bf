"""GPU: two handles of one lane kernel whose blocks take different amounts of shared memory
(tetrahedra at p = 3: two tiles a block on the larger mesh, one on the smaller), stepped in
turn and from two threads at once.  The limit of a kernel's shared memory belongs to the
process: one handle's launch must not lower it under the other's."""
import threading

import numpy as np
import pytest

import hpgem_b200

pytestmark = pytest.mark.gpu


def make(n):
    s = hpgem_b200.AcousticWave(3, 3, c_inv=0.8, tableau="RK4_4", flux="upwind")
    s.readMesh(hpgem_b200.structured_description([n] * 3, [0.0] * 3, [1.0] * 3, True, True))
    s.handle.set_state(0, np.random.default_rng(n).standard_normal(s.handle.vector_length))
    return s


def test_in_turn():
    a, b, ref = make(16), make(8), make(16)
    ref.handle.step(0.0, 1e-5, 3)
    for _ in range(3):
        a.handle.step(0.0, 1e-5, 1)
        b.handle.step(0.0, 1e-5, 1)
    a.handle.synchronize()
    assert np.array_equal(a.handle.get_state(0), ref.handle.get_state(0))


def test_from_two_threads():
    solvers = [make(16), make(8)]
    failures = []

    def work(s):
        try:
            for i in range(400):
                s.handle.time_derivative(0, 1)
                if i % 8 == 0:
                    s.handle.step(0.0, 1e-6 * (1 + i), 1)  # a new dt: a new capture
        except Exception as e:  # (a thread's exception does not reach the test by itself)
            failures.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in solvers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
