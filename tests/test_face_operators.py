"""CPU: the lane kernels' face operators.  Operators are merged, and functions left out of a
face, only where they are equal, or zero, up to the rounding they are tabulated with (a few
1e-16): a difference of 1e-13, or a trace of 1e-14, is a user's own and stays."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HOST = os.path.join(ROOT, "hpgem_b200", "csrc", "host")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("face") / "face_operators")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", HOST, os.path.join(ROOT, "tests", "host", "face_operators.cpp")] +
                   [os.path.join(HOST, f) for f in ("operators.cpp", "setup.cpp")] + ["-o", out], check=True, timeout=300)
    return out


def counts(program, dim, tri, order, change=0.0, value=0.0):
    out = subprocess.run([program, str(dim), str(int(tri)), str(order), repr(change), repr(value)], check=True,
                         capture_output=True, text=True, timeout=120)
    return [int(v) for v in out.stdout.split()]


def trace_size(dim, tri, p):
    return p + 1 if dim == 2 else (p + 1) * (p + 2) // 2 if tri else (p + 1) ** 2


@pytest.mark.parametrize("dim,tri,order", [(2, True, p) for p in range(1, 6)] + [(3, True, p) for p in range(1, 6)] +
                         [(2, False, 5), (3, False, 2), (3, False, 3)])
def test_copies_merge_and_trace_functions_are_found(program, dim, tri, order):
    pairs, distinct, trace = counts(program, dim, tri, order)
    assert trace == pairs * trace_size(dim, tri, order)
    # the three distinct self operators of a triangle, four of a tetrahedron, and the neighbours'
    assert distinct <= pairs and (not tri or distinct < pairs)


@pytest.mark.parametrize("dim,order", [(2, 2), (3, 2), (3, 3)])
def test_operators_that_differ_are_kept_apart(program, dim, order):
    pairs, distinct, _ = counts(program, dim, True, order)
    assert counts(program, dim, True, order, change=1e-13)[1] > distinct


@pytest.mark.parametrize("dim,tri,order", [(2, True, 3), (3, True, 2), (3, False, 2)])
def test_small_traces_are_kept(program, dim, tri, order):
    pairs, _, trace = counts(program, dim, tri, order)
    assert counts(program, dim, tri, order, value=1e-14)[2] > trace
