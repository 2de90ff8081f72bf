"""CPU: which elements the lane kernels' host set-up takes as equal.  Elements share one
element's geometry only where they differ by the rounding of their vertex coordinates: a
mesh whose cells vary by more, in whichever axis, however flat the cells, is refused (sum-
factorised form) or split into groups (simplices and the wave).  The deviation of any
element from the one it steps with stays below rounding: 2^-50 of the mesh's extent over a
cell's, twice (both ends of an edge), times the entries of the inverse Jacobian (below 4)."""
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
    out = str(tmp_path_factory.mktemp("lane") / "lane_groups")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", HOST, os.path.join(ROOT, "tests", "host", "lane_groups.cpp")] +
                   [os.path.join(HOST, f) for f in ("lane.cpp", "operators.cpp", "setup.cpp")] + ["-o", out],
                   check=True, timeout=300)
    return out


def groups(program, cells, upper, tri, order, wave, fp32=False, axis=-1, by=0.0, lower=None):
    args = [len(cells)] + list(cells) + list(lower or [0.0] * len(cells)) + list(upper) + \
           [int(tri), order, int(wave), int(fp32), axis, by]
    out = subprocess.run([program] + [repr(a) for a in args], check=True, capture_output=True, text=True, timeout=120)
    return out.stdout.split()


# (cells, upper corner, simplices, wave): equal cells, flat and long ones among them
EQUAL = [([32, 32], [1.0, 1.0], False, False), ([150, 210], [1.0, 1e-6], False, False), ([1000, 3], [1.0, 1.0], False, False),
         ([8, 8, 8], [1.0, 1.0, 1e-5], False, False), ([30, 26], [1.0, 1e-6], True, False), ([26, 22], [1.0, 1.0], True, True),
         ([8, 8, 8], [1.0, 1e-5, 1.0], True, True), ([9, 7], [1.0, 1.0], False, True)]


@pytest.mark.parametrize("cells,upper,tri,wave", EQUAL)
def test_equal_cells_share_their_geometry(program, cells, upper, tri, wave):
    for fp32 in (False, True):
        got = groups(program, cells, upper, tri, 2, wave, fp32)
        assert got[1] == "1", got
        if got[0] == "groups" and not fp32:
            assert int(got[2]) <= 128  # ten simplices, their parities and the odd sides' wrap
            assert float(got[3]) <= 8 * 2.0 ** -50 * max(cells)


# (cells, upper corner, simplices, wave, axis, by): every other node plane moved by `by` cells.  The
# first ones hide below a bound relative to the largest entry: the moved axis is the long one of
# flat cells, so its entries are the small ones.
UNEQUAL = [([8, 8, 8], [1.0, 1.0, 1e-5], False, False, 0, 1e-8), ([32, 32], [1.0, 1e-4], True, False, 0, 1e-9),
           ([32, 32], [1.0, 1e-6], True, True, 0, 1e-7), ([8, 8, 8], [1.0, 1.0, 1e-5], True, True, 0, 1e-8),
           ([16, 12], [1.0, 1e-5], False, True, 0, 1e-8), ([32, 32], [1.0, 1.0], False, False, 0, 1e-13),
           ([32, 32], [1.0, 1.0], True, False, 1, 1e-13), ([32, 32], [1.0, 1.0], False, True, 1, 1e-13),
           ([32, 32], [1.0, 1.0], False, False, 1, 1e-3)]


@pytest.mark.parametrize("cells,upper,tri,wave,axis,by", UNEQUAL)
def test_cells_that_differ_keep_their_own(program, cells, upper, tri, wave, axis, by):
    got = groups(program, cells, upper, tri, 2, wave, False, axis, by)
    if got[0] == "tensor":
        assert got[1] == "0", got
    else:
        alike = groups(program, cells, upper, tri, 2, wave)
        assert got[1] == "1" and int(got[2]) > int(alike[2]), (got, alike)
        assert float(got[3]) <= 8 * 2.0 ** -50 * max(cells)


def test_graded_cells_are_refused(program):
    # every cell of its own size: more groups than tiles of them could fill
    assert groups(program, [60, 64], [1.0, 1.0], True, 2, False, False, 2, 1e-4) == ["groups"] + ["0"] * 6
    assert groups(program, [60, 64], [1.0, 1.0], True, 2, False, False, 2, 1e-11) == ["groups"] + ["0"] * 6
    assert groups(program, [33, 31], [1.0, 1.0], False, 2, False, False, 2, 1e-4) == ["tensor", "0"]


@pytest.mark.parametrize("cells,tri", [([26, 22], True), ([9, 7], False), ([8, 6, 10], True)])
@pytest.mark.parametrize("fp32", [False, True])
def test_padding_stays_at_zero(program, cells, tri, fp32):
    """A tile's padding slots are their own neighbours (they start at zero: their derivative
    is zero), with a face normal the upwind wave can divide by."""
    got = groups(program, cells, [1.0] * len(cells), tri, 2, True, fp32)
    assert got[1] == "1" and int(got[4]) > 0 and got[5] == got[4], got
    if fp32:
        assert float(got[6]) > 0.0
