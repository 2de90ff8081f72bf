"""CPU: what the chained stage kernels may read through the non-coherent path.

A chained stage is resident while the previous stage still writes the solution and the
stage vectors.  Non-coherent loads (ld.global.nc, __ldg) are defined only for memory that
nobody writes while the kernel lives, and one in an asm without a memory clobber may be
moved ahead of the wait.  So in the sources of those kernels such loads take operators,
geometry and indices only, and no kernel lets the next one start before its own wait (three
stages would be resident together)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hpgem_b200", "csrc")
CHAINED = ["tensor_slice.cuh", "tensor_lane.cuh", "lane_stage.cuh", "stage_lane.cu", "batch_lane.cu", "batch_items.cuh"]
# the tables no stage kernel writes
TABLES = ("geo", "geo_nu", "g.nbr", "gcols", "head", "cols")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def functions_with_nc(text):
    """Names of the functions whose body has a non-coherent load."""
    names = set()
    for m in re.finditer(r"(\w+)\s*\([^()]*\)\s*\{([^{}]*)\}", text):
        if "ld.global.nc" in m.group(2):
            names.add(m.group(1))
    return names


@pytest.mark.parametrize("name", CHAINED)
def test_non_coherent_loads_read_tables_only(name):
    loaders = functions_with_nc(source("tensor_slice.cuh")) | {"__ldg"}
    wrappers = True
    while wrappers:  # functions that hand their argument on to one of them
        wrappers = {m.group(1) for n in CHAINED for m in
                    re.finditer(r"(\w+)\(const (?:double|float) \*(\w+)\) \{ return [^;{}]*\b(?:%s)\(\2\); \}" %
                                "|".join(map(re.escape, loaders)), source(n))} - loaders
        loaders |= wrappers
    text = source(name)
    for loader in loaders:
        for m in re.finditer(r"\b%s\(\s*([\w.]+)" % re.escape(loader), text):
            if m.group(1) == "const":  # the definition
                continue
            assert m.group(1) in TABLES or m.group(1) == "p", (name, loader, text[m.start():m.start() + 60])
    for m in re.finditer(r"asm\b([^;]*)\bld\.global\b(?!\.nc)", text):  # a coherent load in asm stays behind the wait
        statement = text[m.start():text.index(";", m.end())]
        assert "volatile" in m.group(1) and '"memory"' in statement, statement


@pytest.mark.parametrize("name", ["tensor_slice.cuh", "tensor_lane.cuh", "lane_stage.cuh"])
def test_no_stage_lets_the_next_start_before_its_own_wait(name):
    text = source(name)
    for m in re.finditer(r"__global__[^;{]*\{", text):  # kernels hand over to a body that waits
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        body = text[m.end():at]
        assert "chain_next" not in body or 0 <= body.find("chain_wait") < body.find("chain_next"), body
    assert "chain_wait()" in text
