"""Kernels that may start while the kernel before them still runs (programmatic dependent launch) must not let the compiler
assume that nobody writes their inputs: checked on the sources, since a load moved above the wait is a race that no run has to
show."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "polarai-framework_b200", "csrc")


def code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


OVERLAPPING = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and
                     re.search(r"\blaunch(_clusters)?\(\"|ProgrammaticStreamSerialization", code(f)))


def test_the_overlapping_sources_are_found():
    assert {"elementwise.cu", "extra_builtins.cu", "gemm_skinny.cu", "gemm_tc_mid.cu", "program.cu"} <= set(OVERLAPPING)


@pytest.mark.parametrize("name", OVERLAPPING)
def test_inputs_are_read_after_the_wait(name):
    text = code(name)
    # a restrict-qualified input may be read through the read-only path and from above the wait, and so may the
    # intrinsics for loads with a cache hint, which are no volatile accesses
    assert not re.search(r"__restrict__|\b__ld(g|cs|cg|ca|lu|cv)\b|\b__st(cs|cg|wb|wt)\b", text)
    kernels = re.split(r"\b__global__\b", text)[1:]
    assert kernels and all("pdl_enter()" in k for k in kernels)
