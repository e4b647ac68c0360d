"""Kernels that launch_dependent starts may run beside the kernel before them in their stream. The
sources keep the two rules that follow from it (sgnb_device.h): such a kernel waits before it
touches global memory, and reads nothing through the non-coherent path."""
from __future__ import annotations

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sgn-hyperbolic-gpu_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


SOURCES = {n: source(n) for n in sorted(os.listdir(CSRC)) if n.endswith((".cu", ".cuh", ".h"))}
KERNELS = sorted({k for s in SOURCES.values() for k in re.findall(r"launch_dependent\((k_\w+)", s)})


def definition(kernel):
    """(file, parameters, body) of a kernel."""
    for name, s in SOURCES.items():
        m = re.search(r"__global__[^;{]*?\b" + kernel + r"\(([^{]*?)\)\s*\{", s)
        if m:
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(s[end], 0)
                end += 1
            return name, m.group(1), s[m.end():end]
    raise AssertionError(kernel)


def test_there_are_such_kernels():
    assert {"k_line", "k_line_exact", "k_fused", "k_controller_loop"} <= set(KERNELS)


@pytest.mark.parametrize("kernel", KERNELS)
def test_waits_first(kernel):
    _, params, body = definition(kernel)
    before, wait, _ = body.partition("wait_for_previous();")
    assert wait
    for p in re.findall(r"(\w+)\s*(?:,|$)", params.replace("\n", " ")):
        assert not re.search(r"\b" + p + r"\b", before), (kernel, p)


@pytest.mark.parametrize("name", sorted({definition(k)[0] for k in KERNELS} | {"sgnb_kernels_line.cuh", "sgnb_kernels.cuh",
                                                                                "sgnb_device.h"}))
def test_ordinary_loads(name):
    s = SOURCES[name]
    dependent = {k for k in KERNELS if definition(k)[0] == name}
    for k in set(re.findall(r"__global__[^;{]*?\b(k_\w+)\(", s)) - dependent:  # launched in stream order
        s = s.replace(definition(k)[1], "")
    assert not re.search(r"ld\.global\.nc|__ldg\(|const double\* ?__restrict__", s)
