"""Every function that sgnb_device.h declares for the kernels' launch and set-up has a caller."""
from __future__ import annotations

import re

import pytest

from test_dependent_launch import SOURCES

DECLARED = sorted(set(re.findall(r"\b(?:cudaError_t|int|size_t|long long)\s+(\w+)\([^;{]*\);", SOURCES["sgnb_device.h"])))


def test_declarations_are_found():
    assert {"launch_line", "launch_controller_loop", "line_grid_blocks", "launch_cells_back"} <= set(DECLARED)


@pytest.mark.parametrize("name", DECLARED)
def test_is_called(name):
    uses = sum(len(re.findall(r"\b" + name + r"\(", s)) for s in SOURCES.values())
    assert uses > 2, "declared and defined only"
