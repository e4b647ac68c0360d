"""What the checked build covers, from the sources: every kernel that indexes a mesh's arrays checks
its indices, and the count that a test reads sums all translation units."""
from __future__ import annotations

import re

import pytest

from test_dependent_launch import SOURCES

COUNTERS = sorted(set(re.findall(r"\b(read_oob_\w+)\(", SOURCES["sgnb_device.h"])))
CELLS = re.findall(r"__global__[^;{]*?\b(k_\w+)\(", SOURCES["sgnb_cells.cu"])


@pytest.mark.parametrize("counter", COUNTERS)
def test_counter_is_summed(counter):
    assert counter in SOURCES["sgnb_api.cu"]


@pytest.mark.parametrize("kernel", CELLS)
def test_cells_check_their_indices(kernel):
    """Reads and writes go through the checked helpers, or follow a check of the same index."""
    s = SOURCES["sgnb_cells.cu"]
    body = s[s.index(kernel + "("):]
    body = body[:body.index("\n}\n")]
    assert re.search(r"\bat\(|\bput\(|\bdepth_at\(|SGNB_INB\(", body)
    arrays = re.findall(r"double\* __restrict__ (\w+)", body)
    unchecked = [a for a in arrays if re.search(r"\b" + a + r"\[", body.split("{", 1)[1])]
    assert set(unchecked) <= ({"Hb"} if "SGNB_INB(node" in body else {"grad"})


def test_cells_count():
    assert "read_oob_cells" in COUNTERS
