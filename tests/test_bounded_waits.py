"""Waits for copies are bounded; one that gives up waits as long again before its CTA goes on (a
copy must not land in shared memory that the CTA has left), and then writes NaN. From the sources: a
copy that never lands cannot be made."""
from __future__ import annotations

import re

import pytest

from test_dependent_launch import SOURCES

WAIT = r"for \(int it = 0; it < kTmaTries && !landed; \+\+it\) landed = mbar_try_wait\(mbar, 0\);"


@pytest.mark.parametrize("name", [n for n, s in SOURCES.items() if "mbar_try_wait(mbar" in s])
def test_second_wait(name):
    s = SOURCES[name]
    assert len(re.findall(r"mbar_try_wait\(mbar", s)) == len(re.findall(WAIT, s))
    assert re.search(WAIT + r"\s*if \(!landed\) \{\s*" + WAIT + r"[^}]*0x7ff8000000000000LL", s)
