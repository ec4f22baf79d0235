"""The library keeps what it finds out about a device in the context: a variable
that a function keeps between calls would be shared by the threads of all
contexts (the server's lanes launch side by side) without ordering."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "atrbvh_b200" / "csrc"


@pytest.mark.parametrize("src", sorted(p.name for p in CSRC.iterdir() if p.suffix in (".cu", ".cpp", ".cuh", ".h")))
def test_no_function_keeps_a_variable(src):
    kept = [line.strip() for line in (CSRC / src).read_text().splitlines()
            if re.match(r"\s+(static|thread_local)\s(?!.*\bconst(expr)?\b)[^()]*;", line)]
    assert not kept, kept
