"""Kernels that may start while the previous one still writes read global memory with plain loads only."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "iree-turbine_b200" / "csrc"


@pytest.mark.parametrize("path", sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]), ids=lambda p: p.name)
def test_no_load_asks_for_constant_memory(path):
    code = re.sub(r"//[^\n]*", "", path.read_text())
    assert not re.search(r"__ldg|__restrict__|ld\.global\.nc|ldu\.global", code)
