"""Rules on the CUDA sources that no run shows."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "varrcwa_b200" / "csrc"


@pytest.mark.parametrize("src", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_math_functions_are_called(src):
    """Reciprocals, roots and exponentials are CUDA's own functions: none is
    rebuilt from the hardware's approximation in inline assembly."""
    text = (CSRC / src).read_text()
    assert not re.search(r"\b(rcp|rsqrt|sqrt|div|ex2|lg2|sin|cos|tanh)\.(approx|full)\b", text)
