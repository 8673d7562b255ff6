"""A context's work goes on its own streams, which do not wait for the default stream: copies and clears without a
stream argument would run on the default stream, in no order with the context's runs."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cms-julia_b200" / "csrc"


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_no_default_stream_commands(source):
    text = re.sub(r"//[^\n]*", "", (CSRC / source).read_text())
    assert not re.findall(r"\bcuda(?:Memset|Memcpy)(?:2D|3D)?\s*\(", text)
