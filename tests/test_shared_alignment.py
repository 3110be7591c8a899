"""Dynamic shared memory of kernels with asynchronous copies has to say the 16
bytes of alignment that cp.async.bulk needs, or round its address up to more:
the element type alone promises less, and the placement beside static arrays
then decides whether the copies fault."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "nalu-wind_gb300" / "csrc"


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu") if "cp.async" in p.read_text()))
def test_declared_or_rounded_alignment(source):
    found = re.findall(r"extern __shared__\s+(.*?)(\w+)\[\];(.{0,200})", (CSRC / source).read_text(), re.S)
    assert found
    for qualifiers, name, after in found:
        declared = re.search(r"__align__\((\d+)\)", qualifiers)
        rounded = re.search(name + r"\)\s*\+\s*(\d+)\)\s*&", after)
        assert (declared and int(declared.group(1)) >= 16) or (rounded and int(rounded.group(1)) >= 15), (name, qualifiers)
