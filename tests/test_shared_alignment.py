"""Dynamic shared memory that is read as 16-byte vectors is declared with that
alignment: beside a static shared variable nothing else promises it."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "prym_green_ancillary_b200" / "csrc"
DECLARED = re.compile(r"extern\s+__shared__\s+(?:__align__\((\d+)\)\s+)?(\w+)\s+(\w+)\s*\[\]")
VECTORS = {"int4", "uint4", "float4"}


@pytest.mark.parametrize("path", sorted(p for p in CSRC.glob("*.cu*") if "extern __shared__" in p.read_text()),
                         ids=lambda p: p.name)
def test_arrays_read_as_vectors_are_aligned(path):
    text = path.read_text()
    declared = DECLARED.findall(text)
    assert len(declared) == len(re.findall(r"extern\s+__shared__", text))
    for align, element, name in declared:
        as_vectors = re.search(rf"reinterpret_cast<(?:const )?u?int4\s*\*>\(\s*{name}\b", text)
        assert element in VECTORS or int(align or 0) >= 16 or not as_vectors, f"{path.name}: {element} {name}[]"
