"""What the comparison of the resident rounds rests on: BW_CYCLIC_PERSISTENT=0 has
a round launched kernel by kernel (ten of the two applications, two of moments),
and without it whole rounds take one launch."""
import json

import pytest

from perf.cases import _cyclic_instance
from prym_green_ancillary_b200 import CyclicEngine

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("genus,rounds", [(12, 10), (16, 40), (22, 5)])
def test_launches_of_either_path(genus, rounds, tmp_path, monkeypatch):
    monkeypatch.delenv("BW_CYCLIC_GENERIC", raising=False)
    path = tmp_path / f"g{genus}.json"
    path.write_text(json.dumps(_cyclic_instance(genus, 2)))
    launches = {}
    for persistent in ("0", "1"):
        monkeypatch.setenv("BW_CYCLIC_PERSISTENT", persistent)
        with CyclicEngine(path, 0, seed=9) as eng:
            before = eng.launch_count
            eng.generate(1 + 4 * rounds)
            launches[persistent] = eng.launch_count - before
    assert launches["0"] >= 12 * rounds
    assert launches["1"] <= 5
