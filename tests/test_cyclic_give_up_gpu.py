"""The paper operator's resident rounds when their grid barriers run out of tries
at any of their places (BW_TEST_WAIT_LIMIT of a few tries: a barrier takes about
as long): every call ends, with the exact sequence or with status 2, and the
context goes on from there.
"""
import json

import numpy as np
import pytest

from perf.cases import _cyclic_instance
from prym_green_ancillary_b200 import CyclicEngine, EngineError

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _instance(tmp_path, genus):
    path = tmp_path / f"g{genus}.json"
    path.write_text(json.dumps(_cyclic_instance(genus, 2)))
    return path


@pytest.mark.parametrize("genus", [14, 18, 22])
@pytest.mark.parametrize("limit", [1, 2, 3, 4, 6, 8, 16])
def test_barriers_of_few_tries(genus, limit, tmp_path, monkeypatch):
    for name in ("BW_CYCLIC_GENERIC", "BW_CYCLIC_PERSISTENT", "BW_TEST_HOLD_FIRST_STAGE", "BW_TEST_WAIT_LIMIT"):
        monkeypatch.delenv(name, raising=False)
    path = _instance(tmp_path, genus)
    with CyclicEngine(path, 1, seed=9) as eng:
        eng.generate(33)
        want = eng.download()
    monkeypatch.setenv("BW_TEST_WAIT_LIMIT", str(limit))
    with CyclicEngine(path, 1, seed=9) as eng:
        for _ in range(8):
            try:
                eng.generate(33)
            except EngineError as err:
                assert err.status == 2 and "gave up waiting" in str(err)
                continue
            for a, b in zip(eng.download(), want):
                np.testing.assert_array_equal(a, b)
