"""The paper operator's sequence with whole rounds in one cooperative launch
(small sectors) against the same sequence launched kernel by kernel: every
moment and the final block.  Bit-exact.

The instances have the published ones' character blocks; the sizes go from one
CTA of a few subsets to a full GPU, at both ends of the sectors, with odd
counts, and with more rounds than one launch takes.
"""
import json

import numpy as np
import pytest

from perf.cases import _cyclic_instance
from prym_green_ancillary_b200 import CyclicEngine, EngineError

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _instance(tmp_path, genus, seed=2):
    path = tmp_path / f"g{genus}.json"
    path.write_text(json.dumps(_cyclic_instance(genus, seed)))
    return path


def _sequence(path, sector, nlen, **kw):
    with CyclicEngine(path, sector, seed=9, **kw) as eng:
        eng.generate(nlen)
        first = eng.download()
        launches = eng.launch_count
        eng.generate(nlen)      # again from the initial block, on the same context
        second = eng.download()
        again = eng.launch_count - launches
    for a, b in zip(first, second):
        np.testing.assert_array_equal(a, b)
    return first, again


@pytest.mark.parametrize("genus,sector,nlen", [
    (8, 0, 13), (10, 4, 5), (12, 0, 2), (12, 5, 41), (14, 6, 37), (16, 3, 4 * 1030 + 1), (18, 0, 21), (20, 9, 61),
    (22, 10, 33),
])
def test_rounds_in_one_launch_match_the_kernels(genus, sector, nlen, tmp_path, monkeypatch):
    monkeypatch.delenv("BW_CYCLIC_GENERIC", raising=False)
    path = _instance(tmp_path, genus)
    monkeypatch.setenv("BW_CYCLIC_PERSISTENT", "0")
    want, many = _sequence(path, sector, nlen)
    monkeypatch.delenv("BW_CYCLIC_PERSISTENT")
    got, few = _sequence(path, sector, nlen)
    rounds = (nlen + 2) // 4
    assert few <= 4 + rounds // 1024 + 1 < many + 5   # the launches of whole rounds, not of their kernels
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("rowmix_rounds", [0, 1, 3])
def test_other_rowmix_rounds_keep_the_kernels(rowmix_rounds, tmp_path, monkeypatch):
    monkeypatch.delenv("BW_CYCLIC_GENERIC", raising=False)
    path = _instance(tmp_path, 14)
    got, _ = _sequence(path, 2, 25, rowmix_rounds=rowmix_rounds)
    monkeypatch.setenv("BW_CYCLIC_GENERIC", "1")
    want, _ = _sequence(path, 2, 25, rowmix_rounds=rowmix_rounds)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


def test_grid_barrier_that_runs_out_returns_status_2(tmp_path, monkeypatch):
    monkeypatch.delenv("BW_CYCLIC_GENERIC", raising=False)
    monkeypatch.delenv("BW_CYCLIC_PERSISTENT", raising=False)
    path = _instance(tmp_path, 16)
    want, _ = _sequence(path, 1, 25)
    monkeypatch.setenv("BW_TEST_WAIT_LIMIT", "20000")
    monkeypatch.setenv("BW_TEST_HOLD_FIRST_STAGE", "1")
    with CyclicEngine(path, 1, seed=9) as eng:
        with pytest.raises(EngineError) as err:
            eng.generate(25)
        assert err.value.status == 2 and "gave up waiting" in str(err.value)
    monkeypatch.delenv("BW_TEST_WAIT_LIMIT")
    monkeypatch.delenv("BW_TEST_HOLD_FIRST_STAGE")
    got, _ = _sequence(path, 1, 25)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
