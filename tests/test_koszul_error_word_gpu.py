"""The INT8 contexts' error words (mapped host memory, shared out of pages of
64): a word is its context's alone until that context's kernels are done, and
one context's give-up is no other's.

A kernel gives up here because CTA 0 of d never sees its first stage
(BW_TEST_HOLD_FIRST_STAGE) and its bounded wait runs out; nothing faults.
"""
import threading
import time

import numpy as np
import pytest

import oracle
from prym_green_ancillary_b200 import EngineError, KoszulEngine

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPE = (8, 4, 6, 5, 32003, 16, 16)   # r, k, dim_in, dim_out, p, n, m


def _problem():
    shape = oracle.KoszulShape(*SHAPE)
    maps, diag, X, Y = oracle.seeded_problem(shape, 41)
    x, y = (torch.from_numpy(a.view(np.int32)).cuda() for a in (X, Y))
    z = torch.empty((shape.n_tgt, shape.nb), dtype=torch.int32, device="cuda")
    return maps, diag, x, y, z, oracle.forward(shape, maps, Y)


def _holding_engine(monkeypatch, maps, diag):
    monkeypatch.setenv("BW_TEST_WAIT_LIMIT", "20000")
    monkeypatch.setenv("BW_TEST_HOLD_FIRST_STAGE", "1")
    engine = KoszulEngine(*SHAPE, maps=maps, diag=diag, form="int8")
    monkeypatch.delenv("BW_TEST_WAIT_LIMIT")
    monkeypatch.delenv("BW_TEST_HOLD_FIRST_STAGE")
    return engine


def test_word_of_a_context_closed_in_flight_is_not_reused_before_its_kernels_end(monkeypatch):
    """A context is closed while its steps wait behind a long kernel; another is
    created meanwhile, by a second thread.  The steps then give up."""
    maps, diag, x, y, z, want = _problem()
    stream = torch.cuda.Stream()
    with KoszulEngine(*SHAPE, maps=maps, diag=diag, form="int8") as warm, \
            torch.cuda.stream(stream):   # loads every kernel, and keeps the page of words
        warm.forward(y, z, stream=stream)
        seq = torch.empty((4, SHAPE[6], SHAPE[5]), dtype=torch.int32, device="cuda")
        warm.seq_start(x, y, seq, stream=stream)
        warm.seq_step(1, stream=stream)
        warm.seq_finish(stream=stream)
        torch.cuda.synchronize()
        closing = _holding_engine(monkeypatch, maps, diag)
        closing.seq_start(x, y, seq, stream=stream)
        torch.cuda._sleep(1_000_000_000)   # about half a second
        closing.seq_step(1, stream=stream)
        thread = threading.Thread(target=closing.close)
        thread.start()
        time.sleep(0.05)
        with KoszulEngine(*SHAPE, maps=maps, diag=diag, form="int8") as fresh:
            thread.join()
            torch.cuda.synchronize()
            fresh.forward(y, z, stream=stream)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(z.cpu().numpy().view(np.uint32), want)


def test_give_up_is_reported_by_its_own_context_alone(monkeypatch):
    """More contexts than a page has words, one of which gives up."""
    maps, diag, x, y, z, want = _problem()
    engines = [KoszulEngine(*SHAPE, maps=maps, diag=diag, form="int8") for _ in range(66)]
    held = _holding_engine(monkeypatch, maps, diag)
    try:
        for _ in range(2):
            with pytest.raises(EngineError) as err:
                held.forward(y, z)
            assert err.value.status == 2
        for engine in engines:
            z.zero_()
            engine.forward(y, z)
            torch.cuda.synchronize()
            np.testing.assert_array_equal(z.cpu().numpy().view(np.uint32), want)
    finally:
        for engine in [held, *engines]:
            engine.close()
