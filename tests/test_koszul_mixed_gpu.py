"""The INT8 form with the union kernel in one direction and a dense kernel in the
other, as the set-up's timings may choose where the maps fill shared memory:
dense kernels read the limbs the union kernel stores (any representative that two
limbs hold, not the balanced one) and the other way round, and a union d that
does not wait for the projection before it precedes a dense d^T.  Against the CPU
oracle, bit-exact, with enough steps for the captured and the single ones.
"""
import numpy as np
import pytest

import oracle
from prym_green_ancillary_b200 import KoszulBatch, KoszulEngine

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

PAIRS = ["union,cpasync", "union,hybrid", "cpasync,union", "hybrid,union"]
NAMES = {"union": "union", "cpasync": "cp.async", "hybrid": "hybrid"}
SHAPES = [
    # r, k, ci, co, p, nb, m
    (8, 4, 20, 28, 32749, 16, 16),
    (7, 3, 33, 41, 32749, 32, 32),
    (10, 8, 24, 3, 32003, 8, 4),
    (6, 2, 3, 48, 101, 4, 8),
]
STEPS = 21   # a graph of 16 and five single ones


def _problem(dims):
    shape = oracle.KoszulShape(*dims)
    maps, diag, X, Y = oracle.seeded_problem(shape, 7)
    # the largest magnitudes too: residues and coefficients whose balanced value is +-(p - 1) / 2
    Y[:, 0] = (shape.p - 1) // 2
    Y[:, 1] = (shape.p + 1) // 2
    maps[: shape.co * shape.ci] = (shape.p - 1) // 2
    return shape, maps, diag, X, Y


@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("pair", PAIRS)
def test_mixed_directions_match_oracle(dims, pair, monkeypatch):
    monkeypatch.setenv("BW_I8_PRODUCER", pair)
    shape, maps, diag, X, Y = _problem(dims)
    with KoszulEngine(*dims, maps=maps, diag=diag, form="int8") as eng:
        plans = [part.split(": ", 1)[1] for part in eng.plan.replace("d^T: ", "\nd^T: ").splitlines()]
        for plan, name in zip(plans, pair.split(",")):
            assert plan.startswith(NAMES[name]), eng.plan
        seq, last = eng.sequence_host(X, Y, STEPS + 1)
    want, yf = oracle.sequence(shape, maps, diag, X, Y, STEPS + 1)
    np.testing.assert_array_equal(seq, want)
    np.testing.assert_array_equal(last, yf)


@pytest.mark.parametrize("pair", PAIRS)
def test_mixed_directions_in_a_batch(pair, monkeypatch):
    monkeypatch.setenv("BW_I8_PRODUCER", pair)
    problems = [_problem(dims) for dims in SHAPES[:2]]
    specs = [dict(r=s.r, k=s.k, dim_in=s.ci, dim_out=s.co, prime=s.p, block_width=s.nb, proj_width=s.m, maps=maps,
                  diag=diag, form="int8") for s, maps, diag, _, _ in problems]
    xs, ys = ([torch.from_numpy(p[i].view(np.int32)).cuda() for p in problems] for i in (3, 4))
    seqs = [torch.empty((STEPS + 1, s.m, s.nb), dtype=torch.int32, device="cuda") for s, *_ in problems]
    outs = [torch.empty_like(y) for y in ys]
    with KoszulBatch(specs) as batch:
        batch.seq_start(xs, ys, seqs)
        batch.seq_step(STEPS)
        batch.seq_finish(outs)
        torch.cuda.synchronize()
    for (shape, maps, diag, X, Y), seq, out in zip(problems, seqs, outs):
        want, yf = oracle.sequence(shape, maps, diag, X, Y, STEPS + 1)
        np.testing.assert_array_equal(seq.cpu().numpy().view(np.uint32), want)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), yf)
