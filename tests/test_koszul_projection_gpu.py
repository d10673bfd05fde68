"""The INT8 form's projection (moments of a sequence) at the edges of its stages,
and steps whose d runs beside the projection before it, against the CPU oracle.
Bit-exact.

Shapes: 32-column blocks (boxes of a tensor map) with a ragged last stage, more
blocks than one box can hold (256), one-row runs, the longest runs and a padded
K; 16-column blocks (plain bulk copies); 4 to 32 projection columns.  20 steps:
16 in a graph, four launched one by one.
"""
import numpy as np
import pytest

import oracle
from prym_green_ancillary_b200 import KoszulEngine

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [
    # r, k, ci, co, p, nb, m
    (12, 6, 1, 2, 32749, 32, 32),      # 924 one-row blocks: boxes of 256
    (9, 4, 5, 3, 32003, 32, 16),       # 126 blocks of 5 rows: K padded
    (7, 3, 64, 3, 32749, 32, 32),      # the longest runs, widest X
    (8, 4, 32, 40, 32749, 32, 4),      # 70 blocks, 8 or 16 a stage: ragged
    (11, 5, 7, 6, 101, 16, 32),
    (10, 4, 16, 24, 32003, 8, 8),
    (5, 5, 3, 2, 32003, 32, 32),       # one source block
]


@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("steps", [(20,), (3, 17)])
def test_moments_match_oracle(dims, steps):
    shape = oracle.KoszulShape(*dims)
    maps, diag, X, Y = oracle.seeded_problem(shape, 19)
    X[:, 0] = (shape.p - 1) // 2       # largest magnitudes
    Y[:, -1] = (shape.p + 1) // 2
    total = sum(steps)
    with KoszulEngine(*dims, maps=maps, diag=diag, form="int8") as eng:
        x, y = (torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda() for a in (X, Y))
        seq = torch.empty((total + 1, shape.m, shape.nb), dtype=torch.int32, device="cuda")
        eng.seq_start(x, y, seq)
        for n in steps:
            eng.seq_step(n)
        eng.seq_finish()
        torch.cuda.synchronize()
    want, _ = oracle.sequence(shape, maps, diag, X, Y, total + 1)
    np.testing.assert_array_equal(seq.cpu().numpy().view(np.uint32), want)
