"""The plain form's gathers at tile heights of 5, 6 and 7 rows (forced) and its
projection, against the CPU oracle.  Bit-exact.

Output rows at the tiles' edges, inner dims around the chunk of eight products
between two folds, every block width with every projection width, primes from
3 to the largest below 2^15, and residues of the largest balanced magnitude
throughout (the folded sums' bound).
"""
import numpy as np
import pytest

import oracle
from prym_green_ancillary_b200 import KoszulEngine

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [
    # r, k, ci, co, p, nb, m
    (7, 3, 1, 3, 3, 4, 4),
    (8, 4, 7, 9, 101, 8, 32),
    (8, 3, 8, 17, 32749, 16, 8),
    (9, 4, 25, 16, 32003, 32, 16),
    (7, 4, 33, 28, 32749, 4, 16),
    (6, 3, 65, 5, 32749, 8, 8),
    (5, 5, 4, 72, 10007, 16, 4),
    (9, 2, 20, 12, 32003, 32, 32),
]


@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("extreme", [False, True])
@pytest.mark.parametrize("rows", [5, 6, 7])
def test_tile_heights_match_oracle(dims, rows, extreme, monkeypatch):
    monkeypatch.setenv("BW_PLAIN_TILE", str(rows))
    shape = oracle.KoszulShape(*dims)
    maps, diag, X, Y = oracle.seeded_problem(shape, 5)
    if extreme:   # every product of the largest magnitude, all of one sign or alternating
        maps[:] = (shape.p - 1) // 2
        Y[:] = (shape.p - 1) // 2
        Y[::2, 1] = (shape.p + 1) // 2
        X[:] = (shape.p + 1) // 2
    dev = torch.device("cuda", 0)
    y = torch.from_numpy(Y.view(np.int32)).to(dev)
    out_z = torch.empty((shape.n_tgt, shape.nb), dtype=torch.int32, device=dev)
    out_s = torch.empty((shape.n_src, shape.nb), dtype=torch.int32, device=dev)
    with KoszulEngine(*dims, maps=maps, diag=diag, form="plain") as eng:
        assert eng.plan.startswith("plain: %d output rows" % rows), eng.plan
        eng.forward(y, out_z)
        eng.apply(y, out_s)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out_z.cpu().numpy().view(np.uint32), oracle.forward(shape, maps, Y))
        np.testing.assert_array_equal(out_s.cpu().numpy().view(np.uint32), oracle.apply(shape, maps, diag, Y))
        seq, yf = eng.sequence_host(X, Y, 5)
    want, yf_want = oracle.sequence(shape, maps, diag, X, Y, 5)
    np.testing.assert_array_equal(seq, want)
    np.testing.assert_array_equal(yf, yf_want)
