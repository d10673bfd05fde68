"""The union kernel's tile order (stars of four blocks, the rest four by four)
against the CPU oracle.  Bit-exact.

Sectors with more tiles than the GPU has SMs, so that the order is built: tiles
of four and eight blocks, block counts that are no multiple of either, few and
many elements in a block, r with and without a partial quad of elements, and one
direction in lexicographic order beside the other's stars.
"""
import numpy as np
import pytest

import oracle
from prym_green_ancillary_b200 import KoszulEngine

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [
    # r, k, ci, co, p, nb, m
    (14, 7, 3, 5, 32749, 32, 32),
    (15, 7, 2, 3, 32003, 16, 16),
    (13, 6, 5, 2, 101, 32, 8),
    (20, 3, 2, 1, 32749, 32, 4),       # d: 48 tiles, lexicographic
    (17, 14, 1, 2, 32003, 32, 16),
    (16, 8, 3, 3, 32749, 8, 8),
    (24, 2, 1, 4, 32003, 32, 4),       # d: six tiles; d^T: 69
    (12, 6, 9, 7, 3, 32, 32),
]


@pytest.mark.parametrize("dims", SHAPES)
def test_star_order_matches_oracle(dims, monkeypatch):
    monkeypatch.setenv("BW_I8_PRODUCER", "union")
    shape = oracle.KoszulShape(*dims)
    maps, diag, X, Y = oracle.seeded_problem(shape, 23)
    rng = np.random.default_rng(5)
    Z = rng.integers(0, shape.p, (shape.n_tgt, shape.nb), dtype=np.uint32)
    y, z = (torch.from_numpy(a.view(np.int32)).cuda() for a in (Y, Z))
    out_z = torch.empty((shape.n_tgt, shape.nb), dtype=torch.int32, device="cuda")
    out_w = torch.empty((shape.n_src, shape.nb), dtype=torch.int32, device="cuda")
    with KoszulEngine(*dims, maps=maps, diag=diag, form="int8") as eng:
        eng.forward(y, out_z)
        eng.transpose(z, out_w, scale_by_diag=True)
        torch.cuda.synchronize()
        seq, yf = eng.sequence_host(X, Y, 5)
    np.testing.assert_array_equal(out_z.cpu().numpy().view(np.uint32), oracle.forward(shape, maps, Y))
    want_w = oracle.transpose(shape, maps, Z).astype(np.int64) * diag[:, None] % shape.p
    np.testing.assert_array_equal(out_w.cpu().numpy().view(np.uint32), want_w.astype(np.uint32))
    want, yf_want = oracle.sequence(shape, maps, diag, X, Y, 5)
    np.testing.assert_array_equal(seq, want)
    np.testing.assert_array_equal(yf, yf_want)
