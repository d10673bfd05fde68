"""The INT8 form's union kernel (K over the generators a tile has, both limbs in
K), forced, against the CPU oracle.  Bit-exact.

Shapes at its edges: generators of an odd and an even number of 16-row chunks
(2 * dim rounded up to 16), one-row dims, dims at 8, 16 and 64, tiles of 8 and 4
blocks with a ragged last tile, more than 500 rows a block (the epilogue's
wider reduction), one tile, and the largest prime.
"""
import numpy as np
import pytest

import oracle
from prym_green_ancillary_b200 import EngineError, KoszulEngine

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [
    # r, k, ci, co, p, nb, m
    (9, 4, 20, 28, 32003, 16, 16),
    (8, 4, 32, 40, 32749, 32, 32),
    (10, 5, 1, 1, 3, 8, 8),
    (7, 3, 8, 7, 32749, 16, 4),
    (9, 5, 9, 16, 10007, 32, 16),
    (6, 3, 64, 3, 32749, 16, 16),
    (6, 2, 3, 64, 32749, 32, 8),
    (11, 2, 17, 33, 101, 4, 4),
    (13, 1, 41, 5, 32003, 16, 32),
    (5, 5, 2, 3, 32003, 16, 16),
    (15, 13, 47, 9, 32749, 16, 16),    # d^T: 13 * 9 rows; d: 3 * 47
    (14, 2, 44, 48, 32749, 16, 16),    # d: 13 * 44 = 572 rows a block
]


@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("tune", ["0", "1"])
def test_union_matches_oracle(dims, tune, monkeypatch):
    monkeypatch.setenv("BW_I8_PRODUCER", "union")
    monkeypatch.setenv("BW_I8_TUNE", tune)      # 0: the first plan that fits, two MMA warps where they can be
    shape = oracle.KoszulShape(*dims)
    maps, diag, X, Y = oracle.seeded_problem(shape, 7)
    # largest magnitudes too: residues whose balanced value is +-(p - 1) / 2 in every place of two columns
    Y[:, 0] = (shape.p - 1) // 2
    Y[:, 1] = (shape.p + 1) // 2
    maps[: shape.co * shape.ci] = (shape.p - 1) // 2
    rng = np.random.default_rng(3)
    Z = rng.integers(0, shape.p, (shape.n_tgt, shape.nb), dtype=np.uint32)
    Z[:, 0] = (shape.p - 1) // 2
    dev = torch.device("cuda", 0)
    y, z = (torch.from_numpy(a.view(np.int32)).to(dev) for a in (Y, Z))
    out_z = torch.empty((shape.n_tgt, shape.nb), dtype=torch.int32, device=dev)
    out_w = torch.empty((shape.n_src, shape.nb), dtype=torch.int32, device=dev)
    with KoszulEngine(*dims, maps=maps, diag=diag, form="int8") as eng:
        assert eng.plan.count("union stage=") >= 2, eng.plan
        eng.forward(y, out_z)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out_z.cpu().numpy().view(np.uint32), oracle.forward(shape, maps, Y))
        for scale in (False, True):
            eng.transpose(z, out_w, scale_by_diag=scale)
            torch.cuda.synchronize()
            want = oracle.transpose(shape, maps, Z).astype(np.int64)
            if scale:
                want = want * diag[:, None] % shape.p
            np.testing.assert_array_equal(out_w.cpu().numpy().view(np.uint32), want.astype(np.uint32))
        seq, yf = eng.sequence_host(X, Y, 6)
    want, yf_want = oracle.sequence(shape, maps, diag, X, Y, 6)
    np.testing.assert_array_equal(seq, want)
    np.testing.assert_array_equal(yf, yf_want)


def test_union_wait_that_runs_out_returns_status_2(monkeypatch):
    dims = (8, 4, 6, 5, 32003, 16, 16)
    shape = oracle.KoszulShape(*dims)
    maps, diag, X, Y = oracle.seeded_problem(shape, 41)
    y = torch.from_numpy(Y.view(np.int32)).cuda()
    z = torch.empty((shape.n_tgt, shape.nb), dtype=torch.int32, device="cuda")
    monkeypatch.setenv("BW_I8_PRODUCER", "union")
    monkeypatch.setenv("BW_TEST_WAIT_LIMIT", "100000")
    monkeypatch.setenv("BW_TEST_HOLD_FIRST_STAGE", "1")
    with KoszulEngine(*dims, maps=maps, diag=diag, form="int8") as eng:
        with pytest.raises(EngineError) as err:
            eng.forward(y, z)
        assert err.value.status == 2 and "gave up waiting (ERR_WAIT_" in str(err.value)
    monkeypatch.delenv("BW_TEST_WAIT_LIMIT")
    monkeypatch.delenv("BW_TEST_HOLD_FIRST_STAGE")
    with KoszulEngine(*dims, maps=maps, diag=diag, form="int8") as eng:
        eng.forward(y, z)
        torch.cuda.synchronize()
    np.testing.assert_array_equal(z.cpu().numpy().view(np.uint32), oracle.forward(shape, maps, Y))
