"""BW_PLAIN_TILE heights that pad a tile's coefficients beyond shared memory: the
context takes a height that fits, as it does without the setting."""
import numpy as np
import pytest

import oracle
from prym_green_ancillary_b200 import KoszulEngine

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,rows,forced", [
    ((13, 9, 36, 79, 7, 16, 8), 5, False),        # d's tiles of five rows, padded to eight: 234 KB
    ((12, 6, 79, 36, 32749, 8, 16), 5, False),    # d^T's
    ((13, 9, 36, 79, 7, 16, 8), 8, True),
    ((10, 4, 20, 28, 32003, 16, 16), 5, True),
])
def test_forced_heights(dims, rows, forced, monkeypatch):
    monkeypatch.setenv("BW_PLAIN_TILE", str(rows))
    shape = oracle.KoszulShape(*dims)
    maps, diag, X, Y = oracle.seeded_problem(shape, 3)
    with KoszulEngine(*dims, maps=maps, diag=diag, form="plain") as eng:
        assert eng.plan.startswith(f"plain: {rows} output rows a thread (forced)") == forced, eng.plan
        seq, last = eng.sequence_host(X, Y, 4)
    want, yf = oracle.sequence(shape, maps, diag, X, Y, 4)
    np.testing.assert_array_equal(seq, want)
    np.testing.assert_array_equal(last, yf)
