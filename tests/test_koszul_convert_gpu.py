"""The engine's conversions between a caller's residues and its own layouts:
buffers that are not 16-byte aligned, residues that are not reduced, counts
that are not a multiple of four, and every block width.  Bit-exact."""
import numpy as np
import pytest

import oracle
from prym_green_ancillary_b200 import KoszulEngine

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _shifted(a, shift):
    """The array in a CUDA buffer that starts `shift` residues into an allocation."""
    buf = torch.empty(a.size + shift, dtype=torch.int32, device="cuda")
    view = buf[shift:].view(a.shape)
    view.copy_(torch.from_numpy(a.view(np.int32)))
    return view


@pytest.mark.parametrize("form", ["plain", "int8"])
@pytest.mark.parametrize("nb,m", [(4, 32), (8, 4), (16, 8), (32, 16)])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_unaligned_and_unreduced_buffers(form, nb, m, shift):
    shape = oracle.KoszulShape(7, 3, 5, 3, 32749, nb, m)
    maps, diag, X, Y = oracle.seeded_problem(shape, 23)
    want, yf_want = oracle.sequence(shape, maps, diag, X, Y, 5)
    # the same residues with multiples of p added, up to the top of 32 bits
    top = (2 ** 32 - 1 - shape.p) // shape.p
    rng = np.random.default_rng(1)
    lift = lambda a: (a + rng.integers(0, top + 1, a.shape, dtype=np.uint64) * shape.p).astype(np.uint32)  # noqa: E731
    x, y = _shifted(lift(X), shift), _shifted(lift(Y), shift)
    seq = _shifted(np.zeros((5, m, nb), dtype=np.uint32), shift)
    last = _shifted(np.zeros((shape.n_src, nb), dtype=np.uint32), shift)
    d = _shifted(lift(diag), shift)
    assert shape.n_src % 4 and d.data_ptr() % 16 == 4 * shift
    with KoszulEngine(shape.r, shape.k, shape.ci, shape.co, shape.p, nb, m, maps=maps, diag=d, form=form) as eng:
        eng.seq_start(x, y, seq)
        eng.seq_step(4)
        eng.seq_finish(last)
        torch.cuda.synchronize()
    np.testing.assert_array_equal(seq.cpu().numpy().view(np.uint32), want)
    np.testing.assert_array_equal(last.cpu().numpy().view(np.uint32), yf_want)
