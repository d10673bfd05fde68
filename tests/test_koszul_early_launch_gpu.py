"""INT8 steps behind a kernel that lets its dependents begin long before it ends:
the steps' kernels are then resident while it runs, and the limit of their
bounded waits must not count its time.
"""
import numpy as np
import pytest

import oracle
from prym_green_ancillary_b200 import KoszulEngine

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SOURCE = r"""
extern "C" __global__ void early() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long start = clock64();
    while (clock64() - start < 2000000000ll) {}   // about a second
}
"""


@pytest.mark.parametrize("dims", [(8, 4, 6, 5, 32003, 16, 16), (9, 4, 20, 28, 32749, 32, 32)])
def test_waits_do_not_count_the_kernel_before(dims, monkeypatch):
    monkeypatch.setenv("BW_I8_PRODUCER", "union")
    monkeypatch.setenv("BW_TEST_WAIT_LIMIT", "20000")
    early = torch.cuda._compile_kernel(SOURCE, "early")
    shape = oracle.KoszulShape(*dims)
    maps, diag, X, Y = oracle.seeded_problem(shape, 41)
    x, y = (torch.from_numpy(a.view(np.int32)).cuda() for a in (X, Y))
    seq = torch.empty((4, shape.m, shape.nb), dtype=torch.int32, device="cuda")
    out = torch.empty_like(y)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with KoszulEngine(*dims, maps=maps, diag=diag, form="int8") as eng:
        eng.seq_start(x, y, seq, stream=stream)
        for _ in range(3):   # a step a call: its first kernel follows the early one directly
            early((1, 1, 1), (32, 1, 1), stream=stream)
            eng.seq_step(1, stream=stream)
        eng.seq_finish(out, stream=stream)
        torch.cuda.synchronize()
    want, last = oracle.sequence(shape, maps, diag, X, Y, 4)
    np.testing.assert_array_equal(seq.cpu().numpy().view(np.uint32), want)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), last)
