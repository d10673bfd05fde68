"""Engine contexts across cudaDeviceReset: one that was left open takes nothing
with it that a later one needs.  In a child process, whose device contexts the
reset destroys.
"""
import os
import subprocess
import sys
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes
import os

import numpy as np

import oracle
from prym_green_ancillary_b200 import KoszulEngine

DIMS = (8, 4, 6, 5, 32003, 16, 16)
shape = oracle.KoszulShape(*DIMS)
maps, diag, X, Y = oracle.seeded_problem(shape, 41)
want, last = oracle.sequence(shape, maps, diag, X, Y, 5)


def check(engine):
    seq, final = engine.sequence_host(X, Y, 5)
    np.testing.assert_array_equal(seq, want)
    np.testing.assert_array_equal(final, last)


left_open = [KoszulEngine(*DIMS, maps=maps, diag=diag, form="int8") for _ in range(2)]
check(left_open[1])
assert ctypes.CDLL("libcudart.so.12").cudaDeviceReset() == 0
for _ in range(2):
    later = [KoszulEngine(*DIMS, maps=maps, diag=diag, form="int8") for _ in range(2)]
    for engine in later:
        check(engine)
    for engine in later:
        engine.close()
print("done", flush=True)
os._exit(0)     # the contexts left open are not closed: their device memory is gone
"""


def test_contexts_after_a_reset():
    libs = [str(Path(torch.__file__).resolve().parents[1] / "nvidia" / "cuda_runtime" / "lib"), "/usr/local/cuda/lib64"]
    env = dict(os.environ, LD_LIBRARY_PATH=":".join([*libs, os.environ.get("LD_LIBRARY_PATH", "")]))
    child = subprocess.run([sys.executable, "-c", CHILD], cwd=Path(__file__).resolve().parents[1], env=env,
                           capture_output=True, text=True, timeout=300)
    assert child.returncode == 0 and "done" in child.stdout, child.stderr
