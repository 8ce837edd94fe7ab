"""FP64 handles whose pair-force slots cannot be allocated evaluate each pair twice: nothing is refused, and the results
are those with slots, bit for bit.  The allocations fail on the host, in a child process whose cudaMalloc refuses them
(tests/programs/malloc_refuse.cpp)."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

CHILD = """
import ctypes as C
import sys

import numpy as np

sys.path[:0] = [%r, %r]
from helpers import make_gpu
from parm_gb300 import workloads as W

shim = C.CDLL(None)
shim.refuse.argtypes = [C.c_size_t]
w = W.lj_lattice(shape=(26, 26, 26))


def run(sizes):
    n0 = shim.refuse_none()
    for b in sizes:
        shim.refuse(b)
    g = make_gpu(w)
    caps = [g.capacity()]
    g.nlist_update(False)
    g.verlet(0.002, 5)
    g.set_capacity(caps[0] + 32)
    caps.append(g.capacity())
    g.verlet(0.002, 5)
    return g.get_atoms(), caps, shim.refuse_none() - n0


ref, caps, refused = run([])
assert refused == 0
slots = [w.n * m // 2 * 32 + 32 for m in caps]      # 32 bytes for half of the list entries, and one more
indices = [w.n * m * 4 for m in caps]
for sizes in (slots, indices, slots[:1], indices[1:]):
    got, _, refused = run(sizes)
    assert refused == len(sizes)
    for k in ("x", "v", "f"):
        assert np.array_equal(got[k], ref[k])
print("ok")
"""


def test_slots_that_cannot_be_allocated(tmp_path):
    lib = tmp_path / "malloc_refuse.so"
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", str(ROOT / "tests/programs/malloc_refuse.cpp"),
                        "-o", str(lib), "-ldl"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([sys.executable, "-c", CHILD % (str(ROOT), str(ROOT / "tests"))], capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, LD_PRELOAD=str(lib)))
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
