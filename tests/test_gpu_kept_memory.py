"""Host memory that solves hand on is given back with the last assembler.

A solve follows its problems through a block of pinned memory, which the next
batch takes over. While an assembler is alive at most eight blocks are kept,
afterwards one; threads that solve at the same time take one each. Counted in a
process of its own, where no other test's objects are alive.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = """
import threading
import torch
from gpu_fem_b200 import _lib as L, mesh as M
from gpu_fem_b200.assembler import ElementAssembler, createBsrMat, direct_solve
kept = L.lib().gf_test_kept_blocks
m = M.plate(4, 3, 1.0, 0.75, lambda x, y: 0.006 + 0 * x, "all_edges", lambda q: 1e3 + 0 * q[:, 0])
b = torch.tensor(m.loads, device="cuda")
def make():
    A = ElementAssembler.from_mesh(m)
    K = createBsrMat(A)
    A.add_jacobian(None, K, fuse_bcs=True)
    return A, K
for again in range(2):
    objects = [make() for _ in range(10)]
    torch.cuda.synchronize()
    x = [torch.zeros_like(b) for _ in objects]
    assert kept() == again, kept()
    direct_solve(*objects[0], b, x[0])
    assert kept() == 1, kept()
    threads = [threading.Thread(target=direct_solve, args=(A, K, b, x[k].zero_()))
               for k, (A, K) in enumerate(objects)]
    torch.cuda.synchronize()
    for t in threads: t.start()
    for t in threads: t.join()
    del threads
    torch.cuda.synchronize()
    assert 1 <= kept() <= 8, kept()
    assert all(torch.equal(x[0], y) for y in x) and float(x[0].abs().max()) > 0
    K = objects[3][1]
    objects.clear()  # K keeps its assembler alive
    assert kept() >= 1, kept()
    del K
    assert kept() == 1, kept()
print("ok")
"""


def test_blocks_live_as_long_as_an_assembler():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
