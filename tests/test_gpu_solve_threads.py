"""Solves whose kernels need different amounts of shared memory, first used by
several threads at once in a fresh process, each on its own stream."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import threading
import numpy as np, torch
import remifa_b200 as rb
from remifa_b200.batch import BatchPlan, MatrixBatch, RhsBatch

n = 300
lu = rb.colmajor(2.0 * torch.eye(n, device="cuda"))
batches = []
for top in (40, 170, 300, 512):
    sizes = np.array([top, top // 2], np.int32)
    m = MatrixBatch(sizes)
    for i in range(2):
        m.matrix(i).copy_(2.0 * torch.eye(int(sizes[i]), device="cuda"))
    batches.append((sizes, m, BatchPlan(sizes, outer=rb.FP32)))
torch.cuda.synchronize()
gate, bad = threading.Barrier(8), []

def work(k):
    try:
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            gate.wait()
            for rep in range(20):
                if k < 4:
                    x = torch.ones((k + 1, n), dtype=torch.float64, device="cuda").t()
                    rb.lu_solve(lu, x)
                    got = x
                else:
                    sizes, m, plan = batches[k - 4]
                    x = RhsBatch(sizes, 1)
                    x.data.fill_(1.0)
                    plan.solve(m, x)
                    got = x.data
                s.synchronize()
                if not bool((got == 0.5).all()):
                    raise RuntimeError("wrong solution")
    except Exception as e:
        bad.append((k, repr(e)))

threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
[t.start() for t in threads]
[t.join() for t in threads]
assert not bad, bad
print("ok")
"""


def test_first_use_from_several_threads(built):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, capture_output=True, text=True,
                       timeout=240)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr
