"""Staged host copies start threads for the CPUs that the process may run on:
none in a process bound to one CPU, whose results arrive all the same."""
import os
import subprocess
import sys

import pytest

from _common import HERE

REPO = os.path.dirname(HERE)

CODE = """
import os, sys, threading, time
os.sched_setaffinity(0, {min(os.sched_getaffinity(0))})
sys.path[:0] = [%r, %r]
import numpy as np
import gausslectronitegrate_b200 as gli
from _common import g10, sym_grid
rng, spec = np.random.default_rng(1), sym_grid(17)
real = gli.compute_sparse_erida_gausslet_integrals(g10(), spec, 1e-3).indices
idx = np.unique(np.concatenate([real, rng.integers(0, 17 ** 6, 3_000_000)]))
s = gli.SparseERIDA._make(g10(), spec, idx, rng.standard_normal(idx.size), 1e-3)
grid = [(-2, 5), (0, 2), (-1, 3)]
s.fill_matrix(grid)  # the driver's and the library's own threads
seen, stop = [], False
def watch():
    while not stop:
        seen.append(len(os.listdir('/proc/self/task')))
        time.sleep(2e-4)
w = threading.Thread(target=watch)
w.start()
time.sleep(0.05)
before = max(seen)
for _ in range(10):
    got = s.fill_matrix(grid)
stop = True
w.join()
pts = [(x, y, z) for x in range(-2, 3) for y in range(2) for z in range(-1, 2)]
assert np.array_equal(got, [[s.integral_value([p, q]) for q in pts] for p in pts])
print('threads', before, max(seen), len(seen))
assert max(seen) == before
"""


@pytest.mark.gpu
def test_one_cpu_starts_no_threads():
    r = subprocess.run([sys.executable, "-c", CODE % (REPO, HERE)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
