"""Contexts of one process traced from several host threads at once.

Every thread has a context of its own, as st_b200.h allows; each must get what the same run gives
alone.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# the first runs of a process, started together: what the library finds out on first use (resident
# blocks per kernel) must be ready for every thread
FIRST_RUNS = r"""
import sys, threading
sys.path.insert(0, sys.argv[1])
import numpy as np
from soltrace_b200 import scenes
from soltrace_b200.lib import load
api = load()
N = 8
gate = threading.Barrier(N)
got = [None] * N

def trace(k):
    ctx = api.st_create_context()
    scenes.push(api, ctx, scenes.trough_scene(70_000))
    api.st_b200_set_precision(ctx, 0)
    gate.wait()
    n = api.run(ctx, 3)
    got[k] = (n, api.records(ctx) if n > 0 else api.messages(ctx))
    api.st_free_context(ctx)

ts = [threading.Thread(target=trace, args=(k,)) for k in range(N)]
[t.start() for t in ts]
[t.join() for t in ts]
assert all(n == got[0][0] > 0 for n, _ in got), got
for _, r in got[1:]:
    assert all(np.array_equal(r[k], got[0][1][k]) for k in r)
print("ok")
"""


def test_first_runs_of_a_process_on_eight_threads():
    r = subprocess.run([sys.executable, "-c", FIRST_RUNS, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
