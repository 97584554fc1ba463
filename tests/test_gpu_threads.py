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


def test_fields_with_bitmaps_of_different_sizes_on_two_threads(product):
    """The flat-rectangle probe's shared memory follows the scene's occupancy bitmap, and its limit is
    shared by all threads of a device: two fields, one with a far larger bitmap, traced over and over
    side by side leave what they leave alone."""
    import threading

    import numpy as np

    from soltrace_b200 import scenes
    from test_gpu_flat_probe import _elem, _scene

    up = np.array([0.0, 0.0, 1.0])
    small = _scene([_elem((x, y, 0.0), up, (1.0, 1.0)) for x in (0, 2) for y in (0, 2)], up, 2000)
    large = scenes.field_scene(1500, 2000)
    runs = 150

    def trace(ctx, seed):
        assert product.run(ctx, seed) > 0, product.messages(ctx)
        r = product.records(ctx)
        return {k: np.array(v) for k, v in r.items()}

    def context(sc):
        ctx = product.st_create_context()
        scenes.push(product, ctx, sc)
        product.st_b200_set_precision(ctx, 1)
        return ctx

    ctxs = [context(small), context(large)]
    try:
        want = [trace(c, 7) for c in ctxs]
        gate, wrong = threading.Barrier(2), []

        def work(k):
            gate.wait()
            for _ in range(runs):
                try:
                    got = trace(ctxs[k], 7)
                except AssertionError as ex:
                    wrong.append((k, str(ex)))
                    return
                if not all(np.array_equal(got[q], want[k][q]) for q in got):
                    wrong.append((k, "records differ"))
                    return

        ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        [t.start() for t in ts]
        [t.join() for t in ts]
        assert not wrong, wrong
    finally:
        [product.st_free_context(c) for c in ctxs]
