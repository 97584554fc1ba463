"""Ranks of one run whose contexts come with record buffers of different sizes.

Rank 0's context has traced a larger run before, so it holds more record room than rank 1's; the
run over both must leave the single run's records (the buffers' bookkeeping itself is checked on the
host, test_record_room.py).
"""
import os
import subprocess
import sys

import numpy as np
import pytest

from test_gpu_ranks import ROOT, _free_port, _sorted

HITS, EARLIER, SEED = 200_000, 500_000, 31

pytestmark = pytest.mark.gpu


def _worker(rank, world, port, out):
    import datetime

    import torch.distributed as dist
    sys.path.insert(0, ROOT)
    from soltrace_b200 import parallel, scenes
    from soltrace_b200.lib import load

    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
    dist.init_process_group("gloo", rank=rank, world_size=world, timeout=datetime.timedelta(seconds=120))
    try:
        api = load()
        ctx = api.st_create_context()
        scenes.push(api, ctx, scenes.field_scene(300, EARLIER, dynamic_group=False))
        if rank == 0:
            assert api.run(ctx, 1) > 0
        api.st_sim_params(ctx, HITS, 2_000_000_000, 0)
        ex = parallel.RankExchange(device="cpu")
        assert ex.attach(api, ctx) == 1
        assert api.run(ctx, SEED) > 0, api.messages(ctx)
        assert not ex.errors
        np.savez(out, **api.records(ctx))
        api.st_free_context(ctx)
    finally:
        dist.destroy_process_group()


def test_ranks_with_different_record_buffers(product, tmp_path):
    from soltrace_b200 import scenes
    ctx = product.st_create_context()
    try:
        sc = scenes.field_scene(300, EARLIER, dynamic_group=False)
        sc.raycount, sc.raymax = HITS, 2_000_000_000
        scenes.push(product, ctx, sc)
        assert product.run(ctx, SEED) > 0
        one = _sorted(product.records(ctx))
    finally:
        product.st_free_context(ctx)
    port = _free_port()
    outs = [str(tmp_path / f"rank{r}.npz") for r in range(2)]
    procs = [subprocess.Popen([sys.executable, __file__, str(r), "2", str(port), outs[r]]) for r in range(2)]
    for p in procs:
        assert p.wait(timeout=300) == 0
    parts = [np.load(o) for o in outs]
    both = _sorted({k: np.concatenate([p[k] for p in parts]) for k in one})
    for k in one:
        assert np.array_equal(both[k], one[k]), k


if __name__ == "__main__":
    _worker(int(sys.argv[1]), int(sys.argv[2]), int(sys.argv[3]), sys.argv[4])
