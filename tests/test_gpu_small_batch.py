"""Small batches (first and finishing kernel alone) against the wavefront's rounds.

A run of few rays is traced without rounds and without the sort by element; a run of more than
65,536 takes both.  Every ray has its own random stream, so the first rays of the large run must
leave the very records of the small one, on every surface, aperture and stage flag of the zoo (the
small run's last rays are left out: the reference's end-of-run rules drop records there).
"""
import numpy as np
import pytest

from helpers import run_scene
from soltrace_b200 import scenes
from test_gpu_parity import ZOO_NAMES, _fp64

pytestmark = pytest.mark.gpu

LARGE = 66_000


def _scene(name, zoo_scenes):
    if name in zoo_scenes:
        return zoo_scenes[name]
    return {"dish": scenes.dish_scene(1000), "trough": scenes.trough_scene(1000),
            "field": scenes.field_scene(300, 1000, elevation_deg=20.0),
            "beam_down": scenes.beam_down_scene(300, 1000)}[name]


@pytest.mark.parametrize("name", [n for n in ZOO_NAMES if n != "fe_surface"] + ["dish", "trough", "field", "beam_down"])
def test_small_batch_equals_rounds(product, zoo_scenes, name):
    sc = _scene(name, zoo_scenes)
    rows = {}
    for hits in (1500, LARGE):
        sc.raycount, sc.raymax = hits, 2_000_000_000 - 1
        n, rec, _, msg = run_scene(product, sc, 23, _fp64)[:4]
        assert n > 0, msg
        keep = rec["raynum"] < 1490
        order = np.lexsort((np.arange(keep.sum()), rec["stage"][keep], rec["raynum"][keep]))
        rows[hits] = {k: v[keep][order] for k, v in rec.items()}
    for k in rows[LARGE]:
        assert np.array_equal(rows[1500][k], rows[LARGE][k]), k
