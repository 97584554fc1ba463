"""Batched runs that cannot be set up name the same reason whichever way their grids are built.

First stages of flat rectangles have their grids built on the device, others on the host.
"""
import numpy as np
import pytest

from test_gpu_flat_probe import _scene
from test_gpu_hit_rate import _elements

pytestmark = pytest.mark.gpu

SUN = (0.0, 0.0, 1e4)
ORIGIN = (0.0, 0.0, 0.0)
# suns, tracking target, elements enabled, the message (after the call's name)
CASES = {
    "no sun": ([SUN, ORIGIN], None, True, "sun position 1: error calculating sun position in primary stage, dtot = 0.0\n"),
    "no sun, tracking": ([SUN, ORIGIN], (0.0, 0.0, 50.0), True, "sun position 1: sun position at the origin"),
    "target opposite the sun": ([(1e4, 0.0, 0.0)], (-1e9, 40.0, 0.0), True,
                                "sun position 0: a tracking element cannot bisect the sun and target directions"),
    # the context's own set-up comes before any position's
    "none enabled": ([ORIGIN], (0.0, 0.0, 50.0), False,
                     "error calculating sun position in primary stage because no elements were enabled"),
}


@pytest.mark.parametrize("surface", ["f", "p"])
@pytest.mark.parametrize("name", list(CASES))
def test_reason_of_a_refused_batch(product, surface, name):
    from soltrace_b200 import scenes
    suns, target, enabled, message = CASES[name]
    els = _elements(surface, 4.0)
    for e in els:
        e.enabled = enabled
        if name.startswith("target"):  # exactly opposite: the element lies on the line
            e.origin, e.aim = (e.origin[0], 40.0, 0.0), (e.origin[0], 40.0, 100.0)
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, _scene(els, (0.0, 0.0, 1.0), 100))
        product.st_b200_set_records(ctx, 0)
        assert product.run_batch(ctx, 1, suns, [100] * len(suns), target) == -1
        assert product.messages(ctx)[-1] == ("st_b200_sim_run_batch: " if enabled else "") + message
    finally:
        product.st_free_context(ctx)
