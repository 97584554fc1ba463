"""Sun rays queued for a scene that replaces another in the same context.

A run plans its batches from the last run's hits per sun ray.  That rate says nothing about another
scene: after elements of 5 cm, of which one sun ray in a few hundred thousand finds one, elements of
30 m must not be given the former's billions of sun rays, and the other way round both runs leave what
a fresh context leaves.
"""
import numpy as np
import pytest

from soltrace_b200.scenes import Element
from test_gpu_flat_probe import _scene

pytestmark = pytest.mark.gpu

UP = (0.0, 0.0, 1.0)
HITS = 20_000


def _elements(surface, size):
    xy = [(x, y) for x in (-40.0, 40.0) for y in (-40.0, 40.0)]
    params = (0.001, 0.001) if surface == "p" else ()
    return [Element(origin=(x, y, 0.0), aim=(x, y, 100.0), aperture="r", aperture_params=(size, size), surface=surface,
                    surface_params=params, interaction=2, optic="m") for x, y in xy]


def _trace(product, ctx, surface, size, hits, seed):
    from soltrace_b200 import scenes
    product.st_clear_stages(ctx)
    product.st_clear_optics(ctx)
    scenes.push(product, ctx, _scene(_elements(surface, size), UP, hits))
    product.st_b200_set_records(ctx, 0)
    assert product.run(ctx, seed) >= 0, product.messages(ctx)
    return product.stats(ctx), product.element_counts(ctx, 1, 4)


@pytest.mark.parametrize("surface", ["f", "p"])
def test_another_scenes_rate_does_not_plan_the_run(product, surface):
    fresh = {}
    for size, hits in ((0.05, 50), (30.0, HITS)):
        ctx = product.st_create_context()
        try:
            fresh[size] = _trace(product, ctx, surface, size, hits, 4)
        finally:
            product.st_free_context(ctx)
    ctx = product.st_create_context()
    try:
        for size, hits in ((0.05, 50), (30.0, HITS), (0.05, 50), (30.0, HITS)):
            st, counts = _trace(product, ctx, surface, size, hits, 4)
            assert st["sun_rays"] == fresh[size][0]["sun_rays"]
            assert all(np.array_equal(a, b) for a, b in zip(counts, fresh[size][1]))
            if size == 30.0:  # half the box's rays hit; a batch takes 2^26
                assert st["batches"] <= 2
    finally:
        product.st_free_context(ctx)
