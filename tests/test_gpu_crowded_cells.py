"""Batched grids whose cells hold many elements.

One distant element stretches the sun box, and the batch's cell budget then puts the whole field into
a few cells.  The device lists a crowded cell's entries in element order through a bitmap of 32,768
elements at a time; cells of up to 32 entries are sorted by one thread.  Positions must number the rays
of single runs (whose grids the host builds), and the grids must not cost seconds.
"""
import numpy as np
import pytest

from test_gpu_flat_probe import _elem, _scene

pytestmark = pytest.mark.gpu

UP = np.array([0.0, 0.0, 1.0])


def _field(n, far, spread=400.0):
    """n rectangles, overlapping where they are many, within `spread` of the origin and one far away."""
    rng = np.random.default_rng(n)
    xy = rng.uniform(-spread, spread, (n - 1, 2))
    return [_elem((x, y, rng.uniform(0, 30)), UP + rng.normal(0, 0.1, 3), (4.0, 4.0)) for x, y in xy] + \
        [_elem((far, far, 0.0), UP, (4.0, 4.0))]


@pytest.mark.parametrize("n,far,spread", [(33, 4.0e4, 20.0), (34, 4.0e4, 20.0), (500, 5.0e4, 60.0),
                                          (10_001, 2.0e5, 300.0), (33_000, 4.0e4, 400.0), (70_000, 4.0e4, 400.0)])
def test_crowded_cells_number_the_single_runs_rays(product, n, far, spread):
    from soltrace_b200 import scenes
    hits = 40
    els = _field(n, far, spread)
    sun = 1e4 * np.array([0.1, -0.05, 0.99])
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, _scene(els, sun / 1e4, hits))
        product.st_b200_set_precision(ctx, 1)
        product.st_b200_set_records(ctx, 0)
        assert product.run_batch(ctx, 5, [sun], [hits]) == 1, product.messages(ctx)
        rays, absorbed = product.batch_stats(ctx, 0)["sun_rays"], product.batch_absorbed(ctx, 0, 1, n)
        product.st_sun_xyz(ctx, *map(float, sun))
        assert product.run(ctx, 5) >= 0, product.messages(ctx)
        assert product.stats(ctx)["sun_rays"] == rays
        assert np.array_equal(product.element_counts(ctx, 1, n)[1], absorbed)
    finally:
        product.st_free_context(ctx)


def test_a_crowded_cell_costs_no_seconds(product):
    """10,000 elements in one or two cells: a thread's insertion sort of a cell took seconds, as
    long as the square of its entries says.  The least of four repeated runs, without first allocations
    and whatever else the host does."""
    from soltrace_b200 import scenes
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, _scene(_field(10_001, 2.0e5, 100.0), UP, 4))
        product.st_b200_set_records(ctx, 0)
        setup = []
        for _ in range(5):
            assert product.run_batch(ctx, 5, [1e4 * UP], [4]) == 1, product.messages(ctx)
            setup.append(product.batch_stats(ctx, -1)["setup_ms"])
        assert min(setup[1:]) < 300.0, setup
    finally:
        product.st_free_context(ctx)
