"""Single runs and batches in turn on one context.

A context keeps the tables of its last scene on the device; a batch writes its own over them.  Whatever the
order of calls, each leaves what it leaves on a fresh context.
"""
import numpy as np
import pytest

from soltrace_b200 import scenes

pytestmark = pytest.mark.gpu

GM = scenes.GROUND_MAP
SUNS, HITS = scenes.annual_suns(3, seed=11)[0], [9000, 70_000, 20_000]
OTHER = (3000.0, -2000.0, 9000.0)


def _context(product, prec):
    ctx = product.st_create_context()
    scenes.push(product, ctx, scenes.beam_down_scene(400, 30_000))
    product.st_b200_set_precision(ctx, prec)
    product.st_b200_add_flux_map(ctx, *GM)
    return ctx


def _batch(product, ctx):
    assert product.run_batch(ctx, 5, SUNS, HITS, scenes.beam_down_target()) == 1, product.messages(ctx)
    return [product.batch_flux(ctx, 0, k, GM[3], GM[4]) for k in range(3)]


def _single(product, ctx):
    assert product.run(ctx, 5) > 0, product.messages(ctx)
    return [product.flux(ctx, 0, GM[3], GM[4]), *product.records(ctx).values()]


def _moved(product, ctx):
    x, y, z = 0.0, 0.0, 1e4
    product.st_sun_xyz(ctx, *OTHER)
    got = _single(product, ctx)
    product.st_sun_xyz(ctx, x, y, z)
    return got


def _refused(product, ctx):  # a batch that stops at the ray limit after its first positions were queued
    product.st_sim_params(ctx, 30_000, 200_000, 0)
    assert product.run_batch(ctx, 5, SUNS, HITS, scenes.beam_down_target()) == -1
    product.st_sim_params(ctx, 30_000, 2_000_000_000, 0)
    return []


@pytest.mark.parametrize("prec", [0, 1])
def test_calls_in_turn_leave_what_each_leaves_alone(product, prec):
    calls = {"batch": _batch, "single": _single, "moved": _moved, "refused": _refused}
    alone = {}
    for name, call in calls.items():
        ctx = _context(product, prec)
        try:
            product.st_sun_xyz(ctx, 0.0, 0.0, 1e4)
            alone[name] = call(product, ctx)
        finally:
            product.st_free_context(ctx)
    ctx = _context(product, prec)
    try:
        product.st_sun_xyz(ctx, 0.0, 0.0, 1e4)
        for name in ("single", "batch", "single", "single", "batch", "batch", "moved", "single", "refused", "single",
                     "refused", "batch", "moved", "batch", "single"):
            for a, b in zip(calls[name](product, ctx), alone[name]):
                assert np.array_equal(a, b), name
    finally:
        product.st_free_context(ctx)
