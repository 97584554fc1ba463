"""First-stage rectangles up-sun of the plane that sun rays start from.

Sun rays start 10,000 m up-sun of the first stage's origin and an element behind that plane is
never met, nor does it hide one in front of it.  The flat-rectangle probe must keep to that, in
single runs and in batches (whose grids are built on the device).
"""
import ctypes as C

import numpy as np
import pytest

from helpers import assert_same_records, run_scene
from test_gpu_flat_probe import _elem, _scene
from test_gpu_parity import PHILOX, _fp64, _mixed
from test_zz_no_alloc import _bind, _first_elements

pytestmark = pytest.mark.gpu

UP = np.array([0.0, 0.0, 1.0])
GRID = [(x, y) for x in range(0, 40, 10) for y in range(0, 40, 10)]


def _behind():
    sc = _scene([_elem((x, y, 11_000.0), UP, (4.0, 4.0)) for x, y in GRID], UP, 100)
    sc.raymax = 20_000
    return sc


def _mixed_depths(hits):
    """Ground rectangles, half of them under one behind the plane, one 300 m long rectangle that
    crosses the plane and one that ends a millimetre short of it."""
    els = [_elem((x, y, 0.0), UP, (4.0, 4.0)) for x, y in GRID]
    els += [_elem((x, y, 10_500.0), UP, (5.0, 5.0)) for x, y in GRID[::2]]
    els += [_elem((80.0, 20.0, 10_000.0), (1.0, 0.0, 0.2), (300.0, 6.0)),
            _elem((120.0, 20.0, 9_999.999), UP, (6.0, 6.0))]
    return _scene(els, UP, hits)


@pytest.mark.parametrize("setup", [_fp64, _mixed], ids=["fp64", "mixed"])
def test_elements_behind_the_start_plane_are_not_hit(product, oracle, setup):
    want = run_scene(oracle, _behind(), 3, PHILOX)
    got = run_scene(product, _behind(), 3, setup)
    assert want[0] < 0 and got[0] == want[0]
    assert "generated sun rays reached maximum count" in got[3][-1]


def test_elements_behind_the_start_plane_hide_nothing(product, oracle):
    sc = _mixed_depths(3000)
    want = run_scene(oracle, sc, 5, PHILOX)
    got = run_scene(product, sc, 5, _fp64)
    assert got[0] == want[0] and got[2] == want[2], got[3]
    assert_same_records(got[1], want[1], pos_tol=1e-9, rel_tol=2e-12, dir_tol=1e-9)
    mixed = run_scene(product, sc, 5, _mixed)
    assert mixed[2] == want[2]
    assert np.array_equal(_first_elements(mixed[1], 3000), _first_elements(want[1], 3000))


def test_general_probe_agrees_across_the_start_plane(product):
    import torch
    from soltrace_b200 import scenes
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, _mixed_depths(3000))
        assert product.run(ctx, 5) > 0, product.messages(ctx)
        first, n = _first_elements(product.records(ctx), 3000), product.stats(ctx)["sun_rays"]
        sid = torch.zeros(n, dtype=torch.int64, device="cuda")
        el = torch.zeros(n, dtype=torch.int32, device="cuda")
        cnt = C.c_uint()
        assert _bind(product)(ctx, 5, 0, n, sid.data_ptr(), el.data_ptr(), C.byref(cnt), None) == 1
        assert cnt.value == 3000
        assert np.array_equal(el[:3000].cpu().numpy() + 1, first)
    finally:
        product.st_free_context(ctx)


@pytest.mark.parametrize("prec", [0, 1])
def test_batched_grids_keep_to_the_start_plane(product, prec):
    from soltrace_b200 import scenes
    sc = _mixed_depths(3000)
    suns = [1e4 * UP, 1e4 * np.array([0.02, 0.0, np.sqrt(1 - 0.0004)])]
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, sc)
        product.st_b200_set_precision(ctx, prec)
        product.st_b200_set_records(ctx, 0)
        n = len(sc.stages[0].elements)
        assert product.run_batch(ctx, 9, suns, [3000] * 2) == 1, product.messages(ctx)
        got = [(product.batch_stats(ctx, k)["sun_rays"], product.batch_absorbed(ctx, k, 1, n)) for k in range(2)]
        sc.raycount = 3000
        for k, (rays, absorbed) in enumerate(got):
            product.st_sun_xyz(ctx, *map(float, suns[k]))
            assert product.run(ctx, 9 + k) >= 0, product.messages(ctx)
            assert product.stats(ctx)["sun_rays"] == rays
            assert np.array_equal(product.element_counts(ctx, 1, n)[1], absorbed)
    finally:
        product.st_free_context(ctx)


def test_batch_behind_the_start_plane_ends_at_the_ray_limit(product):
    from soltrace_b200 import scenes
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, _behind())
        product.st_b200_set_records(ctx, 0)
        assert product.run_batch(ctx, 9, [1e4 * UP], [100]) == -1
        assert "generated sun rays reached maximum count" in product.messages(ctx)[-1]
    finally:
        product.st_free_context(ctx)
