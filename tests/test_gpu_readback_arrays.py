"""Record columns read into arrays that overlap.

Long columns are copied by several threads.  A caller that wants one column only may pass the same array
for all three: the columns are then written in their order, so that the last one stays.
"""
import numpy as np
import pytest

from soltrace_b200 import scenes
from soltrace_b200.capi import dptr

pytestmark = pytest.mark.gpu


def test_overlapping_arrays_hold_the_last_columns(product):
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, scenes.dish_scene(600_000))
        assert product.run(ctx, 2) > 0, product.messages(ctx)
        n = product.st_num_intersections(ctx)
        x, y, z = (np.zeros(n) for _ in range(3))
        assert product.st_locations(ctx, dptr(x), dptr(y), dptr(z)) == 1
        cx, cy, cz = (np.zeros(n) for _ in range(3))
        assert product.st_cosines(ctx, dptr(cx), dptr(cy), dptr(cz)) == 1
        assert n * 8 > 4 << 20 and len({a.tobytes() for a in (x, y, z, cx, cy, cz)}) == 6
        one = np.zeros(n + 1000)
        for _ in range(20):
            assert product.st_locations(ctx, dptr(one), dptr(one), dptr(one)) == 1
            assert np.array_equal(one[:n], z)
            assert product.st_cosines(ctx, dptr(one), dptr(one), None) == 1
            assert np.array_equal(one[:n], cy)
            # shifted by a thousand values: y over x's tail
            assert product.st_locations(ctx, dptr(one), dptr(one[1000:]), None) == 1
            assert np.array_equal(one[:1000], x[:1000]) and np.array_equal(one[1000:], y)
    finally:
        product.st_free_context(ctx)
