"""Bytes that a run of many batches brings back.

A run with records waits for every batch.  Its accumulators (element counts, flux bins) are read once the
work queued may be the last, not after every batch.
"""
import numpy as np
import pytest

from test_gpu_hit_rate import _elements
from test_gpu_flat_probe import _scene

pytestmark = pytest.mark.gpu

NX = NY = 240


@pytest.mark.parametrize("callback", [False, True])
def test_accumulators_come_back_once(product, callback):
    """Elements of 5 cm in a box of 80 m: 1,000 hits take about ten batches of 2^26 sun rays."""
    from soltrace_b200 import scenes
    seen = []

    def progress(*a):
        seen.append(a[1])
        return 1

    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, _scene(_elements("f", 0.05), (0.0, 0.0, 1.0), 1000))
        product.st_b200_add_flux_map(ctx, 1, 1, 0, NX, NY, -0.03, 0.03, -0.03, 0.03, 0)
        assert product.run(ctx, 3, progress if callback else None) > 0, product.messages(ctx)
        st = product.stats(ctx)
        assert st["batches"] >= 5 and len(seen) == (st["batches"] if callback else 0)
        first, absorbed, delivered = product.element_counts(ctx, 1, 4)
        assert first.sum() == 1000
        rec = product.records(ctx)
        on_first = np.sum((rec["stage"] == 1) & (np.abs(rec["element"]) == 1))
        assert product.flux(ctx, 0, NX, NY).sum() == on_first > 0
        assert st["d2h_bytes"] < 3 * 8 * NX * NY
    finally:
        product.st_free_context(ctx)
