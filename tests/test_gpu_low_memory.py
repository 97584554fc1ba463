"""Runs on a device whose memory is nearly full."""
import pytest

from soltrace_b200 import scenes

pytestmark = pytest.mark.gpu


def _run(product):
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, scenes.dish_scene(1_000_000))
        product.st_b200_set_records(ctx, 0)
        rc = product.run(ctx, 5)
        return (rc, product.stats(ctx)["sun_rays"]) if rc >= 0 else product.messages(ctx)
    finally:
        product.st_free_context(ctx)


def _with_memory_left(product, left_mb):
    """The run's outcome in an empty device and with `left_mb` left; kernels are loaded first, so that
    their memory does not count."""
    import torch
    want = _run(product)
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (left_mb << 20), dtype=torch.uint8, device="cuda")
    try:
        return want, _run(product)
    finally:
        del hold
        torch.cuda.empty_cache()


def test_a_run_that_found_no_memory_leaves_the_next_one_alone(product):
    want, got = _with_memory_left(product, 20)
    assert want[0] >= 0 and "out of memory" in got[-1]
    assert _run(product) == want


@pytest.mark.parametrize("left_mb", [190, 210, 230, 250, 270, 300, 400])
def test_first_run_with_little_memory_left(product, left_mb):
    """A context's first run of unknown hit rate reserves its next run's buffers (about 300 MB here);
    where that room is not to be had, it still gets what it needs itself (about 150 MB)."""
    want, got = _with_memory_left(product, left_mb)
    assert want[0] >= 0 and got == want
