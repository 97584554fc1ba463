"""Flat-rectangle probe of more than 2^32 sun rays.

The probe makes part of a ray's random words once per segment of 1,024 rays, from the upper half of the
64-bit ray index; segments that cross a multiple of 2^32 take another path.  Every ray of such a run is
checked against the general double-precision probe through the hits that each element gets.
"""
import ctypes as C

import numpy as np
import pytest

from test_gpu_flat_probe import _elem, _scene
from test_zz_no_alloc import _bind

pytestmark = pytest.mark.gpu

UP = np.array([0.0, 0.0, 1.0])
CHUNK = 1 << 22


def test_hits_of_every_element_past_two_to_the_32(product):
    """Each rectangle lies above another, so the run's first plan takes the hit rate for twice what it
    is and its second group of batches begins at an odd ray: a segment crosses 2^32."""
    import torch

    from soltrace_b200 import scenes
    xy = [(28.0 * i, 28.0 * j) for i in range(6) for j in range(6)]
    els = [_elem((x, y, z), UP, (4.0, 4.0)) for z in (0.0, 2.0) for x, y in xy]
    hits = int(36 * 16.0 / (28.0 * 5 + 4 * 2**0.5) ** 2 * 1.01 * 2**32)
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, _scene(els, UP, hits))
        product.st_b200_set_records(ctx, 0)
        product.st_b200_set_max_sun_rays(ctx, 10**11)
        got = []
        for prec in (0, 1):
            product.st_b200_set_precision(ctx, prec)
            assert product.run(ctx, 77) >= 0, product.messages(ctx)
            got.append((product.stats(ctx)["sun_rays"], product.element_counts(ctx, 1, len(els))[0]))
        n = got[0][0]
        assert n > 2**32 + 2**24 and got[1][0] == n
        sid = torch.zeros(CHUNK, dtype=torch.int64, device="cuda")
        el = torch.zeros(CHUNK, dtype=torch.int32, device="cuda")
        want = torch.zeros(len(els), dtype=torch.int64, device="cuda")
        fn, cnt, last = _bind(product), C.c_uint(), -1
        for s0 in range(0, n, CHUNK):
            assert fn(ctx, 77, s0, min(CHUNK, n - s0), sid.data_ptr(), el.data_ptr(), C.byref(cnt), None) == 1
            want += torch.bincount(el[:cnt.value], minlength=len(els))
            last = int(sid[cnt.value - 1]) if cnt.value else last
        want = want.cpu().numpy().astype(np.uint64)
        assert last == n - 1 and want.sum() == hits
        for _, first in got:
            assert np.array_equal(first, want)
    finally:
        product.st_free_context(ctx)
