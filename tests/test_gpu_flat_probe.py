"""The flat-rectangle probe (k_sun_probe_flat) against the general grid probe.

st_sim_run's probe of a first stage of flat rectangles decides rays in float outside its
rounding margins and leaves the rest to the double search; st_b200_probe_noalloc runs the general
double-precision grid probe on the same sun rays.  Both must list the same rays with the same
elements, on layouts where the float test can go wrong: grids much coarser than the elements,
kilometre-long rows (bitmaps coarser than the cells), coplanar duplicates (every ray undecided),
elements near edge-on, narrow rotated rectangles, disabled elements, and a last tile of one ray.
Batched runs build the same grids on the device: their positions must number the rays of single
runs on those layouts.
"""
import ctypes as C
import math

import numpy as np
import pytest

from soltrace_b200.scenes import Element, OpticFace, OpticSet, Scene, Stage, Sun
from test_zz_no_alloc import _bind, _first_elements

pytestmark = pytest.mark.gpu

MIRROR = OpticSet("m", OpticFace("g", refl=0.9, slope=1.5), OpticFace("g", refl=0.9, slope=1.5))


def _scene(elements, sun, hits):
    return Scene(Sun("p", 4.65, tuple(1e4 * np.asarray(sun))), [MIRROR], [Stage(elements)], raycount=hits,
                 raymax=2_000_000_000 - 1)


def _elem(pos, normal, size, zrot=0.0, enabled=True):
    pos, normal = np.asarray(pos, float), np.asarray(normal, float)
    return Element(origin=tuple(pos), aim=tuple(pos + 100.0 * normal / np.linalg.norm(normal)), zrot=zrot,
                   aperture="r", aperture_params=size, surface="f", interaction=2, optic="m", enabled=enabled)


def _layout(name):
    """(elements, unit vector to the sun, hits)"""
    rng = np.random.default_rng(len(name))
    up = np.array([0.0, 0.0, 1.0])
    if name == "sparse":  # 0.1 m elements over 3 km: cells hundreds of times their size
        p = rng.uniform(-1500, 1500, (4000, 2))
        return [_elem((x, y, rng.uniform(0, 3)), up + rng.normal(0, 0.2, 3), (0.1, 0.1)) for x, y in p], up, 1
    if name == "row":  # 6 km x 2 m
        return [_elem((x, rng.uniform(-0.5, 0.5), 1.0), up, (2.0, 1.0)) for x in np.arange(-3000, 3000, 2.5)], up, 4000
    if name == "duplicates":
        e = [_elem((x, y, 0.0), up, (4.0, 4.0)) for x in range(0, 40, 5) for y in range(0, 40, 5)]
        return e + e, np.array([0.0, 0.6, 0.8]), 3000
    if name == "edge-on":  # normals within 2 degrees of edge-on among ordinary ones, some disabled
        els = []
        for k, (x, y) in enumerate(rng.uniform(-60, 60, (120, 2))):
            t = math.radians(rng.uniform(88.0, 92.0)) if k % 3 == 0 else rng.uniform(0.0, 1.4)
            a = rng.uniform(0, 2 * math.pi)
            n = (math.sin(t) * math.cos(a), math.sin(t) * math.sin(a), math.cos(t))
            els.append(_elem((x, y, rng.uniform(0, 20)), n, (6.0, 3.0), zrot=rng.uniform(0, 180), enabled=k % 7 != 0))
        return els, up, 3001
    if name == "negative":  # a negative size accepts nothing
        e = [_elem((x, y, 0.0), up, (3.0, 3.0)) for x in range(0, 40, 5) for y in range(0, 40, 5)]
        return e + [_elem((x, 50.0, 0.0), up, (-3.0, 3.0)) for x in range(0, 40, 5)], up, 3000
    if name == "narrow":
        return [_elem((x, y, rng.uniform(0, 5)), up + rng.normal(0, 0.4, 3), (12.0, 0.3), zrot=rng.uniform(0, 180))
                for x, y in rng.uniform(-50, 50, (200, 2))], np.array([0.3, 0.4, math.sqrt(0.75)]), 4097
    return [_elem((x, y, 0.0), up, (1.0, 1.0)) for x in (0, 2) for y in (0, 2)], up, 1  # "four"


@pytest.mark.parametrize("name", ["sparse", "row", "duplicates", "edge-on", "narrow", "four", "negative"])
def test_flat_probe_lists_the_general_probes_hits(product, name):
    import torch

    from soltrace_b200 import scenes
    els, sun, hits = _layout(name)
    sc = _scene(els, sun, hits)
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, sc)
        product.st_b200_set_precision(ctx, 0)
        assert product.run(ctx, 11) > 0, product.messages(ctx)
        first = _first_elements(product.records(ctx), hits)
        nsun = product.stats(ctx)["sun_rays"]
        product.st_b200_set_precision(ctx, 1)
        assert product.run(ctx, 11) > 0, product.messages(ctx)
        assert product.stats(ctx)["sun_rays"] == nsun
        fn = _bind(product)
        got_sid, got_el = [], []
        for s0 in range(0, nsun, 2_000_000):
            n = min(2_000_000, nsun - s0)
            sid = torch.zeros(n, dtype=torch.int64, device="cuda")
            el = torch.zeros(n, dtype=torch.int32, device="cuda")
            cnt = C.c_uint()
            assert fn(ctx, 11, s0, n, sid.data_ptr(), el.data_ptr(), C.byref(cnt), None) == 1, product.messages(ctx)
            got_sid.append(sid[:cnt.value].cpu().numpy())
            got_el.append(el[:cnt.value].cpu().numpy())
        got_sid, got_el = np.concatenate(got_sid), np.concatenate(got_el)
        assert len(got_sid) == hits and got_sid[-1] == nsun - 1
        assert np.array_equal(got_el + 1, first)
    finally:
        product.st_free_context(ctx)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("name", ["sparse", "row", "duplicates", "edge-on", "narrow", "four", "negative"])
def test_batched_grids_number_the_single_runs_rays(product, name, prec):
    from soltrace_b200 import scenes
    els, sun, hits = _layout(name)
    suns = [1e4 * np.asarray(sun), 1e4 * np.asarray([0.2, -0.3, math.sqrt(1 - 0.13)]), 1e4 * np.asarray([0.0, 0.8, 0.6])]
    ctx = product.st_create_context()
    try:
        scenes.push(product, ctx, _scene(els, sun, hits))
        product.st_b200_set_precision(ctx, prec)
        product.st_b200_set_records(ctx, 0)
        assert product.run_batch(ctx, 5, suns, [hits] * 3) == 1, product.messages(ctx)
        got = [(product.batch_stats(ctx, k)["sun_rays"], product.batch_absorbed(ctx, k, 1, len(els))) for k in range(3)]
        for k, (n, absorbed) in enumerate(got):
            product.st_sun_xyz(ctx, *map(float, suns[k]))
            assert product.run(ctx, 5 + k) >= 0, product.messages(ctx)
            assert product.stats(ctx)["sun_rays"] == n
            assert np.array_equal(product.element_counts(ctx, 1, len(els))[1], absorbed)
    finally:
        product.st_free_context(ctx)
