"""Packing of proposals, metadata and plan tables for many sources or views at
once against the record-by-record form: all results are bit for bit the same."""

import ctypes

import numpy as np
import pytest

from forcepho_b200 import _native as N
from forcepho_b200 import synthetic
from forcepho_b200.sources import Galaxy, Scene, pack_proposal


class Shifted(Galaxy):
    """A source that packs its own record."""

    def proposal(self):
        p = super().proposal().copy()
        p["ra"] += 1.0
        return p


def galaxies(n, rng, cls=Galaxy):
    out = []
    for _ in range(n):
        g = cls(["a", "b", "c"])
        g.flux = rng.uniform(0.1, 9.0, 3)
        g.ra, g.dec = rng.normal(size=2) * 1e-4
        g.q, g.pa = rng.uniform(0.3, 1.0), rng.uniform(-1.5, 1.5)
        g.sersic, g.rhalf = rng.uniform(1.0, 5.0), rng.uniform(0.03, 1.0)
        out.append(g)
    return out


@pytest.mark.parametrize("n,mixed", [(1, False), (2, False), (17, False), (5, True)])
def test_proposals_together_or_one_by_one(n, mixed):
    rng = np.random.default_rng(n)
    srcs = galaxies(n, rng)
    if mixed:
        srcs[2:4] = galaxies(2, rng, Shifted)
    want = np.concatenate([s.proposal().copy() for s in srcs])
    got = pack_proposal(srcs)
    assert got.dtype == want.dtype and got.tobytes() == want.tobytes()


def test_metadata_of_several_scenes():
    patch = synthetic.config_multiband(n_sources=5, size=20)
    scenes = [Scene([g]) for g in patch.scene.sources]
    for many in (scenes, scenes[:1], scenes + [patch.scene]):
        for got, sc in zip(patch.metas_for(many), many):
            want = patch.meta_for(sc)
            assert set(got) == set(want)
            for k, w in want.items():
                assert np.asarray(got[k]).dtype == np.asarray(w).dtype
                assert np.array_equal(np.asarray(got[k]), np.asarray(w)), k


def shape_of(x, y):
    start, n = np.array([0], np.int32), np.array([len(x)], np.int32)
    one = np.array([1], np.int16)
    keep = [start, n, np.array([0], np.int16), one, np.array([1], np.int32), x, y]
    s = N.PatchShape(1, 1, 1, len(x), *[a.ctypes.data for a in keep])
    s._keep = keep
    return s


def order_of(x, y, tile_pixels):
    """Stable order by grid cell (row by row; pixels without a finite position last)."""
    w, h = {64: (8, 8), 1024: (32, 32)}[tile_pixels]
    ok = np.isfinite(x) & np.isfinite(y)
    xd, yd = x.astype(np.float64), y.astype(np.float64)
    x0, x1 = (xd[ok].min(), xd[ok].max()) if ok.any() else (0.0, 0.0)
    y0, y1 = (yd[ok].min(), yd[ok].max()) if ok.any() else (0.0, 0.0)
    ncx, ncy = int((x1 - x0) / w) + 1, int((y1 - y0) / h) + 1
    key = np.full(len(x), ncx * ncy, np.int64)
    cx = np.minimum(((xd[ok] - x0) * (1.0 / w)).astype(np.int64), ncx - 1)
    cy = np.minimum(((yd[ok] - y0) * (1.0 / h)).astype(np.int64), ncy - 1)
    key[ok] = cy * ncx + cx
    order = np.argsort(key, kind="stable")
    sizes = []
    for n in np.unique(key, return_counts=True)[1]:
        sizes += [min(tile_pixels, n - k) for k in range(0, n, tile_pixels)]
    return order, sizes


def layout(kind, rng):
    yy, xx = np.mgrid[0:41, 0:53]
    x, y = xx.ravel().astype(np.float32), yy.ravel().astype(np.float32)
    if kind == "negative":
        x, y = x - 30.25, y - 1000.5
    elif kind == "shuffled":
        p = rng.permutation(len(x))
        x, y = x[p], y[p]
    elif kind == "not finite":
        x[::97], y[5::131], x[7] = np.nan, np.inf, -np.inf
    elif kind == "none finite":
        x[:] = np.nan
    elif kind == "sparse":
        x, y = x * 1e4, y * 1e3
    elif kind == "stacked":
        x, y = np.zeros_like(x), np.zeros_like(y)
    elif kind == "one":
        x, y = x[:1], y[:1]
    return np.ascontiguousarray(x, np.float32), np.ascontiguousarray(y, np.float32)


@pytest.mark.parametrize("copies", [1, 3])
@pytest.mark.parametrize("tile_pixels", [64, 1024])
@pytest.mark.parametrize("kind", ["rows", "negative", "shuffled", "not finite", "none finite", "sparse", "stacked",
                                  "one"])
def test_pixel_order_against_a_stable_sort(kind, tile_pixels, copies):
    """`copies` views share the coordinate arrays; a patch of other arrays
    with the same values stands between them."""
    L = N.load()
    x, y = layout(kind, np.random.default_rng(3))
    shapes = [shape_of(x, y) for _ in range(copies)]
    shapes.insert(1, shape_of(x.copy(), y.copy()))
    arr = (N.PatchShape * len(shapes))(*shapes)
    rule, z = N.tile_rule([(0, tile_pixels)]), N.PlanSizes()
    N.check(L.fp_plan_count_rule(ctypes.addressof(arr), len(shapes), ctypes.byref(rule), ctypes.byref(z)))
    expos, bands = np.zeros(z.n_exposures, N.exposure_desc_dtype), np.zeros(z.n_band_outputs, N.band_desc_dtype)
    tiles, run = np.zeros(z.n_tiles, N.tile_dtype), np.zeros(z.n_tiles, np.int32)
    perm = np.zeros(z.n_perm, np.int32)
    N.check(L.fp_plan_fill_rule(ctypes.addressof(arr), len(shapes), ctypes.byref(rule), expos.ctypes.data,
                                tiles.ctypes.data, bands.ctypes.data, run.ctypes.data, perm.ctypes.data))
    order, sizes = order_of(x, y, tile_pixels)
    assert np.array_equal(perm, np.tile(order, len(shapes)))
    assert np.array_equal(tiles["n_pix"], np.tile(sizes, len(shapes)))
