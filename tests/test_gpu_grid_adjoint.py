"""The adjoint over a tile's dense weight grid against the one over its pixel
list, and both against the FP64 oracle: tile classes, cells cut off at the
right and lower edge, one-pixel columns, last groups of every replication,
masked pixels, and the pixel layouts that must fall back to the list (duplicate
positions, fractional coordinates, sparse and unordered pixels, weights that
are not finite).

Both forms evaluate each pair in FP32, so each is held to the tiled path's
FP64 tolerance, and they may differ by the two together.  The forward pass is
the same code for both: chi2 is bitwise equal."""

import numpy as np
import pytest

from tolerances import GRAD_F64, grad_err

pytestmark = pytest.mark.gpu


def make(width, height, n_sources, seed=5, n_psf=2):
    from forcepho_b200 import synthetic as S
    rng = np.random.default_rng(seed)
    p = S.make_patch(rng, n_sources=n_sources, exp_per_band=[1, 2], exp_pix=[(width, height)] * 3, n_psf=n_psf,
                     source_params=S._broad_source)
    S.add_noise(p, rng, rng.uniform(0.5, 2.0, p.n_exp))
    p.return_residual = False
    return p


def evaluate(p, tile_pixels, flags):
    from forcepho_b200.proposal import B200Proposer
    p.send_to_device()
    return B200Proposer(tile_pixels=tile_pixels, flags=flags).evaluate_proposal(p.scene.get_proposal(), patch=p)


def check(p, tile_pixels):
    from forcepho_b200 import _native as N
    from oracle import oracle as O
    cg, gg = evaluate(p, tile_pixels, 0)
    cl, gl = evaluate(p, tile_pixels, N.FLAG_PIXEL_LIST)
    assert np.array_equal(cg, cl)
    _, g64 = O.evaluate(p, p.scene.get_proposal(), precision="f64")[:2]
    assert grad_err(gg, g64) < GRAD_F64
    assert grad_err(gl, g64) < GRAD_F64
    assert grad_err(gg, gl) < 2 * GRAD_F64


@pytest.mark.parametrize("tile_pixels", [256, 512, 1024])
@pytest.mark.parametrize("width,height", [(64, 64), (33, 47), (22, 15), (1, 40), (70, 3), (31, 33)])
def test_grid_matches_list_and_oracle(width, height, tile_pixels):
    check(make(width, height, 3), tile_pixels)


@pytest.mark.parametrize("n_psf", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("n_sources", [1, 2, 5, 16])
def test_groups_of_every_size(n_sources, n_psf):
    check(make(40, 36, n_sources, seed=n_sources, n_psf=n_psf), 1024)


@pytest.mark.parametrize("keep", [0.9, 0.6, 0.2])
def test_masked_pixels(keep):
    """Bad pixels have no weight; few left make the list the cheaper form."""
    p = make(64, 50, 4)
    p.ierr[np.random.default_rng(1).random(p.npix) > keep] = 0.0
    check(p, 1024)


def _shuffle(p):
    for e in range(p.n_exp):
        s = slice(int(p.exposure_start[e]), int(p.exposure_start[e]) + int(p.exposure_N[e]))
        o = np.random.default_rng(e).permutation(int(p.exposure_N[e]))
        for name in ("xpix", "ypix", "data", "ierr"):
            getattr(p, name)[s] = getattr(p, name)[s][o]


def _duplicate(p):
    p.xpix[100], p.ypix[100] = p.xpix[101], p.ypix[101]
    p.xpix[2000], p.ypix[2000] = p.xpix[2001], p.ypix[2001]


def _fraction(p):
    p.xpix += np.float32(0.25)


def _half_row(p):
    p.ypix[:900] += np.float32(0.5)


@pytest.mark.parametrize("change", [_shuffle, _duplicate, _fraction, _half_row], ids=lambda f: f.__name__[1:])
@pytest.mark.parametrize("tile_pixels", [256, 1024])
def test_pixel_layouts(change, tile_pixels):
    p = make(48, 40, 4)
    change(p)
    check(p, tile_pixels)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_weights_that_are_not_finite(bad):
    """A bad data value leaves the sources out of its reach untouched, as over the list."""
    from forcepho_b200 import _native as N
    p = make(150, 40, 6)
    p.data[75] = bad
    cg, gg = evaluate(p, 1024, 0)
    cl, gl = evaluate(p, 1024, N.FLAG_PIXEL_LIST)
    assert np.array_equal(cg, cl, equal_nan=True)
    assert np.array_equal(np.isfinite(gg), np.isfinite(gl)) and not np.isfinite(gg).all()
