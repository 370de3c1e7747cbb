"""The adjoint over the weight grid on thin, oblique sources near a mode, and the
inputs that must leave it for the pixel list.

Near a mode the weights are white noise, so that a gradient is what is left of
terms that cancel; sums of plain pixel offsets lose two to four digits there for
axis ratios that the samplers' bounds include.  In ridge coordinates an FP32
emulation of this path stays below 5e-6 of the gradient in every column down to
axis ratios of 0.08; the FP64 bound of the tiled path is 1e-5.  Sources are faint, so
that the residual's own rounding does not enter.

A tile that must take the list gives the list's result bit for bit; a tile that
may take the grid does not, as the two round differently."""

import numpy as np
import pytest

from tolerances import GRAD_F64, grad_err

pytestmark = pytest.mark.gpu


def thin_patch(q, pa, rhalf, sersic, size=96, n_sources=3, psf_sigma=0.6, seed=11):
    from forcepho_b200 import synthetic as S
    from oracle import oracle as O
    rng = np.random.default_rng(seed)
    p = S.make_patch(rng, n_sources=n_sources, exp_per_band=[1, 1], exp_pix=[(size, size)] * 2, n_psf=1,
                     psf_offsets=False,
                     source_params=lambda r, nb: dict(flux=np.full(nb, 0.1), q=q, pa=pa, sersic=sersic, rhalf=rhalf))
    for name, value in (("Cxx", psf_sigma ** 2), ("Cyy", psf_sigma ** 2), ("Cxy", 0.0)):
        p.psfgauss[name] = value
    S.add_noise(p, rng, 1.0, O.render(p, p.scene.get_proposal()))
    p.return_residual = False
    return p


def evaluate(p, tile_pixels, flags=0):
    from forcepho_b200.proposal import B200Proposer
    p.send_to_device()
    return B200Proposer(tile_pixels=tile_pixels, flags=flags).evaluate_proposal(p.scene.get_proposal(), patch=p)


def both(p, tile_pixels):
    """(grid wherever it may be, list) gradients; chi2 does not depend on the choice."""
    from forcepho_b200 import _native as N
    (cg, gg), (cl, gl) = evaluate(p, tile_pixels), evaluate(p, tile_pixels, N.FLAG_PIXEL_LIST)
    assert np.array_equal(cg, cl, equal_nan=True)
    return gg, gl


@pytest.mark.parametrize("tile_pixels", [256, 512, 1024])
@pytest.mark.parametrize("q,rhalf,sersic", [(0.2, 0.2, 2.0), (0.2, 0.6, 4.0), (0.1, 0.3, 2.0), (0.9, 0.03, 1.0)])
@pytest.mark.parametrize("pa", [0.3, np.pi / 4, 1.4, -1.1])
def test_thin_sources_near_a_mode(q, rhalf, sersic, pa, tile_pixels):
    from oracle import oracle as O
    p = thin_patch(q, pa, rhalf, sersic)
    _, g64 = O.evaluate(p, p.scene.get_proposal(), precision="f64")[:2]
    _, g = evaluate(p, tile_pixels)
    assert grad_err(g, g64) < GRAD_F64


@pytest.mark.parametrize("tile_pixels", [256, 512, 1024])
def test_dense_rasters_take_the_grid(tile_pixels):
    gg, gl = both(thin_patch(0.6, 0.5, 0.2, 2.0), tile_pixels)
    assert not np.array_equal(gg, gl)


def _half_columns(p):
    p.xpix[1::2] += np.float32(0.5)


def _sparse(p):
    p.ierr[np.random.default_rng(3).random(p.npix) > 0.1] = 0.0


def _heavy(p):
    p.ierr *= np.float32(2.0 ** 32)         # weights beyond 2^60


def _growing(p):
    for name, value in (("Cxx", -3e4), ("Cyy", -3e4)):      # below every radius: exponents that grow
        p.psfgauss[name] = value


def _wide(p):
    p.psfgauss["Cxx"] = 2.0 ** 26           # a width of 8192 pixels


def _steep(p):
    for name, value in (("Cxx", 1.0), ("Cyy", 2.0 ** 23), ("Cxy", 2047.0)):   # F of slope -2047
        p.psfgauss[name] = value
    p.rad2[:] = 0.0


@pytest.mark.parametrize("change", [_half_columns, _sparse, _heavy, _growing, _wide, _steep],
                         ids=lambda f: f.__name__[1:])
@pytest.mark.parametrize("tile_pixels", [256, 1024])
def test_what_the_grid_refuses_is_the_list(change, tile_pixels):
    p = thin_patch(0.6, 0.5, 0.2, 2.0, size=64)
    change(p)
    gg, gl = both(p, tile_pixels)
    assert np.isfinite(gl).all() and np.abs(gl).max() > 0
    np.testing.assert_array_equal(gg, gl)


@pytest.mark.parametrize("ierr", [2.0 ** 26, 2.0 ** 52])
def test_large_weights_stay_finite(ierr):
    """The largest weights the grid takes, and ones whose fourth moments leave FP32: the
    gradient scales with their square (both are powers of two)."""
    p = thin_patch(0.6, 0.5, 0.2, 2.0, size=64)
    _, one = evaluate(p, 1024)
    p.ierr *= np.float32(ierr)
    _, g = evaluate(p, 1024)
    assert grad_err(np.asarray(g, np.float64) / ierr ** 2, one) < 2 * GRAD_F64


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_bad_pixel_out_of_reach(bad):
    """The widest Gaussian of a source ends 6 x 1.5 arcsec / q = 316 pixels from it."""
    from forcepho_b200 import _native as N
    from forcepho_b200 import synthetic as S
    rng = np.random.default_rng(2)
    far = iter([(850.0, 3.0), (60.0, 4.0)])
    p = S.make_patch(rng, n_sources=2, exp_per_band=[1], exp_pix=[(900, 8)], n_psf=2, perturb_wcs=False,
                     source_params=lambda r, nb: dict(flux=np.full(nb, 5.0), q=0.95, pa=0.4, sersic=2.0, rhalf=0.2,
                                                      pix=next(far)))
    S.add_noise(p, rng, 1.0)
    p.return_residual = False
    p.send_to_device()
    clean = evaluate(p, 1024)[1]
    p.data[2 * 900 + 10] = bad
    gg, gl = both(p, 1024)
    assert not np.isfinite(gg[:, 1]).any() and not np.isfinite(gl[:, 1]).any()
    assert np.isfinite(gg[:, 0]).all()
    np.testing.assert_array_equal(gg[:, 0], clean[:, 0])
    assert grad_err(gg[:, 0], gl[:, 0]) < 2 * GRAD_F64
