"""The forward pass at the edges of its work split: tiles of every class whose
pixels fill one warp, a few, or all eight (the others then take further runs of
Gaussians), rows of 4 pixels or not, one run of Gaussians to several chunks.
Each pair is evaluated in FP32, so residuals and chi2 are held to the tiled
path's FP64 tolerances; a forward-only launch gives the same bits as a full one."""

import numpy as np
import pytest

from tolerances import CHI2_F64, band_scales, chi2_raw_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile_pixels", [256, 512, 1024])
@pytest.mark.parametrize("n_sources,n_psf", [(1, 3), (4, 4), (16, 4)])
@pytest.mark.parametrize("width", [16, 32, 22, 3])
def test_sets_of_warps(width, n_sources, n_psf, tile_pixels):
    from forcepho_b200 import _native as N
    from forcepho_b200 import synthetic as S
    from forcepho_b200.proposal import B200Proposer
    from oracle import oracle as O
    rng = np.random.default_rng(width + n_sources)
    pix = [1, 31, 32, 33, 127, 128, 129, 255, 257, 511, 513, 1023, 1024]
    p = S.make_patch(rng, n_sources=n_sources, exp_per_band=[6, 7], exp_pix=pix, n_psf=n_psf,
                     source_params=S._broad_source, raster_width=width)
    S.add_noise(p, rng, rng.uniform(0.5, 2.0, p.n_exp))
    p.return_residual = True
    p.send_to_device()
    prop = p.scene.get_proposal()
    chi2, _, res = B200Proposer(tile_pixels=tile_pixels).evaluate_proposal(prop, patch=p, unpack=False)
    c64, _, r64 = O.evaluate(p, prop, precision="f64", return_residual=True)
    peak = np.abs(p.data.astype(np.float64) - r64).max()
    np.testing.assert_allclose(res, r64, rtol=0, atol=1e-5 * peak + 1e-6)
    assert chi2_raw_err(chi2, c64, band_scales(p, r64)) < CHI2_F64
    only = B200Proposer(tile_pixels=tile_pixels, flags=N.FLAG_FORWARD_ONLY).evaluate_proposal(prop, patch=p, unpack=False)
    assert np.array_equal(only[0], chi2) and np.array_equal(only[2], res)
