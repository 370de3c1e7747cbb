"""The per-band reduction over tiles: bands of 0, 1 and just below, at and above
a multiple of the warps' shares and of the loads in flight, against the FP64
oracle at the tiled path's tolerances (the sums themselves are FP64)."""

import numpy as np
import pytest

from tolerances import CHI2_F64, GRAD_F64, band_scales, chi2_raw_err, grad_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sources", [1, 5, 30])
@pytest.mark.parametrize("tiles", [(0, 1, 2, 7), (8, 9, 16, 17), (63, 64, 65), (72, 1, 129)])
def test_band_sums(tiles, n_sources):
    from forcepho_b200 import synthetic as S
    from forcepho_b200.proposal import B200Proposer
    from oracle import oracle as O
    rng = np.random.default_rng(sum(tiles))
    # an empty band cannot place sources, so the first band always has a tile of its own
    p = S.make_patch(rng, n_sources=n_sources, exp_per_band=[1] * (1 + len(tiles)), n_psf=1, raster_width=16,
                     exp_pix=[256] + [256 * t for t in tiles], source_params=S._broad_source)
    S.add_noise(p, rng, rng.uniform(0.5, 2.0, p.n_exp))
    p.return_residual = False
    p.send_to_device()
    prop = p.scene.get_proposal()
    chi2, grad = B200Proposer(tile_pixels=256).evaluate_proposal(prop, patch=p)
    c64, g64, r64 = O.evaluate(p, prop, precision="f64", return_residual=True)
    empty = np.array([False] + [t == 0 for t in tiles])
    assert np.all(chi2[empty] == 0) and np.all(grad[empty] == 0)
    assert chi2_raw_err(chi2[~empty], c64[~empty], band_scales(p, r64)[~empty]) < CHI2_F64
    assert grad_err(grad[~empty], g64[~empty]) < GRAD_F64
