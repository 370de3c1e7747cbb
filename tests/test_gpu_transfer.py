"""A batch's proposals and results through the transfer kernels: patches with no
source, one, and MAXSOURCES, uneven bands, proposals shorter than the patch's
scene, and repeated calls, bit for bit against one patch at a time."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(n_sources, bands, seed):
    from forcepho_b200 import synthetic as S
    rng = np.random.default_rng(seed)
    p = S.make_patch(rng, n_sources=n_sources, exp_per_band=[1] * bands, exp_pix=[(24, 20)] * bands, n_psf=1,
                     source_params=S._broad_source)
    S.add_noise(p, rng, 1.0)
    p.return_residual = False
    p.send_to_device()
    return p


def test_batch_matches_single_calls():
    from forcepho_b200.batch import BatchedProposer
    from forcepho_b200.proposal import B200Proposer
    from forcepho_b200.structs import source_struct_dtype
    patches = [make(ns, nb, 10 * ns + nb) for ns, nb in ((3, 2), (0, 1), (30, 5), (1, 1), (2, 30))]
    full = [p.scene.get_proposal().copy() if int(p.n_sources) else np.zeros(0, source_struct_dtype) for p in patches]
    short = [q[:max(len(q) - 1, 0)] for q in full]
    bp = BatchedProposer(patches, tile_pixels=256)
    for props in (full, short, full):
        padded = [np.concatenate([q, np.zeros(int(p.n_sources) - len(q), source_struct_dtype)])
                  for p, q in zip(patches, props)]
        for p, q, (chi2, grad) in zip(patches, padded, bp.evaluate_proposals(props)):
            c, g = B200Proposer(tile_pixels=256).evaluate_proposal(q, patch=p)
            assert chi2.shape == (p.n_bands,) and grad.shape == (p.n_bands, int(p.n_sources), 7)
            assert np.array_equal(chi2, c, equal_nan=True) and np.array_equal(grad, g, equal_nan=True)
    assert bp.h2d_bytes == 36 * source_struct_dtype.itemsize
    assert bp.d2h_bytes == 39 * 8 + (6 + 150 + 1 + 60) * 7 * 4


def test_residual_is_a_fresh_copy_of_the_current_buffer():
    """Also after a swap, which moves the residual to the other buffer."""
    from forcepho_b200.proposal import B200Proposer
    p = make(3, 2, 1)
    p.return_residual = True
    p.send_to_device()
    q, pr = p.scene.get_proposal(), B200Proposer(tile_pixels=256)
    first = pr.evaluate_proposal(q, patch=p, unpack=False)[2]
    assert np.array_equal(first, p.retrieve_array("residual"))
    kept = first.copy()
    p.swap_on_device()
    second = pr.evaluate_proposal(q, patch=p, unpack=False)[2]
    assert np.array_equal(second, p.retrieve_array("residual")) and not np.array_equal(first, second)
    assert np.array_equal(first, kept)
