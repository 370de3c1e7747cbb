"""The GPU checks that compare with the compiled reference kernel, with the
oracle's FP32 restatement of that kernel in its place: their FP64 assertions then
run where the reference's sources are not at hand."""

import pytest

import test_gpu_autograd_hmc
import test_gpu_edges
import test_gpu_limits
import test_gpu_parity
import test_gpu_shapes
from oracle import oracle as O
from test_gpu_limits import limits_patch  # noqa: F401

pytestmark = pytest.mark.gpu

SHAPES = [dict(q=0.21, rhalf=0.2, sersic=2.0), dict(q=0.9, rhalf=0.03, sersic=1.0),
          dict(q=0.5, rhalf=0.6, sersic=6.0), dict(q=0.35, rhalf=0.1, sersic=0.85)]


@pytest.fixture(autouse=True)
def restated(monkeypatch):
    def ref_evaluate(patch, proposal, return_residual=False, bands=None):
        return O.evaluate(patch, proposal, precision="f32", return_residual=return_residual, bands=bands)
    monkeypatch.setattr(O, "ref_evaluate", ref_evaluate)


@pytest.mark.parametrize("kind", ["tiled", "plain"])
@pytest.mark.parametrize("shape", SHAPES)
def test_extreme_shapes(kind, shape):
    test_gpu_shapes.test_extreme_shapes(kind, shape)


@pytest.mark.parametrize("kind", ["tiled", "plain"])
def test_max_bands_and_sources(kind):
    test_gpu_edges.test_max_bands_and_sources(kind)


@pytest.mark.parametrize("kind", ["tiled", "plain"])
def test_limits_parity(limits_patch, kind):
    test_gpu_limits.test_limits_parity(limits_patch, kind)


def test_unpadded_and_empty_exposures():
    test_gpu_parity.test_unpadded_and_empty_exposures()


def test_autograd_backward_vs_fd_and_restatement():
    test_gpu_autograd_hmc.test_autograd_backward_vs_fd_and_reference()
