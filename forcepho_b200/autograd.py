"""chi2 as a differentiable torch function of the scene parameters, on the device.

``BatchChi2(patches)`` maps the flat scene-parameter vector theta of many
device patches (per patch, per active source, the reference's order
``[flux_1..flux_nb, ra, dec, q, pa, sersic, rhalf]``, forcepho/sources.py:559-605)
to the per-band chi2 of every patch, concatenated patch by patch:

    f = BatchChi2(patches)
    chi2 = f(theta)                          # float64[sum of n_bands]
    (-0.5 * chi2.sum()).backward()           # theta.grad = dlnlike/dtheta

``PatchChi2(patch)`` is the one-patch form (chi2 float64[n_bands]).

Everything stays on the GPU, with no host synchronisation in forward or
backward, so both can be captured in a CUDA graph:

* forward: the proposal records are built on the device from theta
  (``fp_hmc_prepare``: the Sersic mixture amplitudes and their sersic / rhalf
  derivatives from the device B-spline tables), then one batched evaluation
  (``fp_evaluate_batch``: Gaussian setup, the persistent tile kernel with its
  hand-written adjoint, the fixed-order reduction) gives chi2 and every
  d chi2[band] / d(source parameter) in one pass; those of the rows that
  exist are kept for backward;
* backward: the vector-Jacobian product with those per-band derivatives,
  assembled like ``stack_grad`` (forcepho/model.py:370-387) but kept per band,
  so any function of the band chi2s differentiates correctly: a band's flux
  moves only that band's chi2, the six shape parameters move every band's.
"""

import ctypes

import numpy as np
import torch

from . import _native as N
from .device import Plan, current_stream_ptr, result_rows, to_device_bytes
from .kernel_limits import NPARAMS

__all__ = ["BatchChi2", "PatchChi2"]


def _in_memory(t):
    """``t`` with its values in memory: kernels read addresses, which show neither
    the pending sign of a negated view nor anything of a zero tensor."""
    return t.clone() if t._is_zerotensor() else t.resolve_neg()


class _Chi2Fn(torch.autograd.Function):

    @staticmethod
    def forward(ctx, theta, owner):
        chi2, grads = owner._evaluate(theta.detach())
        ctx.owner = owner
        ctx.theta_meta = (theta.device, theta.dtype)
        ctx.save_for_backward(grads)
        return chi2

    @staticmethod
    def backward(ctx, grad_chi2):
        (grads,) = ctx.saved_tensors
        dev, dt = ctx.theta_meta
        g = ctx.owner._vjp(grad_chi2.to(ctx.owner.device), grads)
        return g.to(device=dev, dtype=dt), None


class BatchChi2(torch.nn.Module):
    """Per-band chi2 of many device patches as one differentiable function.

    Parameters
    ----------
    patches : device patches (``send_to_device``-ed, B200PatchMixin)
    tile_pixels, ctas_per_sm : launch parameters of the tile kernel
    splines : the Sersic amplitude splines (default: the package's table)
    """

    def __init__(self, patches, tile_pixels=1024, ctas_per_sm=4, splines=None):
        super().__init__()
        from .hmc import spline_table
        self.L = N.load()
        self.patches = list(patches)
        self.n = len(self.patches)
        self.plan = Plan(self.patches, tile_pixels=tile_pixels)
        self.launch = self.plan.launch(ctas_per_sm=ctas_per_sm)
        dev = self.plan.device
        self.device = dev
        hp = np.zeros(self.n, dtype=N.hmc_patch_dtype)
        first = np.zeros(self.n, dtype=np.int32)
        off = nrow = 0
        self.slices, self.band_slices = [], []
        for i, p in enumerate(self.patches):
            ns, nb = int(p.n_sources), int(p.n_bands)
            nper = nb + NPARAMS - 1
            hp[i] = (off, ns, nb)
            first[i] = nrow
            self.slices.append(slice(off, off + ns * nper))
            self.band_slices.append(slice(nrow, nrow + nb))
            off += ns * nper
            nrow += nb
        self.n_params = off
        self.n_rows = nrow
        self.d_hp = to_device_bytes(hp, dev)
        self._h_rows, self._n_grads = result_rows(self.patches)
        self._rows = to_device_bytes(self._h_rows, dev)
        self._first_row = torch.from_numpy(first).to(dev)
        self._theta_buf = torch.zeros(max(off, 1), dtype=torch.float64, device=dev)
        self._jac_buf = torch.zeros(max(off, 1), dtype=torch.float64, device=dev)
        self.tab = spline_table(dev, splines)
        self.ncall = 0

    def _evaluate(self, theta):
        """Queue proposal construction and one evaluation at theta; returns
        (chi2 rows, their derivatives), as ``fp_fetch_results`` lays them out."""
        if theta.shape != (self.n_params,):
            raise ValueError("theta has shape %s, expected (%d,)" % (tuple(theta.shape), self.n_params))
        th = _in_memory(theta.to(device=self.device, dtype=torch.float64)).contiguous()
        s = current_stream_ptr()
        pl = self.plan
        N.check(self.L.fp_hmc_prepare(self.d_hp.data_ptr(), self.n, th.data_ptr(), None, None,
                                      ctypes.byref(self.tab), pl.proposals.data_ptr(),
                                      self._theta_buf.data_ptr(), self._jac_buf.data_ptr(), s), "fp_hmc_prepare")
        pl.evaluate(self.launch)
        self.ncall += 1
        chi2 = torch.empty(self.n_rows, dtype=torch.float64, device=self.device)
        grads = torch.empty(max(self._n_grads, 1), dtype=torch.float32, device=self.device)
        N.check(self.L.fp_fetch_results(pl.chi2.data_ptr(), pl.response.data_ptr(), self._rows.data_ptr(),
                                        self.n_rows, chi2.data_ptr(), grads.data_ptr(), s), "fp_fetch_results")
        return chi2, grads

    def _vjp(self, grad_chi2, grads):
        """theta gradient of sum_rows grad_chi2[row] * chi2[row], in one launch
        of 2 us (15 torch kernels over every slot took 40 us of the device and
        bound small patches by their launches)."""
        if grads.device != self.device or grads.shape != (max(self._n_grads, 1),):
            # only a saved-tensor hook can have changed them
            raise RuntimeError("the saved derivatives came back as %s on %s, expected [%d] on %s"
                               % (list(grads.shape), grads.device, max(self._n_grads, 1), self.device))
        if (torch.is_grad_enabled() and grad_chi2.requires_grad) or grads.dtype != torch.float32:
            return self._vjp_differentiable(grad_chi2, grads)
        g = _in_memory(grad_chi2.detach().to(torch.float64))
        grads = _in_memory(grads).contiguous()
        out = torch.empty(self.n_params, dtype=torch.float64, device=self.device)
        N.check(self.L.fp_chi2_vjp(self.d_hp.data_ptr(), self.n, self._rows.data_ptr(), self._first_row.data_ptr(),
                                   g.data_ptr(), g.stride(0), grads.data_ptr(), out.data_ptr(),
                                   current_stream_ptr()), "fp_chi2_vjp")
        return out

    def _vjp_differentiable(self, grad_chi2, grads):
        """The same product in torch operations, for a backward pass that is
        itself differentiated by grad_chi2 (create_graph), and for derivatives
        that a saved-tensor hook returned in another type."""
        i64 = dict(dtype=torch.int64, device=self.device)
        out = torch.zeros(self.n_params, dtype=torch.float64, device=self.device)
        for p, sl, rows in zip(self.patches, self.slices, self.band_slices):
            ns, nb = int(p.n_sources), int(p.n_bands)
            if ns == 0 or nb == 0:
                continue
            g0 = int(self._h_rows["grad_offset"][rows.start])
            r = grads[g0:g0 + nb * ns * NPARAMS].view(nb, ns, NPARAMS).to(torch.float64)
            g = grad_chi2[rows].to(torch.float64).view(nb, 1, 1)
            whole = torch.cat([(g[..., 0] * r[..., 0]).T, (g * r[..., 1:]).sum(dim=0)], dim=1)
            out = out.index_copy(0, torch.arange(sl.start, sl.stop, **i64), whole.reshape(-1))
        return out

    def forward(self, theta):
        return _Chi2Fn.apply(theta, self)

    def split(self, chi2):
        """Per-patch views of a chi2 row vector."""
        return [chi2[sl] for sl in self.band_slices]


class PatchChi2(BatchChi2):
    """Per-band chi2 of one device patch as a torch function of theta
    (float64[n_sources * (n_bands + 6)] -> float64[n_bands])."""

    def __init__(self, patch, tile_pixels=None, ctas_per_sm=4, splines=None):
        if tile_pixels is None:
            from .autotune import default_tile_pixels
            tile_pixels = default_tile_pixels(patch)
        super().__init__([patch], tile_pixels=tile_pixels, ctas_per_sm=ctas_per_sm, splines=splines)
        self.patch = patch
        self.scene = getattr(patch, "scene", None)
        self.n_sources = int(patch.n_sources)
        self.n_bands = patch.n_bands
