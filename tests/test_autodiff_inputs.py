"""What reaches the differentiable chi2's backward kernel by address: upstream
gradients of every stride, with a pending sign or without storage, and saved
derivatives that a hook has moved, converted or cut.  On the CPU the kernel is
a stand-in that reads the addresses it is given, and only those of whole float32
buffers; on the GPU the same forms go through the kernel."""

import ctypes

import numpy as np
import pytest
import torch

from forcepho_b200 import autograd
from forcepho_b200 import _native as N
from forcepho_b200.device import result_rows
from forcepho_b200.kernel_limits import NPARAMS

SHAPES = ((2, 3), (0, 1), (1, 2))            # (sources, bands) of each patch
ROWS = sum(nb for _, nb in SHAPES)


class Patch:
    def __init__(self, ns, nb):
        self.n_sources, self.n_bands = ns, nb


def expected(grads, g):
    """The product, written out."""
    out, at, row = [], 0, 0
    for ns, nb in SHAPES:
        d = np.asarray(grads[at:at + nb * ns * NPARAMS], np.float64).reshape(nb, ns, NPARAMS)
        w = np.asarray(g[row:row + nb], np.float64)[:, None]
        for s in range(ns):
            out += list(w[:, 0] * d[:, s, 0]) + list((w * d[:, s, 1:]).sum(0))
        at, row = at + nb * ns * NPARAMS, row + nb
    return np.array(out)


class Kernel:
    """Stands for the library's fp_chi2_vjp."""

    def __init__(self, n_grads):
        self.n_grads, self.buffers = n_grads, []

    def fp_chi2_vjp(self, hp, n, rows, first, g, g_stride, grads, out, stream):
        known = [t for t in self.buffers if t.data_ptr() == grads and t.dtype == torch.float32 and t.is_contiguous()
                 and t.numel() == self.n_grads]
        if not g or not known:
            return 1
        up = [ctypes.c_double.from_address(g + 8 * g_stride * i).value for i in range(ROWS)]
        d = np.ctypeslib.as_array((ctypes.c_float * self.n_grads).from_address(grads))
        want = expected(d, up)
        np.ctypeslib.as_array((ctypes.c_double * len(want)).from_address(out))[:] = want
        return 0

    @staticmethod
    def fp_error_string():
        return b"not a buffer of the call"


@pytest.fixture
def chi2(monkeypatch):
    monkeypatch.setattr(autograd, "current_stream_ptr", lambda: None)
    f = autograd.BatchChi2.__new__(autograd.BatchChi2)
    torch.nn.Module.__init__(f)
    f.patches = [Patch(*s) for s in SHAPES]
    f.n, f.device, f.n_rows = len(SHAPES), torch.device("cpu"), ROWS
    f.slices, f.band_slices, off, row = [], [], 0, 0
    for ns, nb in SHAPES:
        size = ns * (nb + NPARAMS - 1)
        f.slices.append(slice(off, off + size))
        f.band_slices.append(slice(row, row + nb))
        off, row = off + size, row + nb
    f.n_params = off
    f._h_rows, f._n_grads = result_rows(f.patches)
    f.d_hp = f._rows = f._first_row = torch.zeros(1)
    f.L = Kernel(f._n_grads)
    f.grads = torch.randn(f._n_grads, generator=torch.Generator().manual_seed(1))
    f.L.buffers.append(f.grads)
    f._evaluate = lambda theta: (torch.arange(ROWS, dtype=torch.float64), f.grads)
    return f


def upstream(kind, device="cpu"):
    v = torch.linspace(-1.5, 2.0, ROWS, dtype=torch.float64, device=device)
    if kind == "expanded":
        return torch.tensor(0.75, dtype=torch.float64, device=device).expand(ROWS)
    if kind == "strided":
        return torch.stack([v, -v], 1).reshape(-1)[::2]
    if kind == "negated":
        return torch.complex(torch.zeros_like(v), v).conj().imag
    if kind == "zero":
        return torch._efficientzerotensor((ROWS,), dtype=torch.float64, device=device)
    return v


KINDS = ["plain", "expanded", "strided", "negated", "zero"]


@pytest.mark.parametrize("kind", KINDS)
def test_upstream_gradients(chi2, kind):
    g = upstream(kind)
    theta = torch.zeros(chi2.n_params, dtype=torch.float64, requires_grad=True)
    chi2(theta).backward(g)
    np.testing.assert_allclose(theta.grad, expected(chi2.grads, (g + 0).tolist()), rtol=1e-15)


def moved(t):
    return t.clone()


def strided(t):
    return torch.stack([t, t], 1)[:, 0]


def half(t):
    return t.half()


def double(t):
    return t.double()


def short(t):
    return t[:-1]


def elsewhere(t):
    return t.to("meta")


@pytest.mark.parametrize("change", [moved, strided, half, double], ids=lambda f: f.__name__)
def test_saved_derivatives_in_another_form(chi2, change):
    g = upstream("plain")

    def unpack(t):
        chi2.L.buffers.append(t)
        return t

    contiguous = torch.Tensor.contiguous

    def kept(t):
        chi2.L.buffers.append(contiguous(t))
        return chi2.L.buffers[-1]

    with pytest.MonkeyPatch.context() as m, torch.autograd.graph.saved_tensors_hooks(change, unpack):
        m.setattr(torch.Tensor, "contiguous", kept)
        theta = torch.zeros(chi2.n_params, dtype=torch.float64, requires_grad=True)
        chi2(theta).backward(g)
    np.testing.assert_allclose(theta.grad, expected(change(chi2.grads), g.tolist()), rtol=1e-14)


@pytest.mark.parametrize("change", [short, elsewhere], ids=lambda f: f.__name__)
def test_saved_derivatives_that_do_not_fit(chi2, change):
    theta = torch.zeros(chi2.n_params, dtype=torch.float64, requires_grad=True)
    with torch.autograd.graph.saved_tensors_hooks(change, lambda t: t):
        out = chi2(theta)
    with pytest.raises(RuntimeError, match="saved derivatives"):
        out.backward(upstream("plain"))


def test_batched_gradients_stay_refused(chi2):
    theta = torch.zeros(chi2.n_params, dtype=torch.float64, requires_grad=True)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(chi2(theta), theta, torch.eye(ROWS, dtype=torch.float64), is_grads_batched=True)


@pytest.mark.gpu
def test_the_same_forms_on_the_device():
    from forcepho_b200 import synthetic as S
    rng = np.random.default_rng(3)
    patches = []
    for ns, nb in SHAPES:
        p = S.make_patch(rng, n_sources=ns, exp_per_band=[1] * nb, exp_pix=[(24, 20)] * nb, n_psf=1,
                         source_params=S._broad_source)
        S.add_noise(p, rng, 1.0)
        p.return_residual = False
        p.send_to_device()
        patches.append(p)
    f = autograd.BatchChi2(patches, tile_pixels=256)
    th = np.concatenate([p.scene.get_all_source_params() for p in patches if int(p.n_sources)])
    theta = torch.tensor(th, dtype=torch.float64, device="cuda", requires_grad=True)

    def gradient(t, g, pack=None, unpack=None):
        t.grad = None
        if pack is None:
            f(t).backward(g)
        else:
            with torch.autograd.graph.saved_tensors_hooks(pack, unpack or (lambda x: x)):
                f(t).backward(g)
        return t.grad.cpu().numpy()

    with torch.no_grad():
        grads = f._evaluate(theta)[1].cpu()
    for kind in KINDS:
        g = upstream(kind, "cuda")
        np.testing.assert_allclose(gradient(theta, g), expected(grads, (g + 0).tolist()), rtol=1e-13, atol=1e-300)
    g = upstream("plain", "cuda")
    want = gradient(theta, g)
    np.testing.assert_array_equal(gradient(theta, g, lambda t: t.cpu(), lambda t: t.cuda()), want)
    np.testing.assert_allclose(gradient(theta, g, lambda t: t.double()), want, rtol=1e-13)
    with pytest.raises(RuntimeError, match="saved derivatives"):
        gradient(theta, g, lambda t: t.cpu())
    negated = torch.complex(torch.zeros_like(theta.detach()), -theta.detach()).conj().imag
    np.testing.assert_array_equal(gradient(negated.requires_grad_(), g), want)
