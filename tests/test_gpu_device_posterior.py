"""The warp-per-source proposal construction against the host splines, at the
edges of the knot range, and the one-launch vector-Jacobian product of the band
chi2s against the same sum in torch, with every kind of upstream gradient."""

import ctypes

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


@pytest.mark.parametrize("n_sources,bands", [(1, 1), (2, 3), (30, 30)])
def test_prepare_matches_host_splines(n_sources, bands):
    """f32 records of the host's FP64 amplitudes: two FP64 evaluations of one
    spline differ by far less than the records' rounding, so by at most one unit
    of it (and 1e-12 of the largest amplitude where they cancel)."""
    import torch
    from forcepho_b200 import _native as N
    from forcepho_b200.device import to_device_bytes
    from forcepho_b200.hmc import spline_table
    from forcepho_b200.structs import source_struct_dtype
    p = make(n_sources, bands, 3)
    rng = np.random.default_rng(n_sources)
    sp = p.splines
    for i, g in enumerate(p.scene.sources):
        g.sersic = rng.uniform(*sp.sersic_range)
        g.rhalf = rng.uniform(*sp.rh_range)
        if i % 5 == 1:      # the ends of the knots, and past them (both clamp)
            g.sersic, g.rhalf = sp.sersic_range[i % 2], sp.rh_range[(i // 2) % 2]
        if i % 5 == 2:
            g.sersic, g.rhalf = sp.sersic_range[1] + 1, sp.rh_range[0] - 0.01
    want = p.scene.get_proposal()
    theta = torch.from_numpy(p.scene.get_all_source_params()).cuda()
    hp = np.zeros(1, N.hmc_patch_dtype)
    hp[0] = (0, n_sources, bands)
    d_hp, tab = to_device_bytes(hp, theta.device), spline_table(theta.device)
    rec = torch.zeros(30 * source_struct_dtype.itemsize, dtype=torch.uint8, device="cuda")
    th, jac = torch.empty_like(theta), torch.empty_like(theta)
    N.check(N.load().fp_hmc_prepare(d_hp.data_ptr(), 1, theta.data_ptr(), None, None, ctypes.byref(tab),
                                    rec.data_ptr(), th.data_ptr(), jac.data_ptr(),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "fp_hmc_prepare")
    got = rec.cpu().numpy().view(source_struct_dtype)[:n_sources]
    assert torch.equal(th, theta) and torch.equal(jac, torch.ones_like(jac))
    for name in ("ra", "dec", "q", "pa", "nsersic", "rh", "fluxes"):
        assert np.array_equal(got[name], want[name]), name
    for name in ("mixture_amplitudes", "damplitude_drh", "damplitude_dnsersic"):
        a, b = got[name].astype(np.float64), want[name].astype(np.float64)
        assert np.all(np.abs(a - b) <= np.spacing(np.abs(want[name])) + 1e-12 * np.abs(b).max()), name


def test_vjp_kernel():
    import torch
    from forcepho_b200.autograd import BatchChi2
    f = BatchChi2([make(ns, nb, 7 * ns + nb) for ns, nb in ((3, 2), (1, 5), (30, 1), (4, 30))], tile_pixels=256)
    theta = torch.cat([torch.from_numpy(p.scene.get_all_source_params()) for p in f.patches]).cuda()
    _, grads = f._evaluate(theta)
    rng = torch.Generator(device="cuda").manual_seed(1)
    w = torch.randn(f.n_rows, dtype=torch.float64, device="cuda", generator=rng)
    wide = torch.randn(2 * f.n_rows, dtype=torch.float64, device="cuda", generator=rng)
    for g in (w, wide[::2], w[:1].expand(f.n_rows), w.float()):
        got = f._vjp(g, grads)
        want = f._vjp_differentiable(g, grads)
        # FP64 sums of at most 30 terms in two orders
        assert torch.all((got - want).abs() <= 1e-13 * f._vjp_differentiable(g.abs(), grads.abs()))


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_backward_of_the_backward(dtype):
    """create_graph: the gradient is linear in the upstream weights, so its
    derivative by them is the Jacobian applied to the cotangent."""
    import torch
    from forcepho_b200.autograd import BatchChi2
    f = BatchChi2([make(2, 3, 1), make(1, 2, 2)], tile_pixels=256)
    theta = torch.cat([torch.from_numpy(p.scene.get_all_source_params()) for p in f.patches]).cuda()
    theta = theta.to(getattr(torch, dtype)).requires_grad_(True)
    v = torch.ones(f.n_rows, dtype=torch.float64, device="cuda", requires_grad=True)
    (g,) = torch.autograd.grad(f(theta), theta, v, create_graph=True)
    (plain,) = torch.autograd.grad(f(theta), theta, v.detach())
    # float32 rounds both once; the sums themselves are FP64
    assert torch.allclose(g, plain, rtol=1e-6 if dtype == "float32" else 1e-12, atol=0)
    u = torch.linspace(-1, 1, len(theta), dtype=theta.dtype, device="cuda")
    (jvp,) = torch.autograd.grad(g, v, u)
    rows = [torch.autograd.grad(f(theta)[i], theta)[0].double() @ u.double() for i in range(f.n_rows)]
    scale = torch.stack([torch.autograd.grad(f(theta)[i], theta)[0].double().abs() @ u.double().abs()
                         for i in range(f.n_rows)])
    assert torch.all((jvp - torch.stack(rows)).abs() <= 1e-6 * scale)
