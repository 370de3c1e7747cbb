"""Workloads that stand for what users of this framework have it do.

Every case goes through the public calls a program makes: the proposers, the
batched proposer, the reference's kernel ABI, the differentiable chi2, renders,
the linear flux solve and the device sampler, on synthetic patches of the
repository's own generator (pixel scale, PSF mixtures, source and noise
distributions of its workloads).  Data are a model of the scene plus noise;
the model is rendered here in 64 bits with torch, so that inputs depend on the
seed alone.

A case is a dict with

``kind``      which call: proposer, abi, batch, chi2, render, fluxes, hmc
``sources``   sources of a patch (the upper end of 1..sources in a batch)
``bands``, ``exposures``   bands, and exposures of each band (upper ends in a batch)
``width``, ``height``      pixels of an exposure (in a batch, exposures are the
              first n pixels of a ``width`` wide raster, n up to width x height)
``psf``       Gaussians of the PSF mixture; each is convolved with 9 radii
``patches``   patches of the call
and, where they apply, ``residual`` (the residual image comes back too) and
``steps`` (leapfrog steps of the trajectory).
"""

import ctypes
import math

import numpy as np
import torch

from forcepho_b200 import _native, synthetic
from forcepho_b200.autograd import BatchChi2, PatchChi2
from forcepho_b200.batch import BatchedProposer
from forcepho_b200.fitting import optimize_fluxes
from forcepho_b200.hmc import DeviceHMC
from forcepho_b200.kernel_limits import MAXSOURCES, NPARAMS
from forcepho_b200.proposal import B200Proposer
from forcepho_b200.splines import default_splines
from forcepho_b200.structs import source_struct_dtype

RADII = 9                 # Sersic mixture radii
CUTOFF = 36.0             # Gaussians end at dx^T F dx = 36
WITHIN = 0.22             # share of a patch's (pixel, Gaussian) pairs inside that, on the 512-patch workload
PAIR_FLOPS = 84           # of a value and its gradient; 21 of a value alone
VALUE_FLOPS = 21


def listed():
    return [
        # the smallest call: one source on a 64x64 stamp, where latency is all
        dict(name="proposer_stamp", kind="proposer", sources=1, bands=1, exposures=1, width=64, height=64, psf=3,
             patches=1, residual=False),
        # an odd-sized cutout whose residual image is looked at after the fit
        dict(name="proposer_odd_residual", kind="proposer", sources=5, bands=3, exposures=2, width=97, height=113,
             psf=3, patches=1, residual=True),
        # an ordinary patch of the host sampler: 16 sources, 5 bands x 2 exposures of 150x150 px
        dict(name="proposer_multiband", kind="proposer", sources=16, bands=5, exposures=2, width=150, height=150,
             psf=4, patches=1, residual=False),
        # a patch at the kernel's limits: 30 sources, 8 bands x 4 exposures of 256x256 px, 6-Gaussian PSFs
        dict(name="proposer_limits", kind="proposer", sources=30, bands=8, exposures=4, width=256, height=256,
             psf=6, patches=1, residual=False),
        # the reference's own kernel arguments, from a binding that holds device pointers
        dict(name="abi_patch", kind="abi", sources=8, bands=4, exposures=2, width=120, height=120, psf=4, patches=1),
        # many small stamps at once, as a survey of isolated galaxies has them
        dict(name="batch_stamps", kind="batch", sources=4, bands=3, exposures=2, width=64, height=64, psf=3,
             patches=128),
        # the uneven field patches of the batched benchmark
        dict(name="batch_field", kind="batch", sources=30, bands=8, exposures=4, width=256, height=256, psf=4,
             patches=48),
        # chi2 as a torch function, forward and backward: one patch of an optimiser
        dict(name="chi2_patch", kind="chi2", sources=12, bands=4, exposures=2, width=100, height=130, psf=4,
             patches=1),
        # the same over a batch of uneven patches
        dict(name="chi2_batch", kind="chi2", sources=16, bands=5, exposures=2, width=160, height=160, psf=4,
             patches=24),
        # model images of a catalog (forward only), planned anew for each scene as the call does
        dict(name="render_scene", kind="render", sources=15, bands=5, exposures=2, width=150, height=150, psf=4,
             patches=1),
        # maximum-likelihood fluxes of a scene at fixed shapes
        dict(name="flux_fit", kind="fluxes", sources=10, bands=4, exposures=2, width=128, height=128, psf=4,
             patches=1),
        # one sampler trajectory of patches at the limits
        dict(name="hmc_limits", kind="hmc", sources=30, bands=8, exposures=4, width=256, height=256, psf=6,
             patches=2, steps=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["proposer", "proposer", "proposer", "abi", "batch", "batch", "chi2", "render", "fluxes", "hmc"])
    c = dict(kind=kind, sources=_log(rng, 1, 30), bands=_log(rng, 1, 8), exposures=rng.randint(1, 4),
             width=_log(rng, 32, 256), height=_log(rng, 32, 256), psf=rng.randint(2, 6), patches=1)
    if kind == "proposer":
        c["residual"] = rng.random() < 0.3
    elif kind == "batch":
        c["patches"] = _log(rng, 4, 48)
    elif kind == "chi2":
        c["patches"] = _log(rng, 1, 16)
    elif kind in ("render", "fluxes"):
        c["sources"] = _log(rng, 2, 15)
        c["width"], c["height"] = min(c["width"], 160), min(c["height"], 160)
    elif kind == "hmc":
        c["patches"], c["steps"] = rng.randint(1, 2), rng.randint(4, 16)
    return c


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _shape(case, i):
    """Sources, exposures per band, and each exposure's pixels, of patch i: the field's layout, the same for every seed."""
    if case["kind"] in ("batch", "chi2") and case["patches"] > 1:
        rng = np.random.default_rng([4, i])
        ns = int(rng.integers(1, case["sources"] + 1))
        epb = [int(v) for v in rng.integers(1, case["exposures"] + 1, int(rng.integers(1, case["bands"] + 1)))]
        most = case["width"] * case["height"]
        return ns, epb, [int(v) for v in rng.integers(max(most // 64, 512), most + 1, sum(epb))], case["width"]
    epb = [case["exposures"]] * case["bands"]
    return case["sources"], epb, [(case["width"], case["height"])] * sum(epb), None


def _patches(case, seed):
    """The case's patches (host) and a proposal of each, a little off the truth."""
    out = []
    for i in range(case["patches"]):
        rng = np.random.default_rng([int(seed), i])
        ns, epb, pix, raster = _shape(case, i)
        p = synthetic.make_patch(rng, n_sources=ns, exp_per_band=epb, exp_pix=pix, n_psf=case["psf"],
                                 source_params=synthetic._broad_source, raster_width=raster)
        truth = _parameters(p)
        model = np.zeros(p.npix, np.float32)
        for b, e, sl in _exposures(p):
            model[sl] = _exposure(p, truth, b, e)["model"].float().cpu().numpy()
        synthetic.add_noise(p, rng, rng.uniform(0.5, 2.0, p.n_exp), model)
        theta = _theta(p)
        theta[:, -6:-4] += rng.normal(0, 2e-6, (ns, 2))
        theta[:, -4] = np.clip(theta[:, -4] * rng.uniform(0.95, 1.05, ns), 0.2, 0.99)
        out.append((p, theta.astype(np.float32)))
    return out


def _theta(p):
    """The scene's parameters, a row for each source: fluxes, ra, dec, q, pa, sersic, rhalf."""
    return np.array([np.concatenate([g.flux, [g.ra, g.dec, g.q, g.pa, g.sersic, g.rhalf]]) for g in p.scene.sources])


def _proposal(p, theta):
    """The source records of a parameter table, as a host program packs them."""
    p.scene.set_all_source_params(theta.reshape(-1))
    return p.scene.get_proposal().copy()


def prepare(case, seed):
    kind = case["kind"]
    made = _patches(case, seed)
    patches = [p for p, _ in made]
    for p in patches:
        p.return_residual = bool(case.get("residual", False))
    if kind in ("render", "fluxes"):
        catalog = patches[0].catalog()
        patches[0].send_to_device()
        return dict(kind=kind, patch=patches[0], catalog=catalog)
    thetas = [t for _, t in made]
    for p in patches:
        p.send_to_device()
    if kind == "proposer":
        return dict(kind=kind, patch=patches[0], proposal=_proposal(patches[0], thetas[0]), proposer=B200Proposer())
    if kind == "abi":
        p, dev = patches[0], patches[0].device_patch.device
        rec = torch.from_numpy(_proposal(p, thetas[0]).view(np.uint8).copy()).to(dev)
        return dict(kind=kind, patch=p, lib=_native.load(), records=rec,
                    chi2=torch.zeros(p.n_bands, dtype=torch.float64, device=dev),
                    response=torch.zeros((p.n_bands, MAXSOURCES, NPARAMS), dtype=torch.float32, device=dev))
    if kind == "batch":
        return dict(kind=kind, proposer=BatchedProposer(patches),
                    proposals=[_proposal(p, t) for p, t in zip(patches, thetas)])
    if kind == "chi2":
        f = PatchChi2(patches[0]) if len(patches) == 1 else BatchChi2(patches)
        theta = torch.from_numpy(np.concatenate([t.reshape(-1) for t in thetas])).to(f.device)
        return dict(kind=kind, f=f, theta=theta.requires_grad_(True))
    # a step size small enough for unit masses: the chain moves and is accepted
    hmc = DeviceHMC(patches, [t.astype(np.float64).reshape(-1) for t in thetas], n_steps=case["steps"], max_traj=1024,
                    seed=int(seed), step_size=1e-3)
    return dict(kind=kind, hmc=hmc, done=0)


# --------------------------------------------------------------------------
# the calls
# --------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "proposer":
        return state["proposer"].evaluate_proposal(state["proposal"], patch=state["patch"])
    if kind == "abi":
        p = state["patch"]
        rc = state["lib"].fp_evaluate_proposal(
            p.device_patch_ptr, state["records"].data_ptr(), int(p.n_sources), p.n_bands, state["chi2"].data_ptr(),
            state["response"].data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(state["lib"].fp_error_string().decode())
        return state["chi2"], state["response"]
    if kind == "batch":
        results = state["proposer"].evaluate_proposals(state["proposals"])
        return (np.concatenate([c for c, _ in results]), np.concatenate([d.reshape(-1) for _, d in results]))
    if kind == "chi2":
        theta = state["theta"]
        theta.grad = None
        chi2 = state["f"](theta)
        (-0.5 * chi2.sum()).backward()
        return chi2.detach(), theta.grad
    if kind == "render":
        return state["patch"].render(state["catalog"])
    if kind == "fluxes":
        fluxes, precisions = optimize_fluxes(state["patch"], state["catalog"])
        return np.array(fluxes), np.array(precisions)
    hmc = state["hmc"]
    if state["done"] == hmc.max_traj:          # the drawn momenta begin again
        hmc.traj.zero_()
        state["done"] = 0
    hmc.run(1)
    state["done"] += 1
    records = hmc.proposals()                  # the draw, as the source records of its last position
    return records.view(np.float32), hmc.accepted


def work(case):
    kind, ns, nb, ne = case["kind"], case["sources"], case["bands"], case["bands"] * case["exposures"]
    npix = ne * case["width"] * case["height"] * case["patches"]
    if kind in ("batch", "chi2") and case["patches"] > 1:       # uniform draws up to these
        ns, nb, ne = (1 + ns) / 2, (1 + nb) / 2, (1 + nb) / 2 * (1 + case["exposures"]) / 2
        npix = ne * case["width"] * case["height"] * (1 + 1 / 64) / 2 * case["patches"]
    pairs = npix * ns * RADII * case["psf"] * WITHIN
    records = case["patches"] * ns * source_struct_dtype.itemsize
    results = case["patches"] * nb * (8 + 4 * NPARAMS * ns)
    if kind in ("render", "fluxes"):
        # pixel positions in and models out; the solve reads data and errors instead and writes n x n per band
        moved = 8 * npix + (4 * npix if kind == "render" else 8 * npix + 8 * nb * ns * (ns + 1))
        normal = 2 * npix * ns * (ns + 1) if kind == "fluxes" else 0
        return {"bytes": int(moved + records), "flops": int(VALUE_FLOPS * pairs + normal)}
    moved = 16 * npix + records + results + (4 * npix if case.get("residual") else 0)
    times = case.get("steps", 1)
    return {"bytes": int(moved * times), "flops": int(PAIR_FLOPS * pairs * times)}


# --------------------------------------------------------------------------
# the same in 64 bits, with torch and numpy alone
# --------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _f64(a):
    return torch.tensor(np.asarray(a, np.float64), device=_device())


def _exposures(p):
    """(band, exposure, its pixels) in order."""
    for b in range(p.n_bands):
        for e in range(int(p.band_start[b]), int(p.band_start[b]) + int(p.band_N[b])):
            s = int(p.exposure_start[e])
            yield b, e, slice(s, s + int(p.exposure_N[e]))


def _basis(t, k, x):
    """The B-splines of degree k on the knots t at x, and their derivatives (Cox and de Boor)."""
    n = len(t) - k - 1
    x = min(max(float(x), t[k]), t[n])
    last = max(i for i in range(k, n) if t[i] <= x)
    b = [np.array([1.0 if i == last else 0.0 for i in range(len(t) - 1)])]
    for d in range(1, k + 1):
        c = np.zeros(len(t) - 1 - d)
        for i in range(len(c)):
            if t[i + d] > t[i]:
                c[i] += (x - t[i]) / (t[i + d] - t[i]) * b[-1][i]
            if t[i + d + 1] > t[i + 1]:
                c[i] += (t[i + d + 1] - x) / (t[i + d + 1] - t[i + 1]) * b[-1][i + 1]
        b.append(c)
    der = np.zeros(n)
    for i in range(n):
        if t[i + k] > t[i]:
            der[i] += k / (t[i + k] - t[i]) * b[-2][i]
        if t[i + k + 1] > t[i + 1]:
            der[i] -= k / (t[i + k + 1] - t[i + 1]) * b[-2][i + 1]
    return b[-1], der


def _parameters(p, theta=None):
    """Differentiable 64-bit parameters of a scene, with the mixture amplitudes to first order in sersic and rhalf."""
    theta = np.asarray(_theta(p) if theta is None else theta, np.float64)
    tx, ty, c, kx, ky = default_splines().tck()
    c = np.asarray(c).reshape(len(c), len(tx) - kx - 1, len(ty) - ky - 1)
    value, by_n, by_r = [], [], []
    for row in theta:
        (bx, dx), (by, dy) = _basis(tx, kx, row[-2]), _basis(ty, ky, row[-1])
        value.append(np.einsum("rij,i,j->r", c, bx, by))
        by_n.append(np.einsum("rij,i,j->r", c, dx, by))
        by_r.append(np.einsum("rij,i,j->r", c, bx, dy))
    leaf = _f64(theta).requires_grad_(True)
    held = leaf.detach()
    amplitude = (_f64(value) + _f64(by_n) * (leaf[:, -2:-1] - held[:, -2:-1])
                 + _f64(by_r) * (leaf[:, -1:] - held[:, -1:]))
    return dict(leaf=leaf, amplitude=amplitude)


def _gaussians(p, par, band, e):
    """Amplitude, centre and inverse covariance of every image Gaussian of an exposure, by source and PSF component."""
    leaf, n = par["leaf"], int(p.n_psf_per_source[band])
    ns = leaf.shape[0]
    first = int(p.psfgauss_start[e])
    psf = p.psfgauss[first:first + n]
    radius = torch.tensor(psf["sersic_bin"].astype(np.int64), device=_device())
    flux, (ra, dec, q, pa) = leaf[:, band], leaf[:, -6:-2].unbind(1)
    D, CW = _f64(p.D).reshape(-1, ns, 2, 2)[e], _f64(p.CW).reshape(-1, ns, 2, 2)[e]
    crpix, crval = _f64(p.crpix).reshape(-1, ns, 2)[e], _f64(p.crval).reshape(-1, ns, 2)[e]
    turn = torch.stack([torch.cos(pa), -torch.sin(pa), torch.sin(pa), torch.cos(pa)], 1).reshape(ns, 2, 2)
    T = D @ turn * torch.stack([1 / q, q], 1)[:, None, :]
    TT = T @ T.transpose(1, 2)
    centre = (CW @ (torch.stack([ra, dec], 1) - crval)[:, :, None])[:, :, 0] + crpix
    r2 = _f64(p.rad2)[radius]
    sxx = r2 * TT[:, 0, 0, None] + _f64(psf["Cxx"])
    sxy = r2 * TT[:, 0, 1, None] + _f64(psf["Cxy"])
    syy = r2 * TT[:, 1, 1, None] + _f64(psf["Cyy"])
    det = sxx * syy - sxy * sxy
    amp = (float(p.G[e]) * _f64(psf["amp"]) * flux[:, None] * par["amplitude"][:, radius]
           / (2 * math.pi * torch.sqrt(det)))
    return (amp, centre[:, :1] + _f64(psf["xcen"]), centre[:, 1:] + _f64(psf["ycen"]), syy / det, -sxy / det,
            sxx / det)


def _exposure(p, par, band, e, gradient=False, by_source=False):
    """An exposure's model, and chi2 with its gradient by the parameters where that is asked for."""
    image = _gaussians(p, par, band, e)
    ns = image[0].shape[0]
    A, xc, yc, fxx, fxy, fyy = (g.detach().expand(ns, -1).reshape(1, -1) for g in image)
    s = slice(int(p.exposure_start[e]), int(p.exposure_start[e]) + int(p.exposure_N[e]))
    x, y = _f64(p.xpix[s])[:, None], _f64(p.ypix[s])[:, None]
    d, ierr = _f64(p.data[s]), _f64(p.ierr[s])
    total = [torch.zeros_like(A[0]) for _ in range(6)]
    model, chi2 = [], 0.0
    rows = max(1, (1 << 22) // max(1, A.numel()))
    for i in range(0, x.shape[0], rows):
        j = slice(i, i + rows)
        dx, dy = x[j] - xc, y[j] - yc
        vx, vy = fxx * dx + fxy * dy, fxy * dx + fyy * dy
        E = dx * vx + dy * vy
        g = torch.where(E > CUTOFF, 0.0, torch.exp(-0.5 * E))
        h = 1 + (vx * vx + vy * vy - fxx - fyy) / 24
        counts = A * g * h
        model.append(counts.reshape(-1, ns, A.numel() // max(ns, 1)).sum(2) if by_source else counts.sum(1))
        if not gradient:
            continue
        r = d[j] - model[-1]
        chi2 = chi2 + float(((r * r - d[j] * d[j]) * ierr[j] ** 2).sum())
        k = (-2 * r * ierr[j] ** 2)[:, None] * g
        c = k * A
        for t, v in zip(total, (k * h, c * (h * vx - (fxx * vx + fxy * vy) / 12),
                                c * (h * vy - (fyy * vy + fxy * vx) / 12),
                                -c * (0.5 * h * dx * dx + (1 - 2 * dx * vx) / 24),
                                -c * (h * dx * dy - (dy * vx + dx * vy) / 12),
                                -c * (0.5 * h * dy * dy + (1 - 2 * dy * vy) / 24))):
            t += v.sum(0)
    out = dict(model=torch.cat(model).detach())
    if gradient:
        out["chi2"] = chi2
        full = [g.expand(ns, -1) for g in image]
        out["grad"] = torch.autograd.grad(full, par["leaf"], [t.reshape(full[0].shape) for t in total],
                                          retain_graph=True)[0]
    return out


def _evaluate(p, theta):
    """Per band chi2 and its gradient by (flux of the band, ra, dec, q, pa, sersic, rhalf) of each source, and the residual."""
    par = _parameters(p, theta)
    chi2, grad = np.zeros(p.n_bands), np.zeros((p.n_bands, len(theta), NPARAMS))
    residual = []
    for b, e, sl in _exposures(p):
        r = _exposure(p, par, b, e, gradient=True)
        chi2[b] += r["chi2"]
        g = r["grad"].cpu().numpy()
        grad[b] += np.concatenate([g[:, b:b + 1], g[:, -6:]], 1)
        residual.append(p.data[sl].astype(np.float64) - r["model"].cpu().numpy())
    return chi2, grad, residual


def exact(case, seed):
    kind = case["kind"]
    if kind == "hmc":
        return None            # every step is a gradient of all pairs: minutes in 64 bits
    made = _patches(case, seed)
    if kind in ("render", "fluxes"):
        p = made[0][0]
        par = _parameters(p)
        if kind == "render":
            return [_exposure(p, par, b, e)["model"].cpu().numpy() for b, e, _ in _exposures(p)]
        normal = [[0.0, 0.0] for _ in range(p.n_bands)]
        for b, e, sl in _exposures(p):
            w = _f64(p.ierr[sl])
            X = _exposure(p, par, b, e, by_source=True)["model"].T / par["leaf"].detach()[:, b:b + 1] * w
            normal[b][0] = normal[b][0] + X @ X.T
            normal[b][1] = normal[b][1] + X @ (_f64(p.data[sl]) * w)
        return (np.array([np.linalg.solve(a.cpu().numpy(), v.cpu().numpy()) for a, v in normal]),
                np.array([a.cpu().numpy() for a, _ in normal]))
    results = [_evaluate(p, t) for p, t in made]
    if kind == "proposer":
        chi2, grad, residual = results[0]
        return (chi2, grad, residual) if case["residual"] else (chi2, grad)
    if kind == "abi":
        chi2, grad, _ = results[0]
        response = np.zeros((len(chi2), MAXSOURCES, NPARAMS))
        response[:, :grad.shape[1]] = grad
        return chi2, response
    if kind == "batch":
        return (np.concatenate([c for c, _, _ in results]), np.concatenate([g.reshape(-1) for _, g, _ in results]))
    whole = []                 # d(-chi2 / 2) / dtheta
    for _, g, _ in results:
        whole.append(-0.5 * np.concatenate([g[:, :, 0].T, g[:, :, 1:].sum(0)], 1).reshape(-1))
    return np.concatenate([c for c, _, _ in results]), np.concatenate(whole)
