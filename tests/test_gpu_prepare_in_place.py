"""fp_hmc_prepare with theta written over z, with and without bounds: the
records, theta and Jacobian of the call with buffers of its own."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bounded", [False, True])
@pytest.mark.parametrize("bands", [1, 5, 30])                # 30: a source's parameters take two turns of a warp
def test_theta_over_z(bands, bounded):
    import torch
    from forcepho_b200 import _native as N
    from forcepho_b200.device import to_device_bytes
    from forcepho_b200.hmc import spline_table
    from forcepho_b200.structs import source_struct_dtype
    n_sources, nper = 7, bands + 6
    rng = np.random.default_rng(bands)
    lo = np.tile(np.r_[np.zeros(bands), -1.0, -1.0, 0.2, -2.0, 0.81, 0.03], n_sources)
    hi = np.tile(np.r_[np.full(bands, 9.0), 1.0, 1.0, 1.0, 2.0, 6.19, 0.6], n_sources)
    if bounded:
        start = rng.normal(0, 1, n_sources * nper)
    else:
        start = rng.uniform(lo, hi)
    dev = torch.device("cuda")
    hp = np.zeros(1, N.hmc_patch_dtype)
    hp[0] = (0, n_sources, bands)
    d_hp, tab = to_device_bytes(hp, dev), spline_table(dev)
    lower, upper = torch.tensor(lo, device=dev), torch.tensor(hi, device=dev)

    def prepare(in_place):
        z = torch.tensor(start, device=dev)
        theta, jac = z if in_place else torch.empty_like(z), torch.empty_like(z)
        rec = torch.zeros(30 * source_struct_dtype.itemsize, dtype=torch.uint8, device=dev)
        N.check(N.load().fp_hmc_prepare(d_hp.data_ptr(), 1, z.data_ptr(), lower.data_ptr() if bounded else None,
                                        upper.data_ptr() if bounded else None, ctypes.byref(tab), rec.data_ptr(),
                                        theta.data_ptr(), jac.data_ptr(),
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "fp_hmc_prepare")
        return rec.cpu().numpy(), theta.cpu().numpy(), jac.cpu().numpy()

    for got, want in zip(prepare(True), prepare(False)):
        np.testing.assert_array_equal(got, want)
