"""fp_evaluate_proposal from several threads: work queued on one caller's stream
holds up no other caller, and calls that run side by side give the results of
single ones."""

import ctypes
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Caller:
    """A patch, a stream and the call's buffers."""

    def __init__(self, seed):
        import torch
        from forcepho_b200 import _native as N
        from forcepho_b200 import synthetic as S
        from forcepho_b200.kernel_limits import MAXSOURCES, NPARAMS
        self.L = N.load()
        self.p = S.config_multiband(seed=seed, n_sources=3, n_bands=2, exp_per_band=2, size=40)
        self.p.return_residual = False
        self.p.send_to_device()
        self.prop = torch.from_numpy(self.p.scene.get_proposal().view(np.uint8).copy()).cuda()
        self.chi2 = torch.zeros(2, dtype=torch.float64, device="cuda")
        self.resp = torch.zeros((2, MAXSOURCES * NPARAMS), dtype=torch.float32, device="cuda")
        self.stream = torch.cuda.Stream()
        torch.cuda.synchronize()

    def call(self):
        assert self.L.fp_evaluate_proposal(
            self.p.device_patch_ptr, self.prop.data_ptr(), 3, 2, self.chi2.data_ptr(), self.resp.data_ptr(),
            ctypes.c_void_p(self.stream.cuda_stream)) == 0, self.L.fp_error_string()

    def result(self):
        self.stream.synchronize()
        return self.chi2.cpu().numpy(), self.resp.cpu().numpy()


def test_a_busy_stream_holds_up_no_other_thread():
    import torch
    a, b = Caller(1), Caller(2)
    a.call()
    b.call()                                    # both plans made
    torch.cuda.synchronize()
    with torch.cuda.stream(a.stream):
        torch.cuda._sleep(1_500_000_000)        # most of a second
    busy = torch.cuda.Event()
    busy.record(a.stream)
    t = threading.Thread(target=a.call)
    t.start()
    time.sleep(0.1)                             # into its wait
    b.call()
    b.stream.synchronize()
    assert not busy.query()
    t.join()
    a.stream.synchronize()


def test_calls_side_by_side():
    callers = [Caller(10 + i) for i in range(12)]           # more than the landing places kept
    want = []
    for c in callers:
        c.call()
        want.append(c.result())
        c.chi2.zero_()
        c.resp.zero_()

    def repeat(c):
        for _ in range(20):
            c.call()

    threads = [threading.Thread(target=repeat, args=(c,)) for c in callers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c, (chi2, resp) in zip(callers, want):
        got = c.result()
        np.testing.assert_array_equal(got[0], chi2)
        np.testing.assert_array_equal(got[1], resp)
    assert callers[0].L.fp_evaluate_proposal_release() == 0
    callers[0].call()
    np.testing.assert_array_equal(callers[0].result()[0], want[0][0])
