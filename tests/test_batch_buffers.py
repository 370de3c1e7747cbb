"""The transfer buffers of a batched proposer: kernels address them directly, so
they outlive the proposer until its queued transfers are through, and the
transfers are launched on their stream's device."""

import gc
import weakref

import numpy as np
import pytest

from forcepho_b200 import batch


class Event:
    """Stands for a CUDA event; notes whether the buffer is alive when waited for."""

    def __init__(self, buffer=None):
        self.alive, self.waits, self.seen = None if buffer is None else weakref.ref(buffer), 0, []

    def record(self, stream):
        pass

    def synchronize(self):
        self.waits += 1
        self.seen.append(self.alive is None or self.alive() is not None)


class Buffer:
    pass


class Owner:
    pass


def owner_of(buffer, event):
    o = Owner()
    weakref.finalize(o, batch._release, {"d2h": event}, (buffer,))
    return o


def test_buffers_stay_until_their_transfers_are_through(monkeypatch):
    monkeypatch.setattr(batch.torch.cuda, "is_current_stream_capturing", lambda: False)
    buffer = Buffer()
    gone, event = weakref.ref(buffer), Event(buffer)
    o = owner_of(buffer, event)
    del buffer
    assert gone() is not None
    del o
    gc.collect()
    assert event.seen == [True] and gone() is None and not batch._RETIRED


def test_nothing_waits_during_a_capture(monkeypatch):
    capturing = [True]
    monkeypatch.setattr(batch.torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    first, second = Event(), Event()
    o = owner_of(Buffer(), first)
    del o
    assert first.waits == 0 and len(batch._RETIRED) == 1
    capturing[0] = False
    o = owner_of(Buffer(), second)
    del o
    assert first.waits == second.waits == 1 and not batch._RETIRED


def test_transfers_are_launched_on_their_streams_device(monkeypatch):
    """With fakes for the device and the library: a stream of another device than the current one."""
    current, launches = [0], []

    class device:
        def __init__(self, d):
            self.d = d

        def __enter__(self):
            self.saved, current[0] = current[0], self.d

        def __exit__(self, *exc):
            current[0] = self.saved

    class stream:
        device = 1
        cuda_stream = 0

    class library:
        @staticmethod
        def fp_upload_proposals(*args):
            launches.append(("up", current[0]))
            return 0

        @staticmethod
        def fp_fetch_results(*args):
            launches.append(("down", current[0]))
            return 0

    class tensor:
        @staticmethod
        def data_ptr():
            return 0

        @staticmethod
        def numel():
            return 0

    class plan:
        L = library
        proposals = chi2 = response = tensor

        @staticmethod
        def check_current(s):
            pass

    monkeypatch.setattr(batch.torch.cuda, "device", device)
    monkeypatch.setattr(batch.torch.cuda, "Event", Event)
    bp = batch.BatchedProposer.__new__(batch.BatchedProposer)
    bp.n, bp.plan, bp._done = 1, plan, {}
    bp._prop_slots, bp._prop_len = np.zeros((1, 30), batch._RECORD), [0]
    bp._pin_prop = bp._counts = bp._rows = bp._pin_chi2 = bp._pin_grad = tensor
    bp.set_proposals_async([], stream())
    bp.fetch_async(stream())
    assert launches == [("up", 1), ("down", 1)] and current == [0]


@pytest.mark.gpu
def test_dropping_a_proposer_with_queued_work():
    import torch
    from forcepho_b200 import synthetic as S
    p = S.config_multiband(seed=12, n_sources=3, n_bands=2, exp_per_band=1, size=40)
    p.return_residual = False
    p.send_to_device()
    bp = batch.BatchedProposer([p])
    prop = [p.scene.get_proposal().copy()]
    want = bp.evaluate_proposals(prop)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        torch.cuda._sleep(100_000_000)              # some 50 ms
    bp.set_proposals_async(prop, s)
    bp.run(s)
    bp.fetch_async(s)
    events, sizes = list(bp._done.values()), [bp._pin_prop.numel(), bp._pin_chi2.numel(), bp._pin_grad.numel()]
    del bp
    assert all(e.query() for e in events)
    new = [torch.full((n,), 7, dtype=dt).pin_memory()
           for n, dt in zip(sizes, (torch.uint8, torch.float64, torch.float32))]
    s.synchronize()
    assert all(bool((t == 7).all()) for t in new)
    again = batch.BatchedProposer([p]).evaluate_proposals(prop)
    np.testing.assert_array_equal(again[0][1], want[0][1])


@pytest.mark.gpu
@pytest.mark.parametrize("use_graph", [True, False])
def test_a_single_call_that_fails_half_way_waits_for_its_kernels(use_graph, monkeypatch):
    """The reduction writes the proposer's pinned buffers: none of it may be queued once the call is over."""
    import torch
    from forcepho_b200 import synthetic as S
    from forcepho_b200.proposal import B200Proposer
    p = S.config_multiband(seed=13, n_sources=3, n_bands=2, exp_per_band=1, size=40)
    p.return_residual = True
    p.send_to_device()
    proposer, prop = B200Proposer(use_graph=use_graph), p.scene.get_proposal().copy()
    want = proposer.evaluate_proposal(prop, patch=p, unpack=False)

    def fails(*args, **kwargs):
        raise MemoryError("no page-locked memory")

    proposer._pinned_res = None                     # its buffer is made after the launches
    with monkeypatch.context() as m:
        m.setattr(torch.Tensor, "pin_memory", fails)
        torch.cuda._sleep(100_000_000)              # some 50 ms
        with pytest.raises(MemoryError):
            proposer.evaluate_proposal(prop, patch=p)
        assert torch.cuda.current_stream().query()
    got = proposer.evaluate_proposal(prop, patch=p, unpack=False)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
