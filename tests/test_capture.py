"""device.capture_graph on the host: what it does to the process around the capture, with the CUDA graph
and the streams replaced by stand-ins.  No GPU needed."""

import contextlib
import gc
import threading

import pytest

from pyvl_b200 import device


class _Stream:
    cuda_stream = 0

    def wait_stream(self, other):
        pass


class _Graph:
    def capture_begin(self):
        pass

    def capture_end(self):
        pass


@pytest.fixture
def stand_ins(monkeypatch):
    monkeypatch.setattr(device.torch.cuda, "CUDAGraph", _Graph)
    monkeypatch.setattr(device.torch.cuda, "Stream", _Stream)
    monkeypatch.setattr(device.torch.cuda, "current_stream", lambda *a: _Stream())
    monkeypatch.setattr(device.torch.cuda, "stream", lambda s: contextlib.nullcontext())
    on = gc.isenabled()
    yield
    (gc.enable if on else gc.disable)()


@pytest.mark.parametrize("on", [True, False])
def test_collector_stays_off_until_the_last_capture_ends(stand_ins, on):
    """Two threads capture at once and the first to begin ends first."""
    (gc.enable if on else gc.disable)()
    first_in, second_in, first_out, done = (threading.Event() for _ in range(4))
    seen = []

    def first():
        first_in.set()
        assert second_in.wait(10)
        seen.append(gc.isenabled())

    def second():
        second_in.set()
        assert first_out.wait(10)
        seen.append(gc.isenabled())

    def run_first():
        device.capture_graph(first)
        first_out.set()

    def run_second():
        assert first_in.wait(10)
        device.capture_graph(second)
        done.set()

    threads = [threading.Thread(target=f) for f in (run_first, run_second)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(20)
    assert done.is_set() and seen == [False, False]
    assert gc.isenabled() == on


def test_collector_is_back_after_a_capture_that_fails(stand_ins):
    gc.enable()

    def fails():
        assert not gc.isenabled()
        raise RuntimeError("in the capture")

    with pytest.raises(RuntimeError, match="in the capture"):
        device.capture_graph(fails)
    assert gc.isenabled()
