"""device.capture_graph on the host: what it does to the process around the capture, with the CUDA graph
and the streams replaced by stand-ins.  No GPU needed."""

import contextlib
import gc
import threading
from pathlib import Path

import pytest

from pyvl_b200 import device


class _Stream:
    def __init__(self, handle=0, device=None):
        self.handle = handle

    def wait_stream(self, other):
        pass


class _Graph:
    def capture_begin(self):
        pass

    def capture_end(self):
        pass


@pytest.fixture
def stand_ins(monkeypatch):
    entered, made = [], []

    def create(name, out):
        assert name == "pvl_stream_create"
        made.append(len(made) + 1)
        out._obj.value = made[-1]

    @contextlib.contextmanager
    def enter(s):
        entered.append(s.handle)
        yield

    monkeypatch.setattr(device._lib, "call", create)
    monkeypatch.setattr(device, "require_cuda", lambda: device.torch.device("cuda", 0))
    monkeypatch.setattr(device._CaptureStreams, "_free", {})
    monkeypatch.setattr(device.torch.cuda, "CUDAGraph", _Graph)
    monkeypatch.setattr(device.torch.cuda, "ExternalStream", _Stream)
    monkeypatch.setattr(device.torch.cuda, "current_stream", lambda *a: _Stream())
    monkeypatch.setattr(device.torch.cuda, "stream", enter)
    on = gc.isenabled()
    yield entered
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


def test_a_capture_has_its_stream_to_itself(stand_ins):
    """One after the other, also after one that failed: the same stream.  One inside the other: another."""
    def fails():
        raise RuntimeError("in the capture")

    device.capture_graph(lambda: None)
    with pytest.raises(RuntimeError):
        device.capture_graph(fails)
    device.capture_graph(lambda: device.capture_graph(lambda: None))
    device.capture_graph(lambda: None)
    assert stand_ins[:4] == [1, 1, 1, 2] and stand_ins[4] in (1, 2)


def test_captures_take_one_route():
    sources = sorted((Path(device.__file__).parent).rglob("*.py"))
    assert sources and not [p.name for p in sources if "cuda.graph(" in p.read_text()]


def test_a_capture_that_finds_the_memory_full_is_repeated(stand_ins, monkeypatch):
    import torch

    emptied, tries = [], []
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: emptied.append(len(tries)))

    def full_once():
        tries.append(gc.isenabled())
        if len(tries) == 1:
            raise torch.OutOfMemoryError("full")

    device.capture_graph(full_once)
    assert emptied == [1] and tries == [False, False]

    def always_full():
        raise torch.OutOfMemoryError("full")

    with pytest.raises(torch.OutOfMemoryError):
        device.capture_graph(always_full)
