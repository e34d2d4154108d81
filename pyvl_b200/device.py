"""PyTorch plumbing for the C ABI: device tensors, raw pointers, streams, workspaces.

PyTorch only moves memory here; every computation is a kernel of libpvl_b200.so.
"""

from __future__ import annotations

import ctypes
import gc
import threading

import numpy as np
import torch

from . import _lib


def require_cuda() -> torch.device:
    """Return the current CUDA device or raise: the hot path has no CPU fallback."""
    if torch.cuda.is_initialized() and _cur_device is not None:  # then a GPU was available
        return torch.device("cuda", _cur_device())
    if not torch.cuda.is_available():
        raise RuntimeError("pyvl_b200 runs its kernels on a CUDA GPU (B200); no GPU is available")
    return torch.device("cuda", torch.cuda.current_device())


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_cur_device = getattr(torch._C, "_cuda_getDevice", None)


def stream_ptr(stream: torch.cuda.Stream | None = None) -> int:
    """The stream handle as an integer for a void* argument (the current stream by default;
    read through torch's raw-stream query, which costs far less per call than building a
    Stream object: a step makes dozens of these calls)."""
    if stream is not None:
        return stream.cuda_stream
    if _raw_stream is not None and _cur_device is not None:
        return _raw_stream(_cur_device())
    return torch.cuda.current_stream().cuda_stream


def ptr(t: torch.Tensor | None) -> int | None:
    """Device address of a tensor as an integer for a void* argument (None -> NULL)."""
    return None if t is None else t.data_ptr()


def to_device(a, dtype=torch.float64, device=None) -> torch.Tensor:
    """Contiguous device tensor of `dtype` (no copy when already one)."""
    dev = device or require_cuda()
    if isinstance(a, torch.Tensor):
        if a.dtype is dtype and a.device == dev and a.is_contiguous():
            return a
        t = a.to(device=dev, dtype=dtype)
        return t.contiguous()
    arr = np.ascontiguousarray(a)
    return torch.from_numpy(arr).to(device=dev, dtype=dtype, non_blocking=False).contiguous()


def to_device_u32(a, device=None) -> torch.Tensor:
    """uint32 host array -> int32 device tensor with the same bit pattern."""
    dev = device or require_cuda()
    arr = np.ascontiguousarray(np.asarray(a, np.uint32)).view(np.int32)
    return torch.from_numpy(arr.copy()).to(dev)


class _CollectorHeld:
    """The cyclic collector off, for all threads, from the first one's entry to the last one's exit;
    then as it was."""

    _lock = threading.Lock()
    _inside = 0
    _was_on = False

    def __enter__(self):
        cls = _CollectorHeld
        with cls._lock:
            if cls._inside == 0:
                cls._was_on = gc.isenabled()
                gc.disable()
            cls._inside += 1

    def __exit__(self, *exc):
        cls = _CollectorHeld
        with cls._lock:
            cls._inside -= 1
            if cls._inside == 0 and cls._was_on:
                gc.enable()


class _CaptureStreams:
    """Streams that only captures use, each by one capture at a time: as many per device as captures
    have been under way at once.  (torch.cuda.Stream() hands out the same few dozen handles in turn,
    so that its stream may be one on which another thread is enqueuing work, which would end up in
    the graph.)"""

    _lock = threading.Lock()
    _free: dict = {}

    def __init__(self, device: int):
        self.device = device

    def __enter__(self):
        with self._lock:
            free = self._free.setdefault(self.device, [])
            self.stream = free.pop() if free else None
        if self.stream is None:
            handle = ctypes.c_void_p()
            _lib.call("pvl_stream_create", ctypes.byref(handle))
            self.stream = torch.cuda.ExternalStream(handle.value, device=self.device)
        return self.stream

    def __exit__(self, *exc):
        with self._lock:
            self._free[self.device].append(self.stream)


def capture_graph(fn) -> torch.cuda.CUDAGraph:
    """``fn`` (launches on fixed buffers, no host reads) captured as a CUDA graph.

    torch.cuda.graph without the device-wide synchronisation, garbage collection and emptied
    allocator cache of its entry (~1 ms a capture, more than a short run's steps take).  The
    cyclic collector is held off instead, so that nothing it frees reaches the CUDA runtime while
    the stream captures (until the last of several threads' captures has ended).  The allocator
    gives no cached block back while a stream captures, so a capture that finds the memory full is
    repeated after the collection and with the cache emptied."""
    try:
        return _capture(fn)
    except torch.OutOfMemoryError:
        pass  # the failed capture's tensors go with the exception
    gc.collect()
    torch.cuda.empty_cache()
    return _capture(fn)


def _capture(fn) -> torch.cuda.CUDAGraph:
    g = torch.cuda.CUDAGraph()
    cur = torch.cuda.current_stream()
    with _CaptureStreams(require_cuda().index) as side:
        side.wait_stream(cur)
        with _CollectorHeld(), torch.cuda.stream(side):
            g.capture_begin()
            try:
                fn()
            finally:
                g.capture_end()
        cur.wait_stream(side)
    return g


class Workspace:
    """Grow-only device scratch buffer, one per (device, stream)."""

    _pool: dict = {}

    @classmethod
    def get(cls, nbytes: int, stream: torch.cuda.Stream | None = None) -> tuple[ctypes.c_void_p, int]:
        dev = require_cuda()
        key = (dev.index, stream_ptr(stream))
        buf = cls._pool.get(key)
        nbytes = max(int(nbytes), 256)
        if buf is None or buf.numel() < nbytes:
            buf = torch.empty(int(nbytes * 1.25) + 256, dtype=torch.uint8, device=dev)
            cls._pool[key] = buf
        return ctypes.c_void_p(buf.data_ptr()), buf.numel()

    @classmethod
    def clear(cls) -> None:
        cls._pool.clear()
