"""Stream/event plumbing shared by every collective call.

``EventHandle`` is a CUDA event recorded on a stream at construction; ``EventOverlap`` is the object
the public API returns: ``current_stream_wait()`` makes the caller's stream wait for the communication
kernels, and used as a context manager it does that on exit, so compute issued inside the ``with``
block overlaps the communication.

Reference counterparts: ``EventHandle`` (csrc/event.hpp:9-40) and ``EventOverlap``
(deep_ep/utils.py:10-61).
"""
from __future__ import annotations

from typing import Any, Dict, Optional, Tuple

import torch


_HAS_CUDA: Optional[bool] = None


def _has_cuda() -> bool:
    """``torch.cuda.is_available()``, asked once: it queries the driver on every call."""
    global _HAS_CUDA
    if _HAS_CUDA is None:
        _HAS_CUDA = torch.cuda.is_available()
    return _HAS_CUDA


_STREAMS: Dict[Tuple[int, int], "torch.cuda.Stream"] = {}


def current_stream() -> "torch.cuda.Stream":
    """``torch.cuda.current_stream()``, which builds an object on every call (1.5 us, of which a call on the communication stream asks for four): the object
    of a CUDA stream is kept by its address. PyTorch's streams live as long as the process, and for others the address is all that the object holds."""
    device = torch.cuda.current_device()
    key = (device, torch._C._cuda_getCurrentRawStream(device))
    stream = _STREAMS.get(key)
    if stream is None:
        if len(_STREAMS) >= 256:
            _STREAMS.clear()
        stream = _STREAMS[key] = torch.cuda.current_stream(device)
    return stream


class EventHandle:
    """A CUDA event recorded on ``stream`` (default: the current stream) when created.

    On a machine without CUDA the handle is inert, which keeps the CPU/gloo backend API-compatible."""

    def __init__(self, stream: Optional["torch.cuda.Stream"] = None, record: bool = True) -> None:
        self.event = None
        if _has_cuda():
            self.event = torch.cuda.Event(enable_timing=False)
            if record:
                self.event.record(stream if stream is not None else current_stream())

    def current_stream_wait(self) -> None:
        if self.event is not None:
            current_stream().wait_event(self.event)


class EventOverlap:
    """Wrapper returned by every collective; see the module docstring.

    Attributes:
        event: the underlying :class:`EventHandle` (``None`` when the call was synchronous).
        extra_tensors: tensors kept alive until this object dies (their memory may still be in use by
            the communication stream).
    """

    def __init__(self, event: Optional[EventHandle] = None, extra_tensors: Optional[Tuple[Any, ...]] = None) -> None:
        self.event = event
        self.extra_tensors = extra_tensors

    def current_stream_wait(self) -> None:
        if self.event is not None:
            self.event.current_stream_wait()

    def __enter__(self) -> "EventOverlap":
        return self

    def __exit__(self, exc_type, exc, tb) -> None:
        if self.event is not None:
            self.event.current_stream_wait()
