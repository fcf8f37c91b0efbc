"""Stream policy of an EP buffer: which stream a launch goes to and what has to wait for what.

Result pools are overwritten in place, so the buffer must know every stream that may still be reading
an earlier result.  All dependencies set up here are device-side (``wait_stream`` / ``wait_event``);
nothing blocks the calling CPU thread.
"""

from __future__ import annotations

import sys
from typing import Any, Dict, List, Optional, Tuple

import torch


_POOLED_EVENTS = 16


def _references_of_list_only() -> Optional[int]:
    """What ``sys.getrefcount(objects[index])`` says of an object that nothing but the list holds.  How many references the
    expression adds is the interpreter's affair, so it is counted, not assumed; None where one more holder does not count as
    exactly one more."""
    objects, index = [object()], 0
    alone = sys.getrefcount(objects[index])
    holder = objects[index]
    counted = sys.getrefcount(objects[index]) == alone + 1
    del holder
    return alone if counted and sys.getrefcount(objects[index]) == alone else None


class NullStream:
    """Stands in for a CUDA stream on the CPU transport: every operation is already ordered."""

    cuda_stream = 0

    def wait_stream(self, other: Any) -> None:
        pass

    def wait_event(self, event: Any) -> None:
        pass

    def synchronize(self) -> None:
        pass


def stream_key(stream: Any) -> Tuple[int, int]:
    return (stream.device.index, int(stream.cuda_stream))


class StreamPolicy:
    """Owns the communication stream and the registry of consumer streams of one buffer.

    A *synchronous* call without a producer event means "the communication stream waits for the compute
    stream and the compute stream waits for the result", which is plain in-order execution: the kernel
    is put on the compute stream itself and both cross-stream hand-offs (tens of microseconds of device
    latency per call) disappear.  Asynchronous calls and calls with a producer event go to the
    communication stream.
    """

    def __init__(self, device: Any, on_gpu: bool) -> None:
        self.on_gpu = on_gpu
        self.device = device
        self.comm = torch.cuda.Stream(device=device) if on_gpu else NullStream()
        self.consumers: Dict[Tuple[int, int], Any] = {}
        self._reader: Any = None  # the last stream of the callers' that a synchronous call ran on
        self._reader_raw, self._reader_key = -1, None
        # stream objects by raw handle: torch builds a new one per query (1.3 us), and with one object per stream "the only
        # reader is the stream itself" is a comparison of identities
        self._known: Dict[int, Any] = {}
        self._events: List[Any] = []
        self._unheld = _references_of_list_only()
        self._next_event = 0
        # work was queued on the communication stream that the compute stream has not waited for yet
        self._comm_ahead = False

    def current(self) -> Any:
        if not self.on_gpu:
            return NullStream()
        raw = torch._C._cuda_getCurrentRawStream(self.device)
        stream = self._known.get(raw)
        if stream is None:
            if len(self._known) >= 64:
                self._known.clear()
            stream = self._known[raw] = torch.cuda.current_stream(self.device)
        return stream

    def event(self) -> Any:
        """A CUDA event that nothing but this pool refers to: creating, first recording and destroying one costs 2 to 5 us,
        recording one that exists 0.7.  An event that somebody still holds (a token, a handle, a watchdog) is never recorded again."""
        events = self._events
        for _ in range(len(events)):
            self._next_event = (self._next_event + 1) % len(events)
            if sys.getrefcount(events[self._next_event]) == self._unheld:
                return events[self._next_event]
        event = torch.cuda.Event()
        if self._unheld is not None and len(events) < _POOLED_EVENTS:
            events.append(event)
        return event

    def is_comm(self, stream: Any) -> bool:
        """Also true for a caller that has made the communication stream its current one."""
        return stream is self.comm or stream.cuda_stream == self.comm.cuda_stream

    # -- readers of result pools ---------------------------------------------------------------
    def add_consumer(self, stream: Any) -> None:
        """Remember a stream that reads results; it outlives the Python tensors it reads."""
        if not self.on_gpu:
            return
        key = stream_key(stream)
        if key != stream_key(self.comm):
            self.consumers[key] = stream

    def _after_consumers(self, target: Any, *already_ordered: Any) -> None:
        """Make ``target`` wait for every registered reader except the streams given."""
        if len(self.consumers) == 1 and target in self.consumers.values():
            return
        done = {stream_key(s) for s in already_ordered}
        done.add(stream_key(target))
        for key, reader in self.consumers.items():
            if key not in done:
                target.wait_stream(reader)

    def sole(self) -> Any:
        """The caller's current stream if a synchronous launch on it has nothing to be ordered with: it alone reads results, and the
        communication stream is not ahead of it.  Else None."""
        if self._comm_ahead or torch._C._cuda_getCurrentRawStream(self.device) != self._reader_raw:
            return None
        return self._reader if len(self.consumers) == 1 and self._reader_key in self.consumers else None

    def first(self) -> Any:
        """The same for the first launch on a buffer: nobody reads results yet, and the caller's stream is about to."""
        if self._reader is not None or self.consumers or self._comm_ahead:
            return None
        stream = self.current()
        self.finish(stream, stream, None, False)
        return self.sole()

    def raw(self, stream: Any) -> int:
        return self._reader_raw if stream is self._reader else int(stream.cuda_stream)

    # -- one launch ------------------------------------------------------------------------------
    def begin(self, compute: Any, previous_event: Any, run_async: bool) -> Any:
        """Return the stream the next kernel is launched on, with its input dependencies in place."""
        if not self.on_gpu:
            return compute
        if not run_async and previous_event is None:
            if self._comm_ahead:
                compute.wait_stream(self.comm)
                self._comm_ahead = False
            self._after_consumers(compute, self.comm)
            return compute
        if previous_event is None:
            self.comm.wait_stream(compute)
            self._after_consumers(self.comm, compute)
        else:
            self._wait_for_producer(previous_event)
            self._after_consumers(self.comm)
        self._comm_ahead = True
        return self.comm

    def _wait_for_producer(self, previous_event: Any) -> None:
        raw = getattr(previous_event, "event", None)
        if raw is not None:
            self.comm.wait_event(raw)  # an EventOverlap: the communication stream is the one that waits
        elif hasattr(previous_event, "current_stream_wait"):
            with torch.cuda.stream(self.comm):
                previous_event.current_stream_wait()
        else:
            self.comm.wait_event(previous_event)

    def finish(self, compute: Any, launched_on: Any, event: Optional[Any], run_async: bool) -> None:
        """After the launch of a synchronous call: the caller's stream sees the result and is recorded as a reader."""
        if not self.on_gpu or run_async:
            return
        if launched_on is not compute and event is not None:
            compute.wait_event(event)
            self._comm_ahead = False
        if not (len(self.consumers) == 1 and compute in self.consumers.values()):
            self.add_consumer(compute)
        if compute is not self._reader and not self.is_comm(compute):
            self._reader, self._reader_raw, self._reader_key = compute, int(compute.cuda_stream), stream_key(compute)

    def drain(self, last_event: Optional[Any]) -> None:
        """Blocking: used by ``close`` only."""
        if not self.on_gpu:
            return
        if last_event is not None:
            last_event.synchronize()
        self.comm.synchronize()
