"""The stream every call of the package runs on, and CUDA-graph capture of it.

The reference routes all work to one "active stream" that a capture context swaps
(``src/quark/graph.py:47-49``, ``:105-173``).  Here a single non-blocking stream is created on
first use and used for every launch and copy, so capture needs no stream switch: entering
``capture_graph()`` starts capturing that stream, leaving it instantiates the graph.
"""

from __future__ import annotations

import ctypes as C

from .. import _lib

_stream: int | None = None


def active_stream() -> int:
    global _stream
    if _stream is None:
        p = C.c_void_p()
        _lib.check(_lib.load().qb_stream_create(C.byref(p)))
        _stream = int(p.value)
    return _stream


# Called as (old, new) when the active stream changes, and as (graph,) when a capture has ended: the scratch memory of
# ``functional`` belongs to a stream, or to the graph that was captured with it.
on_stream_change: list = []
on_captured: list = []


def set_stream(handle: int) -> None:
    """Run on a caller-owned ``cudaStream_t`` instead (must not be the legacy default stream when graphs are captured).

    The choice is the process's, for all its threads.  Work on different streams may overlap, with these exceptions: a module's
    output buffers are its own whatever the stream, and ``patchify``, ``unpatchify`` and attention that casts its caches have one
    intermediate buffer per shape."""
    global _stream
    old, _stream = _stream, int(handle)
    for f in on_stream_change:
        f(old, _stream)


def synchronize() -> None:
    _lib.check(_lib.load().qb_stream_sync(C.c_void_p(active_stream())))


class Event:
    def __init__(self):
        p = C.c_void_p()
        _lib.check(_lib.load().qb_event_create(C.byref(p)))
        self.handle = int(p.value)

    def record(self) -> "Event":
        _lib.check(_lib.load().qb_event_record(C.c_void_p(self.handle), C.c_void_p(active_stream())))
        return self

    def synchronize(self) -> None:
        _lib.check(_lib.load().qb_event_sync(C.c_void_p(self.handle)))

    def elapsed_ms(self, later: "Event") -> float:
        ms = C.c_float(0)
        _lib.check(_lib.load().qb_event_elapsed_ms(C.c_void_p(self.handle), C.c_void_p(later.handle), C.byref(ms)))
        return float(ms.value)

    def __del__(self):
        try:
            _lib.load().qb_event_destroy(C.c_void_p(self.handle))
        except Exception:
            pass


class SideStream:
    """A second stream for work beside the active one, joined again before what follows may be captured or timed as a whole."""

    def __init__(self):
        p = C.c_void_p()
        _lib.check(_lib.load().qb_stream_create(C.byref(p)))
        self.handle = int(p.value)
        self._fork, self._join = Event(), Event()

    def fork(self) -> int:
        """The side stream, behind everything the active stream has been given so far."""
        self._fork.record()
        _lib.check(_lib.load().qb_stream_wait_event(C.c_void_p(self.handle), C.c_void_p(self._fork.handle)))
        return self.handle

    def join(self) -> None:
        """What the active stream is given from now on comes after the side stream's work."""
        lib = _lib.load()
        _lib.check(lib.qb_event_record(C.c_void_p(self._join.handle), C.c_void_p(self.handle)))
        _lib.check(lib.qb_stream_wait_event(C.c_void_p(active_stream()), C.c_void_p(self._join.handle)))

    def __del__(self):
        try:
            _lib.load().qb_stream_destroy(C.c_void_p(self.handle))
        except Exception:
            pass


_capturing = False


def capturing() -> bool:
    """Whether ``capture_graph`` is recording the active stream."""
    return _capturing


class Graph:
    """An instantiated CUDA graph; ``launch()`` replays it on the active stream."""

    def __init__(self, handle: int):
        self.handle = handle
        self.scratch = None  # memory that the kernels of the graph use besides their arguments

    def launch(self) -> None:
        _lib.check(_lib.load().qb_graph_launch(C.c_void_p(self.handle), C.c_void_p(active_stream())))

    def __del__(self):
        try:
            _lib.load().qb_graph_destroy(C.c_void_p(self.handle))
        except Exception:
            pass


class capture_graph:
    """``with capture_graph() as cap: ...`` then ``cap.graph.launch()``.

    Nothing inside the block may allocate or synchronise; run the same calls once eagerly
    first so that every cached buffer exists (the reference has the same rule,
    ``src/quark/models/waypoint_15.py:729-753``).
    """

    def __init__(self):
        self.graph: Graph | None = None

    def __enter__(self):
        global _capturing
        synchronize()
        _lib.check(_lib.load().qb_graph_begin(C.c_void_p(active_stream())))
        _capturing = True
        return self

    def __exit__(self, exc_type, exc, tb):
        global _capturing
        _capturing = False
        p = C.c_void_p()
        rc = _lib.load().qb_graph_end(C.c_void_p(active_stream()), C.byref(p))
        if exc_type is None:
            _lib.check(rc)
            self.graph = Graph(int(p.value))
            for f in on_captured:
                f(self.graph)
        return False
