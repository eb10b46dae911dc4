"""What a module derives from its parameters and keeps between calls: transfer tables, packed 1x1 weights."""
import threading
from collections import OrderedDict

from . import _cabi

_LOCK = threading.Lock()      # guards the slow path of every cache: a look-up that missed the entry used last


class _Entry:
    __slots__ = ("value", "tensors", "ready", "streams")

    def __init__(self, value, tensors, ready, streams):
        self.value, self.tensors, self.ready, self.streams = value, tensors, ready, streams


class Kept:
    """A few values by key, each for one state of the parameters it was made from.

    The last element of a key is `host.state(*params)`: the parameters' addresses and version counters, then the current
    stream.  An entry keeps its parameters' storages alive, so that no other tensor can come to their addresses and pass
    for them.  It is used on the stream it was made on; any other stream first waits for it, and the allocator learns that
    this stream uses it.  While a CUDA graph is captured nothing is kept: a value made there exists only when the graph is
    replayed (and a capture cannot wait for another stream's work, so values that it uses are made before it begins).

    Copies and pickles of a module start with an empty cache: the addresses are those of the original's parameters."""

    def __init__(self, slots=1):
        self.slots = slots
        self.entries = OrderedDict()
        self.last = None         # (key, value, entry) used last; callers look here first

    def __reduce__(self):
        return Kept, (self.slots,)

    def __deepcopy__(self, memo):
        return Kept(self.slots)

    def values(self):
        """Every value kept now (a captured graph holds on to those that its kernels read)."""
        with _LOCK:
            return [e.value for e in self.entries.values()] + ([] if self.last is None else [self.last[1]])

    def clear(self):
        with _LOCK:
            self.entries.clear()
            self.last = None

    def get(self, key, params, build):
        """The value for `key`; `build()` makes it: a tensor or a tuple of tensors that share a device and a stream."""
        host, state = _cabi.host(), key[-1]
        if state is None:        # inference tensors: nothing says when they change
            return build()
        own, stream = key[:-1] + (state[:-8],), state[-8:]
        with _LOCK:
            e = self.entries.get(own)
            if e is None:
                value = build()
                tensors = value if isinstance(value, tuple) else (value,)
                ready = host.ready(tensors[0], *params)
                if ready is None:        # capturing
                    return value
                self.entries[own] = e = _Entry(value, tensors, ready, {stream})
                while len(self.entries) > self.slots:
                    self.entries.popitem(last=False)
            else:
                self.entries.move_to_end(own)
                if stream not in e.streams:
                    if not host.join(e.ready, *e.tensors):      # capturing
                        return e.value
                    e.streams.add(stream)
            self.last = (key, e.value, e)
            return e.value
