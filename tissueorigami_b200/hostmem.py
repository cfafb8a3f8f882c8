"""Page-locked memory for large result arrays.

A device-to-host copy into fresh pageable memory is bound by its page faults and by CUDA's staging
(14 MB of Jacobian: 2.1 ms, 0.28 ms into page-locked memory). Results of at least 1 MB therefore live in
page-locked blocks that go back to a bounded pool when the last view of the array is gone.
"""
from __future__ import annotations

import collections
import ctypes
import mmap
import os
import threading
import weakref

import numpy as np

MIN_BYTES = 1 << 20    # below, a pageable copy costs less than 0.1 ms
LIMIT = 256 << 20      # page-locked bytes, handed out and kept; beyond, results are ordinary arrays
KEEP = 64 << 20        # of these, bytes kept for the next results


class _Pool:
    def __init__(self):
        self._reset()

    def _reset(self):
        """Also in a forked child, where the parent's registrations do not count."""
        self._lock = threading.Lock()
        self._free = []  # (size, block), oldest first; only the lock's holder touches it
        self._back = collections.deque()  # (lib, size, block) dropped and not yet in _free
        self._bytes = 0
        self._pid = os.getpid()

    def _kept(self):
        return sum(size for size, _ in self._free)

    def _drop(self, lib, need):
        """Gives kept blocks back until `need` bytes fit below LIMIT."""
        while self._free and self._bytes + need > LIMIT:
            self._unregister(lib, *self._free.pop(0))

    def _unregister(self, lib, size, block):
        view = ctypes.c_char.from_buffer(block)
        lib.tf_host_unregister(ctypes.addressof(view))
        del view
        self._bytes -= size

    def take(self, lib, handle, shape):
        """A float64 array of `shape` in page-locked memory (contents undefined), or None."""
        n = 8 * int(np.prod(shape, dtype=np.int64))
        size = -(-n // MIN_BYTES) * MIN_BYTES
        if n < MIN_BYTES or size > LIMIT:
            return None
        try:
            with self._lock:
                self._settle()
                size, block = self._block(lib, handle, size)
        finally:
            self._settle_unless_held()
        if block is None:
            return None
        owner = (ctypes.c_char * n).from_buffer(block)
        weakref.finalize(owner, self._give, lib, size, block, self._pid).atexit = False
        return np.frombuffer(owner, dtype=np.float64).reshape(shape)

    def _block(self, lib, handle, size):
        """A kept block of about `size` bytes or a new one, or None; and its size."""
        for i, (have, block) in enumerate(self._free):
            if size <= have <= size + size // 4:
                del self._free[i]
                return have, block
        self._drop(lib, size)
        if self._bytes + size > LIMIT:
            return size, None
        try:
            block = mmap.mmap(-1, size, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
        except OSError:  # no address space or mapping left
            return size, None
        try:
            block.madvise(mmap.MADV_HUGEPAGE)
        except (AttributeError, OSError):  # a kernel without huge pages
            pass
        view = ctypes.c_char.from_buffer(block)
        ok = lib.tf_host_register(handle, ctypes.addressof(view), size) == 0
        del view
        if not ok:
            return size, None
        self._bytes += size
        return size, block

    def _give(self, lib, size, block, pid):
        """The last view of a block is gone. A finalizer: the garbage collector may run it between any two
        instructions, those of the lock's holder on the same thread among them, so it only queues the block."""
        if pid != self._pid:
            return
        self._back.append((lib, size, block))
        self._settle_unless_held()

    def _settle_unless_held(self):
        while self._back and self._lock.acquire(blocking=False):
            try:
                self._settle()
            finally:
                self._lock.release()

    def _settle(self):
        """Queued blocks into _free, the oldest given back beyond KEEP."""
        while self._back:
            lib, size, block = self._back.popleft()
            self._free.append((size, block))
            while self._kept() > KEEP:
                self._unregister(lib, *self._free.pop(0))


_pool = _Pool()
if hasattr(os, "register_at_fork"):
    os.register_at_fork(after_in_child=_pool._reset)


def result(lib, handle, shape):
    """An uninitialised float64 array for a result of the context `handle`."""
    out = _pool.take(lib, handle, shape)
    return np.empty(shape) if out is None else out
