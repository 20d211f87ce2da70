"""Host memory of the tables that the drop-in calls return.

A fresh host table costs its page faults: 32 MB take 2.3 ms to fill from the device (14 GB/s, whatever the copy), against
0.19 ms into memory that has been written before (175 GB/s); the charges of 1,000 events are 160 MB.  So a large table
lies in memory that goes back to a bounded pool when the last array on it is gone, and the next table of its size class
takes it from there.  A table's memory is never shared while any array on it lives.

Tables that the host fills (the waveform matrix) stay ordinary arrays: memory that the device has read is slower for the
host to write than fresh memory (52 MB: 8.5 against 5.8 ms for the call).

The pool keeps at most LIMIT bytes (the least recently returned go first) and nothing above that; release() gives all of
it back.  It never waits: when another thread, or a destructor that interrupted this one, holds it, a table gets fresh
memory and a returned block is freed.
"""
from __future__ import annotations

import threading

import numpy as np

SMALL = 1 << 20          # bytes: below, a table is an ordinary array (the allocator reuses such memory itself)
LIMIT = 1 << 30          # bytes kept for later tables


class _Block:
    """The owner of a table's memory while arrays on it live."""

    def __init__(self, pool, raw):
        self.__array_interface__ = raw.__array_interface__
        self._pool, self._raw = pool, raw

    def __del__(self):
        self._pool._put(self._raw)


class HostPool:
    def __init__(self, limit=LIMIT):
        self.limit, self.kept = int(limit), 0
        self._free = []                       # returned blocks, oldest first
        self._lock = threading.Lock()

    @staticmethod
    def size_class(nbytes):
        """Bytes of the block for a table: up to an eighth of a power of two more (its tail is never touched)."""
        step = 1 << max(int(nbytes).bit_length() - 4, 0)
        return -(-int(nbytes) // step) * step

    def empty(self, shape, dtype):
        """np.empty(shape, dtype), from a returned block when one of its size class is there."""
        dtype = np.dtype(dtype)
        n = int(np.prod(shape, dtype=np.int64)) * dtype.itemsize
        if n < SMALL:
            return np.empty(shape, dtype)
        size, raw = self.size_class(n), None
        if self._lock.acquire(blocking=False):
            try:
                for i in range(len(self._free) - 1, -1, -1):
                    if self._free[i].nbytes == size:
                        raw = self._free.pop(i)
                        self.kept -= size
                        break
            finally:
                self._lock.release()
        if raw is None:
            raw = np.empty(size, np.uint8)
        return np.asarray(_Block(self, raw))[:n].view(dtype).reshape(shape)

    def _put(self, raw):
        if raw.nbytes > self.limit or not self._lock.acquire(blocking=False):
            return
        try:
            self._free.append(raw)
            self.kept += raw.nbytes
            while self.kept > self.limit:
                self.kept -= self._free.pop(0).nbytes
        finally:
            self._lock.release()

    def release(self):
        """Free what the pool keeps."""
        with self._lock:
            self._free, old, self.kept = [], self._free, 0
        del old


POOL = HostPool()


def empty(shape, dtype):
    return POOL.empty(shape, dtype)


def to_host(t):
    """t.cpu().numpy() of a device tensor."""
    import torch
    if not t.is_cuda or t.numel() * t.element_size() < SMALL:
        return t.cpu().numpy()
    out = empty(tuple(t.shape), np.dtype(str(t.dtype).replace("torch.", "")))
    torch.from_numpy(out).copy_(t)
    return out


def release():
    """Free the memory that is kept for later tables."""
    POOL.release()
