"""Host memory of large results that came and went, kept for the next ones.

The reference's calling convention returns a new CPU tensor per call.  For a result of tens of megabytes the page
faults of fresh memory cost more than the copy from the device (33 MB: 1.7 against 0.6 ms), and the C library gives
such blocks back to the system every time.  Blocks handed out here return to a list when the last tensor
over them is gone; at most KEEP_BYTES wait there, the oldest go first, release() lets all of them go.

They are never page-locked: a copy from page-locked memory may still be under way when the tensor is gone, and nothing
would keep the block from the next result until then.
"""
from __future__ import annotations

import math
import mmap
import threading
import weakref

import numpy as np
import torch

MIN_BYTES = 1 << 20      # below, the C library reuses memory itself
KEEP_BYTES = 256 << 20
_BLOCK = 2 << 20         # large pages

_adapted = False

_lock = threading.RLock()   # re-entrant: a collection inside _take() may give blocks back
_idle: list = []            # oldest first


class _Block:
    def __init__(self, n: int):
        self.bytes = -(-n // _BLOCK) * _BLOCK
        self.memory = mmap.mmap(-1, self.bytes)
        self.address = np.frombuffer(self.memory, dtype=np.uint8).ctypes.data
        if hasattr(mmap, "MADV_HUGEPAGE"):
            try:
                self.memory.madvise(mmap.MADV_HUGEPAGE)
            except OSError:   # a kernel without large pages
                pass


def _give_back(block):
    with _lock:
        _idle.append(block)
        waiting = sum(b.bytes for b in _idle)
        while waiting > KEEP_BYTES:
            waiting -= _idle.pop(0).bytes


def _take(n: int):
    with _lock:
        fits = [i for i, b in enumerate(_idle) if n <= b.bytes <= n + n // 4 + _BLOCK]
        block = _idle.pop(min(fits, key=lambda i: _idle[i].bytes)) if fits else None
    return _Block(n) if block is None else block


def empty(shape, dtype: torch.dtype) -> torch.Tensor:
    """An uninitialised CPU tensor."""
    count = math.prod(shape)
    n = count * dtype.itemsize
    if n < MIN_BYTES or n > KEEP_BYTES:
        return torch.empty(shape, dtype=dtype)
    global _adapted
    if not _adapted:
        # The C library takes blocks up to the largest one freed so far (32 MB at most) from its heap, larger ones from the
        # system each time.  Results used to raise that mark; without them a program's own arrays of a few
        # megabytes would fault their pages in anew on every allocation.
        _adapted = True
        torch.empty(31 << 20, dtype=torch.uint8)
    block = _take(n)
    owner = np.frombuffer(block.memory, dtype=np.uint8, count=n)   # lives as long as the tensor's storage
    weakref.finalize(owner, _give_back, block).atexit = False
    return torch.from_numpy(owner).view(dtype).view(shape)


def release():
    with _lock:
        _idle.clear()
