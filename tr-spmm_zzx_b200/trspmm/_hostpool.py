"""Host memory of large results that came and went, kept for the next ones.

The reference's calling convention returns a new CPU tensor per call.  For a result of tens of megabytes the page
faults of fresh memory cost more than the copy from the device (33 MB: 1.7 against 0.6 ms), and the C library gives
such blocks back to the system every time.  So the storages of the last results, KEEP_BYTES of them at most, are kept, and
one that no tensor holds any more serves the next result of its size; release() lets all of them go.

A result is an ordinary tensor on ordinary memory of torch's: private to the process (a fork's child has its own), it can
be resized or moved to shared memory, and it is never page-locked, because a copy from page-locked memory may still be
under way when the tensor is gone.
"""
from __future__ import annotations

import math
import sys
import threading

import torch

MIN_BYTES = 1 << 20      # below, the C library reuses memory itself
KEEP_BYTES = 256 << 20

_use_count = getattr(torch._C, "_storage_Use_Count", None)

_lock = threading.Lock()
_idle: list = []         # storages idle or still in use, oldest first


class _Block:
    def __init__(self, n: int):
        self.bytes = n
        # The C library serves arrays up to the largest one freed so far (32 MB at most) from its heap, which keeps their
        # pages.  A result that is kept is never freed, so it is once in advance, as it would be by any program that drops
        # it: otherwise the program's own arrays of such sizes fault their pages in every time (a format's copy to
        # the CPU, 45 MB in 29 arrays: 38 against 8 ms).
        torch.empty(n, dtype=torch.uint8, device="cpu")
        self.storage = torch.empty(n, dtype=torch.uint8, device="cpu").untyped_storage()

    def in_use(self) -> bool:
        """By a tensor, or by a caller who holds the storage itself."""
        return _use_count(self.storage._cdata) > 1 or sys.getrefcount(self.storage) > 2

    def changed(self) -> bool:
        """Resized, moved to shared memory, or pinned to its size by an array over it."""
        s = self.storage
        return s.nbytes() != self.bytes or not s.resizable() or s.is_shared()


def _take(n: int) -> _Block:
    for block in _idle[:]:
        if block.bytes == n and not block.in_use():
            _idle.remove(block)
            if not block.changed():
                return block
    return _Block(n)


def empty(shape, dtype: torch.dtype) -> torch.Tensor:
    """An uninitialised CPU tensor."""
    n = math.prod(shape) * dtype.itemsize
    if n < MIN_BYTES or n > KEEP_BYTES or _use_count is None:
        return torch.empty(shape, dtype=dtype, device="cpu")
    with _lock:
        block = _take(n)
        out = torch.empty(0, dtype=dtype, device="cpu").set_(block.storage, 0, shape)
        _idle.append(block)
        kept = sum(b.bytes for b in _idle)
        while kept > KEEP_BYTES:
            kept -= _idle.pop(0).bytes
    return out


def release():
    with _lock:
        _idle.clear()
