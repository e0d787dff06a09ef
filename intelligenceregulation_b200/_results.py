"""Host memory for large results.

A fresh array of some megabytes costs more in page faults than the copy into it (the lookup columns of 2 M queries, 33 MB of them at once,
take 2.0 ms into pages that are there, 4.2 ms into fresh ones and 16 ms at a process's first call).  ``empty`` hands out memory of results
that the caller has dropped: a block goes back when the last array over it is gone, at most ``KEEP`` bytes wait for reuse, ``release`` gives
them all back.  A caller that keeps every result gets fresh pages every time.
"""
from __future__ import annotations

import math
import threading
from typing import List

import numpy as np

SMALL = 256 << 10  # below this the C library's heap keeps its pages by itself
KEEP = 192 << 20   # a few results of the largest calls (some 70 MB at a time): a caller usually holds one while it computes the next

_lock = threading.RLock()  # a block may come back from a garbage collection inside `empty`
_idle: List[np.ndarray] = []
_late: List[np.ndarray] = []  # came back while `empty` was looking through `_idle`
_looking = False
_bytes = 0


def _back(block: np.ndarray) -> None:
    global _bytes
    _idle.append(block)
    _bytes += block.nbytes
    while _bytes > KEEP:
        _bytes -= _idle.pop(0).nbytes


class _Hold:
    """What the arrays over a block have for a base: when the last of them is gone, so is this, and the block goes back."""

    __slots__ = ("block", "__array_interface__")

    def __init__(self, block: np.ndarray, shape, dtype: np.dtype):
        self.block = block
        self.__array_interface__ = {"shape": shape, "typestr": dtype.str, "data": (block.__array_interface__["data"][0], False), "version": 3}

    def __del__(self):
        with _lock:
            if _looking:
                _late.append(self.block)
            else:
                _back(self.block)


def empty(shape, dtype) -> np.ndarray:
    """``np.empty(shape, dtype)``, over reused memory where it is large"""
    global _bytes, _looking
    dtype, shape = np.dtype(dtype), tuple(shape) if isinstance(shape, (tuple, list)) else (int(shape),)
    nbytes = math.prod(shape) * dtype.itemsize
    if nbytes < SMALL:
        return np.empty(shape, dtype)
    block = None
    with _lock:
        _looking, best = True, -1
        for i, b in enumerate(_idle):
            if nbytes <= b.nbytes <= nbytes + (nbytes >> 2) and (best < 0 or b.nbytes < _idle[best].nbytes):
                best = i
        if best >= 0:
            block = _idle.pop(best)
            _bytes -= block.nbytes
        _looking = False
        while _late:
            _back(_late.pop())
    if block is None:
        block = np.empty(nbytes, np.uint8)
    return np.asarray(_Hold(block, shape, dtype))


def release() -> None:
    global _bytes
    with _lock:
        _idle.clear()
        _bytes = 0
