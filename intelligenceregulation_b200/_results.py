"""Host memory for large results.

A fresh array of some megabytes costs more in page faults than the copy into it (measured on the B200 hosts: 33 MB from the device take
0.65 ms into pages that are there and 15 ms into pages that are not).  ``empty`` hands out memory of results that the caller has dropped:
a block goes back when the last array over it is gone, at most ``KEEP`` bytes wait for reuse, ``release`` gives them all back.
"""
from __future__ import annotations

import ctypes as C
import threading
import weakref
from typing import List

import numpy as np

SMALL = 256 << 10  # below this the C library's heap keeps its pages by itself
KEEP = 192 << 20   # a block's logup columns twice over (the caller holds one result while it computes the next), and the opening's vectors

_lock = threading.RLock()  # a block may come back from a garbage collection inside `empty`
_idle: List[np.ndarray] = []


def _back(block: np.ndarray) -> None:
    with _lock:
        _idle.append(block)
        while sum(b.nbytes for b in _idle) > KEEP:
            _idle.pop(0)


def empty(shape, dtype) -> np.ndarray:
    """``np.empty(shape, dtype)``, over reused memory where it is large"""
    dtype = np.dtype(dtype)
    nbytes = int(np.prod(shape, dtype=np.int64)) * dtype.itemsize
    if nbytes < SMALL:
        return np.empty(shape, dtype)
    block = None
    with _lock:
        fits = [b for b in _idle if nbytes <= b.nbytes <= nbytes + (nbytes >> 2)]
        if fits:
            best = min(fits, key=lambda b: b.nbytes)
            block = _idle.pop(next(i for i, b in enumerate(_idle) if b is best))
    if block is None:
        block = np.empty(nbytes, np.uint8)
    hold = (C.c_ubyte * nbytes).from_buffer(block)
    weakref.finalize(hold, _back, block).atexit = False
    return np.frombuffer(hold, dtype=dtype).reshape(shape)


def release() -> None:
    with _lock:
        _idle.clear()
