"""Copies between host and device at the sizes where the path changes: the bounce area's limit, one ring piece, more pieces than the
ring has slots; pageable and page-locked; two contexts copying at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
P = 0xFFFFFFFF00000001


def _same_back(ctx, a):
    out = ctx.probe_field(a, np.zeros_like(a))  # (a + 0, a - 0, a * 0)
    assert (out[:, 0] == a).all() and (out[:, 1] == a).all() and not out[:, 2].any()


def _words(n, seed):
    return np.random.default_rng(seed).integers(0, P, size=n, dtype=np.uint64)


@pytest.mark.parametrize("n", [1, 8191, 8192, 8193, 16384, 16385, 32768, 32769, 49152, 49153, 24575, 24576, 24577, 131072, 131073, (1 << 20) + 5, (5 << 20) + 1])
@pytest.mark.parametrize("locked", [False, True])
def test_round_trip(n, locked):
    import torch
    from intelligenceregulation_b200 import backend

    ctx = backend.Context(0)
    a = _words(n, n)
    if locked:
        keep = torch.from_numpy(a.view(np.int64)).pin_memory()
        a = keep.numpy().view(np.uint64)
    for _ in range(3):
        _same_back(ctx, a)
    ctx.close()


def test_two_contexts_at_once():
    from intelligenceregulation_b200 import backend

    bad = []

    def work(seed):
        try:
            ctx = backend.Context(0)
            for i in range(6):
                _same_back(ctx, _words((1 << 19) + 77 * i + seed, seed + i))
            ctx.close()
        except BaseException as e:  # noqa: BLE001 - handed to the test's thread
            bad.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in (1, 2, 3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


@pytest.mark.parametrize("extra", [16384 - 1, 16384, 16384 + 1, 3 * 16384 + 1])
def test_last_piece_of_whole_and_short_shares(extra):
    from intelligenceregulation_b200 import backend

    ctx = backend.Context(0)
    _same_back(ctx, _words(2 * 65536 + extra, extra))  # pieces of 64 Ki words, each filled and emptied in four shares
    ctx.close()
