"""Row combinations of vectors with few entries around the number whose words are asked for together, at every word's extremes, and
dense ones over few columns, whose many row ranges are added by several warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
P = 0xFFFFFFFF00000001


@pytest.fixture(scope="module")
def dev():
    from intelligenceregulation_b200 import backend

    d = backend.B200Backend(device=0)
    yield d
    d.ctx.close()


@pytest.mark.parametrize("entries", [0, 1, 7, 8, 9, 16, 17, 100, 1000])
@pytest.mark.parametrize("extreme", [False, True])
def test_fold(dev, oracle, entries, extreme):
    rows, n, nn = 1000, 16, 32
    rng = np.random.default_rng(entries)
    data = np.full(rows * n, P - 1, dtype=np.uint64) if extreme else rng.integers(0, P, size=rows * n, dtype=np.uint64)
    rho = np.zeros((2, rows, 2), dtype=np.uint64)
    at = rng.permutation(rows)[:entries]
    rho[0, at] = P - 1 if extreme else rng.integers(0, P, size=(entries, 2), dtype=np.uint64)
    rho[1, -1] = 1
    want = oracle.fold_rows(oracle.encode_rows_plain(data, rows, n, nn, 18), rows, n, nn, 2, rho)
    store, _ = dev.try_commit(4, 2, data, 18)
    got = store.fold_rows(rho)
    store.free()
    assert (got == want).all()
