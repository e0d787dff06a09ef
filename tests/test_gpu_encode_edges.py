"""Encoded rows at the edges of the row encoder's forms: one CTA per (row, residue) against one per row on both sides of a CTA an SM,
every transform size, and rows of two and four transforms (one output residue, pads above twice the row)."""
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


CASES = [(n, 2, rows, 33) for n in range(8, 15) for rows in (1, 74, 75)]
CASES += [(9, 4, 38, 600), (14, 1, 2, 0), (15, 1, 2, 0), (16, 1, 1, 0), (15, 2, 3, 1), (16, 4, 1, 150000)]
CASES += [(12, 2, 148, 5), (12, 2, 149, 5), (10, 4, 297, 5), (15, 2, 75, 70000 // 4), (15, 2, 149, 40)]
CASES += [(12, 2, 110, 5), (12, 2, 111, 5), (11, 4, 184, 5), (11, 4, 185, 5), (10, 8, 332, 5), (10, 8, 333, 5), (8, 2, 887, 5), (8, 2, 888, 5)]  # where a row's residues stop being apart


@pytest.mark.parametrize("log_cols,inv_rate,rows,q", CASES)
def test_encoded_rows_match_the_oracle(dev, oracle, log_cols, inv_rate, rows, q):
    n, nn = 1 << log_cols, inv_rate << log_cols
    rng = np.random.default_rng(log_cols * 1000 + rows)
    data = rng.integers(0, P, size=rows * n, dtype=np.uint64)
    if q:
        pads, pows = rng.integers(0, P, size=rows * q, dtype=np.uint64), oracle.coset_powers(7, nn)
        want = oracle.encode_rows_zk(data, rows, n, pads, q, pows, 18)
        store, leaves = dev.try_commit_zk_keyed(log_cols, inv_rate, data, pads, pows, 18, None)
    else:
        want = oracle.encode_rows_plain(data, rows, n, nn, 18)
        store, leaves = dev.try_commit(log_cols, inv_rate, data, 18)
    assert (leaves == oracle.hash_columns(want, rows, nn)).all()
    store.free()
