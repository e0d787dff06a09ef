"""Column hashes at the edges of the chunk merge's forms (two chunks and three, 64 and 65, 4,096 columns and more) and table
multiplicities where a warp's queries are all alike, mixed, or fewer than a warp."""
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


@pytest.mark.parametrize("log_cols,rows", [(4, 256), (4, 257), (4, 385), (4, 8192), (4, 8193), (11, 257), (12, 257)])
def test_column_hashes(dev, oracle, log_cols, rows):
    n, nn = 1 << log_cols, 2 << log_cols
    data = np.random.default_rng(rows + log_cols).integers(0, P, size=rows * n, dtype=np.uint64)
    store, leaves = dev.try_commit(log_cols, 2, data, 18)
    assert (leaves == oracle.hash_columns(oracle.encode_rows_plain(data, rows, n, nn, 18), rows, nn)).all()
    store.free()


@pytest.mark.parametrize("size,table", [(1, 1), (31, 7), (33, 256), (100003, 65536), (1 << 18, 4)])
@pytest.mark.parametrize("runs", [False, True])
def test_multiplicities(dev, size, table, runs):
    idx = np.random.default_rng(size).integers(0, table, size=size, dtype=np.int32)
    if runs:
        idx = np.sort(idx)
    assert (dev.ctx.logup_histogram(idx, table) == np.bincount(idx, minlength=table)).all()


@pytest.mark.parametrize("masks", [148, 149])
def test_masking_rows_in_one_pass_and_by_residue(dev, oracle, masks):
    """2 x 148 rows of eight residues are 16 a multiprocessor on 148 of them; one mask more takes a row at a time"""
    from intelligenceregulation_b200 import backend

    tag = oracle.HashTag.for_profile("hashline-zk-mr1/b200-mask/1")
    mc = oracle.mask_commit([(5, 3)] * masks, oracle.ZkRng(masks, b"mask"), tag, 9, 12, 256)
    dm = backend.mask_commit(dev.ctx, mc.msgs, np.stack([mc.b[0], mc.b[1], mc.u[0], mc.u[1]]), oracle.coset_powers(7, 4096), tag.column, 9, 12)
    assert (dm.a_coefs == mc.a_coefs).all() and (dm.leaves == oracle.hash_columns(mc.encoded, 2 * masks + 4, 4096, tag.column)).all()
    dm.free()
