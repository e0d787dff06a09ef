"""The tensor-core row encoder at the edges of its forms: full and short batches of rows per 2^14 words, one residue or all of them a CTA, pads that
reach most of a row and beyond it, rates 1 to 1/64, packed rows of every width, and rows that do not start on 32-byte boundaries; and
what reads an encoding that lies residue by residue."""
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


# log_cols, inv_rate, rows, q: (10 .. 13) just above the line where the tensor cores take over, a last batch of one row
CASES = [(10, 2, 2369, 33), (11, 2, 1185, 320), (12, 2, 593, 1), (12, 4, 601, 40), (13, 2, 149, 281), (13, 4, 41, 8000),
         (14, 2, 3, 280), (14, 2, 149, 5), (14, 4, 38, 40001), (14, 4, 2, 1), (14, 1, 2, 0), (14, 2, 75, 0),
         # rates that keep many residues' words, whole batches and split ones
         (14, 8, 3, 280), (14, 8, 79, 17), (14, 16, 75, 0), (14, 64, 2, 20001), (13, 8, 21, 9), (12, 8, 593, 12), (10, 16, 2353, 5)]


@pytest.mark.parametrize("log_cols,inv_rate,rows,q", CASES)
def test_commitments_and_columns(dev, oracle, log_cols, inv_rate, rows, q):
    n, nn = 1 << log_cols, inv_rate << log_cols
    top = max(18, nn.bit_length() - 1)
    rng = np.random.default_rng(log_cols * 1000 + rows)
    data = rng.integers(0, P, size=rows * n, dtype=np.uint64)
    data[:n] = P - 1
    data[-n:] = 0
    if q:
        pads, pows = rng.integers(0, P, size=rows * q, dtype=np.uint64), oracle.coset_powers(7, nn)
        want = oracle.encode_rows_zk(data, rows, n, pads, q, pows, top)
        store, leaves = dev.try_commit_zk_keyed(log_cols, inv_rate, data, pads, pows, top, None)
    else:
        want = oracle.encode_rows_plain(data, rows, n, nn, top)
        store, leaves = dev.try_commit(log_cols, inv_rate, data, top)
    assert (leaves == oracle.hash_columns(want, rows, nn)).all()
    idx = np.array([0, nn - 1, nn // 2, 1 % nn, 5 % nn, nn // 3], dtype=np.uint64)
    cols = oracle.gather_columns(want, rows, nn, idx)
    assert (store.columns(idx) == cols).all()
    if not q:  # a plain store folds the systematic positions of its encoding
        rhos = rng.integers(0, P, size=(2, rows, 2), dtype=np.uint64)
        assert (store.fold_rows(rhos) == oracle.fold_rows(np.ascontiguousarray(want.reshape(rows, nn)[:, ::inv_rate]).reshape(-1), rows, n, n, 1, rhos)).all()
    if rows < 200 and nn <= 1 << 18:  # in the columns' own order, for callers on the device, and what reads it afterwards
        import torch
        from intelligenceregulation_b200 import backend

        out = torch.empty((nn, 32), dtype=torch.uint8, device="cuda")
        backend.hash_columns_static(store.encoded_dev(), rows, nn, None, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert (out.cpu().numpy() == leaves).all()
        assert (store.columns(idx) == cols).all()
    store.free()


@pytest.mark.parametrize("log_cols,inv_rate,rows,q", [(12, 2, 593, 64), (13, 2, 150, 33), (14, 2, 40, 280), (14, 4, 75, 7)])
def test_packed_rows_of_every_width(dev, oracle, log_cols, inv_rate, rows, q):
    n, nn = 1 << log_cols, inv_rate << log_cols
    rng = np.random.default_rng(rows)
    widths = rng.choice(np.array([1, 2, 4, 8], dtype=np.uint8), size=rows)
    parts, wide = [], []
    for w in map(int, widths):
        if w == 8:
            row = rng.integers(0, P, size=n, dtype=np.uint64)
            wide.append(row)
        else:
            row = rng.integers(-(1 << (8 * w - 1)), 1 << (8 * w - 1), size=n).astype({1: np.int8, 2: np.int16, 4: np.int32}[w])
            row[:2] = [-(1 << (8 * w - 1)), (1 << (8 * w - 1)) - 1]
            wide.append(np.where(row < 0, row.astype(np.int64).astype(np.uint64) + np.uint64(P), row.astype(np.uint64)))
        parts.append(row.view(np.uint8))
    data = np.concatenate(wide).astype(np.uint64)
    pads, pows = rng.integers(0, P, size=rows * q, dtype=np.uint64), oracle.coset_powers(7, nn)
    want = oracle.encode_rows_zk(data, rows, n, pads, q, pows, 18)
    salts = rng.integers(0, 256, size=(nn, 32), dtype=np.uint8)
    store, leaves, _ = dev.try_commit_zk_packed(log_cols, inv_rate, np.concatenate(parts), widths, pads, pows, 18, None, salts, None, None)
    assert (leaves == oracle.hash_columns(want, rows, nn)).all()
    rhos = rng.integers(0, P, size=(1, rows, 2), dtype=np.uint64)
    assert (store.fold_rows(rhos) == oracle.fold_rows(data, rows, n, n, 1, rhos)).all()  # the widened rows
    store.free()


def test_rows_on_8_byte_boundaries(dev, oracle):
    import torch

    rows, q, n = 9, 31, 1 << 14
    rng = np.random.default_rng(3)
    data, pads = rng.integers(0, P, size=rows * n, dtype=np.uint64), rng.integers(0, P, size=rows * q, dtype=np.uint64)
    pows = oracle.coset_powers(7, 2 * n)
    up = lambda a, off: torch.from_numpy(np.concatenate([np.zeros(off, dtype=np.uint64), a]).view(np.int64)).cuda()
    d, p, h = up(data, 1), up(pads, 1), up(pows, 1)
    out = torch.empty((2 * n, 32), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    store = dev.commit_zk_dev(14, 2, d.data_ptr() + 8, rows, p.data_ptr() + 8, q, h.data_ptr() + 8, None, d_leaves=out.data_ptr())
    idx = np.arange(0, 2 * n, 4097, dtype=np.uint64)
    want = oracle.encode_rows_zk(data, rows, n, pads, q, pows, 18)
    assert (store.columns(idx) == oracle.gather_columns(want, rows, 2 * n, idx)).all()
    assert (out.cpu().numpy() == oracle.hash_columns(want, rows, 2 * n)).all()
    store.free()


def test_a_wait_that_runs_out_is_told_to_its_own_store(dev, oracle):
    """The kernel looks at its barriers no more than it is let: its CTAs give up, walk to their end and leave the machine as it was.  The store
    answers nothing but that status, another store made beside it and one made afterwards are whole."""
    from intelligenceregulation_b200 import backend

    rows, n, ctx = 160, 1 << 14, dev.ctx
    rng = np.random.default_rng(11)
    data = rng.integers(0, P, size=rows * n, dtype=np.uint64)
    idx = np.array([0, 5, 2 * n - 1], dtype=np.uint64)
    want = oracle.gather_columns(oracle.encode_rows_plain(data, rows, n, 2 * n, 18), rows, 2 * n, idx)

    import torch

    d = torch.from_numpy(data.view(np.int64)).cuda()
    p, h = torch.zeros(rows, dtype=torch.int64, device="cuda"), torch.ones(2 * n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    commit = lambda: dev.commit_zk_dev(14, 2, d.data_ptr(), rows, p.data_ptr(), 1, h.data_ptr(), None)
    fine = commit()
    ctx.check(ctx.lib.hl_b200_set_encoder_wait_limit(ctx.h, 0))
    try:
        lost, gone = commit(), commit()
        gone.free()
        assert dev.try_commit(14, 2, data, 18) is None and "wait" in dev.ctx.declines[-1][1]
    finally:
        ctx.check(ctx.lib.hl_b200_set_encoder_wait_limit(ctx.h, 1 << 22))
    assert (fine.columns(idx) == want).all()
    later, _ = dev.try_commit(14, 2, data, 18)
    assert (later.columns(idx) == want).all()
    for _ in range(2):
        for ask in (lambda: lost.columns(idx), lambda: lost.merkle(None, None, None), lambda: lost.fold_rows(np.ones((1, rows, 2), dtype=np.uint64))):
            with pytest.raises(backend.DeviceError) as e:
                ask()
            assert e.value.code == -4
    with pytest.raises(backend.DeviceError) as e:
        ctx.sync()
    assert e.value.code == -4
    ctx.sync()
    for s in (fine, later, lost):
        s.free()


# log_cols, inv_rate, rows, q, whole batches, the scratch they are left in MB: few rows never keep the other residues' words, and where there is no memory
# for them many rows do without
@pytest.mark.parametrize("log_cols,inv_rate,rows,q,left", [(14, 64, 4, 280, 2), (14, 256, 2, 5, 1), (14, 8, 140, 31, 16), (14, 2, 149, 7, 16), (13, 4, 296, 40, 16)])
def test_scratch_does_not_grow_with_the_rate(oracle, log_cols, inv_rate, rows, q, left):
    from intelligenceregulation_b200 import backend

    n, nn = 1 << log_cols, inv_rate << log_cols
    dev = backend.B200Backend(device=0)
    rng = np.random.default_rng(rows)
    data, pads = rng.integers(0, P, size=rows * n, dtype=np.uint64), rng.integers(0, P, size=rows * q, dtype=np.uint64)
    pows = oracle.coset_powers(7, nn)
    dev.ctx.set_alloc_cap((rows * (n + q + nn) + 5 * nn) * 8 + (rows + 127) // 128 * nn * 32 + (left << 20))  # what the call has to hold, and that
    got = dev.try_commit_zk(log_cols, inv_rate, data, pads, pows, log_cols + inv_rate.bit_length() - 1)
    assert got is not None, dev.ctx.declines
    store, leaves = got
    assert (leaves == oracle.hash_columns(oracle.encode_rows_zk(data, rows, n, pads, q, pows, log_cols + inv_rate.bit_length() - 1), rows, nn)).all()
    store.free()
    dev.ctx.close()


@pytest.mark.parametrize("fit", [0, 1, 3, 40])
def test_the_columns_order_with_little_memory(oracle, fit):
    """the encoding is put into the columns' order with as many rows of scratch as there is memory for; with none that is an error, not an
    address of 0, and the store stays as it was"""
    import torch
    from intelligenceregulation_b200 import backend

    rows, n, q = 40, 1 << 14, 12
    nn = 2 * n
    dev = backend.B200Backend(device=0)
    rng = np.random.default_rng(fit)
    data, pads = rng.integers(0, P, size=rows * n, dtype=np.uint64), rng.integers(0, P, size=rows * q, dtype=np.uint64)
    store, leaves = dev.try_commit_zk(14, 2, data, pads, oracle.coset_powers(7, nn), 18)
    dev.ctx.set_alloc_cap((rows * (n + q + nn) + 4 * nn + fit * nn) * 8 + 64)  # what the store holds, and that many rows
    out = torch.empty((nn, 32), dtype=torch.uint8, device="cuda")
    if fit == 0:
        with pytest.raises(backend.DeviceError):
            store.encoded_dev()
        dev.ctx.set_alloc_cap(0)
    backend.hash_columns_static(store.encoded_dev(), rows, nn, None, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert (out.cpu().numpy() == leaves).all()
    dev.ctx.set_alloc_cap(0)
    store.free()
    dev.ctx.close()
