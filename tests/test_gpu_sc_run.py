"""The launch that takes a sumcheck's short rounds together, where its forms part: one chunk of pairs and one pair past it, tables at and
above the length it takes over at, batches that end inside it, and programs whose live values do not fit its shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from intelligenceregulation_b200 import backend

    c = backend.Context(0)
    yield c
    c.close()


def _check(ctx, o, poly, tables, deg, n, batches, what=None, coefs=None):
    from intelligenceregulation_b200 import backend

    tr = o.Transcript(b"sc-run")
    t_cpu = tr.clone()
    want = o.sc_prove(poly, tables, deg, t_cpu, coefs=coefs)
    ev = backend.B200Rounds(ctx, what if what is not None else poly, tables, deg)
    got, st, ctr = [], tr.state, tr.counter
    for b in batches:
        r = ev.batched(b, st, ctr, None)
        got.append(r[0])
        st, ctr = r[3], r[4]
    assert sum(batches) == n and (np.concatenate(got) == want.rounds).all() and st == t_cpu.state
    assert (ev.finals() == want.finals).all()
    ev.free()


@pytest.mark.parametrize("n,batches", [(1, [1]), (6, [6]), (7, [6, 1]), (8, [1] * 8), (18, [18]), (18, [3, 15]), (19, [1, 17, 1]), (20, [2, 18])])
@pytest.mark.parametrize("k,deg", [(2, 2), (3, 3)])
def test_closed_forms(ctx, oracle, n, batches, k, deg):
    tables = oracle.ZkRng(n, b"sc-run").fp2_vec(k << n).reshape(k, 1 << n, 2)
    _check(ctx, oracle, 0, tables, deg, n, batches)


def _program(o, nodes):
    """every node is used twice, at the end: all of them live at once"""
    from intelligenceregulation_b200 import backend

    SP = backend.SlotProgram
    cf = [tuple(map(int, c)) for c in o.ZkRng(nodes, b"sc-run-ir").fp2_vec(3 * nodes)]
    p = SP(4)
    ids = [p.sum([(cf[3 * i], [1 + i % 3, 1 + i // 3 % 3]), (cf[3 * i + 1], [1 + i % 3])]) for i in range(nodes)]
    a = p.sum([(cf[3 * i + 2], [SP.node(d)]) for i, d in enumerate(ids)])
    b = p.sum([(SP.NEG_ONE if i % 2 else SP.ONE, [SP.node(d)]) for i, d in enumerate(ids)])
    p.term(SP.ONE, [0], [SP.node(a)])
    p.term(cf[0], [], [SP.node(b)])
    return p


@pytest.mark.parametrize("nodes,n,batches", [(1, 5, [5]), (1, 6, [5, 1]), (2, 14, [14]), (2, 15, [15]), (30, 11, [11]), (30, 12, [1, 10, 1]), (120, 9, [9]),
                                             (120, 12, [12])])
def test_programs(ctx, oracle, nodes, n, batches):
    p = _program(oracle, nodes)
    tables = oracle.ZkRng(n, b"sc-run-tabs").fp2_vec(4 << n).reshape(4, 1 << n, 2)
    c = p.coef_array()
    oracle.ir_set(p.words(), p.n_nodes, p.n_terms)
    _check(ctx, oracle, oracle.POLY_IR, tables, 3, n, batches, what=p, coefs=c if c.size else None)


@pytest.mark.parametrize("limits,nd", [((0, 1 << 22), 13), ((1 << 12, 0), 13), ((1 << 12, 0), 1), ((1 << 12, 0), 2)])
@pytest.mark.parametrize("parts", [False, True])
def test_a_wait_that_runs_out_is_reported(ctx, oracle, limits, nd, parts):
    """CTA 0's wait for a round's sums, or the others' for a challenge: in the middle of a batch, and for the last challenge of one that ends
    before the last round, when CTA 0 has gone.  The evaluator then answers nothing but that status; the context goes on."""
    from intelligenceregulation_b200 import backend

    n, k, deg = 13, 4, 3
    what = _program(oracle, 30) if parts else backend.POLY_ZC
    tables = oracle.ZkRng(n, b"sc-run-wait").fp2_vec(k << n).reshape(k, 1 << n, 2)
    if parts:
        n, tables = 11, np.ascontiguousarray(tables[:, : 1 << 11])
        nd = min(nd, n)
    tr = oracle.Transcript(b"sc-run-wait")
    ev = backend.B200Rounds(ctx, what, tables, deg)
    ctx.check(ctx.lib.hl_b200_set_wait_limits(ctx.h, *limits))
    try:
        with pytest.raises(backend.DeviceError) as e:
            ev.batched(nd, tr.state, tr.counter, None)
        assert e.value.code == -4 and "wait" in str(e.value)
        for again in (ev.finals, lambda: ev.batched(1, tr.state, tr.counter, None), lambda: ev.round(0), lambda: ev.fold((1, 2))):
            with pytest.raises(backend.DeviceError) as e:
                again()
            assert e.value.code == -4
        ev.free()
    finally:
        ctx.check(ctx.lib.hl_b200_set_wait_limits(ctx.h, 1 << 22, 1 << 22))
    c = None
    if parts:
        c = what.coef_array()
        oracle.ir_set(what.words(), what.n_nodes, what.n_terms)
    _check(ctx, oracle, oracle.POLY_IR if parts else oracle.POLY_ZC, tables, deg, n, [n], what=what if parts else None, coefs=c)


@pytest.mark.parametrize("n", [6, 13])  # the one launch's evaluator, and the long rounds' before it
def test_products_of_words_at_the_carries(ctx, oracle, n):
    """Extension products whose partial sums carry, or do not, in every column: entries from the ends of the 32-bit halves."""
    from intelligenceregulation_b200 import backend

    P = 0xFFFFFFFF00000001
    edge = np.array([0, 1, 7, 2**32 - 1, 2**32, 2**32 + 1, 2**63, P - 2**32, P - 2**32 + 1, P - 2, P - 1], dtype=np.uint64)
    tables = np.random.default_rng(n).choice(edge, size=(4, 1 << n, 2))
    p = backend.SlotProgram(4)
    p.term((P - 1, P - 1), [0], [1, 2, 3])
    o, tr = oracle, oracle.Transcript(b"sc-run")
    scaled = tables.copy()  # the coefficient goes with the first table in the oracle
    scaled[0] = np.array([o.fp2_mul((P - 1, P - 1), tuple(map(int, x))) for x in tables[0]], dtype=np.uint64)
    t_cpu = tr.clone()
    want = o.sc_prove(0, scaled, 4, t_cpu)
    ev = backend.B200Rounds(ctx, p, tables, 4)
    got = ev.batched(n, tr.state, tr.counter, None)
    assert (got[0] == want.rounds).all() and got[3] == t_cpu.state
    ev.free()
