"""Timed workloads of the prover's device path: what a block prover (and its verifier) calls, through the public entry points.

One case is one call sequence of a user's program at one size.  The kinds, and what each stands for in a run:

  commit_host   the hiding commitment with its salted tree from host rows: a boundary plane of a few rows (one per pair of
                blocks), a block's witness matrix `A` (narrow rows, page-locked), a fork's matrix; leaves and tree come back
  commit_dev    the same from rows that are on the device already (the helper matrix `H`): encode, column hash, tree
  open          the opening of a commitment: one combination per claim group (living on a plane's rows and two mask rows), the
                dense proximity combination, and the sampled columns
  verify        the verifier's part of that opening: clear vectors encoded, columns hashed, walked to the root and combined
  mask          the masking commitment `M` with its tree, and its opening
  matmul        the claim of one integer product C = A B: both weight folds and the masked product sumcheck
  logup         the lookup columns of an activation: multiplicities, query helpers, table helpers
  check         the LogUp zero-check of those columns: tables from device planes, masked sumcheck
  slot          one of a block's 23 slot sumchecks, polynomial as data: tables from device planes, masked sumcheck
  witness       one weight product of the block's forward pass, weights and activations resident

Sizes: a block of W16R2_8B_T128_H24 (128 tokens, width 4096, hidden 14336, rows of 2^14 words), the recorded slot graphs of
a W16R2 block core, the boundary planes and forks of the block-sharded run.  All results are exact.
"""
import functools
import json
import os

import numpy as np
import torch

import intelligenceregulation_b200
from intelligenceregulation_b200 import backend

P = 0xFFFFFFFF00000001
GRAPHS = os.path.join(os.path.dirname(intelligenceregulation_b200.__file__), "slot_graphs", "w16r2.json")
WIDE_ROW_STEP = 313  # of a witness matrix, every 313th row holds full-width words (digests, masks), the others int16 values


def listed():
    return [
        # a boundary plane between two blocks: 32 data rows, two reserved pairs and a proximity pair (latency)
        {"name": "commit_plane", "kind": "commit_host", "rows": 38, "log_cols": 12, "inv_rate": 2, "q": 64, "words": "narrow", "keyed": True, "pinned": False},
        # a block's witness matrix `A`, as the prover sends it: narrow rows, page-locked
        {"name": "commit_block_A", "kind": "commit_host", "rows": 2504, "log_cols": 14, "inv_rate": 2, "q": 280, "words": "narrow", "keyed": True, "pinned": True},
        # the block's helper matrix `H`, resident
        {"name": "commit_block_H", "kind": "commit_dev", "rows": 2606, "log_cols": 14, "inv_rate": 2, "q": 280, "words": "field", "keyed": True},
        # the opening of `A`: 37 claim groups, the proximity combination, 280 sampled columns
        {"name": "open_block_A", "kind": "open", "rows": 2504, "log_cols": 14, "inv_rate": 2, "q": 280, "groups": 37, "cols": 280, "keyed": True},
        # the verifier on that opening
        {"name": "verify_block_A", "kind": "verify", "rows": 2504, "log_cols": 14, "inv_rate": 2, "q": 280, "groups": 37, "cols": 280, "keyed": True},
        # the block's masking commitment, 24 masks, committed and opened at 256 columns
        {"name": "mask_block_M", "kind": "mask", "masks": 24, "cols": 256, "keyed": True},
        # one claim of an integer product of 128 tokens, 4096 x 4096 int8 weights
        {"name": "matmul_claim", "kind": "matmul", "tokens": 128, "inner": 4096, "outer": 4096, "keyed": False},
        # the activation lookup of 128 x 14336 values in a table of 2^16
        {"name": "logup_columns", "kind": "logup", "tokens": 128, "hidden": 14336, "log_table": 16},
        # and its zero-check
        {"name": "logup_check", "kind": "check", "n_vars": 21, "keyed": True},
        # a short slot (the row-scale check, 2^14 points) and the heaviest one (the width check, 37 tables, degree 5, 2^19 points)
        {"name": "slot_short", "kind": "slot", "slot": 3, "n_vars": 14, "keyed": True},
        {"name": "slot_width", "kind": "slot", "slot": 14, "n_vars": 19, "keyed": True},
        # the gate projection of the block's forward pass
        {"name": "witness_gate", "kind": "witness", "tokens": 128, "inner": 4096, "outer": 14336, "in_out": False},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["commit_host", "commit_dev", "open", "verify", "mask", "matmul", "logup", "check", "slot", "witness"])
    c = {"kind": kind}
    if kind in ("commit_host", "commit_dev", "open", "verify"):
        c["log_cols"] = rng.randint(10, 14) if kind != "commit_dev" else rng.randint(10, 16)
        c["inv_rate"] = rng.choice([2, 2, 2, 4])
        cap = (41 << 20 >> c["log_cols"]) * 2 // c["inv_rate"]
        c["rows"] = _log_uniform(rng, 24, min(cap, 2606 if c["log_cols"] <= 14 else cap))
        c["q"] = rng.randint(33, 320)
        c["keyed"] = rng.random() < 0.75
        if kind == "commit_host":
            c["words"] = rng.choice(["narrow", "narrow", "field"])
            c["pinned"] = rng.random() < 0.5
            if c["words"] == "field":
                c["rows"] = min(c["rows"], 512)
        elif kind == "commit_dev":
            c["words"] = rng.choice(["narrow", "field"])
        else:
            c["rows"] = max(c["rows"], 96)
            c["groups"] = rng.randint(1, 37)
            c["cols"] = rng.randint(64, 280)
    elif kind == "mask":
        c.update(masks=rng.randint(2, 48), cols=rng.randint(32, 256), keyed=rng.random() < 0.75)
    elif kind == "matmul":
        # the inner axis is the sumcheck's: a power of two in this protocol (the callers pad); tokens and outputs are ragged
        c.update(tokens=_log_uniform(rng, 4, 512), inner=1 << rng.randint(8, 12), outer=_log_uniform(rng, 200, 4096), keyed=rng.random() < 0.5)
    elif kind == "logup":
        c.update(tokens=_log_uniform(rng, 4, 128), hidden=_log_uniform(rng, 300, 14336), log_table=rng.choice([8, 12, 16]))
    elif kind == "check":
        c.update(n_vars=rng.randint(8, 21), keyed=rng.random() < 0.75)
    elif kind == "slot":
        s = rng.randrange(len(_graphs()))
        k, top = len(_graphs()[s]["tables"]), 21
        while k << top > 37 << 19:
            top -= 1
        c.update(slot=s, n_vars=rng.randint(7, top), keyed=rng.random() < 0.75)
    else:
        c.update(tokens=_log_uniform(rng, 1, 300), inner=_log_uniform(rng, 200, 14336), outer=_log_uniform(rng, 100, 4096), in_out=rng.random() < 0.3)
    return c


@functools.lru_cache(None)
def _graphs():
    with open(GRAPHS) as f:
        return json.load(f)["slots"]


@functools.lru_cache(None)
def _backend():
    """One context for the process, as a prover keeps it."""
    return backend.B200Backend()


@functools.lru_cache(None)
def _coset_powers(nn):
    out, x = np.empty(nn, dtype=np.uint64), 1
    for i in range(nn):
        out[i] = x
        x = x * 7 % P
    return out


class _Rand:
    """Seeded inputs: field words, witness words, host arrays and bytes."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.np = np.random.default_rng(seed)

    def field_dev(self, n):
        """uniform canonical words on the device, as int64 (p = 2^64 - 2^32 + 1: the words from p up are -2^32 + 1 .. -1)"""
        x = torch.randint(-(1 << 63), (1 << 63) - 1, (n,), dtype=torch.int64, device="cuda", generator=self.gen)
        return torch.where((x < 0) & (x > -(1 << 32)), x & 0x7FFFFFFFFFFFFFFF, x)

    def int16_dev(self, n):
        """int16 values of a quantised activation"""
        return (torch.randn(n, device="cuda", generator=self.gen) * 4096).round().clamp(-32768, 32767).to(torch.int16)

    def witness_dev(self, n):
        """the same as field words: x >= 0 as x, x < 0 as p + x"""
        v = self.int16_dev(n).to(torch.int64)
        return torch.where(v < 0, v + (1 - (1 << 32)), v)

    def field(self, *shape):
        x = self.np.integers(0, 1 << 63, size=shape, dtype=np.uint64) * np.uint64(2)
        return x % np.uint64(P)

    def pair(self):
        return tuple(int(v) for v in self.field(2))

    def key(self):
        return self.np.bytes(32)


def _host(t):
    return t.cpu().numpy()


def _signed(a):
    """uint64 words as int64, whole"""
    return np.ascontiguousarray(a).view(np.int64)


def _matrix_dev(r, case):
    rows, n = case["rows"], 1 << case["log_cols"]
    if case.get("words", "narrow") == "field":
        return r.field_dev(rows * n)
    data = r.witness_dev(rows * n).view(rows, n)
    wide = range(0, rows, WIDE_ROW_STEP)
    data[::WIDE_ROW_STEP] = r.field_dev(len(wide) * n).view(len(wide), n)
    return data.view(-1)


def _packed(r, case):
    """(packed bytes, widths) of a witness matrix: int16 rows, every WIDE_ROW_STEP-th row 64-bit words"""
    rows, n = case["rows"], 1 << case["log_cols"]
    parts, widths = [], np.full(rows, 2, dtype=np.uint8)
    widths[::WIDE_ROW_STEP] = 8
    for at in range(0, rows, WIDE_ROW_STEP):
        parts.append(r.field_dev(n).view(torch.uint8))
        parts.append(r.int16_dev((min(at + WIDE_ROW_STEP, rows) - at - 1) * n).view(torch.uint8))
    return torch.cat(parts).cpu(), widths


def _keys(r, case):
    return [r.key() if case["keyed"] else None for _ in range(3)]


def _prepare_commit_host(case, r):
    rows, n = case["rows"], 1 << case["log_cols"]
    nn = n * case["inv_rate"]
    s = {"pows": _coset_powers(nn)}
    if case["words"] == "narrow":
        data, s["widths"] = _packed(r, case)
    else:
        data = r.field_dev(rows * n).cpu()
    pads = r.field_dev(rows * case["q"]).cpu()
    salts = r.field_dev(nn * 4).cpu()
    levels = torch.empty(((2 * nn - 1), 32), dtype=torch.uint8)
    if case["pinned"]:
        data, pads, salts, levels = (t.pin_memory() for t in (data, pads, salts, levels))
    s["hold"] = (data, pads, salts, levels)
    s.update(data=data.numpy(), pads=pads.numpy().view(np.uint64), salts=salts.numpy().view(np.uint8), levels=levels.numpy())
    if "widths" not in s:
        s["data"] = s["data"].view(np.uint64)
    s["keys"] = _keys(r, case)
    return s


def _run_commit_host(case, s):
    be, lc, ir, top = _backend(), case["log_cols"], case["inv_rate"], case["log_cols"] + case["inv_rate"].bit_length() - 1
    col, leaf, node = s["keys"]
    if "widths" in s:
        got = be.try_commit_zk_packed(lc, ir, s["data"], s["widths"], s["pads"], s["pows"], top, col, s["salts"], leaf, node, levels_out=s["levels"], want_leaves=False)
    else:
        got = be.try_commit_zk_tree(lc, ir, s["data"], s["pads"], s["pows"], top, col, s["salts"], leaf, node, levels_out=s["levels"], want_leaves=False)
    store, _, levels = got
    store.free()
    return levels


def _prepare_commit_dev(case, r):
    nn = case["inv_rate"] << case["log_cols"]
    return {"data": _matrix_dev(r, case), "pads": r.field_dev(case["rows"] * case["q"]), "pows": torch.from_numpy(_coset_powers(nn).view(np.int64)).cuda(),
            "salts": r.field_dev(nn * 4), "levels": torch.empty((2 * nn - 1, 32), dtype=torch.uint8, device="cuda"), "keys": _keys(r, case)}


def _commit_dev(case, s):
    be = _backend()
    col, leaf, node = s["keys"]
    store = be.commit_zk_dev(case["log_cols"], case["inv_rate"], s["data"].data_ptr(), case["rows"], s["pads"].data_ptr(), case["q"], s["pows"].data_ptr(), col)
    store.merkle_dev(s["salts"].data_ptr(), leaf, node, s["levels"].data_ptr())
    return store


def _run_commit_dev(case, s):
    _commit_dev(case, s).free()
    return s["levels"]


def _row_weights(r, case, dense):
    """one vector per claim group, living on its claim's 32 plane rows and two mask rows, then `dense` full ones"""
    rows, g = case["rows"], case["groups"]
    w = np.zeros((g + dense, rows, 2), dtype=np.uint64)
    for i in range(g):
        r0 = (i * 64) % (rows - 40)
        w[i, r0:r0 + 32] = r.field(32, 2)
        w[i, rows - 3:rows - 1] = r.field(2, 2)
    w[g:] = r.field(dense, rows, 2)
    return w


def _prepare_open(case, r):
    s = _prepare_commit_dev(case, r)
    s["store"] = _commit_dev(case, s)
    s["rhos"] = _row_weights(r, case, 1)
    s["idx"] = r.np.integers(0, s["store"].nn, size=case["cols"], dtype=np.uint64)
    return s


def _run_open(case, s):
    return {"vectors": _signed(s["store"].fold_rows_with_pads(s["rhos"])), "columns": _signed(s["store"].columns(s["idx"]))}


def _prepare_verify(case, r):
    """What a verifier receives.  A few columns were tampered with, at seeded places: it meets those too, and the verdicts name them."""
    s = _prepare_commit_dev(case, r)
    store = _commit_dev(case, s)
    rhos = _row_weights(r, case, 2)
    vecs = store.fold_rows_with_pads(rhos)
    idx = r.np.integers(0, store.nn, size=case["cols"], dtype=np.uint64)
    cols = store.columns(idx)
    torch.cuda.synchronize()
    levels, salts = _host(s["levels"]), _host(s["salts"].view(torch.uint8)).reshape(-1, 32)
    store.free()
    nn = case["inv_rate"] << case["log_cols"]
    depth = nn.bit_length() - 1
    paths = np.empty((case["cols"], depth, 32), dtype=np.uint8)
    at, off, width = idx.astype(np.int64), 0, nn
    for level in range(depth):  # the sibling at every level below the root
        paths[:, level] = levels[off + (at ^ 1)]
        at, off, width = at >> 1, off + width, width // 2
    bad = r.np.choice(case["cols"], size=1 + case["cols"] // 32, replace=False)
    cols[bad, r.np.integers(0, case["rows"], size=bad.size)] ^= np.uint64(1)
    return {"pows": _coset_powers(nn), "args": (cols, idx, np.ascontiguousarray(salts[idx.astype(np.int64)]), paths, bytes(levels[-1]), *s["keys"], rhos, vecs)}


def _run_verify(case, s):
    return _backend().check_opening_columns(case["log_cols"], case["inv_rate"], s["pows"], case["log_cols"] + 2, *s["args"])


def _prepare_mask(case, r):
    m = r.field(2 * case["masks"], 512)
    m[:, 320:] = 0  # coefficients and pads, then zeros
    return {"msgs": m, "coefs": r.field(4, 1024), "pows": _coset_powers(4096), "salts": r.field(4096, 4).view(np.uint8), "ws": r.field(case["masks"], 512, 2),
            "rs": r.field(2 * case["masks"] + 2, 2), "idx": r.np.integers(0, 4096, size=case["cols"], dtype=np.uint64), "keys": _keys(r, case)}


def _run_mask(case, s):
    col, leaf, node = s["keys"]
    m = backend.mask_commit(_backend().ctx, s["msgs"], s["coefs"], s["pows"], col)
    out = {"coefs": _signed(m.a_coefs), "levels": m.merkle(s["salts"], leaf, node), "q": _signed(m.open_q(s["ws"])), "prox": _signed(m.prox(s["rs"])),
           "columns": _signed(m.columns(s["idx"]))}
    m.free()
    return out


def _transcript(r, case):
    return {"state": r.key(), "counter": int(r.np.integers(0, 1 << 20)), "key": r.key() if case["keyed"] else None}


def _sumcheck(ev, n_vars, s, claim):
    """the masked sumcheck as the prover drives it: all rounds in one device batch, then the final table values"""
    sums, absorbed, challenges, state, counter, _ = ev.batched(n_vars, s["state"], s["counter"], s["key"], mask=s["mask"], mask_vars=n_vars + 1, mask_c=s["mask_c"],
                                                               recover_one=True, claim=claim)
    out = {"sums": _signed(sums), "absorbed": _signed(absorbed), "challenges": _signed(challenges), "state": np.frombuffer(state, dtype=np.uint8), "counter": counter,
           "finals": _signed(ev.finals())}
    ev.free()
    return out


def _mask_of(r, n_vars, degree):
    return {"mask": r.field((n_vars + 1) * degree + 2, 2), "mask_c": r.pair()}


def _prepare_matmul(case, r):
    a = r.np.integers(-128, 128, size=(case["tokens"], case["inner"]), dtype=np.int8)
    b = _host((torch.randn(case["inner"], case["outer"], device="cuda", generator=r.gen) * 32).round().clamp(-128, 127).to(torch.int8))
    n = case["inner"].bit_length() - 1
    # the eq weights of the claim's token and output points
    return {"a": a, "b": b, "eq_i": r.field(case["tokens"], 2), "eq_j": r.field(case["outer"], 2), "n": n, **_transcript(r, case), **_mask_of(r, n, 2), "claim": r.pair()}


def _run_matmul(case, s):
    ctx = _backend().ctx
    tables = np.stack([ctx.fold_rows_i8(s["a"], s["eq_i"]), ctx.fold_cols_i8(s["b"], s["eq_j"])])
    ev = backend.B200Rounds(ctx, backend.POLY_PROD, tables, 2)
    return {"tables": _signed(tables), **_sumcheck(ev, s["n"], s, s["claim"])}


def _prepare_logup(case, r):
    size = 1 << case["log_table"]
    mid, padded = size // 2, 1 << (case["hidden"] - 1).bit_length()
    x = (np.arange(size) - mid) / 4096.0
    table = np.clip(np.rint(x / (1.0 + np.exp(-x)) * 4096.0), -32768, 32767).astype(np.int32)  # a quantised SiLU
    v = (torch.randn(case["tokens"], case["hidden"], device="cuda", generator=r.gen) * (size / 16)).round().clamp(-mid, mid - 1).to(torch.int32) + mid
    idx = np.full((case["tokens"], padded), mid, dtype=np.int32)  # padding looks up the entry of value 0
    idx[:, :case["hidden"]] = _host(v)
    idx = idx.reshape(-1)
    return {"idx": idx, "out": table[idx], "table": table, "alpha": r.pair(), "beta": r.pair(), "tag": r.pair()}


def _run_logup(case, s):
    ctx = _backend().ctx
    mult = ctx.logup_histogram(s["idx"], s["table"].size)
    h = ctx.logup_helpers(s["idx"], s["out"], s["alpha"], s["beta"], s["tag"])
    ht = ctx.logup_helpers(None, s["table"], s["alpha"], s["beta"], s["tag"], mult=mult)
    return {"mult": _signed(mult), "h": _signed(h), "ht": _signed(ht)}


def _prepare_check(case, r):
    n = case["n_vars"]
    # h and q as their real and imaginary planes of the resident helper matrix
    return {"rows": r.field_dev(4 << n), "point": r.field(n, 2), "alpha": np.array([r.pair()], dtype=np.uint64), **_transcript(r, case), **_mask_of(r, n, 3)}


def _run_check(case, s):
    ctx, n = _backend().ctx, case["n_vars"]
    rows, cube = (s["rows"].data_ptr(), s["rows"].numel()), [("rho", v) for v in range(n)]
    tabs = backend.B200Tables(ctx, 3, n)
    tabs.plan_eq(0, s["point"], 0)
    tabs.plan_plane(1, rows, cube, [(0, (1, 0)), (1 << n, (0, 1))])
    tabs.plan_plane(2, rows, cube, [(2 << n, (1, 0)), (3 << n, (0, 1))])
    return _sumcheck(backend.B200Rounds(ctx, backend.POLY_LOGUP_Q, tabs, 3, s["alpha"]), n, s, (0, 0))


@functools.lru_cache(None)
def _program(slot):
    g = _graphs()[slot]
    prog = backend.SlotProgram(len(g["tables"]))

    def coef(c):
        return c[2] if c[2] in ("one", "neg-one") else (c[0], c[1])

    def factors(fs):
        return [prog.node(i) if kind == "n" else i for kind, i in fs]

    for node in g["nodes"]:
        if "affine" in node:
            prog.affine(tuple(node["konst"][:2]), [(coef(c), t) for c, t in node["affine"]])
        else:
            prog.sum([(coef(c), factors(fs)) for c, fs in node["sum"]])
    for t in g["terms"]:
        prog.term(coef(t["coef"]), t["wrapper"], factors(t["inner"]))
    return prog


def _prepare_slot(case, r):
    """Each table's source: an eq cube; a helper column (two planes of the helper rows); in the matmul slots (5 .. 13) a public
    table of folded weights, made on the host; otherwise a plane of the witness rows."""
    g, n = _graphs()[case["slot"]], case["n_vars"]
    k, size = len(g["tables"]), 1 << n
    s = {"witness": r.witness_dev(k * size), "helpers": r.field_dev(2 * k * size), "tables": []}
    for t, kind in enumerate(g["tables"]):
        if kind in ("eq", "geq"):
            s["tables"].append(("eq", r.field(n, 2)))
        elif kind == "H":
            s["tables"].append(("helpers", [(2 * t * size, (1, 0)), ((2 * t + 1) * size, (0, 1))]))
        elif kind == "pub" and 5 <= case["slot"] <= 13:
            s["tables"].append(("put", r.field(size, 2)))
        else:
            s["tables"].append(("witness", [(t * size, (1, 0))]))
    return {**s, **_transcript(r, case), **_mask_of(r, n, g["degree"])}


def _run_slot(case, s):
    ctx, n = _backend().ctx, case["n_vars"]
    cube = [("rho", v) for v in range(n)]
    tabs = backend.B200Tables(ctx, len(s["tables"]), n)
    for t, (kind, what) in enumerate(s["tables"]):
        if kind == "eq":
            tabs.plan_eq(t, what, 0)
        elif kind == "put":
            tabs.put(t, what)
        else:
            tabs.plan_plane(t, (s[kind].data_ptr(), s[kind].numel()), cube, what)
    return _sumcheck(backend.B200Rounds(ctx, _program(case["slot"]), tabs, _graphs()[case["slot"]]["degree"]), n, s, (0, 0))


def _prepare_witness(case, r):
    t, k, n = case["tokens"], case["inner"], case["outer"]
    w = (torch.randn(k * n, device="cuda", generator=r.gen) * 32).round().clamp(-128, 127).to(torch.int8)
    return {"x": r.int16_dev(t * k).to(torch.int64), "w": w, "out": torch.empty(t * n, dtype=torch.int64, device="cuda")}


def _run_witness(case, s):
    t, k, n = case["tokens"], case["inner"], case["outer"]
    taken = _backend().ctx.witness_product_dev(t, s["x"].data_ptr(), t * k, k, s["w"].data_ptr(), k * n, k, n, n, t * n, case["in_out"], s["out"].data_ptr())
    return {"taken": taken, "out": s["out"]}


def prepare(case, seed):
    s = globals()["_prepare_" + case["kind"]](case, _Rand(seed))
    s["case"] = case
    return s


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state["case"], state)


def work(case):
    """Bytes each input is read and each output written once with.  The arithmetic of all kinds but `witness` is on whole 64-bit
    field words and hash words, which no floating-point rate bounds: flops stay 0 there."""
    c, kind = case, case["kind"]
    if kind in ("commit_host", "commit_dev", "open", "verify"):
        rows, n = c["rows"], 1 << c["log_cols"]
        nn = n * c["inv_rate"]
        if kind in ("commit_host", "commit_dev"):
            wide = -(-rows // WIDE_ROW_STEP) if c["words"] == "narrow" and kind == "commit_host" else rows
            # rows and pads in, the encoding (which stays for the opening) and the tree out
            return {"bytes": n * (8 * wide + 2 * (rows - wide)) + 8 * rows * c["q"] + 8 * rows * nn + 32 * nn + 64 * nn, "flops": 0}
        if kind == "open":
            vecs = c["groups"] + 1
            return {"bytes": 8 * rows * (n + c["q"]) + 16 * vecs * (rows + n + c["q"]) + 16 * c["cols"] * rows, "flops": 0}
        vecs = c["groups"] + 2
        return {"bytes": 8 * c["cols"] * rows + 16 * vecs * (rows + n + c["q"]) + c["cols"] * 32 * nn.bit_length() + 4 * c["cols"], "flops": 0}
    if kind == "mask":
        m, rows = c["masks"], 2 * c["masks"] + 4
        return {"bytes": 8 * 512 * 2 * m * 2 + 8 * 4096 * rows + 96 * 4096 + 16 * 512 * m + 16 * 1024 * 2 + 8 * c["cols"] * rows, "flops": 0}
    if kind == "matmul":
        return {"bytes": c["inner"] * (c["tokens"] + c["outer"]) + 16 * (c["tokens"] + c["outer"] + 2 * c["inner"]), "flops": 0}
    if kind == "logup":
        queries = c["tokens"] << (c["hidden"] - 1).bit_length()
        return {"bytes": 24 * queries + (28 << c["log_table"]), "flops": 0}
    if kind == "check":
        return {"bytes": 32 << c["n_vars"], "flops": 0}
    if kind == "slot":
        per = [{"eq": 0, "geq": 0, "H": 16}.get(t, 16 if t == "pub" and 5 <= c["slot"] <= 13 else 8) for t in _graphs()[c["slot"]]["tables"]]
        return {"bytes": sum(per) << c["n_vars"], "flops": 0}
    t, k, n = c["tokens"], c["inner"], c["outer"]
    return {"bytes": 8 * t * k + k * n + 8 * t * n, "flops": 2 * t * k * n}


def tolerance(case):
    return "exact"
