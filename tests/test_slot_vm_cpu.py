"""The sumcheck kernels' straight-line programs, compiled and run on the host: the recorded slot graphs and seeded random ones (shared
linear and non-linear nodes, constants, repeated factors, zero coefficients) against the direct evaluation of the graph."""
import ctypes as C
import os
import subprocess
import threading

import numpy as np
import pytest

import ir_util as U

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("vm") / "slot_vm_emul.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", os.path.join(ROOT, "tests", "host_emul", "slot_vm_emul.cpp"), "-o", so])
    return C.CDLL(so)


def _check(emul, prog, desc, n_tables, seed):
    from intelligenceregulation_b200 import backend  # noqa: F401

    rng = np.random.default_rng(seed)
    lo, hi = (rng.integers(0, U.P, size=(n_tables, 2), dtype=np.uint64) for _ in range(2))
    lo[:: 2, 1] = hi[:: 2, 1] = 0  # half of the tables base-valued
    w, cf, info = prog.words(), prog.coef_array(), np.zeros(4, dtype=np.uint32)

    def at(d):
        v = [tuple((int(lo[t][c]) + d * (int(hi[t][c]) - int(lo[t][c]))) % U.P for c in (0, 1)) for t in range(n_tables)]
        return U.py_eval(desc, v)

    for npt, first, skip, parts in ((1, 0, 0, 1), (1, 3, 0, 2), (1, 2, 0, 4), (2, 0, 1, 1), (3, 0, 0, 1), (4, 0, 1, 1), (5, 0, 0, 1), (2, 4, 1, 1)):
        out = np.zeros((npt, 2), dtype=np.uint64)
        emul.emul_vm(w.ctypes.data_as(C.c_void_p), w.size, n_tables, prog.n_nodes, prog.n_terms, cf.ctypes.data_as(C.c_void_p), cf.shape[0],
                     lo.ctypes.data_as(C.c_void_p), hi.ctypes.data_as(C.c_void_p), npt, first, skip, parts, out.ctypes.data_as(C.c_void_p), info.ctypes.data_as(C.c_void_p))
        for j in range(npt):
            d = first + j + (1 if skip and first == 0 and j > 0 else 0)
            assert tuple(int(x) for x in out[j]) == at(d), (npt, first, skip, parts, j)
    return info


@pytest.mark.parametrize("index", range(23))
def test_recorded_graphs(emul, index):
    from intelligenceregulation_b200 import backend

    slot = U.load_slots(os.path.join(ROOT, "tests", "golden"))[index]
    prog, desc = U.build_program(backend, slot, 100 + index)
    info = _check(emul, prog, desc, len(slot["table_fields"]), index)
    assert info[3] == max(U.degrees(slot)[1])
    assert info[1] <= 8 and info[2] <= 24  # what a thread keeps: a fraction of the graph's nodes


@pytest.mark.parametrize("seed", range(12))
def test_random_graphs(emul, seed):
    from intelligenceregulation_b200 import backend

    SP, rng, r = backend.SlotProgram, np.random.default_rng(seed), U.Rand(seed)
    k = int(rng.integers(1, 12))
    prog, desc = SP(k), {"nodes": [], "terms": []}

    def coef():
        return [r.coef("one"), "neg-one", "zero", r.coef("kbase"), r.coef("chal")][int(rng.integers(0, 5))]

    def factors(n_nodes, most):
        return [int(rng.integers(0, k)) if n_nodes == 0 or rng.integers(0, 2) else SP.node(int(rng.integers(0, n_nodes))) for _ in range(int(rng.integers(0, most + 1)))]

    for n in range(int(rng.integers(0, 14))):
        if rng.integers(0, 2):
            terms = [(coef(), int(rng.integers(0, k))) for _ in range(int(rng.integers(0, 4)))]
            konst = coef()
            prog.affine(konst, terms)
            desc["nodes"].append(("affine", konst, terms))
        else:
            subs = [(coef(), factors(n, 2)) for _ in range(int(rng.integers(0, 4)))]
            prog.sum(subs)
            desc["nodes"].append(("sum", subs))
    for _ in range(int(rng.integers(1, 5))):
        c, fs = coef(), factors(prog.n_nodes, 2)
        prog.term(c, [], fs)
        desc["terms"].append((c, fs))
    _check(emul, prog, desc, k, seed)


def _within(seconds, fn):
    """fn() on a thread of its own (the compiler runs without the interpreter's lock), which a compilation without end does not hold up"""
    got = []
    t = threading.Thread(target=lambda: got.append(fn()), daemon=True)
    t.start()
    t.join(seconds)
    assert not t.is_alive(), "still compiling"
    assert got
    return got[0]


@pytest.mark.parametrize("nodes", [4, 24, 126])
def test_every_node_uses_the_one_before_twice(emul, nodes):
    """2^nodes paths through the graph, `nodes` nodes of work"""
    from intelligenceregulation_b200 import backend

    SP, r = backend.SlotProgram, U.Rand(nodes)
    prog, desc = SP(2), {"nodes": [], "terms": []}

    def node(subs):
        desc["nodes"].append(("sum", subs))
        return prog.sum(subs)

    prev = node([(r.coef("chal"), []), (r.coef("chal"), [])])
    for _ in range(nodes):
        prev = node([(r.coef("chal"), [SP.node(prev), SP.node(prev)]), (r.coef("kbase"), [])])
    for t in (0, 1):
        c = r.coef("chal")
        prog.term(c, [], [t, SP.node(prev)])
        desc["terms"].append((c, [t, SP.node(prev)]))
    info = _within(60, lambda: _check(emul, prog, desc, 2, nodes))
    assert info[3] == 1


def test_a_coefficient_replaced_in_place_counts():
    from intelligenceregulation_b200 import backend

    SP = backend.SlotProgram
    prog = SP(2)
    prog.term((5, 7), [0], [1])
    prog.term((11, 0), [], [0])
    w, cf = prog.words(), prog.coef_array()
    assert cf.tolist() == [[5, 7], [11, 0]]
    prog.coefs[0] = (1 << 63, 3)
    assert prog.coef_array().tolist() == [[1 << 63, 3], [11, 0]] and prog._arrays()[1].tolist() == [[1 << 63, 3], [11, 0]]
    assert (prog.words() == w).all()
    prog.coefs[1] = [17, 0]  # a list, which may change without being replaced
    assert prog.coef_array()[1].tolist() == [17, 0]
    prog.coefs[1][0] = 11
    assert prog.coef_array()[1].tolist() == [11, 0]
    prog.term((13, 0), [1], [])
    assert prog.coef_array().tolist() == [[1 << 63, 3], [11, 0], [13, 0]] and prog.words().size > w.size


@pytest.mark.parametrize("nodes", [2, 31, 32, 33, 120])
def test_degrees_that_double_per_node_do_not_wrap(emul, nodes):
    from intelligenceregulation_b200 import backend

    SP = backend.SlotProgram
    prog = SP(1)
    prev = prog.affine((3, 0), [((5, 0), 0)])
    for _ in range(nodes):
        prev = prog.sum([((7, 1), [SP.node(prev), SP.node(prev)])])
    prog.term(SP.ONE, [], [SP.node(prev)])
    w, cf, info = prog.words(), prog.coef_array(), np.zeros(4, dtype=np.uint32)
    tab, out = np.ones((1, 2), dtype=np.uint64), np.zeros((1, 2), dtype=np.uint64)
    _within(60, lambda: [emul.emul_vm(w.ctypes.data_as(C.c_void_p), w.size, 1, prog.n_nodes, prog.n_terms, cf.ctypes.data_as(C.c_void_p), cf.shape[0],
                                      tab.ctypes.data_as(C.c_void_p), tab.ctypes.data_as(C.c_void_p), 1, 0, 0, 1, out.ctypes.data_as(C.c_void_p),
                                      info.ctypes.data_as(C.c_void_p))])
    assert info[3] == min(2 ** nodes, 1 << 20)
