"""Reference-order walks that give subtrees away (td_ordered.cuh), on the host:
the rules of the split and of the endgame table, with a warp always waiting,
against the oracle's one walk.  Status, witness and expansions equal it; among
the walks are some that pass by a level whose remaining children the table
decides, and whose witness lies before them."""
import ctypes as C
import math
import os

import numpy as np
import pytest

SYMBOLS = 11


@pytest.fixture(scope="module")
def split_search(emu):
    from td16_b200 import _lib
    size = sum(math.factorial(q) for q in range(2, SYMBOLS))
    table = np.zeros(size, np.uint16)
    emu.td_emu_endgame.restype = C.c_long
    assert emu.td_emu_endgame(SYMBOLS, C.c_void_p(table.ctypes.data), max(1, min(16, os.cpu_count() or 1))) == 0

    def run(inst, after, every):
        x = np.ascontiguousarray(inst).reshape(1)
        res = np.zeros(1, _lib.RESULT_DTYPE)
        counts = np.zeros(2, np.int64)
        emu.td_emu_split_search(C.c_void_p(x.ctypes.data), C.c_void_p(table.ctypes.data), after, every,
                                C.c_void_p(res.ctypes.data), C.c_void_p(counts.ctypes.data))
        return res[0], counts

    return run


def _check(td, oracle, split_search, cases, settings):
    """cases: (permutation, bound, rate, full)."""
    total = np.zeros(2, np.int64)  # nodes, levels kept
    for p, bound, rate, full in cases:
        perm = np.zeros((1, 16), np.int8)
        perm[0, : len(p)] = p
        inst = td.prepare_perms(perm, len(p), bound, rate, full)
        status, moves, exp = oracle.search(*oracle.perm_to_pair(list(p)), rate, bound, full)
        for after, every in settings:
            r, counts = split_search(inst[0], after, every)
            total += counts
            assert (r["status"], r["expansions"]) == (status, exp + 1), (p, bound, after, every)
            assert td._lib.unpack_moves(r) == moves
    return total


def test_decided_children_after_the_walks_subtree(td, oracle, split_search):
    walks = [([10, 9, 8, 7, 6, 5, 4, 3, 2, 1, 12, 11, 0], 7), ([12, 10, 9, 8, 7, 4, 6, 5, 3, 2, 1, 11, 0], 7),
             ([13, 12, 11, 10, 9, 1, 0, 8, 7, 6, 5, 4, 3, 2], 7)]
    nodes, kept = _check(td, oracle, split_search, [(p, b, 0.0, True) for p, b in walks],
                         [(1, 1), (1, 8), (8, 8), (64, 8)])
    assert nodes > 0 and kept > 0


@pytest.mark.parametrize("n", [8, 11, 12, 13])
def test_near_reverse_walks(td, oracle, split_search, n):
    perms, size = td.synth_perms(700 + n, 40, n, n, 100, 1, 3)
    cases = []
    for p in perms:
        _, _, init = oracle.perm_to_pair(p[:n].tolist())
        cases += [(p[:n].tolist(), min(9, (n + 2 - init) // 2 + over), 0.0, True) for over in (0, 1)]
    assert _check(td, oracle, split_search, cases, [(1, 1), (8, 8)])[0] > 0


@pytest.mark.parametrize("n", [6, 9])
def test_partial_sorting(td, oracle, split_search, n):
    """Children of the root that are accepted when visited."""
    perms, size = td.synth_perms(800 + n, 40, n, n, 30, 1, 3)
    rates = [0.0, 0.5, 1.0, 1.5]
    cases = [(p[:n].tolist(), 2 + q % 3, rates[q % 4], False) for q, p in enumerate(perms)]
    _check(td, oracle, split_search, cases, [(1, 1), (4, 8)])
