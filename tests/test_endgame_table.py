"""The endgame table (td_endgame.cuh): rebuilt on the host, its entries against
the oracle's walks and, on a B200, against the engine's; and the fact the
engine rests on, that one spare move sorts every state the table holds."""
import ctypes as C
import os

import numpy as np
import pytest

SYMBOLS = 11


def _base(m):
    b, f = 0, 1
    for q in range(2, m):
        f *= q
        b += f
    return b


@pytest.fixture(scope="module")
def table(emu):
    out = np.zeros(_base(SYMBOLS), np.uint16)
    emu.td_emu_endgame.restype = C.c_long
    bad = emu.td_emu_endgame(SYMBOLS, C.c_void_p(out.ctypes.data), max(1, min(16, os.cpu_count() or 1)))
    return out, bad


def _glued(rng, m, count):
    """Permutations of S_m whose inverse (the engine's pinned state) has no
    symbol right after its predecessor in the cyclic sense, with the index of
    that state in the table."""
    out = []
    while len(out) < count:
        p = rng.permutation(m).tolist()
        if p[0] != 0 and p[-1] != m - 1 and all(b != a + 1 for a, b in zip(p, p[1:])):
            rank, left = 0, sorted(p)
            for q, v in enumerate(p):
                rank = rank * (m - q) + left.index(v)
                left.remove(v)
            out.append((np.argsort(p).tolist(), _base(m) + rank))
    return out


def test_one_spare_move_sorts_every_state(table):
    out, bad = table
    assert bad == 0
    assert 0 < (out == 0).sum() and out[out != 0xffff].max() == 2249
    assert (out != 0xffff).sum() == 1350069  # glued states of 3..11 symbols


@pytest.mark.parametrize("m", range(2, 11))
def test_entries_are_the_oracles_walks(table, oracle, m):
    """Entry 0: sorted in the missing moves; else the expansions of the walk
    (the oracle does not count the root)."""
    rng = np.random.default_rng(m)
    for p, g in _glued(rng, m, 1 if m == 2 else 20):
        beta, omega, init = oracle.perm_to_pair(p)
        missing = (m + 1 - init) // 2
        st, _, exp = oracle.search(beta, omega, init, 0.0, missing, True)
        assert st == (1 if table[0][g] == 0 else 0)
        if st == 0:
            assert table[0][g] == exp + 1
        assert oracle.search(beta, omega, init, 0.0, missing + 1, True)[0] == 1


@pytest.mark.gpu
@pytest.mark.parametrize("m", [2, 3, 8, 10])
def test_engine_agrees_with_the_table(td, table, m):
    """Glued states at their missing moves: the engine's verdicts in both
    orders, and its expansion counts in the reference order."""
    rng = np.random.default_rng(100 + m)
    states = _glued(rng, m, 1 if m <= 3 else 4000)
    perms = np.zeros((len(states), 16), np.int8)
    perms[:, :m] = [p for p, _ in states]
    want = table[0][[g for _, g in states]]
    td.init_slots(1, [0], 64 << 20)
    try:
        inst = td.prepare_perms(perms, m, 9)
        inst["max_moves"] = (m + 1 - (inst["packed"] & 31).astype(int)) // 2
        ref, _ = td.search_batch(0, inst, td._lib.FLAG_ORDERED | td._lib.FLAG_VERIFY)
        free, _ = td.search_batch(0, inst, td._lib.FLAG_VERIFY)
    finally:
        td.destroy()
    assert (ref["status"] == (want == 0)).all() and (free["status"] == (want == 0)).all()
    assert (ref["expansions"][want != 0] == want[want != 0]).all()
