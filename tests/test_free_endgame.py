"""The free-order search with the endgame table and the moves that fix symbols
first: the host emulation of it against the oracle's verdicts, and, on a B200, a
plain launch against the emulation, record for record."""
import ctypes as C
import math
import os

import numpy as np
import pytest

SYMBOLS = 11


@pytest.fixture(scope="module")
def endgame_emu(emu):
    table = np.zeros(sum(math.factorial(q) for q in range(2, SYMBOLS)), np.uint16)
    emu.td_emu_endgame.restype = C.c_long
    assert emu.td_emu_endgame(SYMBOLS, C.c_void_p(table.ctypes.data), max(1, min(16, os.cpu_count() or 1))) == 0
    emu.td_emu_set_endgame(C.c_void_p(table.ctypes.data))
    yield emu
    emu.td_emu_set_endgame(None)


def _run(emu, td, inst, restart):
    out = np.zeros(len(inst), td._lib.RESULT_DTYPE)
    emu.td_emu_set_restart(C.c_uint32(restart))
    try:
        emu.td_emu_search_batch(len(inst), C.c_void_p(inst.ctypes.data), 0, C.c_void_p(out.ctypes.data), 4)
    finally:
        emu.td_emu_set_restart(C.c_uint32(16))
    return out


def _instances(td, seed, count, n, hard, over, rate=0.0):
    perms, size = td.synth_perms(seed, count, n, n, hard, 1, 3)
    inst = td.prepare_perms(perms, size, 9, rate)
    inst["max_moves"] = np.clip((n + 2 - (inst["packed"] & 31).astype(np.int32)) // 2 + over, 1, 9)
    return perms, inst


@pytest.mark.parametrize("restart", [0, 16])
@pytest.mark.parametrize("n,over", [(5, 0), (8, 0), (8, 1), (10, 0), (12, 0), (12, 1), (13, 0), (13, 1), (14, 0)])
def test_verdicts(td, oracle, endgame_emu, n, over, restart):
    perms, inst = _instances(td, 10 * n + over, 40, n, 60, over)
    seen = set()
    for p, x, r in zip(perms, inst, _run(endgame_emu, td, inst, restart)):
        beta, omega, init = oracle.perm_to_pair(p[:n].tolist())
        bound = int(x["max_moves"])
        status, _, _ = oracle.search(beta, omega, init, 0.0, bound, True)
        assert r["status"] == status, (p[:n].tolist(), bound)
        if status == 1:
            abc = oracle.positions_to_symbols(beta, td._lib.unpack_moves(r))
            assert oracle.validate(beta, omega, abc, bound) is None
        seen.add(status)
    assert 1 in seen


@pytest.mark.gpu
@pytest.mark.parametrize("n,over,rate", [(4, 1, 0.0), (7, 0, 0.0), (9, 1, 0.0), (11, 0, 0.0), (12, 0, 0.0), (12, 1, 0.0),
                                         (13, 1, 1.0), (14, 0, 0.0), (15, 1, 0.0), (16, 0, 0.0), (16, 1, 0.0), (16, 2, 0.0)])
def test_plain_launch_equals_the_emulation(td, endgame_emu, n, over, rate):
    """Searches that end before the emulation's table of explored states comes in
    (a plain launch has none)."""
    _, inst = _instances(td, 20 * n + over, 1000, n, 40, over, rate)
    td.init_slots(1, [0], 64 << 20)
    try:
        got, _ = td.search_batch(0, inst, td._lib.FLAG_PLAIN, 32)
    finally:
        td.destroy()
    short = got["status"] != -2
    want = _run(endgame_emu, td, inst[short], 0)
    assert short.sum() >= 50
    assert got[short].tobytes() == want.tobytes()
