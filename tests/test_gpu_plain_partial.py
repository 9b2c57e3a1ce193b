"""One warp per instance (the plain launch) in the free order where the endgame
table does not apply: partial sorting, and full sorting at a rate that the bound
does not meet.  The records of the host emulation's plain order, word for word,
for searches that end before its table of explored states comes in.  Needs a
B200."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,full,seed", [(6, False, 1), (9, False, 4), (13, False, 10), (16, False, 11), (6, True, 1),
                                         (9, True, 4)])
def test_plain_order_without_the_endgame_table(td, emu, n, full, seed):
    perms, size = td.synth_perms(seed, 3001, n, n, 30, 1, 3)
    inst = td.prepare_perms(perms, size, 9)
    init = (inst["packed"] & 31).astype(np.int32)
    lower = (n + 2 - init) // 2
    inst["max_moves"] = bound = np.clip(lower + (0 if full else 1), 1, 9).astype(np.int32)
    if full:
        inst["min_rate"] = 4.0
    else:
        target = np.random.default_rng(seed).integers(1, np.maximum(2, lower + 1)).astype(np.float32)
        inst["min_rate"] = np.float32(2) / (bound.astype(np.float32) / target)
        inst["packed"] &= 31
    want = np.zeros(len(inst), td._lib.RESULT_DTYPE)
    emu.td_emu_set_restart(C.c_uint32(0))
    try:
        emu.td_emu_search_batch(len(inst), C.c_void_p(inst.ctypes.data), 0, C.c_void_p(want.ctypes.data), 4)
    finally:
        emu.td_emu_set_restart(C.c_uint32(16))
    td.init_slots(1, [0], 64 << 20)
    try:
        got, _ = td.search_batch(0, inst, td._lib.FLAG_PLAIN)
    finally:
        td.destroy()
    short = want["expansions"] <= 32
    assert short.any()
    assert got[short].tobytes() == want[short].tobytes()
