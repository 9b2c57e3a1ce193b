"""td_search_pairs (prepared and unpacked on the device) against one per-call
td_search_ordered per pair: statuses of every class, depths and triples.  Needs
a B200."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(oracle, count, seed):
    rng = np.random.default_rng(seed)
    perms, n = oracle.synth_perms(seed, count, 2, 11, 30, 1, 3)
    beta, omega = rng.integers(0, 40, (count, 17)).astype(np.uint8), rng.integers(0, 40, (count, 17)).astype(np.uint8)
    sym, init = (n + 1).astype(np.uint8), np.zeros(count, np.int32)
    maxd, full = np.zeros(count, np.int32), (rng.random(count) < 0.8).astype(np.uint8)
    rate = rng.choice([0.0, 1.0, 1.5], count).astype(np.float32)
    for i in range(count):
        b, o, init[i] = oracle.perm_to_pair(perms[i, : n[i]].tolist())
        r = int(rng.integers(len(b)))
        beta[i, : len(b)], omega[i, : len(o)] = b[r:] + b[:r], o
        maxd[i] = np.clip((len(b) - init[i] + 1) // 2 + rng.integers(0, 2), 1, 6)
        kind = rng.integers(0, 12)
        if kind == 0:
            beta[i, int(rng.integers(len(b)))] = rng.integers(0, 255)
        elif kind == 1:
            omega[i, [0, 1]] = omega[i, [1, 0]]  # still a permutation; the product may not be one cycle
        elif kind == 2:
            maxd[i] = rng.choice([0, -3, 10])
        elif kind == 3:
            init[i] = rng.choice([-1, 40, 20])
        elif kind == 4:
            sym[i] = rng.choice([0, 1, 2])
    return beta, omega, sym, init, rate, maxd, full


@pytest.mark.parametrize("count", [1, 127, 129, 700])
def test_pairs_match_one_call_each(td, oracle, count):
    beta, omega, sym, init, rate, maxd, full = _pairs(oracle, count, 90 + count)
    L = td._lib.lib()
    td.init_slots(1, [0], 64 << 20)
    try:
        for _ in range(2):  # the second call reuses the slot's buffers
            status, depth, moves = td._lib.search_pairs(0, beta, omega, sym, init, rate, maxd, full, ordered=True)
        err = C.create_string_buffer(256)
        for i in range(count):
            out, d = (C.c_int16 * 27)(), C.c_int(0)
            rc = L.td_search_ordered(0, beta[i].ctypes.data, omega[i].ctypes.data, int(sym[i]), int(init[i]),
                                     float(rate[i]), int(maxd[i]), int(full[i]), out, C.byref(d), err, 256)
            assert status[i] == rc, (i, err.value)
            assert depth[i] == d.value
            assert moves[i].reshape(-1)[: 3 * d.value].tolist() == list(out)[: 3 * d.value]
            assert not moves[i].reshape(-1)[3 * d.value:].any()
    finally:
        td.destroy()
    if count > 100:
        assert {0, 1, 4} <= set(status.tolist())
