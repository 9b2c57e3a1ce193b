"""The pinned-form replay on the device (td_validate_batch_device) against the
same rule on the host: every n, full and partial sorting, rates, broken
witnesses, block edges and buffers at the records' own alignment.  Needs a
B200."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,shift", [(1, 0), (255, 0), (257, 0), (2000, 0), (2000, 8)])
def test_validation_matches_the_host_rule(td, emu, oracle, count, shift):
    import torch
    rng = np.random.default_rng(count + shift)
    perms, n = oracle.synth_perms(61 + count, count, 2, 16, 50, 1, 3)
    beta, omega = np.zeros((count, 17), np.uint8), np.zeros((count, 17), np.uint8)
    init = np.zeros(count, np.int32)
    for i in range(count):
        b, o, init[i] = oracle.perm_to_pair(perms[i, : n[i]].tolist())
        r = int(rng.integers(len(b)))
        b = b[r:] + b[:r]
        beta[i, : len(b)], omega[i, : len(o)] = b, o
    full = (rng.random(count) < 0.7).astype(np.uint8)
    rate = rng.choice([0.0, 1.0, 1.5, 1.9], count).astype(np.float32)
    inst = td.prepare_pairs(beta, omega, n + 1, np.where(full, init, np.maximum(0, init - 1)), rate, 9, full)
    td.init_slots(1, [0], 64 << 20)
    try:
        res, _ = td.search_batch(0, inst, td._lib.FLAG_ORDERED, 500)  # some run out of their budget
    finally:
        td.destroy()
    for i in np.nonzero(rng.random(count) < 0.3)[0]:  # break some
        k = rng.integers(0, 5)
        if k == 0:
            res["moves"][i, int(rng.integers(9))] = rng.integers(0, 1 << 15)
        elif k == 1:
            res["depth"][i] = rng.integers(-1, 10)
        elif k == 2:
            inst["max_moves"][i] = rng.integers(1, 9)
        elif k == 3:
            res["status"][i] = 1
        else:
            inst["min_rate"][i] = 2.0
    want = np.array([emu.td_emu_witness_ok(C.c_void_p(inst[i:].ctypes.data), C.c_void_p(res[i:].ctypes.data))
                     for i in range(count)])
    dev = []
    for a in (inst, res):
        buf = torch.zeros(a.nbytes + 16, dtype=torch.uint8, device="cuda")
        buf[shift: shift + a.nbytes] = torch.from_numpy(a.view(np.uint8).copy()).cuda()
        dev.append(buf)
    ok = torch.full((count + 1,), 7, dtype=torch.uint8, device="cuda")
    td._lib.validate_batch_device(count, dev[0].data_ptr() + shift, dev[1].data_ptr() + shift, ok.data_ptr())
    torch.cuda.synchronize()
    got = ok.cpu().numpy()
    assert got[count] == 7
    assert (got[:count] == want).all(), np.nonzero(got[:count] != want)[0][:10]
    if count > 100:
        assert 0 < want.sum() < count
