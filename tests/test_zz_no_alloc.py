"""The batch search that allocates no device memory (td_search_batch_noalloc).

It serves callers that cannot call cudaMalloc/cudaFree themselves: a slot
worker that must not stall on the device-wide synchronisation those calls can
imply while other searches run, or a process whose device memory is already
held by another allocator.  This file is collected last on purpose; it needs
no state from the other tests and sets up everything it compares against.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MAX_INSTANCES = 65536


def _noalloc(td):
    f = td._lib.lib().td_search_batch_noalloc
    f.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_uint, C.c_uint64, C.c_void_p, C.c_char_p, C.c_size_t]
    f.restype = C.c_int
    return f


def _call(f, count, d_in, d_out, flags, stream):
    err = C.create_string_buffer(512)
    rc = f(count, C.c_void_p(d_in.data_ptr()), C.c_void_p(d_out.data_ptr()), flags, 0, C.c_void_p(stream), err, 512)
    return rc, err.value.decode()


def _results(t):
    import td16_b200 as td
    return t.cpu().numpy().view(td.RESULT_DTYPE)


def test_noalloc_entry_point_matches_the_allocating_one(td):
    import torch
    f = _noalloc(td)
    # the reference move order on 4096 x S_10 at bound 6 (that order is blind,
    # so it is checked where every search ends well inside the deadline); the
    # free order on a mixed-size batch with hard instances (work donation
    # happens) and on an S_16 batch, all run back to back through the scratch
    p1, n1 = td.synth_perms(43, 4096, 10, 10, 0, 0, 0)
    b1 = td.prepare_perms(p1, n1, 6)
    p2, n2 = td.synth_perms(41, 6000, 11, 13, 40, 1, 3)
    b2 = td.prepare_perms(p2, n2, (n2 // 2 + 1).astype(np.int32))
    p3, n3 = td.synth_perms(42, 3000, 16, 16, 50, 1, 4)
    b3 = td.prepare_perms(p3, n3, 9)
    stream = torch.cuda.current_stream().cuda_stream
    td.init_slots(1, [0], 64 << 20)
    try:
        for batch, flags in ((b1, td._lib.FLAG_ORDERED), (b2, td._lib.FLAG_VERIFY), (b3, td._lib.FLAG_VERIFY)):
            count = len(batch)
            d_in = torch.from_numpy(batch.view(np.uint8).copy()).cuda()
            d_ref = torch.zeros(count * 32, dtype=torch.uint8, device="cuda")
            td._lib.search_batch_device(0, count, d_in.data_ptr(), d_ref.data_ptr(), flags, 0, stream)
            outs = []
            for _ in range(2):  # two calls in a row share the scratch
                d_out = torch.full((count * 32,), 0xAB, dtype=torch.uint8, device="cuda")
                rc, msg = _call(f, count, d_in, d_out, flags, stream)
                assert rc == 0, msg
                outs.append(d_out)
            torch.cuda.synchronize()
            ref = _results(d_ref)
            assert (ref["status"] >= 0).all()
            for d_out in outs:
                got = _results(d_out)
                if flags == td._lib.FLAG_ORDERED:
                    # reference move order: bit-identical results
                    assert (got.view(np.uint8) == ref.view(np.uint8)).all()
                else:
                    # free order: identical verdicts; every witness passed the
                    # device replay (a failing one would read -6)
                    assert (got["status"] == ref["status"]).all()
                    ok = torch.zeros(count, dtype=torch.uint8, device="cuda")
                    td._lib.validate_batch_device(count, d_in.data_ptr(), d_out.data_ptr(), ok.data_ptr(), stream)
                    torch.cuda.synchronize()
                    assert ((got["status"] == 1) == (ok.cpu().numpy() == 1)).all()
    finally:
        td.destroy()


def test_noalloc_rejects_batches_beyond_its_scratch(td):
    import torch
    f = _noalloc(td)
    d = torch.zeros(16, dtype=torch.uint8, device="cuda")
    rc, msg = _call(f, MAX_INSTANCES + 1, d, d, 0, 0)
    assert rc == 4 and "65536" in msg


def test_noalloc_calls_leave_device_memory_unchanged(td):
    """After the one-time set-up of the first call, calls take no device
    memory: the device's free bytes are the same before and after two more
    calls (nothing else allocates inside that window)."""
    import torch
    f = _noalloc(td)
    # the free order on a mix of hard instances, and the reference order (one
    # warp per instance, blind) where every search ends quickly
    p1, n1 = td.synth_perms(44, 8192, 13, 16, 50, 1, 3)
    free = td.prepare_perms(p1, n1, (n1 // 2 + 1).astype(np.int32))
    p2, n2 = td.synth_perms(45, 4096, 10, 10, 0, 0, 0)
    ordered = td.prepare_perms(p2, n2, 6)
    cases = []
    for batch, flags in ((free, td._lib.FLAG_VERIFY), (ordered, td._lib.FLAG_ORDERED | td._lib.FLAG_PLAIN)):
        d_in = torch.from_numpy(batch.view(np.uint8).copy()).cuda()
        d_out = torch.zeros(len(batch) * 32, dtype=torch.uint8, device="cuda")
        cases.append((len(batch), d_in, d_out, flags))
    stream = torch.cuda.current_stream().cuda_stream
    for count, d_in, d_out, flags in cases:  # set-up: first use of each kernel
        rc, msg = _call(f, count, d_in, d_out, flags, stream)
        assert rc == 0, msg
    torch.cuda.synchronize()
    free_before, _ = torch.cuda.mem_get_info()
    for count, d_in, d_out, flags in cases:
        rc, msg = _call(f, count, d_in, d_out, flags, stream)
        assert rc == 0, msg
    torch.cuda.synchronize()
    free_after, _ = torch.cuda.mem_get_info()
    assert free_after == free_before
    for count, _, d_out, _ in cases:
        assert (_results(d_out)["status"] >= 0).all()


def test_noalloc_setup_keeps_eight_warp_blocks_launchable(td):
    """The set-up of the first call sets the kernels' shared-memory limit; a
    launch of 8-warp blocks (the tuned shape) must still fit afterwards."""
    import torch
    perms, n = td.synth_perms(46, 512, 8, 10, 50, 1, 2)
    inst = td.prepare_perms(perms, n, 9)
    d_in = torch.from_numpy(inst.view(np.uint8).copy()).cuda()
    d_out = torch.zeros(len(inst) * 32, dtype=torch.uint8, device="cuda")
    rc, msg = _call(_noalloc(td), len(inst), d_in, d_out, 0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0, msg
    torch.cuda.synchronize()
    td.init_slots(1, [0], 64 << 20)
    try:
        td._lib.configure(8, 1)
        for flags in (0, td._lib.FLAG_ORDERED, td._lib.FLAG_PLAIN, td._lib.FLAG_PLAIN | td._lib.FLAG_ORDERED):
            res, _ = td.search_batch(0, inst, flags)
            assert (res["status"] == 1).all()
    finally:
        td._lib.configure(4, 1)
        td.destroy()
