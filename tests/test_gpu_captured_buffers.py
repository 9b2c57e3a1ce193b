"""A captured batch replayed after larger batches of the same slot, and after a
change of the table's and the split's sizes: its records are what they were.
Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ordered", [False, True])
def test_replay_after_larger_batches(td, ordered):
    import torch
    L = td._lib
    flags = L.FLAG_VERIFY | (L.FLAG_ORDERED if ordered else 0)
    td.init_slots(1, [0], 64 << 20)
    try:
        def batch(count):
            perms, n = td.synth_perms(count, count, 9, 12, 50, 1, 3)
            inst = td.prepare_perms(perms, n, 9)
            inst["max_moves"] = np.clip((n.astype(np.int32) + 2 - (inst["packed"] & 31)) // 2, 1, 9)
            return (torch.from_numpy(inst.view(np.uint8).copy()).cuda(),
                    torch.zeros((count, 8), dtype=torch.int32, device="cuda"))

        stream = L.lib().td_slot_stream(0)
        d_in, d_out = batch(64)
        graph = L.BatchGraph(0, 64, d_in.data_ptr(), d_out.data_ptr(), flags)
        graph.launch(stream)
        torch.cuda.synchronize()
        want = d_out.cpu().numpy().copy()
        assert (want[:, 0] >= 0).all()
        for count, bits, records in ((500, 12, 1 << 20), (5000, 8, (1 << 20) + 1), (20000, 14, 3 << 20)):
            L.configure_table(bits)
            L.configure_split(64, records)
            big_in, big_out = batch(count)
            L.search_batch_device(0, count, big_in.data_ptr(), big_out.data_ptr(), flags, 0, stream)
            d_out.zero_()
            torch.cuda.synchronize()
            graph.launch(stream)
            torch.cuda.synchronize()
            got = d_out.cpu().numpy()
            assert (big_out[:, 0] >= 0).all().item()
            assert (got == want).all() if ordered else (got[:, 0] == want[:, 0]).all()
        graph.close()
    finally:
        L.configure_table(12)
        L.configure_split(64)
        td.destroy()
