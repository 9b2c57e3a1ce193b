"""The race of a search against its inverse: each instance queues its inverse at
most once, also where the search can give nothing away (nodes with one child
each, all warps idle, a look at them after every expansion).  Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# at the lower bound the root, its child and its grandchild have one child each
NARROW = [
    [15, 13, 11, 5, 6, 4, 10, 9, 8, 7, 3, 14, 2, 12, 1, 0],
    [14, 12, 11, 3, 2, 1, 0, 5, 10, 9, 8, 13, 7, 6, 4],
    [14, 6, 5, 1, 13, 12, 4, 3, 11, 10, 9, 8, 2, 7, 0],
    [13, 12, 11, 9, 3, 2, 1, 0, 8, 7, 6, 5, 10, 4],
]


@pytest.mark.parametrize("race", [1, 2, 8])
def test_an_instance_queues_its_inverse_once(td, race):
    perms = np.zeros((len(NARROW), 16), np.int8)
    for i, p in enumerate(NARROW):
        perms[i, : len(p)] = p
    inst = td.prepare_perms(perms, [len(p) for p in NARROW], 9)
    inst["max_moves"] = (inst["n_symbols"] + 1 - (inst["packed"] & 31)) // 2
    td.init_slots(1, [0], 64 << 20)
    try:
        td._lib.configure_steal(4, 0, 16)
        td._lib.configure_race(race)
        ref, _ = td.search_batch(0, inst, td._lib.FLAG_ORDERED)
        for _ in range(20):
            for one, want in zip(np.split(inst, len(inst)), ref["status"]):
                res, stats = td.search_batch(0, one, td._lib.FLAG_VERIFY)
                assert res["status"][0] == want
                assert stats.races <= 1
    finally:
        td._lib.configure_steal(4, 2, 64)
        td._lib.configure_race(8)
        td.destroy()
