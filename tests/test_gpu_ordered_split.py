"""Reference-order batches whose walks give subtrees away, against the one-warp
walk of each instance: records equal word for word.  Partial sorting, where the
root's children may be accepted when visited, and full sorting at the lower
bound; splits after 1, 8 and 64 expansions.  Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MiB = 1 << 20


@pytest.fixture(scope="module")
def slots(td):
    td.init_slots(1, [0], 64 * MiB)
    yield td
    td._lib.configure_split(64)
    td.destroy()


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("n", [4, 7, 10, 11])
def test_split_walks_equal_the_one_warp_walk(slots, n, full):
    td = slots
    perms, size = td.synth_perms(17 * n, 400, n - 1, n, 30, 1, 3)
    inst = td.prepare_perms(perms, size, 9)
    init = (inst["packed"] & 31).astype(np.int32)
    lower = (size.astype(np.int32) + 2 - init) // 2
    bound = np.clip(lower + (0 if full else 1), 1, 9).astype(np.int32)
    inst["max_moves"] = bound
    if not full:
        target = np.random.default_rng(n).integers(1, np.maximum(2, lower + 1)).astype(np.float32)
        inst["min_rate"] = np.float32(2) / (bound.astype(np.float32) / target)
        inst["packed"] &= 31
    td._lib.configure_split(0)
    one, _ = td.search_batch(0, inst, td._lib.FLAG_ORDERED | td._lib.FLAG_VERIFY)
    assert (one["status"] >= 0).all()
    for after in (1, 8, 64):
        td._lib.configure_split(after)
        for _ in range(3):  # who splits what differs from run to run
            many, _ = td.search_batch(0, inst, td._lib.FLAG_ORDERED | td._lib.FLAG_VERIFY)
            assert many.tobytes() == one.tobytes()
