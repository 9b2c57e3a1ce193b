"""Expansion counts of reference-order batches whose walks give subtrees away
while whole levels of their remaining children are decided by the endgame table:
such children rank after the subtree a walk is in, so they count only where the
walk gets to them.  n = 13..15, near-reverse, where it happens; records against
the one-warp walk's, word for word.  Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MiB = 1 << 20

# (permutation, bound): walks that pass by a decided level on their way to the witness
WALKS = [
    ([10, 9, 8, 7, 6, 5, 4, 3, 2, 1, 12, 11, 0], 7),
    ([12, 10, 9, 8, 7, 4, 6, 5, 3, 2, 1, 11, 0], 7),
    ([13, 12, 11, 10, 9, 1, 0, 8, 7, 6, 5, 4, 3, 2], 7),
]


@pytest.fixture(scope="module")
def slots(td):
    td.init_slots(1, [0], 64 * MiB)
    yield td
    td._lib.configure_split(64)
    td.destroy()


def _same_in_every_split(td, inst, runs):
    td._lib.configure_split(0)
    one, _ = td.search_batch(0, inst, td._lib.FLAG_ORDERED | td._lib.FLAG_VERIFY)
    assert (one["status"] >= 0).all()
    for after in (1, 8, 64):
        td._lib.configure_split(after)
        for _ in range(runs):  # who splits what differs from run to run
            many, stats = td.search_batch(0, inst, td._lib.FLAG_ORDERED | td._lib.FLAG_VERIFY)
            differ = np.flatnonzero((many.view(np.uint32) != one.view(np.uint32)).reshape(len(one), -1).any(1))
            assert len(differ) == 0, (after, differ[:8], one["expansions"][differ[:8]], many["expansions"][differ[:8]])
            assert stats.expansions == int(one["expansions"].astype(np.uint64).sum())
    return one


def test_decided_children_after_the_walks_subtree(slots, oracle):
    td = slots
    perms = np.zeros((len(WALKS), 16), np.int8)
    for i, (p, _) in enumerate(WALKS):
        perms[i, : len(p)] = p
    inst = td.prepare_perms(perms, np.array([len(p) for p, _ in WALKS]), np.array([b for _, b in WALKS]))
    one = _same_in_every_split(td, inst, 20)
    for r, (p, bound) in zip(one, WALKS):
        status, moves, exp = oracle.search(*oracle.perm_to_pair(p), 0.0, bound, True)
        assert r["status"] == status == 1 and td.unpack_moves(r) == moves
        assert r["expansions"] == exp + 1  # + the root's evaluation


@pytest.mark.parametrize("n", [13, 14, 15])
@pytest.mark.parametrize("over", [0, 1])
def test_near_reverse_walks_of_every_split(slots, n, over):
    td = slots
    perms, size = td.synth_perms(31 * n + over, 4000, n, n, 100, 1, 3)
    inst = td.prepare_perms(perms, size, 9)
    inst["max_moves"] = np.clip((n + 2 - (inst["packed"] & 31).astype(np.int32)) // 2 + over, 1, 9)
    one = _same_in_every_split(td, inst, 3)
    assert (one["status"] == 1).any()
