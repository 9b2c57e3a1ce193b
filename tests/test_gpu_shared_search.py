"""Free-order searches that many warps share (a handful of long instances on the
whole device): verdicts against the reference order's, with and without a
witness.  Bounds around the cycle-graph lower bound, N from the smallest whose
nodes look children up in a batch to the largest.  Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MiB = 1 << 20


@pytest.fixture(scope="module")
def slots(td):
    td.init_slots(1, [0], 64 * MiB)
    yield td
    td.destroy()


@pytest.mark.parametrize("N", [11, 12, 14, 16, 17])
@pytest.mark.parametrize("over", [0, 1])
def test_shared_searches_keep_the_verdict(slots, oracle, N, over):
    td = slots
    perms, _ = oracle.synth_perms(5 + over, 6, N - 1, N - 1, 90, 1, 3)
    cases = [oracle.perm_to_pair(p[: N - 1].tolist()) for p in perms]
    beta = np.zeros((6, 17), np.uint8)
    omega = np.zeros((6, 17), np.uint8)
    for i, (b, o, _init) in enumerate(cases):
        beta[i, :N], omega[i, :N] = b, o
    init = np.array([c[2] for c in cases], np.int32)
    bound = ((N - init + 1) // 2 + over).astype(np.int32)
    inst = td.prepare_pairs(beta, omega, N, init, np.zeros(6, np.float32), bound, np.ones(6, np.uint8))
    ref, _ = td.search_batch(0, inst, td._lib.FLAG_ORDERED | td._lib.FLAG_VERIFY, 200000)
    done = ref["status"] >= 0
    assert done.any()
    for _ in range(8):  # who gives what to whom differs from run to run
        free, _ = td.search_batch(0, inst, td._lib.FLAG_VERIFY)
        assert (free["status"][done] == ref["status"][done]).all()


@pytest.mark.parametrize("count", [1, 73, 74, 75, 295, 297, 1183, 1185, 75775, 75777])
def test_verdicts_at_the_edges_of_the_launch_shapes(td, oracle, count):
    """Around the counts at which a launch leaves its slot's share of the
    device, fills the device, and stops sharing its searches from the start."""
    td.destroy()
    td.init_slots(16, [0], 64 * MiB)
    perms, n = oracle.synth_perms(count, count, 6, 9, 50, 1, 2)
    inst = td.prepare_perms(perms, n, 9)
    init = (inst["packed"] & 31).astype(np.int32)
    inst["max_moves"] = np.clip((n.astype(np.int32) + 2 - init) // 2, 1, 9)
    ref, _ = td.search_batch(0, inst, td._lib.FLAG_ORDERED | td._lib.FLAG_VERIFY)
    free, _ = td.search_batch(0, inst, td._lib.FLAG_VERIFY)
    assert (free["status"] == ref["status"]).all()
    assert (free["status"] >= 0).all()
