"""Expansion budgets of free-order batches that end before a search looks for
idle warps: nothing is given away, so the budget bounds each instance, however few
instances the launch has.  Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 500, 4096])
@pytest.mark.parametrize("budget", [1, 16, 64])
def test_a_small_budget_bounds_the_instance(td, count, budget):
    perms, n = td.synth_perms(count, count, 12, 16, 75, 1, 3)
    inst = td.prepare_perms(perms, n, 9)
    inst["max_moves"] = np.clip((n.astype(np.int32) + 2 - (inst["packed"] & 31)) // 2, 1, 9)
    td.init_slots(1, [0], 64 << 20)
    try:
        td._lib.configure_steal(4, 2, 64)
        full, _ = td.search_batch(0, inst, td._lib.FLAG_VERIFY)
        for _ in range(3):
            res, stats = td.search_batch(0, inst, td._lib.FLAG_VERIFY, budget)
            assert stats.donated_items == 0
            assert (res["expansions"] <= budget).all()
            decided = res["status"] != -2
            assert (res["status"][decided] == full["status"][decided]).all()
            assert (res["expansions"][~decided] == budget).all()
    finally:
        td.destroy()
    if count > 1:
        assert not decided.all()
        assert decided.any() or budget == 1  # a root by itself decides the distances of one move
