"""Expansion counts at the end of their 32 bits, and what a walk that ends there
reports (td_core.cuh): a count saturates, a search without a budget is never
ended by it, and only a walk searched to its end is a "not found"."""
import ctypes as C

import pytest

MAX = 2 ** 32 - 1
NOT_FOUND, FOUND, BUDGET, TIMEOUT = 0, 1, -2, -5
DFS_EXHAUSTED, DFS_FOUND, DFS_BUDGET, DFS_TIMEOUT, DFS_ABORTED = 0, 1, -2, -5, -7


@pytest.mark.parametrize("a,b,total", [(0, 1, 1), (MAX - 2249, 2249, MAX), (MAX - 1, 1, MAX), (MAX - 1, 2249, MAX),
                                       (MAX, 1, MAX), (MAX, 0, MAX), (MAX, MAX, MAX)])
def test_counts_saturate(emu, a, b, total):
    emu.td_emu_add_count.restype = C.c_uint32
    assert emu.td_emu_add_count(C.c_uint32(a), C.c_uint32(b)) == total


@pytest.mark.parametrize("count,budget,over", [
    (0, 0, False), (MAX - 1, 0, False), (MAX, 0, False),  # 0: no budget
    (15, 16, False), (16, 16, True), (17, 16, True), (MAX - 1, MAX - 1, True),
    (MAX - 1, MAX, False), (MAX, MAX, True), (MAX, MAX + 1, False), (MAX, 2 ** 64 - 1, False)])
def test_budgets(emu, count, budget, over):
    assert bool(emu.td_emu_over_budget(C.c_uint32(count), C.c_uint64(budget))) == over


def test_only_an_exhausted_walk_is_a_not_found(emu):
    ends = {DFS_EXHAUSTED: NOT_FOUND, DFS_FOUND: FOUND, DFS_BUDGET: BUDGET, DFS_TIMEOUT: TIMEOUT,
            DFS_ABORTED: TIMEOUT}
    assert {d: emu.td_emu_status_of_dfs(d) for d in ends} == ends
