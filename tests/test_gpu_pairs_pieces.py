"""td_search_pairs with more pairs than its pinned memory holds in one piece:
the answers of one call against those of the same pairs in smaller calls.  4 MiB
hold the inputs of 91,180 pairs and the outputs of 67,650.  Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [67649, 67651, 91181, 190001])
def test_one_call_equals_smaller_calls(td, count):
    perms, n = td.synth_perms(count, count, 3, 7, 30, 1, 2)
    beta, omega = np.zeros((count, 17), np.uint8), np.zeros((count, 17), np.uint8)
    td._lib.lib().td_pairs_from_perms(count, td._lib._ptr(perms), td._lib._ptr(n), td._lib._ptr(beta),
                                      td._lib._ptr(omega))
    rng = np.random.default_rng(count)
    sym = (n + 1).astype(np.uint8)
    init = rng.integers(0, 3, count).astype(np.int32)
    maxd = rng.integers(0, 5, count).astype(np.int32)  # 0: refused
    full = (rng.random(count) < 0.7).astype(np.uint8)
    rate = rng.choice([0.0, 1.0], count).astype(np.float32)
    omega[rng.random(count) < 0.05, 0] = 33  # no permutation
    td.init_slots(1, [0], 64 << 20)
    try:
        whole = td._lib.search_pairs(0, beta, omega, sym, init, rate, maxd, full, ordered=True)
        parts = [td._lib.search_pairs(0, *[a[i: i + 20000] for a in (beta, omega, sym, init, rate, maxd, full)],
                                      ordered=True) for i in range(0, count, 20000)]
    finally:
        td.destroy()
    for got, want in zip(whole, zip(*parts)):
        assert (got == np.concatenate(want)).all()
    assert {0, 1, 4} == set(whole[0].tolist())
