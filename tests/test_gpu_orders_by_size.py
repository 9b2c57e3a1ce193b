"""Both move orders at every symbol count N = 3..17 against the oracle: the
reference order's witness and expansion count bit for bit, the free order's
verdict with a replayed witness; full and partial sorting, arrays that start
anywhere.  The edges: N = 3 (one triple), pair slots that fill one to four
rounds, and child words that end inside a 32-chunk.  Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MiB = 1 << 20


@pytest.fixture(scope="module")
def slots(td):
    td.init_slots(1, [0], 64 * MiB)
    yield td
    td.destroy()


def _cases(oracle, N, seed):
    """(beta, omega, init, rate, bound, full) per case; bounds near the
    cycle-graph lower bound, so that some have no witness."""
    rng = np.random.default_rng(1000 * N + seed)
    perms, n = oracle.synth_perms(seed, 96, N - 1, N - 1, 50, 1, 3)
    out = []
    for p in perms:
        beta, omega, init = oracle.perm_to_pair(p[: N - 1].tolist())
        r = int(rng.integers(N))
        beta = beta[r:] + beta[:r]
        lb = (N - init + 1) // 2
        full = int(rng.random() < 0.7)
        bound = int(np.clip(lb + rng.integers(-1, 3), 1, 9))
        rate = float(rng.choice([0.0, 0.0, 1.0, 1.5, 2.0]))
        out.append((beta, omega, init if full else max(0, init - int(rng.integers(0, 2))), rate, bound, full))
    return out


@pytest.mark.parametrize("N", range(3, 18))
def test_both_orders_match_the_oracle(slots, oracle, N):
    td = slots
    cases = _cases(oracle, N, 77)
    c = len(cases)
    beta = np.zeros((c, 17), np.uint8)
    omega = np.zeros((c, 17), np.uint8)
    for i, (b, o, *_rest) in enumerate(cases):
        beta[i, :N], omega[i, :N] = b, o
    col = lambda k, dt: np.array([v[k] for v in cases], dt)  # noqa: E731
    init, rate, bound, full = col(2, np.int32), col(3, np.float32), col(4, np.int32), col(5, np.uint8)
    sym = np.full(c, N, np.int32)
    oracle.set_expansion_budget(30000)
    try:
        st, depth, moves, exp = oracle.search_batch(beta, omega, sym, init, rate, bound, full, 16)
    finally:
        oracle.set_expansion_budget(0)
    done = st != oracle.BUDGET
    assert done.sum() >= c // 2
    inst = td.prepare_pairs(beta, omega, N, init, rate, bound, full)[done]
    ref, _ = td.search_batch(0, inst, td._lib.FLAG_ORDERED | td._lib.FLAG_VERIFY)
    assert (ref["status"] == st[done]).all()
    assert (ref["depth"] == np.where(st[done] == 1, depth[done], 0)).all()
    assert (ref["moves"] == np.where((st[done] == 1)[:, None], moves[done], 0)).all()
    assert (ref["expansions"] == exp[done] + 1).all()  # + the root's evaluation
    free, _ = td.search_batch(0, inst, td._lib.FLAG_VERIFY)
    assert (free["status"] == st[done]).all()
