"""The device replay of symbol witnesses against the checker's rules taken step
by step (CertificateValidator.java:14-50): every n, arrays in any order,
broken witnesses, arrays that are no permutation, block edges and unaligned
buffers.  Needs a B200."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _steps(beta, omega, abc, n, max_moves, depth):
    """The rules on lists; beta need not be a permutation."""
    if not (3 <= n <= 17 and 1 <= depth <= max_moves and depth <= 9):
        return 0
    b, o = list(beta[:n]), list(omega[:n])
    if any(v >= n for v in b + o):
        return 0
    rho = {}
    for x in range(n):
        rho[b[x]] = o[b[(x + 1) % n]]
    for m in range(depth):
        t = abc[3 * m: 3 * m + 3]
        if len(set(t)) < 3 or max(t) >= n:
            return 0
        pos = [max((x for x in range(n) if b[x] == v), default=-1) for v in t]
        if not 0 <= pos[0] < pos[1] < pos[2]:
            return 0
        o[t[0]], o[t[1]], o[t[2]] = o[t[2]], o[t[0]], o[t[1]]
        i, j, k = pos
        b = b[:i] + b[j:k] + b[i:j] + b[k:]
        if any(o[b[(x + 1) % n]] != rho[b[x]] for x in range(n)):
            return 0
    return int(all(o[x] == x for x in range(n)))


def _record(rng, n):
    """A record whose witness holds, then perhaps one byte of it changed."""
    beta = rng.permutation(n).tolist() if rng.random() < 0.5 else list(range(n))
    cur, abc = list(beta), []
    depth = int(rng.integers(1, 10))
    for _ in range(depth):
        i, j, k = sorted(rng.choice(n, 3, replace=False).tolist())
        abc += [cur[i], cur[j], cur[k]]
        cur = cur[:i] + cur[j:k] + cur[i:j] + cur[k:]
    succ = {cur[x]: cur[(x + 1) % n] for x in range(n)}
    omega = [0] * n
    for x in range(n):
        omega[beta[(x + 1) % n]] = succ[beta[x]]
    max_moves = 9
    kind = rng.integers(0, 10)
    if kind == 0:
        abc[int(rng.integers(len(abc)))] = int(rng.integers(0, 40))
    elif kind == 1:
        omega[int(rng.integers(n))] = int(rng.integers(n))
    elif kind == 2:
        beta[int(rng.integers(n))] = int(rng.integers(n))  # most often no permutation
    elif kind == 3:
        max_moves = depth - 1
    elif kind == 4:
        beta[int(rng.integers(n))] = 200
    return beta, omega, abc, max_moves, depth


def _periodic():
    """beta = (0 1 2 0 1 2) is no permutation: a symbol's place is its last one."""
    return [0, 1, 2, 0, 1, 2], [1, 2, 0, 3, 4, 5], [0, 1, 2], 9, 1


def _replay(td, recs, n_arr, shift):
    import torch
    c = len(recs)
    host = [np.zeros((c, w), np.uint8) for w in (17, 17)] + [np.asarray(n_arr, np.uint8)]
    mm, dep, abc = np.zeros(c, np.uint8), np.zeros(c, np.uint8), np.zeros((c, 27), np.uint8)
    for r, (b, o, t, m, d) in enumerate(recs):
        host[0][r, : len(b)], host[1][r, : len(o)] = b, o
        mm[r], dep[r], abc[r, : len(t)] = m, d, t
    dev = []
    for a in (*host, mm, dep, abc):
        buf = torch.zeros(a.size + 16, dtype=torch.uint8, device="cuda")
        buf[shift: shift + a.size] = torch.from_numpy(a.reshape(-1)).cuda()
        dev.append(buf)
    ok = torch.full((c + 1,), 7, dtype=torch.uint8, device="cuda")
    err = C.create_string_buffer(256)
    rc = td._lib.lib().td_replay_symbols_device(c, *[C.c_void_p(t.data_ptr() + shift) for t in dev],
                                               C.c_void_p(ok.data_ptr()), None, err, 256)
    assert rc == 0, err.value
    torch.cuda.synchronize()
    got = ok.cpu().numpy()
    assert got[c] == 7  # nothing past the last record
    return got[:c]


@pytest.mark.parametrize("count,shift", [(1, 0), (127, 0), (128, 0), (129, 0), (1000, 0), (1000, 1), (385, 4)])
def test_replay_follows_the_rules(td, count, shift):
    rng = np.random.default_rng(count + shift)
    n_arr = rng.integers(2, 19, count)
    recs = [_record(rng, int(max(3, min(17, n)))) for n in n_arr]
    if count > 1:
        recs[1], n_arr[1] = _periodic(), 6
    want = [_steps(b, o, t, int(n), m, d) for (b, o, t, m, d), n in zip(recs, n_arr)]
    got = _replay(td, recs, n_arr, shift)
    assert got.tolist() == want
    if count > 100:
        assert 0 < sum(want) < count
