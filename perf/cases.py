"""Performance cases of the witness-search engine, through its public binding (td16_b200._lib).

A case is a dict of plain values:
  kind        search (a batch), pairs (td_search_pairs on host arrays), percall (blocking td_search /
              td_search_ordered calls), distances (bounds deepened until every permutation is sorted),
              replay (the checker's replay of certificates), validate (the replay in pinned form)
  count       instances, pairs, calls or records of one pass
  n_min/n_max permutations of S_n, n uniform in this range
  hard_pct    share of near-reverse permutations (the reverse composed with 1..hard_max random block
              transpositions); the rest are uniform
  bound       9 (the engine's largest), half (floor(n/2)+1), or lower / lower+1 (the cycle-graph lower bound
              and one more: the questions whose answers give an exact distance)
  form        search: graph (a captured launch that is replayed), device (one launch call), host (host arrays
              in and out), noalloc (the allocation-free entry)
  order       free, or reference (the reference's single-queue move order)
  full        False: partial sorting with the rates that the emitter's callers pass
  threads     percall: native slot threads that call at once; 0: calls from Python, one after the other

Outputs: in the reference order the records (or witnesses) themselves, bit for bit.  In the free order any
witness within the bound is a right answer and several warps race for one, so a pass returns what is defined:
the status of every instance after the device's replay of its witness, and the permutations solved.
"""
import ctypes as C

import numpy as np
import torch

from td16_b200 import _lib, autotune

SLOTS = 16
BUDGET = 256 << 20  # bytes of device scratch a slot may use
MAX_N = 17


def _case(name, **kw):
    return {"name": name, **kw}


def listed():
    return [
        # the benchmark: decide 2^20 permutations of S_16 within 9 moves, in one captured launch
        _case("free_s16_2p20", kind="search", form="graph", order="free", count=1 << 20, n_min=16, n_max=16,
              hard_pct=50, hard_max=4, bound="9", full=True),
        # the uneven mix of the batched configuration; a few instances are searched to the end without a witness
        _case("free_mix_64k", kind="search", form="device", order="free", count=1 << 16, n_min=11, n_max=13,
              hard_pct=25, hard_max=3, bound="half", full=True),
        # is the lower bound the distance?  About three in ten have no witness: their trees are searched whole
        _case("free_s16_lower_2k", kind="search", form="device", order="free", count=2048, n_min=16, n_max=16,
              hard_pct=50, hard_max=4, bound="lower", full=True),
        # a small group of requests of the serving mix, host arrays in and out: launches and latency
        _case("free_8_16_lower1_250", kind="search", form="host", order="free", count=250, n_min=8, n_max=16,
              hard_pct=50, hard_max=3, bound="lower+1", full=True),
        # a case producer's group of reference pairs (near-reverse, odd count), end to end on the host
        _case("pairs_12_14_20k", kind="pairs", order="free", count=20011, n_min=12, n_max=14, hard_pct=100,
              hard_max=4, bound="lower+1", full=True),
        # exact distances of S_10 by deepening the bound in the reference's move order
        _case("distances_s10_4k", kind="distances", order="reference", count=4096, n_min=10, n_max=10, hard_pct=0,
              hard_max=0, bound="6", full=True),
        # reference-order witnesses of S_12, half near-reverse, a fifth without a witness
        _case("reference_s12_16k", kind="search", form="device", order="reference", count=16384, n_min=12,
              n_max=12, hard_pct=50, hard_max=3, bound="6", full=True),
        # partial sorting with the emitter's callers' rates, reference order, host arrays
        _case("reference_partial_3k", kind="search", form="host", order="reference", count=3001, n_min=8, n_max=12,
              hard_pct=30, hard_max=3, bound="lower+1", full=False),
        # the emitter's own shape: one blocking call per pair from every slot thread
        _case("percall_16_threads_2k", kind="percall", order="free", count=2048, n_min=8, n_max=14, hard_pct=50,
              hard_max=3, bound="lower", full=True, threads=16),
        # one caller, one small pair at a time: latency of a call
        _case("percall_reference_32", kind="percall", order="reference", count=32, n_min=5, n_max=9, hard_pct=20,
              hard_max=2, bound="lower+1", full=True, threads=0),
        # every stored certificate is replayed with the checker's rules
        _case("replay_s16_2p20", kind="replay", count=1 << 20, n_min=16, n_max=16),
        # the pinned-form replay that follows every batch
        _case("validate_s16_1m", kind="validate", count=1000003, n_min=16, n_max=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """One more case of the ranges above; the counts shrink as the questions get harder."""
    kind = rng.choice(["search", "search", "search", "search", "search", "pairs", "distances", "percall", "replay",
                       "validate"])
    if kind in ("replay", "validate"):
        n = rng.randint(5, 16)
        return dict(kind=kind, count=_log_int(rng, 1000, 1 << 20), n_min=rng.randint(4, n), n_max=n)
    case = dict(kind=kind, hard_pct=rng.choice([0, 20, 25, 50, 75, 100]), hard_max=rng.randint(1, 4), full=True)
    if kind == "distances":
        n = rng.randint(6, 10)
        return dict(case, order="reference", count=_log_int(rng, 64, 8192), n_min=rng.randint(4, n), n_max=n,
                    bound="6")
    if kind == "pairs":
        n = rng.randint(10, 15)
        return dict(case, order="free", count=_log_int(rng, 500, 20000), n_min=rng.randint(8, n), n_max=n,
                    bound="lower+1")
    if kind == "percall":
        if rng.random() < 0.5:
            n = rng.randint(8, 14)
            return dict(case, order="free", count=_log_int(rng, 256, 2048), n_min=rng.randint(6, n), n_max=n,
                        bound="lower", threads=16)
        n = rng.randint(5, 9)
        return dict(case, order="reference", count=rng.randint(8, 64), n_min=rng.randint(4, n), n_max=n,
                    bound="lower+1", threads=0)
    if rng.random() < 0.35:
        full = rng.random() < 0.6
        n = rng.randint(7, 12)
        return dict(case, form=rng.choice(["device", "host", "noalloc"]), order="reference", full=full,
                    count=_log_int(rng, 64, 16384 if full else 3000), n_min=rng.randint(5, n), n_max=n,
                    bound=rng.choice(["6", "5", "lower"]) if full else "lower+1")
    bound = rng.choice(["9", "half", "lower+1", "lower"])
    if bound in ("9", "half"):
        n, most = rng.randint(10, 16), 1 << 20
    else:
        n, most = rng.randint(8, 16), 2048 if bound == "lower" else 1 << 15
    form = rng.choice(["graph", "device", "host", "noalloc"])
    return dict(case, form=form, order="free", count=_log_int(rng, 16, min(most, 1 << 14) if form == "noalloc" else most),
                n_min=rng.randint(8 if bound == "9" else 6, n), n_max=n, bound=bound)


# ---- inputs -----------------------------------------------------------------

_started = False


def _start():
    global _started
    if not _started:
        _lib.init_slots(SLOTS, [0], BUDGET)
        _started = True


def _mix(seed):
    return (int(seed) * 0x9E3779B97F4A7C15 + 0x632BE59BD9B4E019) & (2 ** 64 - 1)


def _instances(case, seed):
    """(permutations, n, instances) of a case, the bounds in place."""
    perms, n = _lib.synth_perms(_mix(seed), case["count"], case["n_min"], case["n_max"], case["hard_pct"],
                                min(1, case["hard_max"]), case["hard_max"])
    inst = _lib.prepare_perms(perms, n, 9)
    init = (inst["packed"] & 31).astype(np.int32)
    lower = (n.astype(np.int32) + 1 - init + 1) // 2
    bound = {"half": n.astype(np.int32) // 2 + 1, "lower": lower, "lower+1": lower + 1}.get(case["bound"])
    if bound is None:
        bound = np.full(len(n), int(case["bound"]), np.int32)
    bound = np.clip(bound, 1, 9).astype(np.int32)
    inst["max_moves"] = bound
    if not case["full"]:
        # partial sorting: minRate = 2 / (maxMoves / (float) target), as the emitter's callers compute it, with a
        # target of odd cycles to gain
        rng = np.random.default_rng(_mix(seed))
        target = rng.integers(1, np.maximum(2, lower + 1)).astype(np.float32)
        inst["min_rate"] = np.float32(2) / (bound.astype(np.float32) / target)
        inst["packed"] &= 31
    return perms, n, inst, init, bound


def _pairs(perms, n):
    count = len(n)
    beta = np.zeros((count, MAX_N), np.uint8)
    omega = np.zeros((count, MAX_N), np.uint8)
    _lib.lib().td_pairs_from_perms(count, _lib._ptr(perms), _lib._ptr(n), _lib._ptr(beta), _lib._ptr(omega))
    return beta, omega


def _random_witnesses(case, seed):
    """Records whose witness is known by construction: the array 0..n is taken through random block swaps, and
    the array it ends in is the target.  One record in 64 has its last two symbols of a move exchanged."""
    count, dev = case["count"], "cuda"
    g = torch.Generator(device=dev)
    g.manual_seed(_mix(seed) >> 1)
    ri = lambda lo, hi, shape: torch.randint(lo, hi, shape, generator=g, device=dev)  # noqa: E731
    N = ri(case["n_min"] + 1, case["n_max"] + 2, (count,))
    most = min(9, case["n_max"] // 2 + 1)
    depth = ri(max(1, most - 2), most + 1, (count,))
    col = torch.arange(MAX_N, device=dev).expand(count, MAX_N)
    cur = torch.where(col < N[:, None], col, torch.zeros_like(col))
    ijk = torch.zeros((count, 9, 3), dtype=torch.int64, device=dev)
    abc = torch.zeros((count, 9, 3), dtype=torch.int64, device=dev)
    for m in range(most):
        key = torch.rand((count, MAX_N), generator=g, device=dev).masked_fill_(col >= N[:, None], 2.0)
        t = key.topk(3, dim=1, largest=False).indices.sort(dim=1).values
        on = (m < depth)[:, None]
        ijk[:, m] = torch.where(on, t, 0)
        abc[:, m] = torch.where(on, cur.gather(1, t), 0)
        i, j, k = t[:, :1], t[:, 1:2], t[:, 2:]
        inside = (col >= i) & (col < k)
        src = torch.where(col < i + (k - j), col + (j - i), col - (k - j))
        cur = torch.where(on, cur.gather(1, torch.where(inside, src, col)), cur)
    bad = ri(0, 64, (count,)) == 0
    at = (ri(0, 1 << 30, (count,)) % depth)[:, None, None].expand(-1, 1, 3)
    for v in (ijk, abc):
        v.copy_(torch.where(bad[:, None, None], v.scatter(1, at, v.gather(1, at)[:, :, [0, 2, 1]]), v))
    # omega = rho . beta^-1 with beta = (0 1 ...) and rho the cycle that the array ends in
    nxt = torch.where(col + 1 < N[:, None], col + 1, 0)
    rho = torch.zeros_like(cur).scatter(1, torch.where(col < N[:, None], cur, MAX_N - 1),
                                        torch.where(col < N[:, None], cur.gather(1, nxt), 0))
    prev = torch.where(col > 0, col - 1, N[:, None] - 1)
    omega = torch.where(col < N[:, None], rho.gather(1, prev), 0)
    return N, depth, ijk, abc, omega


class State:
    """What a caller keeps for a case; a captured graph is released with it."""

    graph = None

    def __init__(self, case):
        self.case = case

    def __del__(self):
        if self.graph is not None:
            self.graph.close()


def prepare(case, seed):
    _start()
    s = State(case)
    kind = case["kind"]
    if kind in ("replay", "validate"):
        N, depth, ijk, abc, omega = _random_witnesses(case, seed)
        u8 = lambda v: v.to(torch.uint8).contiguous()  # noqa: E731
        count = case["count"]
        s.ok = torch.zeros(count, dtype=torch.uint8, device="cuda")
        if kind == "replay":
            beta = torch.arange(MAX_N, device="cuda").expand(count, MAX_N)
            s.args = [u8(torch.where(beta < N[:, None], beta, 0)), u8(omega), u8(N),
                      torch.full((count,), 9, dtype=torch.uint8, device="cuda"), u8(depth), u8(abc.view(count, 27))]
            return s
        n_host = N.to(torch.uint8).cpu().numpy()
        beta = np.where(np.arange(MAX_N) < n_host[:, None], np.arange(MAX_N), 0).astype(np.uint8)
        inst = _lib.prepare_pairs(beta, u8(omega).cpu().numpy(), n_host, 0, 0.0, 9, 1)
        res = np.zeros(count, _lib.RESULT_DTYPE)
        res["status"], res["depth"] = 1, depth.cpu().numpy()
        res["moves"] = (ijk[:, :, 0] | (ijk[:, :, 1] << 5) | (ijk[:, :, 2] << 10)).cpu().numpy()
        s.inst = torch.from_numpy(inst.view(np.uint8)).cuda()
        s.res = torch.from_numpy(res.view(np.uint8)).cuda()
        return s
    # the launch shape that the autotuner keeps for the S_16 batches and the mix; the library's own otherwise
    big = kind == "search" and case["order"] == "free" and case["count"] >= 1 << 15
    autotune.apply("17" if big and case["n_min"] == 16 else "mix_11_13" if big and case["n_max"] <= 13 else "defaults")
    perms, n, inst, init, bound = _instances(case, seed)
    if kind in ("pairs", "percall"):
        s.beta, s.omega = _pairs(perms, n)
        s.n, s.init, s.bound = (n + 1).astype(np.uint8), init, bound
        s.call = [(i, s.beta[i, : s.n[i]].tobytes(), s.omega[i, : s.n[i]].tobytes()) for i in range(case["count"])] \
            if kind == "percall" and not case["threads"] else None
        return s
    s.inst = inst
    if case.get("form") == "host":
        return s
    s.stream_ptr = _lib.lib().td_slot_stream(0)
    s.stream = torch.cuda.ExternalStream(s.stream_ptr)
    s.flags = _lib.FLAG_VERIFY | (_lib.FLAG_ORDERED if case["order"] == "reference" else 0)
    s.perm = torch.from_numpy(inst["perm"].view(np.int64).copy()).cuda()
    bounds = [None] if kind == "search" else list(range(1, int(case["bound"]) + 1))
    s.d_in, s.d_res = [], []
    for b in bounds:
        if b is not None:
            inst["max_moves"] = b
        s.d_in.append(torch.from_numpy(inst.view(np.uint8).copy()).cuda())
        s.d_res.append(torch.zeros((case["count"], 8), dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    if case.get("form") == "graph":
        s.graph = _lib.BatchGraph(0, case["count"], s.d_in[0].data_ptr(), s.d_res[0].data_ptr(), s.flags)
    return s


# ---- one pass -----------------------------------------------------------------

def _solved(s, found):
    """omega of the solved pairs (the keys of their certificates), 0 for the others."""
    return s.omega * found.view(np.uint8)[:, None]


def _run_percall(s):
    case = s.case
    if case["threads"]:
        entry = _lib.entry_address("td_search" if case["order"] == "free" else "td_search_ordered")
        r = _lib.slot_threads_run(entry, s.beta, s.omega, s.n, s.init, 0.0, s.bound, 1, case["threads"])
        if case["order"] == "free":
            return {"status": r["status"], "solved": _solved(s, r["status"] == 1)}
        return {"status": r["status"], "moves": r["moves"]}
    moves = np.zeros((case["count"], 9, 3), np.int16)
    for i, beta, omega in s.call:
        w = _lib.search(0, beta, omega, s.init[i], 0.0, s.bound[i], True, case["order"] == "reference")
        if w:
            moves[i, : len(w)] = w
    return {"moves": moves}


def run(s):
    case, kind, count = s.case, s.case["kind"], s.case["count"]
    if kind == "replay":
        err = C.create_string_buffer(256)
        _lib.check(_lib.lib().td_replay_symbols_device(count, *[C.c_void_p(t.data_ptr()) for t in s.args],
                                                       C.c_void_p(s.ok.data_ptr()), None, err, 256), err)
        return {"ok": s.ok}
    if kind == "validate":
        _lib.validate_batch_device(count, s.inst.data_ptr(), s.res.data_ptr(), s.ok.data_ptr())
        return {"ok": s.ok}
    if kind == "percall":
        return _run_percall(s)
    if kind == "pairs":
        status, depth, moves = _lib.search_pairs(0, s.beta, s.omega, s.n, s.init, 0.0, s.bound, 1,
                                                 case["order"] == "reference")
        if case["order"] == "free":
            return {"status": status, "solved": _solved(s, status == _lib.OK)}
        return {"status": status, "depth": depth, "moves": moves}
    free = case["order"] == "free"
    if case.get("form") == "host":
        res, _ = _lib.search_batch(0, s.inst, _lib.FLAG_VERIFY | (0 if free else _lib.FLAG_ORDERED))
        if free:
            return {"status": res["status"], "solved": np.where(res["status"] == 1, s.inst["perm"].view(np.int64), -1)}
        return {"records": res.view(np.int32).reshape(count, 8)}
    for d_in, d_res in zip(s.d_in, s.d_res):
        if s.graph is not None:
            s.graph.launch(s.stream_ptr)
        elif case.get("form") == "noalloc":
            err = C.create_string_buffer(256)
            _lib.check(_lib.lib().td_search_batch_noalloc(
                C.c_int(count), C.c_void_p(d_in.data_ptr()), C.c_void_p(d_res.data_ptr()), C.c_uint(s.flags),
                C.c_uint64(0), C.c_void_p(s.stream_ptr), err, C.c_size_t(256)), err)
        else:
            _lib.search_batch_device(0, count, d_in.data_ptr(), d_res.data_ptr(), s.flags, 0, s.stream_ptr)
    with torch.cuda.stream(s.stream):
        if kind == "distances":
            found = torch.stack([r[:, 0] == 1 for r in s.d_res])
            distance = torch.where(found.any(0), found.to(torch.uint8).argmax(0) + 1, 0)
            return {"distance": distance, "records": s.d_res}
        if not free:
            return {"records": s.d_res[0]}
        status = s.d_res[0][:, 0]
        return {"status": status.clone(), "solved": torch.where(status == 1, s.perm, -1)}


# ---- what a pass cannot do without ---------------------------------------------

def work(case):
    """Bytes: each instance (16) or record read and each result (32) or verdict written once.  Operations: a
    witness of about n/2 moves needs the children of that many nodes, C(n+1, 3) each, classified."""
    count, N = case["count"], (case["n_min"] + case["n_max"]) / 2 + 1
    if case["kind"] == "replay":
        return {"bytes": count * (2 * N + 3 + 3 * N / 2 + 1), "flops": count * N * N}
    if case["kind"] == "validate":
        return {"bytes": count * 49, "flops": count * N * N}
    passes = int(case["bound"]) if case["kind"] == "distances" else 1
    triples = N * (N - 1) * (N - 2) / 6
    return {"bytes": passes * count * 48, "flops": passes * count * triples * (N / 2)}


def exact(case, seed):
    """Every output is a whole number, equal from run to run: none is a rounded value."""
    return None
