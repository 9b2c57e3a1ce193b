// td_emu.cc -- serial host emulation of the engine's warp algorithm.
//
// TEST INFRASTRUCTURE ONLY, and not a parity oracle: it restates the engine's
// own algorithm, not the reference's.  It runs the kernel's per-node steps one
// lane at a time, so that the CPU test suite can check the engine's logic
// against the oracle (td_oracle.c) without a GPU, and so that the benchmark's
// CPU baseline can time the free-order algorithm on host cores
// (td_emu_search_batch):
//   reference order: pinned state, pair table, 12-bit class table, per-lane
//     step bitmasks and the single-queue child order;
//   free order: row masks and bit-sliced classes (td_row_classes), pair slots,
//     the +2-first child order, the table of explored states and the restarts
//     with their child orders (td_attempt_budget, td_level_order), and, once
//     td_emu_set_endgame has given it one, the endgame table with the moves that
//     fix symbols first (td_eg_filter, td_eg_look, td_take_fixing).
// It shares the kernel's helpers in td_core.cuh.  The product library does not
// contain or call it.
#include "../td16_b200/csrc/td_core.cuh"

#include <string.h>

#include <atomic>
#include <thread>
#include <vector>

namespace {

struct Emu {
    int N, T, steps, maxd, ordered;
    uint8_t tri_i[TD_MAX_TRIPLES], tri_j[TD_MAX_TRIPLES], tri_k[TD_MAX_TRIPLES];
    uint32_t acc[TD_MAX_DEPTH + 2], reach[TD_MAX_DEPTH + 2];
    uint8_t lut[4096];
    uint8_t pt[TD_MAX_N * TD_PT_STRIDE];
    uint32_t m1[TD_MAX_DEPTH + 1][32], m2[TD_MAX_DEPTH + 1][32];
    // free order (bit-sliced): rows by caller position, masks, pair slots, outcome words
    uint32_t S[32], G[32], P[32], O, F;
    int next[32];  // next caller position along omega
    uint32_t pc[TD_MAX_ROUNDS][32];
    uint32_t pw[TD_MAX_DEPTH + 1][TD_MAX_ROUNDS][32];
    int rounds;
    uint64_t L[TD_MAX_DEPTH + 1];
    int off[TD_MAX_DEPTH + 1];
    uint16_t path[TD_MAX_DEPTH];
    uint32_t expansions;
};

int prepare(Emu &e, uint64_t L, int off) {
    const int N = e.N;
    int B[TD_MAX_N], pos[TD_MAX_N], nxt[TD_MAX_N], lead[TD_MAX_N], dist[TD_MAX_N], len[TD_MAX_N];
    for (int p = 0; p < N; ++p) {
        B[p] = p ? (int)td_nib(L, p - 1) + 1 : 0;
        pos[B[p]] = p;
    }
    for (int p = 0; p < N; ++p) {
        const int q = p ? p - 1 : N - 1;
        int y = B[q] + 1;
        if (y == N) y = 0;
        nxt[p] = pos[y];
    }
    for (int p = 0; p < N; ++p) {
        int m = p, x = nxt[p], l = 1;
        while (x != p) { if (x < m) m = x; x = nxt[x]; ++l; }
        lead[p] = m;
        len[p] = l;
        int d = 0;
        x = p;
        while (x != m) { x = nxt[x]; ++d; }
        dist[p] = d;
    }
    int odd = 0;
    for (int p = 0; p < N; ++p) odd += (lead[p] == p) && (len[p] & 1);
    for (int p = 0; p < N; ++p) {
        const int rp = (p - off + N) % N;
        for (int q = 0; q < N; ++q) {
            const int rq = (q - off + N) % N;
            e.pt[rp * TD_PT_STRIDE + rq] =
                (uint8_t)td_pair_entry(lead[p], dist[p], len[p], lead[q], dist[q]);
        }
    }
    return odd;
}

// Rows of the bit-sliced evaluation, computed the way the kernel does: lane c
// is caller position c, its cycle leader the smallest caller position on the
// cycle, dist the omega steps to it.  Returns the number of odd cycles.
int prepare_rows(Emu &e, uint64_t L, int off) {
    const int N = e.N;
    int B[TD_MAX_N], pos[TD_MAX_N], nxt[32], lead[32], dist[32], len[32];
    for (int p = 0; p < N; ++p) {
        B[p] = p ? (int)td_nib(L, p - 1) + 1 : 0;
        pos[B[p]] = p;
    }
    for (int c = 0; c < 32; ++c) nxt[c] = c;
    for (int c = 0; c < N; ++c) {
        const int p = (c + off) % N;
        const int q = p ? p - 1 : N - 1;
        const int y = (B[q] + 1) % N;
        nxt[c] = (pos[y] - off + N) % N;
    }
    for (int c = 0; c < 32; ++c) e.next[c] = nxt[c];
    for (int c = 0; c < 32; ++c) {
        int m = c, x = nxt[c], l = 1;
        while (x != c) { if (x < m) m = x; x = nxt[x]; ++l; }
        lead[c] = m;
        len[c] = l;
        int d = 0;
        x = c;
        while (x != m) { x = nxt[x]; ++d; }
        dist[c] = d;
    }
    const uint32_t ACT = (1u << N) - 1u;
    e.O = e.F = 0;
    int odd = 0;
    for (int c = 0; c < N; ++c) {
        if (len[c] & 1) e.O |= 1u << c;
        if (len[c] == 1) e.F |= 1u << c;
        odd += lead[c] == c && (len[c] & 1);
    }
    for (int c = 0; c < N; ++c) {
        uint32_t S = 0, lt = 0, D0 = 0;
        for (int q = 0; q < 32; ++q) {
            if (lead[q] == lead[c]) S |= 1u << q;
            if (dist[q] < dist[c]) lt |= 1u << q;
            if (dist[q] & 1) D0 |= 1u << q;
        }
        S &= ACT;
        const uint32_t lodd = 0u - (uint32_t)(len[c] & 1);
        e.S[c] = S;
        e.G[c] = S & lt;
        e.P[c] = S & ((D0 ^ (0u - (uint32_t)(dist[c] & 1))) ^ (lodd & ~lt));
    }
    return odd;
}

// Bit-sliced evaluation of the node at `level`: fills the outcome words and
// returns the found move (i | j<<5 | k<<10) or -1.
int evaluate_rows(Emu &e, int level, int odd) {
    const int D = level + 1;
    const uint32_t f0 = 0u - ((e.acc[D] >> odd) & 1u), f2 = 0u - ((e.acc[D] >> (odd + 2)) & 1u);
    const uint32_t x0 = (D < e.maxd ? 0u - ((e.reach[D] >> odd) & 1u) : 0u) & ~f0;
    const uint32_t x2 = (D < e.maxd ? 0u - ((e.reach[D] >> (odd + 2)) & 1u) : 0u) & ~f2;
    const uint32_t ACT = (1u << e.N) - 1u;
    uint32_t best = 0xffffffffu;
    for (int lane = 0; lane < 32; ++lane) {
        uint32_t key = 0xffffffffu;
        for (int r = 0; r < e.rounds; ++r) {
            const uint32_t code = e.pc[r][lane];
            const int i = code & 31, j = (code >> 5) & 31, ks = (code >> 10) & 31;
            uint32_t plus, zero;
            td_row_classes_x(e.S[i], e.G[i], e.P[i], e.S[j], e.G[j], e.P[j], e.O, e.F, 0u - ((e.O >> i) & 1u),
                             0u - ((e.O >> j) & 1u), 0u - ((e.F >> i) & 1u), 0u - ((e.F >> j) & 1u), (int)(code >> 15),
                             &plus, &zero);
            const uint32_t km = ACT & (0xfffffffeu << ks);
            const uint32_t fnd = km & ((f0 & zero) | (f2 & plus));
            const uint32_t e2 = km & x2 & plus, e0 = km & x0 & zero;
            e.pw[level][r][lane] = (e2 >> 1) | (e0 << 15);
            if (fnd && key == 0xffffffffu)
                key = ((uint32_t)lane << 17) | ((uint32_t)r << 15) | (code & 1023u) | ((uint32_t)(31 - __builtin_clz(fnd)) << 10);
        }
        if (key < best) best = key;
    }
    e.expansions++;
    return best == 0xffffffffu ? -1 : (int)(best & 0x7fffu);
}

// Next child of `level` in the free order: +2 children first; in the plain
// order (ord = 0) the highest pair slot R*lane + r (lexicographically smallest
// pair) and the smallest k.  `ord` (td_order_variant) rotates the lane
// priority, reverses the round order and takes the largest k first, as the
// kernel does.  Returns the move, with bit 15 set for a 0 child, or -1.
int next_child_rows(Emu &e, int level, uint32_t ord) {
    bool any2 = false;
    for (int lane = 0; lane < 32; ++lane)
        for (int r = 0; r < e.rounds; ++r) any2 |= (e.pw[level][r][lane] & 0xffffu) != 0;
    const uint32_t cm = any2 ? 0x0000ffffu : 0xffff0000u;
    const int rot = (int)(ord & 31u);
    int bl = -1, br = -1;
    unsigned bkey = 0;
    for (int lane = 0; lane < 32; ++lane)
        for (int r = 0; r < e.rounds; ++r)
            if (e.pw[level][r][lane] & cm) {
                const unsigned key = ((((unsigned)(lane - rot) & 31u) << 2) | (unsigned)((ord & 32u) ? 3 - r : r)) + 1u;
                if (key > bkey) { bkey = key; bl = lane; br = r; }
            }
    if (bl < 0) return -1;
    const int lane = bl, r = br;
    const uint32_t w = e.pw[level][r][lane] & cm;
    const int b = (ord & 64u) ? 31 - __builtin_clz(w) : __builtin_ctz(w);
    e.pw[level][r][lane] &= ~(1u << b);
    const int k = any2 ? b + 1 : b - 15;
    return (int)((e.pc[r][lane] & 1023u) | ((uint32_t)k << 10) | (any2 ? 0u : 0x8000u));
}

// Evaluate the children of the node at `level` (parent odd count `odd`).
// Returns the found u (>= 0) or -1.
int evaluate(Emu &e, int level, int odd) {
    const int D = level + 1;
    const int f0 = (e.acc[D] >> odd) & 1, f2 = (e.acc[D] >> (odd + 2)) & 1;
    const int x0 = (D < e.maxd) && ((e.reach[D] >> odd) & 1) && !f0;
    const int x2 = (D < e.maxd) && ((e.reach[D] >> (odd + 2)) & 1) && !f2;
    uint32_t nt;  // byte c holds the flags of class c; byte 0 (filtered out) is zero
    if (e.ordered) nt = ((uint32_t)(f0 | (x0 << 1)) << (8 * TD_CLASS_ZERO)) | ((uint32_t)(f2 | (x2 << 1)) << (8 * TD_CLASS_PLUS2));
    else nt = ((uint32_t)(f0 | (x0 << 2)) << (8 * TD_CLASS_ZERO)) | ((uint32_t)(f2 | (x2 << 1)) << (8 * TD_CLASS_PLUS2));
    uint32_t fb[32];
    for (int lane = 0; lane < 32; ++lane) {
        fb[lane] = 0;
        e.m1[level][lane] = 0;
        e.m2[level][lane] = 0;
        for (int s = 0; s < e.steps; ++s) {
            const int u = 32 * s + lane;
            if (u >= e.T) continue;
            const int t = e.T - 1 - u;
            const int i = e.tri_i[t], j = e.tri_j[t], k = e.tri_k[t];
            const int idx = e.pt[i * TD_PT_STRIDE + j] | (e.pt[j * TD_PT_STRIDE + k] << 4) |
                            (e.pt[k * TD_PT_STRIDE + i] << 8);
            const uint32_t tb = (nt >> (8 * e.lut[idx])) & 7u;
            fb[lane] |= (tb & 1u) << s;
            e.m1[level][lane] |= ((tb >> 1) & 1u) << s;
            e.m2[level][lane] |= ((tb >> 2) & 1u) << s;
        }
    }
    e.expansions++;
    if (e.ordered && level == 0) {  // roots are accepted when visited, not when seeded
        for (int lane = 0; lane < 32; ++lane) e.m2[0][lane] = fb[lane];
        return -1;
    }
    int best = -1;
    for (int lane = 0; lane < 32; ++lane) {
        if (!fb[lane]) continue;
        const int u = 32 * __builtin_ctz(fb[lane]) + lane;
        if (best < 0 || u < best) best = u;
    }
    return best;
}

// Next child of `level` in visit order; returns u or -1; *accepted for roots
// that are accepted on visit (ordered mode).
int next_child(Emu &e, int level, int *accepted) {
    *accepted = 0;
    const bool desc_lanes = e.ordered && level > 0;
    int any1 = 0;
    for (int lane = 0; lane < 32; ++lane) any1 |= e.m1[level][lane] != 0;
    uint32_t best = 0;
    for (int lane = 0; lane < 32; ++lane) {
        uint32_t w;
        if (e.ordered) w = level == 0 ? (e.m1[level][lane] | e.m2[level][lane]) : e.m1[level][lane];
        else w = any1 ? e.m1[level][lane] : e.m2[level][lane];
        if (!w) continue;
        const uint32_t s = 31 - __builtin_clz(w);
        const uint32_t key = s * 32 + (desc_lanes ? 31 - lane : lane) + 1;
        if (key > best) best = key;
    }
    if (!best) return -1;
    best -= 1;
    const int s = (int)(best >> 5);
    const int lane = desc_lanes ? 31 - (int)(best & 31) : (int)(best & 31);
    const uint32_t bit = 1u << s;
    if (e.ordered) {
        if (level == 0 && (e.m2[0][lane] & bit)) *accepted = 1;
        e.m1[level][lane] &= ~bit;
        e.m2[level][lane] &= ~bit;
    } else if (any1) {
        e.m1[level][lane] &= ~bit;
    } else {
        e.m2[level][lane] &= ~bit;
    }
    return 32 * s + lane;
}

// The kernel's table of explored states (free order): 2^12 entries, key =
// td_tt_key of the pinned state (nibbles from N-1 on cleared) times an odd
// constant modulo 2^57, the top 12 bits the slot and the rest the tag, a
// 15-bit generation, the depth in the top nibble.  The generation counter
// persists across searches on a thread, as the kernel's does across units.
#define EMU_TT_BITS 12
// restart budget base of the free order (the kernel's default); 0 = none
static uint32_t g_restart_base = 16;
extern "C" void td_emu_set_restart(uint32_t base) { g_restart_base = base; }
// The child order at DFS level `level` of attempt a, its budget for a base,
// and the number of budgeted attempts (td_core.cuh), for the CPU tests.
extern "C" uint32_t td_emu_order(int a, int level) { return td_level_order(td_order_variant(a), a, level); }
extern "C" uint32_t td_emu_budget(uint32_t base, int a) { return td_attempt_budget(base, a); }
extern "C" int td_emu_restarts(void) { return TD_RESTARTS; }
bool tt_visit(uint64_t *tt, uint64_t L, int N, int lv, uint32_t gen) {
    const uint64_t data = N - 1 >= 16 ? ~0ull : ((1ull << (4 * (N - 1))) - 1ull);
    const uint64_t h = (td_tt_key(L & data) * 0x9E3779B97F4A7C15ull) & 0x01ffffffffffffffull;
    const int tag_bits = 57 - EMU_TT_BITS;
    const unsigned slot = (unsigned)(h >> tag_bits);
    const uint64_t want = (h & ((1ull << tag_bits) - 1ull)) | ((uint64_t)gen << tag_bits);
    const uint64_t old = tt[slot];
    if ((old & ((1ull << 60) - 1ull)) == want && (int)(old >> 60) <= lv) return true;
    tt[slot] = want | ((uint64_t)lv << 60);
    return false;
}

// the next generation of the thread's table; clears it when the counter wraps
uint32_t tt_next_gen(uint64_t *tt, uint32_t &counter) {
    if (++counter >= (1u << (EMU_TT_BITS + 3))) {
        for (int q = 0; q < (1 << EMU_TT_BITS); ++q) tt[q] = 0;
        counter = 1;
    }
    return counter;
}

const uint16_t *g_endgame = nullptr;  // td_emu_endgame's for TD_EG_SYMBOLS symbols, or none

// What the endgame table says of the state L: -1 unknown, 0 sorted within the
// moves left, else the expansions of its walk.  `tight`: no spare move.
int endgame_probe(const uint16_t *table, int N, uint64_t L, bool tight) {
    uint32_t kept = 0;
    for (int p = 0; p < N; ++p) {
        const int b = p ? (int)td_nib(L, p - 1) + 1 : 0, q = p ? p - 1 : N - 1;
        const int a = q ? (int)td_nib(L, q - 1) + 1 : 0;
        if (b != (a + 1) % N) kept |= 1u << b;
    }
    const int n = td_popc(kept);
    if (n > TD_EG_SYMBOLS) return -1;
    if (n == 0 || !tight) return 0;
    return table[td_eg_base(n - 1) + td_eg_rank(L, kept)];
}

// The same for the child that `move` makes of the state of `level`.
int endgame_child(const Emu &e, const uint16_t *table, int level, uint32_t move, bool tight) {
    uint64_t nL;
    int noff;
    td_apply_move(e.L[level], e.off[level], e.N, move & 31, (move >> 5) & 31, (move >> 10) & 31, &nL, &noff);
    return endgame_probe(table, e.N, nL, tight);
}

// td_eg_filter: a node without a spare move.  The first child that can be sorted
// becomes its only one (returns true), else those that the table does not hold
// stay.
bool endgame_filter(Emu &e, int level) {
    bool solved = false;
    for (int lane = 0; lane < 32 && !solved; ++lane)
        for (int r = e.rounds - 1; r >= 0 && !solved; --r)
            for (uint32_t w = e.pw[level][r][lane]; w && !solved; w &= w - 1) {
                const int b = __builtin_ctz(w);
                const int v = endgame_child(e, g_endgame, level, (e.pc[r][lane] & 1023u) | ((uint32_t)(b + 1) << 10), true);
                if (v == 0) {
                    solved = true;
                    for (int q = 0; q < e.rounds; ++q)
                        for (int l = 0; l < 32; ++l) e.pw[level][q][l] = 0;
                    e.pw[level][r][lane] = 1u << b;
                } else if (v > 0) {
                    e.pw[level][r][lane] &= ~(1u << b);
                }
            }
    return solved;
}

// td_take_fixing: the move that fixes two symbols or three, of lowest position,
// where it is among the +2 children of `level`; or -1.
int take_fixing(Emu &e, int level) {
    for (int x = 0; x < e.N; ++x) {
        const int y = e.next[x], z = e.next[y];
        if ((x < y) + (y < z) + (z < x) != 2) continue;
        int c[3] = {x, y, z};
        const int s = x < y && x < z ? 0 : y < z ? 1 : 2;
        const int i = c[s], j = c[(s + 1) % 3], k = c[(s + 2) % 3];
        for (int lane = 0; lane < 32; ++lane)
            for (int r = 0; r < e.rounds; ++r)
                if ((e.pc[r][lane] & 1023u) == (uint32_t)(i | j << 5) && ((e.pw[level][r][lane] >> (k - 1)) & 1u)) {
                    e.pw[level][r][lane] &= ~(1u << (k - 1));
                    return i | j << 5 | k << 10;
                }
        return -1;
    }
    return -1;
}

int search_rows(Emu &e, int eg_moves, td_result *res) {
    static thread_local uint64_t tt[1 << EMU_TT_BITS];  // zero-initialised: every word empty
    static thread_local uint32_t tt_counter = 0;
    bool tt_on = false;  // in use after 32 expansions, as in the kernel
    uint32_t tt_gen = 0;
    int attempt = 0;     // restarts, as in the kernel
    uint32_t ord = 0, attempt_exp = 1, attempt_budget = td_attempt_budget(g_restart_base, 0);
    const int NP = (e.N - 1) * (e.N - 2) / 2;
    e.rounds = (NP + 31) / 32;
    for (int r = 0; r < TD_MAX_ROUNDS; ++r)
        for (int lane = 0; lane < 32; ++lane) e.pc[r][lane] = td_pair_code(e.N, r < e.rounds ? e.rounds * lane + r : -1);
    if (!g_endgame) eg_moves = 0;
    int level = 0, spare[TD_MAX_DEPTH];  // -1: the endgame table decides no child
    bool solved = false;
    int found = -1;
    // expands the node at `level`, and lets the table decide its children
    auto expand = [&] {
        const int odd = prepare_rows(e, e.L[level], e.off[level]);
        const int sp = eg_moves - level - ((e.N - odd) >> 1);
        spare[level] = eg_moves > level + 1 && sp >= 0 && e.N - td_popc(e.F) <= TD_EG_SYMBOLS + 3 ? sp : -1;
        found = evaluate_rows(e, level, odd);
        if (found >= 0 || spare[level] != 0) return;
        int children = 0;
        for (int lane = 0; lane < 32; ++lane)
            for (int r = 0; r < e.rounds; ++r) children += td_popc(e.pw[level][r][lane]);
        if (children >= 8) solved |= endgame_filter(e, level);
    };
    expand();
    for (;;) {
        if (found >= 0) {
            for (int d = 0; d < level; ++d) res->moves[d] = e.path[d];
            res->moves[level] = (uint16_t)found;
            res->depth = level + 1;
            res->status = TD_FOUND;
            break;
        }
        if (attempt_exp >= attempt_budget && !solved) {
            ++attempt;
            ord = td_order_variant(attempt);
            attempt_budget = td_attempt_budget(g_restart_base, attempt);
            attempt_exp = 1;
            if (tt_on) tt_gen = tt_next_gen(tt, tt_counter);  // the abandoned attempt's entries no longer match
            level = 0;
            expand();
            continue;
        }
        bool done = false;
        for (bool fresh = attempt + solved == 0 && eg_moves != 0;; fresh = false) {
            int t = fresh ? take_fixing(e, level) : -1;
            if (t < 0) t = next_child_rows(e, level, td_level_order(ord, attempt, level));
            if (t < 0) {
                if (level == 0) { done = true; break; }
                --level;
                continue;
            }
            e.path[level] = (uint16_t)(t & 0x7fff);
            int noff;
            td_apply_move(e.L[level], e.off[level], e.N, t & 31, (t >> 5) & 31, (t >> 10) & 31, &e.L[level + 1], &noff);
            e.off[level + 1] = noff;
            if (spare[level] >= 0) {
                const int v = endgame_probe(g_endgame, e.N, e.L[level + 1], spare[level] == (t >> 15));
                if (v == 0) {
                    solved = true;
                    break;
                }
                if (v > 0) continue;
            }
            if (solved) break;
            if (!tt_on && e.expansions >= 32) {
                tt_gen = tt_next_gen(tt, tt_counter);
                tt_on = true;
            }
            if (tt_on && tt_visit(tt, e.L[level + 1], e.N, level + 1, tt_gen)) continue;  // explored with at least this budget
            break;
        }
        if (done) { res->status = TD_NOT_FOUND; break; }
        ++level;
        expand();
        ++attempt_exp;
    }
    res->expansions = e.expansions;
    return res->status;
}

}  // namespace

// Compares the bit-sliced classes of every triple of the state (L, off) with
// the 12-bit class table; returns the number of triples that differ.
extern "C" int td_emu_row_check(uint64_t L, int off, int N) {
    static thread_local Emu e;
    e.N = N;
    prepare(e, L, off);
    prepare_rows(e, L, off);
    const uint32_t ACT = (1u << N) - 1u;
    int bad = 0;
    for (int i = 0; i < N; ++i)
        for (int j = i + 1; j < N; ++j) {
            uint32_t plus, zero;
            td_row_classes(e.S[i], e.G[i], e.P[i], e.S[j], e.G[j], e.P[j], e.O, e.F, i, j, &plus, &zero);
            plus &= ACT;
            zero &= ACT;
            for (int k = j + 1; k < N; ++k) {
                const int idx = e.pt[i * TD_PT_STRIDE + j] | (e.pt[j * TD_PT_STRIDE + k] << 4) |
                                (e.pt[k * TD_PT_STRIDE + i] << 8);
                const int cls = td_class_of_index(idx);
                const int got = ((plus >> k) & 1) ? TD_CLASS_PLUS2 : (((zero >> k) & 1) ? TD_CLASS_ZERO : TD_CLASS_SKIP);
                if (((plus >> k) & 1) && ((zero >> k) & 1)) ++bad;
                else if (got != cls) ++bad;
            }
        }
    return bad;
}

// Gives later free-order searches the endgame table (td_emu_endgame's for
// TD_EG_SYMBOLS symbols; it must outlive them), or takes it away (null).
extern "C" void td_emu_set_endgame(const uint16_t *table) { g_endgame = table; }

extern "C" int td_emu_search(const td_instance *x, unsigned flags, td_result *res) {
    static thread_local Emu e;
    memset(res, 0, sizeof *res);
    e.N = x->n_symbols;
    e.maxd = x->max_moves;
    e.ordered = (flags & TD_FLAG_ORDERED) != 0;
    if (e.N > TD_MAX_N || e.maxd < 1 || e.maxd > TD_MAX_DEPTH) { res->status = TD_ERR_ARG; return res->status; }
    e.T = td_triple_count(e.N);
    if (e.T == 0) { res->status = TD_NOT_FOUND; return 0; }
    e.steps = (e.T + 31) / 32;
    int t = 0;
    for (int i = 0; i < e.N - 2; ++i)
        for (int j = i + 1; j < e.N - 1; ++j)
            for (int k = j + 1; k < e.N; ++k) { e.tri_i[t] = i; e.tri_j[t] = j; e.tri_k[t] = k; ++t; }
    for (int idx = 0; idx < 4096; ++idx) e.lut[idx] = (uint8_t)td_class_of_index(idx);
    const int init = td_inst_init(*x), full = td_inst_full(*x);
    for (int D = 0; D <= TD_MAX_DEPTH + 1; ++D) {
        e.acc[D] = e.reach[D] = 0;
        for (int o = 0; o < 32; ++o) {
            if (td_accepts(e.N, init, x->min_rate, full, o, D)) e.acc[D] |= 1u << o;
            if (td_can_reach(e.N, init, x->min_rate, e.maxd, full, o, D)) e.reach[D] |= 1u << o;
        }
    }
    e.expansions = 0;
    e.L[0] = x->perm;
    e.off[0] = x->offset;
    if (!e.ordered)
        return search_rows(e, full && td_accepts(e.N, init, x->min_rate, 1, e.N, e.maxd) ? e.maxd : 0, res);
    int level = 0;
    int odd = prepare(e, e.L[0], e.off[0]);
    int found = evaluate(e, 0, odd);
    for (;;) {
        if (found >= 0) {
            const int tt = e.T - 1 - found;
            for (int d = 0; d < level; ++d) res->moves[d] = e.path[d];
            res->moves[level] = td_pack_move(e.tri_i[tt], e.tri_j[tt], e.tri_k[tt]);
            res->depth = level + 1;
            res->status = TD_FOUND;
            break;
        }
        int accepted;
        const int u = next_child(e, level, &accepted);
        if (u < 0) {
            if (level == 0) { res->status = TD_NOT_FOUND; break; }
            --level;
            continue;
        }
        const int tt = e.T - 1 - u;
        const int i = e.tri_i[tt], j = e.tri_j[tt], k = e.tri_k[tt];
        e.path[level] = td_pack_move(i, j, k);
        if (accepted) {
            for (int d = 0; d <= level; ++d) res->moves[d] = e.path[d];
            res->depth = level + 1;
            res->status = TD_FOUND;
            break;
        }
        int noff;
        td_apply_move(e.L[level], e.off[level], e.N, i, j, k, &e.L[level + 1], &noff);
        e.off[level + 1] = noff;
        ++level;
        odd = prepare(e, e.L[level], e.off[level]);
        found = evaluate(e, level, odd);
    }
    res->expansions = e.expansions;
    return res->status;
}

extern "C" int td_emu_prepare_pair(const uint8_t *beta, const uint8_t *omega, int N, int init,
                                   float min_rate, int max_moves, int full, td_instance *out) {
    return td_prepare_pair(beta, omega, N, init, min_rate, max_moves, full, out);
}

extern "C" void td_emu_apply_move(uint64_t L, int off, int N, int i, int j, int k, uint64_t *outL, int *outOff) {
    td_apply_move(L, off, N, i, j, k, outL, outOff);
}

// `count` independent searches on `threads` host threads, one instance per
// thread at a time (the CPU baseline of the free order).  flags as for
// td_emu_search.  Returns 0.
extern "C" int td_emu_search_batch(int count, const td_instance *x, unsigned flags, td_result *res, int threads) {
    std::atomic<int> next{0};
    auto work = [&] {
        for (int i = next.fetch_add(1); i < count; i = next.fetch_add(1)) td_emu_search(&x[i], flags, &res[i]);
    };
    std::vector<std::thread> pool;
    for (int t = 1; t < threads; ++t) pool.emplace_back(work);
    work();
    for (auto &t : pool) t.join();
    return 0;
}

// The engine's device replay of a witness (td_witness_ok, the rule of
// TD_FLAG_VERIFY), for the CPU tests.
extern "C" int td_emu_witness_ok(const td_instance *x, const td_result *r) { return td_witness_ok(*x, *r); }

// The inverse instance and the conversion of its witnesses (td_core.cuh:
// td_inverse_pinned, td_witness_from_inverse), which the batch engine's race
// of a search against the search of its inverse uses; for the CPU tests.
extern "C" void td_emu_inverse_instance(const td_instance *x, td_instance *out) {
    *out = *x;
    out->perm = td_inverse_pinned(x->perm, x->n_symbols);
    out->offset = 0;
}

extern "C" int td_emu_witness_from_inverse(const td_instance *x, const td_result *inv, td_result *out) {
    *out = *inv;
    return td_witness_from_inverse(x->perm, x->offset, x->n_symbols, inv->moves, inv->depth, out->moves);
}

extern "C" int td_emu_pinned_cycles(uint64_t L, int off, int N) {
    uint32_t fixed;
    return td_pinned_cycles(L, off, N, &fixed);
}

// Rebuilds the endgame table (td_endgame.cuh) for glued states of up to
// `symbols` symbols: out[td_eg_base(m) + rank] = 0 where the state's missing
// moves suffice, else the expansions of the reference-order walk that finds
// they do not; 0xffff where the state is not glued.  Returns the number of
// states that one spare move does not let sort either, which the engine takes
// to be 0.  Each state's +2 children miss one move less, so states are taken
// by their missing moves.
extern "C" long td_emu_endgame(int symbols, uint16_t *out, int threads) {
    const uint32_t total = td_eg_base(symbols);  // states of up to `symbols` symbols: m < symbols
    for (uint32_t g = 0; g < total; ++g) out[g] = 0xffff;
    std::atomic<long> bad{0};
    auto glued = [](uint64_t L, int N, uint32_t *kept) {
        uint32_t k = 0;
        for (int p = 0; p < N; ++p) {
            const int b = p ? (int)td_nib(L, p - 1) + 1 : 0, q = p ? p - 1 : N - 1;
            const int a = q ? (int)td_nib(L, q - 1) + 1 : 0;
            if (b != (a + 1) % N) k |= 1u << b;
        }
        *kept = k;
        return td_popc(k);
    };
    auto state = [](uint32_t g, int *N) {
        int m = 2;
        while (g >= td_eg_base(m + 1)) ++m;
        uint32_t r = g - td_eg_base(m), d[16], U = (1u << m) - 1u;
        for (int q = 1; q <= m; ++q) { d[q] = r % q; r /= q; }
        uint64_t L = 0;
        for (int q = m, at = 0; q >= 1; --q, ++at) {
            uint32_t v = U;
            while (d[q]--) v &= v - 1;
            const int x = __builtin_ctz(v);
            U &= ~(1u << x);
            L |= (uint64_t)x << (4 * at);
        }
        for (int at = m; at < 16; ++at) L |= (uint64_t)at << (4 * at);
        *N = m + 1;
        return L;
    };
    // sweep 0: entries of the states missing `M` moves; sweep 1: where no +2
    // child exists, a 0 child must be sorted by its missing moves
    auto pass = [&](int M, int sweep, int t) {
        static thread_local Emu e;
        for (uint32_t g = (uint32_t)t; g < total; g += (uint32_t)threads) {
            if (sweep == 1 && (out[g] == 0 || out[g] == 0xffff)) continue;
            int N;
            const uint64_t L = state(g, &N);
            uint32_t kept;
            if (glued(L, N, &kept) != N) continue;
            e.N = N;
            const int odd = prepare_rows(e, L, 0);
            if ((N - odd) / 2 != M) continue;
            uint32_t sum = 1;
            bool sorted = false, two = false, zero_sorted = false;
            for (int i = 0; i < N; ++i)
                for (int j = i + 1; j < N; ++j) {
                    uint32_t plus, zero;
                    td_row_classes(e.S[i], e.G[i], e.P[i], e.S[j], e.G[j], e.P[j], e.O, e.F, i, j, &plus, &zero);
                    for (int k = j + 1; k < N; ++k) {
                        if (!(((sweep ? plus | zero : plus) >> k) & 1u)) continue;
                        uint64_t nL;
                        int noff;
                        td_apply_move(L, 0, N, i, j, k, &nL, &noff);
                        const int n = glued(nL, N, &kept);
                        const uint32_t v = n ? out[td_eg_base(n - 1) + td_eg_rank(nL, kept)] : 0u;
                        if ((plus >> k) & 1u) { two = true; sum += v; sorted |= v == 0; }
                        else zero_sorted |= v == 0;
                    }
                }
            if (sweep == 0) out[g] = (uint16_t)(sorted ? 0 : sum);
            else if (!two && !zero_sorted) ++bad;
        }
    };
    for (int M = 1; M <= symbols / 2; ++M)
        for (int sweep = 0; sweep < 2; ++sweep) {
            std::vector<std::thread> pool;
            for (int t = 0; t < threads; ++t) pool.emplace_back(pass, M, sweep, t);
            for (auto &t : pool) t.join();
        }
    return bad.load();
}

// ---- reference-order walks with the endgame table and given-away children ------

namespace {

// One search of td_ordered.cuh with a warp always waiting, one unit after the
// other: the rules of td_eg_skip, td_split and td_split_complete.
struct SplitEmu {
    struct Child {
        uint16_t move;
        bool plus2, accepted;
    };
    struct Rec {  // one record of a split node, or an item still to be walked
        bool item, accepted;
        uint32_t exp;
        uint16_t move;
    };
    struct Node {
        int depth;
        uint64_t L;  // of the node whose children were given away
        int off;
        uint16_t path[TD_MAX_DEPTH];
        std::vector<Rec> recs;  // ranks 1, 2, ...
    };
    const uint16_t *table;
    int split_after, check_every, eg_moves;
    long splits = 0, kept = 0;  // nodes made, and levels that kept their children since the table decides them
    Emu e;

    int decide(uint64_t L, int off, int spare, const Child &c) const {
        if (spare < 0) return -1;
        uint64_t nL;
        int noff;
        td_apply_move(L, off, e.N, c.move & 31, (c.move >> 5) & 31, (c.move >> 10) & 31, &nL, &noff);
        return endgame_probe(table, e.N, nL, c.plus2 ? spare == 0 : spare == 1);
    }

    // A walk from (L, off) at depth d0, path[0 .. d0-1] before it; its own record
    // (status, expansions, moves), the nodes it was split into joined.
    td_result walk(uint64_t L0, int off0, int d0, const uint16_t *before, int after) {
        std::vector<Child> kids[TD_MAX_DEPTH];  // still to visit, the next one last
        int spare[TD_MAX_DEPTH];                // -1: the table drops no child
        uint64_t L[TD_MAX_DEPTH + 1];
        int off[TD_MAX_DEPTH + 1];
        uint16_t path[TD_MAX_DEPTH];
        for (int d = 0; d < d0; ++d) path[d] = before[d];
        std::vector<Node> nodes;
        td_result r;
        memset(&r, 0, sizeof r);
        uint64_t exp = 0;
        int level = d0, since = 0;
        bool due = false;
        L[d0] = L0;
        off[d0] = off0;
        auto record = [&](uint16_t last) {
            r.status = TD_FOUND;
            r.depth = level + 1;
            for (int d = 0; d < level; ++d) r.moves[d] = path[d];
            r.moves[level] = last;
        };
        for (bool done = false; !done;) {
            const int odd = prepare(e, L[level], off[level]);
            uint32_t fixed;
            td_pinned_cycles(L[level], off[level], e.N, &fixed);
            const int sp = eg_moves - level - ((e.N - odd) >> 1);
            spare[level] = eg_moves > level + 1 && sp >= 0 && sp < 2 && e.N - td_popc(fixed) <= TD_EG_SYMBOLS + 3 ? sp : -1;
            const int found = evaluate(e, level, odd);
            ++exp;
            auto move_of = [&](int u) {
                const int t = e.T - 1 - u;
                return td_pack_move(e.tri_i[t], e.tri_j[t], e.tri_k[t]);
            };
            if (found >= 0) {
                record(move_of(found));
                break;
            }
            kids[level].clear();
            for (;;) {
                Child c;
                int accepted;
                const int u = next_child(e, level, &accepted);
                if (u < 0) break;
                c.move = move_of(u);
                c.accepted = accepted != 0;
                uint64_t nL;
                int noff;
                uint32_t f;
                td_apply_move(L[level], off[level], e.N, c.move & 31, (c.move >> 5) & 31, (c.move >> 10) & 31, &nL, &noff);
                c.plus2 = td_pinned_cycles(nL, noff, e.N, &f) == odd + 2;
                kids[level].insert(kids[level].begin(), c);
            }
            if (due) {
                due = false;
                split(nodes, kids, spare, L, off, path, d0, level);
            }
            for (;;) {
                while (spare[level] >= 0 && !kids[level].empty()) {
                    const int v = decide(L[level], off[level], spare[level], kids[level].back());
                    if (v <= 0) break;
                    exp += (uint64_t)v;
                    kids[level].pop_back();
                }
                if (kids[level].empty()) {
                    if (level == d0) { done = true; break; }
                    --level;
                    continue;
                }
                const Child c = kids[level].back();
                kids[level].pop_back();
                if (c.accepted) {
                    record(c.move);
                    done = true;
                    break;
                }
                path[level] = c.move;
                td_apply_move(L[level], off[level], e.N, c.move & 31, (c.move >> 5) & 31, (c.move >> 10) & 31,
                              &L[level + 1], &off[level + 1]);
                break;
            }
            if (done) break;
            if (exp >= (uint64_t)after && ++since >= check_every) {
                since = 0;
                due = true;
            }
            ++level;
        }
        // the walk's record is rank 0 of its last node, whose join is rank 0 of the one before
        for (size_t k = nodes.size(); k-- > 0 && r.status != TD_FOUND;) {
            const Node &nd = nodes[k];
            for (const Rec &q : nd.recs) {
                if (!q.item) {
                    exp += q.exp;
                    continue;
                }
                uint16_t p[TD_MAX_DEPTH];
                for (int d = 0; d < nd.depth; ++d) p[d] = nd.path[d];
                p[nd.depth] = q.move;
                if (q.accepted) {
                    r.status = TD_FOUND;
                    r.depth = 1;
                    r.moves[0] = q.move;
                    break;
                }
                uint64_t nL;
                int noff;
                td_apply_move(nd.L, nd.off, e.N, q.move & 31, (q.move >> 5) & 31, (q.move >> 10) & 31, &nL, &noff);
                const td_result sub = walk(nL, noff, nd.depth + 1, p, split_after / 8);
                exp += sub.expansions;
                if (sub.status == TD_FOUND) {
                    r = sub;
                    break;
                }
            }
        }
        r.expansions = (uint32_t)exp;
        return r;
    }

    void split(std::vector<Node> &nodes, std::vector<Child> *kids, const int *spare, const uint64_t *L, const int *off,
               const uint16_t *path, int d0, int level) {
        int lv = d0;
        while (lv <= level && kids[lv].empty()) ++lv;
        if (lv > level) return;
        const int own = lv == level ? 1 : 0;
        Node nd;
        int units = 0, rank = 0;
        for (size_t q = kids[lv].size(); q-- > 0; ++rank) {
            const Child &c = kids[lv][q];
            const int v = c.accepted ? 0 : decide(L[lv], off[lv], spare[lv], c);
            if (rank >= own) {
                nd.recs.push_back(Rec{v <= 0, c.accepted, v > 0 ? (uint32_t)v : 0u, c.move});
                units += v <= 0;
            }
            if (v == 0) break;  // the walk gets no further
        }
        if (units == 0) {  // they count where the walk gets to them
            kept += !nd.recs.empty();
            return;
        }
        nd.depth = lv;
        nd.L = L[lv];
        nd.off = off[lv];
        for (int q = 0; q < lv; ++q) nd.path[q] = path[q];
        if (own) kids[lv].erase(kids[lv].begin(), kids[lv].end() - 1);
        else kids[lv].clear();
        nodes.push_back(nd);
        ++splits;
    }
};

}  // namespace

// A reference-order search whose walks are split as td_ordered_kernel splits
// them while warps wait: from `split_after` expansions on, every `check_every`
// of them.  `table`: td_emu_endgame's, for 11 symbols.  counts: the nodes made,
// and how often a level kept its children since the table decides them all.
extern "C" int td_emu_split_search(const td_instance *x, const uint16_t *table, int split_after, int check_every,
                                   td_result *res, long *counts) {
    static thread_local SplitEmu s;
    Emu &e = s.e;
    e.N = x->n_symbols;
    e.maxd = x->max_moves;
    e.ordered = 1;
    e.T = td_triple_count(e.N);
    e.steps = (e.T + 31) / 32;
    int t = 0;
    for (int i = 0; i < e.N - 2; ++i)
        for (int j = i + 1; j < e.N - 1; ++j)
            for (int k = j + 1; k < e.N; ++k) { e.tri_i[t] = i; e.tri_j[t] = j; e.tri_k[t] = k; ++t; }
    for (int idx = 0; idx < 4096; ++idx) e.lut[idx] = (uint8_t)td_class_of_index(idx);
    const int init = td_inst_init(*x), full = td_inst_full(*x);
    for (int D = 0; D <= TD_MAX_DEPTH + 1; ++D) {
        e.acc[D] = e.reach[D] = 0;
        for (int o = 0; o < 32; ++o) {
            if (td_accepts(e.N, init, x->min_rate, full, o, D)) e.acc[D] |= 1u << o;
            if (td_can_reach(e.N, init, x->min_rate, e.maxd, full, o, D)) e.reach[D] |= 1u << o;
        }
    }
    s.table = table;
    s.split_after = split_after;
    s.check_every = check_every;
    s.eg_moves = full && td_accepts(e.N, init, x->min_rate, 1, e.N, e.maxd) ? e.maxd : 0;
    s.splits = s.kept = 0;
    *res = s.walk(x->perm, x->offset, 0, nullptr, split_after);
    counts[0] = s.splits;
    counts[1] = s.kept;
    return res->status;
}

// The expansion counts, budgets and statuses of the kernels (td_core.cuh).
extern "C" uint32_t td_emu_add_count(uint32_t a, uint32_t b) { return td_add_count(a, b); }
extern "C" int td_emu_over_budget(uint32_t count, uint64_t max_expansions) {
    return td_over_budget(count, td_budget(max_expansions));
}
extern "C" int td_emu_status_of_dfs(int dfs) { return td_status_of_dfs(dfs); }

// The numbers of launches and requests (td_core.cuh).
extern "C" uint32_t td_emu_next_epoch(uint32_t last, uint32_t epochs, int *again) {
    return td_next_epoch(last, epochs, again);
}
extern "C" uint64_t td_emu_request_number(uint64_t claimed, uint32_t low) { return td_request_number(claimed, low); }
