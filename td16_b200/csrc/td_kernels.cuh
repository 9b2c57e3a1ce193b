// td_kernels.cuh -- the sm_100a witness-search warp engine.
//
// One warp owns one search (a DFS over move sequences), or one donated
// subtree of it.  The state of a level is the caller's array, one byte per
// position.  Per node the warp labels the omega cycles by pointer jumping
// (lane c = caller position c) and builds cycle row masks, and each lane then
// classifies the children (i, j, k) of its pair slots for every k at once with
// LOP3 logic (td_prepare_rows, td_row_classes).  The two move orders differ in
// how the children are kept and picked:
//
// Reference order (td_evaluate, td_next_child): one bit per child at its
// position u in the reference's single-queue order, 22 words of 32 per level.
// The next child comes from one ballot over the words.
//
// Free order (td_evaluate_rows, td_next_child_rows): each lane keeps the
// children of its pair slots.  The next child, +2 moves first, comes from
// per-level lane summaries.  A table of explored states skips children reached
// before by another move order, and busy warps donate subtrees to idle ones.
//
// Reference: emitter/src/native/backtracking/sorting_search.cu:478-712.
#pragma once

#include "td_core.cuh"

#define TD_FULL 0xffffffffu
#define TD_TRI_TABLE 3060      // sum over N <= 17 of C(N,3) = C(18,4)

// Limits and tables of the search a warp runs.
struct td_search_limits {
    uint64_t max_expansions;   // per search; TD_ERR_BUDGET when reached (td_budget)
    uint32_t split_after;      // a walk of the reference order may be split after this many expansions
    uint64_t deadline_ns;      // %globaltimer value; 0 = none
    ulonglong2 *tt;            // the launch's table of explored states (free order); null = none
    uint64_t tt_id;            // number of the launch's first search in it
    int tt_shift;              // 64 - log2 of its entries
    uint32_t restart_base;     // free order: base of the restart budgets (td_attempt_budget); 0 = none
    // a subtree of a split ordered search: it stops once *cutoff < rank, or
    // *cutoff2 < rank2 (the lowest rank with a witness so far, at its node and at
    // that node's); null = none
    const int *cutoff, *cutoff2;
    int rank, rank2;
};

// ---- work items (subtree roots handed between warps) ----------------------

// A node that is known to be expandable, with the moves that lead to it.
struct __align__(16) td_item {  // 32 bytes
    uint64_t L;
    uint32_t inst;          // instance index
    uint8_t depth;          // bits 0-3: DFS depth of the node (0 only for the root of an inverse
                            // instance); bit 7: the node belongs to the inverse instance's search;
                            // bits 4-6: low bits of the restart attempt that donated it
    uint8_t off;            // bits 0-4; bits 5-7: high bits of that attempt
    uint16_t path[TD_MAX_DEPTH];
};

// Per-instance bookkeeping when several warps share one search.  A search that
// never gives anything away does not use it.
struct __align__(16) td_inst_state {
    // units (the root search + items) not yet finished: the low 32 bits count
    // the search of the instance, the high 32 bits that of its inverse
    unsigned long long pending;
    unsigned short found;   // 1: a warp recorded the witness; 2: one side of a race was searched
                            // to the end without one (the verdict is known, the other side stops)
    short error;            // first error status seen (timeout)
    unsigned expansions;    // summed over units
};
#define TD_UNIT_INVERSE (1ull << 32)

// Scheduler counters of one launch.
struct td_pool {
    // items reserved by donors, and item tickets taken (the batch engine) or
    // items claimed (the serving loop); read together
    alignas(8) int produced;
    int consumed;
    int inst_ticket;        // next fresh instance
    int outstanding;        // the batch engine: units in progress plus items not yet finished
    int active;             // the serving loop: warps inside a unit or claiming one
    int idle;               // the serving loop: warps waiting for donated work
    int error;              // launch-level error (bounded wait expired)
    int done;               // the batch engine: nothing outstanding, and no instance left
    unsigned long long donations;
    unsigned long long donated_items;
    unsigned long long races;  // inverse roots queued
};

// Donated items live either in a per-launch array (batch launches: index i
// at slot i, ready[i] == epoch once written, ~epoch once the launch has no work
// left for the warp that waits for it) or in a ring (the serving launch:
// index i at slot i % capacity, ready == td_ring_tag(i) once written and
// td_ring_tag(i) | 0x80000000 once its taker has read it, which frees the slot).
__device__ __forceinline__ uint32_t td_ring_tag(long long i) { return (uint32_t)((i + 1) & 0x7fffffff); }

struct td_donate_ctx {
    int ring;
    int tickets;            // takers hold item tickets (the batch engine), see td_steal_kernel
    uint64_t deadline_ns;   // bounds the wait for a ring slot to be freed
    td_pool *pool;
    td_item *items;
    uint32_t *ready;
    uint32_t epoch;
    int capacity;
    int step;               // td_serve_idle_warps: 3 in the batch engine, 2 in the serving loop
    int idle_after;         // a unit calls it at the first idle warps after this many expansions
    int idle_seen;          // it was called for the three settings below
    int grain;              // at most this many items per donation
    int max_level;          // donate only children of levels <= max_level
    int check_every;        // expansions between idle checks
    uint32_t inst;
    td_inst_state *state;
    int side;               // 1: the unit searches the instance's inverse (items carry it on)
    int attempt;            // the restart attempt that donated the unit (0 for a root)
    int gave;               // 0: a root search that has given nothing away (no other warp knows of it)
    int race;               // > 0: the unit queues its inverse when it starts restart attempt
                            // `race` (root units of full-sorting instances in td_steal_kernel),
                            // and 0 once it has
};

// The buffers of a launch of the reference order whose walks may be split
// (td_ordered.cuh).
struct td_split_node;
struct td_split_item;
struct td_split_space {
    td_split_node *nodes;
    int *node_count, *record_count;
    int max_nodes;
    td_split_item *items;  // by item ticket
    td_result *records;    // by node base + rank
    td_result *out;        // by instance
};

// Per-warp shared state.
struct td_warp_smem {
    // per caller position c: the row masks S, G, P and H (positions after c),
    // and the odd-cycle / fixed-point flags as full masks
    uint4 rows[TD_MAX_N];
    uint2 flg[TD_MAX_N];
    // per lane: its four pair slots (td_load_pairs), i | j << 5 each, and the
    // first child number of their run
    ushort4 pair[32];
    uint16_t u0[32];
    union {
        struct {  // reference move order
            // per level: bit u % 32 of word u / 32 is child u still to visit
            uint32_t cw[TD_MAX_DEPTH][TD_MAX_STEPS];
            uint32_t root_found[TD_MAX_STEPS];  // the root's children accepted when visited
            uint32_t cp[TD_MAX_DEPTH][TD_MAX_STEPS];  // the +2 ones, at nodes that also have 0 children
            // a node being split: its children in visiting order (bit 15:
            // accepted when visited), and what the endgame table says of each
            uint16_t kid[TD_MAX_TRIPLES], kid_e[TD_MAX_TRIPLES];
            td_split_space sp;
            int sp_inst, sp_node, sp_rank;  // where the walk's result goes (node -1: to the instance's)
        };
        struct {  // free move order
            // per level and lane: the expandable children of the lane's four
            // pair slots (word r = slot R*lane + r), +2 class at bits k-1
            // (1..15), 0 class at bits k+15 (17..31)
            uint4 pw[TD_MAX_DEPTH][32];
            uint32_t m2[TD_MAX_DEPTH];                 // per level: lanes that hold +2 children
            uint32_t m0[TD_MAX_DEPTH];                 // per level: lanes that hold 0 children
        };
    };
    uint64_t L[TD_MAX_DEPTH + 1];              // pinned state where a search or subtree starts
    uint32_t acc[TD_MAX_DEPTH + 2];            // accept mask over odd counts, per depth
    uint32_t reach[TD_MAX_DEPTH + 2];          // prune mask over odd counts, per depth
    uint16_t path[TD_MAX_DEPTH];               // caller-position move per level
    uint8_t off[TD_MAX_DEPTH + 1];
    uint8_t A[TD_MAX_DEPTH + 1][32];           // per level: the caller's array, one pinned label per position
    uint8_t inv[32];                           // caller position of each label
    // per level: the moves its node can spare, where the endgame table may
    // decide its children; else 255
    uint8_t spare[TD_MAX_DEPTH];
    uint16_t list[32];                         // children looked up in the endgame table
    int pairs_n;                               // the N the pair slots are loaded for
    int eg_moves;                              // the bound where the endgame table applies, else 0
    // shared memory holds what a warp's search reads rarely, so that registers
    // are left for the evaluation
    td_search_limits lim;
    td_donate_ctx dc;
};

// What a warp's donation settings become once it has met idle warps, in the
// batch engine (step 3): it looks for them 16 times as often, gives them 8
// times as many items at once and from 4 levels deeper.  An item per lane and
// counters read behind an expansion make a donation cheap, and the end of a
// launch is all latency: with the settings that suit the time before (4 items,
// level 2, every 64 expansions) 2,048 S_16 at their lower bound took 20 ms,
// with these 2.8 ms; the n = 11..13 mix 10.3 and 1.6 ms, 250 requests of n =
// 8..16 2.8 and 0.23 ms.  The serving loop's warps claim by compare-and-swap,
// so there it is 4 times as often and as many, from 2 levels deeper (step 2).
// Called by one lane.
__device__ __forceinline__ void td_serve_idle_warps(td_donate_ctx &dc) {
    if (dc.idle_seen) return;
    dc.idle_seen = 1;
    dc.grain = min(32, dc.grain << dc.step);
    dc.max_level = min(TD_MAX_DEPTH - 1, dc.max_level + 2 * (dc.step - 1));
    dc.check_every = max(1, dc.check_every >> (2 * (dc.step - 1)));
}

// Lexicographic position triples i|j<<5|k<<10 for every N, at offset C(N,4).
__device__ uint16_t td_tri_table[TD_TRI_TABLE];

TD_HD int td_tri_base(int N) {
    return N < 4 ? 0 : N * (N - 1) * (N - 2) * (N - 3) / 24;
}

// Accept / prune masks of one instance: lane D computes the masks of depth D
// over all odd counts.  With full sorting the accept test only passes at
// odd == N and its f32 rate part depends on D alone, and the prune bound
// D + ceil((N - odd)/2) <= maxDepth is a threshold on odd, so both masks take
// one f32 division per lane.  Partial sorting evaluates every odd count.
__device__ __forceinline__ void td_rate_masks(td_warp_smem &s, const td_instance &x) {
    const int D = threadIdx.x & 31;
    const int N = x.n_symbols, init = td_inst_init(x), full = td_inst_full(x);
    const int maxd = x.max_moves;
    uint32_t a = 0, r = 0;
    if (D <= TD_MAX_DEPTH + 1) {
        if (full) {
            if (td_accepts(N, init, x.min_rate, 1, N, D)) a = 1u << N;
            if (D < maxd) {
                // D + (N - odd + 1) / 2 <= maxd  <=>  odd >= N - 2 * (maxd - D)
                const int lo = N - 2 * (maxd - D);
                r = lo <= 0 ? 0xffffffffu : (0xffffffffu << lo);
            }
        } else {
            for (int o = 0; o < 32; ++o) {
                if (td_accepts(N, init, x.min_rate, 0, o, D)) a |= 1u << o;
                if (D < maxd && td_can_reach(N, init, x.min_rate, maxd, 0, o, D)) r |= 1u << o;
            }
        }
        s.acc[D] = a;
        s.reach[D] = r;
        // the endgame table knows full sorting; it needs every depth up to the
        // bound accepted (the rate falls with the depth)
        if (D == maxd) s.eg_moves = full && a ? maxd : 0;
    }
    __syncwarp();
}

// Orders this thread's earlier accesses before its later ones for the device
// (release and acquire; cheaper than __threadfence, which is sequentially
// consistent).
__device__ __forceinline__ void td_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ uint64_t td_globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---- node evaluation, bit-sliced ---------------------------------------------
//
// The state of a level is the caller's array, one byte per caller position
// holding the pinned label (A[c] = B[(c + off) mod N]).  In these terms omega
// maps A[c] to A[c-1] + 1 (mod N), and a move (i, j, k) is the plain block swap
// A[:i] + A[j:k] + A[i:j] + A[k:] (the pinned form's start-of-array rule is the
// rotation that keeps label 0 first).  Lane l owns pair slots 4 l + r
// (td_pair_code) and classifies the children (i, j, k) of every k at once
// from the node's row masks (td_row_classes).

// Rounds of the bit-sliced evaluation for N: ceil(C(N-1,2) / 32).
TD_HD int td_pair_rounds(int N) {
    const int NP = N < 3 ? 0 : (N - 1) * (N - 2) / 2;
    return (NP + 31) >> 5;
}

// Every lane's pair slots for every N, i | j << 5 each, and the first child
// number of their run (td_pair_row).
struct td_pair_row {
    uint16_t pair[TD_MAX_ROUNDS];
    uint16_t u0;
};
__device__ td_pair_row td_pair_table[TD_MAX_N + 1][32];

// Lane l owns slots R l + r, r < R = td_pair_rounds(N) (the others are empty:
// j = N-1).  Child (i, j, k) is number u = C(N-1-i, 3) + C(N-1-j, 2) + (N-1-k)
// in the reference's reversed triple order (T-1-t, sorting_search.cu:588-590),
// so the children of a lane's slots r = 0, 1, ... are one run of consecutive u.
inline td_pair_row td_make_pair_row(int N, int lane) {
    td_pair_row w;
    const int R = td_pair_rounds(N);
    for (int r = 0; r < TD_MAX_ROUNDS; ++r) w.pair[r] = (uint16_t)(td_pair_code(N, r < R ? R * lane + r : -1) & 1023u);
    const int a = N - 1 - (w.pair[0] & 31), b = N - 1 - (w.pair[0] >> 5);
    w.u0 = (uint16_t)(a * (a - 1) * (a - 2) / 6 + b * (b - 1) / 2);
    return w;
}

__device__ __forceinline__ void td_load_pairs(td_warp_smem &s, int N) {
    const int lane = threadIdx.x & 31;
    const td_pair_row &w = td_pair_table[N][lane];
    s.pair[lane] = make_ushort4(w.pair[0], w.pair[1], w.pair[2], w.pair[3]);
    s.u0[lane] = w.u0;
    __syncwarp();
}

// Pinned state (L, off) -> the caller's array of `level`.
__device__ __forceinline__ void td_unpack_state(td_warp_smem &s, int level, uint64_t L, int off, int N) {
    const int c = threadIdx.x & 31;
    if (c < N) {
        int p = c + off;
        p -= p >= N ? N : 0;
        s.A[level][c] = (uint8_t)(p ? td_nib(L, p - 1) + 1u : 0u);
    }
    __syncwarp();
}

// The caller's array of `level` -> pinned state (L, off): label 0 sits at
// caller position c0, so off = -c0 mod N and L[m] = A[(m + 1 + c0) mod N] - 1.
__device__ __forceinline__ void td_pack_state(const td_warp_smem &s, int level, int N, uint64_t *L, int *off) {
    const int m = threadIdx.x & 31;
    const uint32_t z = __ballot_sync(TD_FULL, m < N && s.A[level][m] == 0);
    const int c0 = __ffs(z) - 1;
    uint32_t lo = 0, hi = 0;
    if (m < 16) {
        uint32_t v = (uint32_t)m;
        if (m < N - 1) {
            int q = m + 1 + c0;
            q -= q >= N ? N : 0;
            v = s.A[level][q] - 1u;
        }
        const uint64_t w = (uint64_t)v << (4 * m);
        lo = (uint32_t)w;
        hi = (uint32_t)(w >> 32);
    }
    lo = __reduce_or_sync(TD_FULL, lo);
    hi = __reduce_or_sync(TD_FULL, hi);
    *L = ((uint64_t)hi << 32) | lo;
    *off = c0 == 0 ? 0 : N - c0;
}

// The caller's array of level+1 = that of `level` after the move t.
__device__ __forceinline__ void td_apply_bytes(td_warp_smem &s, int level, uint32_t t, int N) {
    const int m = threadIdx.x & 31;
    const int i = t & 31, j = (t >> 5) & 31, k = (t >> 10) & 31;
    if (m < N) {
        int src = m;
        if (m >= i && m < k) src = m < i + (k - j) ? m + (j - i) : m - (k - j);
        s.A[level + 1][m] = s.A[level][src];
    }
    __syncwarp();
}

// Row masks of the node at `level` (lane c = caller position c); returns the
// number of odd-length omega cycles and the odd-cycle and fixed-point masks.
__device__ __forceinline__ int td_prepare_rows(td_warp_smem &s, int level, int N, uint32_t &O, uint32_t &F) {
    const int c = threadIdx.x & 31;
    const bool act = c < N;
    const int a = act ? s.A[level][c] : 0;
    const int am1 = __shfl_sync(TD_FULL, a, c == 0 ? N - 1 : c - 1);
    if (act) s.inv[a] = (uint8_t)c;
    __syncwarp();
    // next caller position along omega: the one holding A[c-1] + 1 (mod N)
    const int y = am1 + 1 == N ? 0 : am1 + 1;
    const int nx = act ? (int)s.inv[y] : c;
    // leader (smallest caller position on the cycle) and dist (omega steps to
    // it) in one pointer-jumping pass: each lane keeps the minimum of the
    // window c, next(c), ..., next^(w-1)(c) and its distance; windows double
    // per round and 32 >= any cycle length, so the first occurrence wins.
    int m = c, d = 0, j = nx;
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        const int mB = __shfl_sync(TD_FULL, m, j);
        const int dB = __shfl_sync(TD_FULL, d, j);
        const int jB = __shfl_sync(TD_FULL, j, j);
        if (mB < m) {
            m = mB;
            d = (1 << r) + dB;
        }
        j = jB;
    }
    const int after_leader = __shfl_sync(TD_FULL, nx, m);
    const int len = __shfl_sync(TD_FULL, d, after_leader) + 1;
    const uint32_t ACT = (1u << N) - 1u;
    const uint32_t S = __match_any_sync(TD_FULL, m) & ACT;  // inactive lanes are their own leaders
    // lt bit q: dist(q) < dist(c), by comparing the five bit planes of dist
    uint32_t lt = 0, eq = TD_FULL, D0 = 0;
#pragma unroll
    for (int b = 4; b >= 0; --b) {
        const uint32_t Bb = __ballot_sync(TD_FULL, (d >> b) & 1);
        const uint32_t mb = 0u - (uint32_t)((d >> b) & 1);
        lt |= eq & ~Bb & mb;
        eq &= ~(Bb ^ mb);
        if (b == 0) D0 = Bb;
    }
    const uint32_t lodd = 0u - (uint32_t)(len & 1);
    const uint32_t G = S & lt;
    // walk c -> q: dist(c) - dist(q), plus the cycle length when q is further
    const uint32_t P = S & ((D0 ^ (0u - (uint32_t)(d & 1))) ^ (lodd & ~lt));
    O = __ballot_sync(TD_FULL, act && (len & 1));
    F = __ballot_sync(TD_FULL, act && len == 1);
    const int odd = __popc(__ballot_sync(TD_FULL, act && m == c && (len & 1)));
    if (act) {
        s.rows[c] = make_uint4(S, G, P, ACT & (0xfffffffeu << c));
        s.flg[c] = make_uint2(lodd, len == 1 ? 0xffffffffu : 0u);
    }
    __syncwarp();
    return odd;
}

// Classifies every child of the node at `level`; fills the level's outcome
// words and lane summaries and returns a found move (i | j<<5 | k<<10) or -1.
__device__ __forceinline__ int td_evaluate_rows(td_warp_smem &s, int N,
                                                int level, int odd, uint32_t O, uint32_t F) {
    const int lane = threadIdx.x & 31;
    const int D = level + 1;
    const uint32_t accD = s.acc[D], reachD = s.reach[D];
    const uint32_t f0 = 0u - ((accD >> odd) & 1u), f2 = 0u - ((accD >> (odd + 2)) & 1u);
    const uint32_t x0 = (0u - ((reachD >> odd) & 1u)) & ~f0;
    const uint32_t x2 = (0u - ((reachD >> (odd + 2)) & 1u)) & ~f2;
    const bool accepting = (f0 | f2) != 0;  // warp-uniform
    const int R = td_pair_rounds(N);  // warp-uniform
    const ushort4 pq = s.pair[lane];
    const uint32_t code[TD_MAX_ROUNDS] = {pq.x, pq.y, pq.z, pq.w};
    uint32_t key = 0xffffffffu;
    uint32_t W[TD_MAX_ROUNDS] = {0u, 0u, 0u, 0u};
    // A node without a spare move only has +2 children, and nearly always odd
    // cycles only (99% of such nodes on near-reverse S_16, and 80% to 100% of
    // all nodes have no spare move): a third of the work, see td_row_plus2_odd.
    // 2^19 near-reverse S_16 at bound 9: 26.8 -> 23.7 ms.
    if (!(x0 | f0) && O == (1u << N) - 1u) {
#pragma unroll
        for (int r = 0; r < TD_MAX_ROUNDS; ++r) {
            if (r >= R) break;
            const uint32_t pc = code[r];
            const int sh = 31 - (int)(pc >> 5);  // brings bit j to the sign bit
            const uint4 ri = s.rows[pc & 31], rj = s.rows[pc >> 5];
            const uint32_t plus =
                rj.w & (uint32_t)((int32_t)(ri.x << sh) >> 31) &
                td_row_plus2_odd(ri.x, ri.y, ri.z, rj.y, rj.z, (uint32_t)((int32_t)(ri.y << sh) >> 31),
                                 (uint32_t)((int32_t)(ri.z << sh) >> 31));
            W[r] = (plus & x2) >> 1;
            if (accepting && plus && key == 0xffffffffu)  // then every +2 child is accepted
                key = ((uint32_t)lane << 17) | ((uint32_t)r << 15) | pc | ((uint32_t)(31 - __clz(plus)) << 10);
        }
    } else {
#pragma unroll
        for (int r = 0; r < TD_MAX_ROUNDS; ++r) {
            if (r >= R) break;
            const uint32_t pc = code[r];
            const int i = pc & 31, j = pc >> 5;
            const uint4 ri = s.rows[i], rj = s.rows[j];
            const uint2 fi = s.flg[i], fj = s.flg[j];
            uint32_t plus, zero;
            td_row_classes_x(ri.x, ri.y, ri.z, rj.x, rj.y, rj.z, O, F, fi.x, fj.x, fi.y, fj.y, 31 - j, &plus,
                             &zero);
            const uint32_t km = rj.w;  // k > j (empty slots: j's row with an empty mask is never read)
            // +2 children at bits k-1, 0 children at bits k+15; the fields do not
            // overlap, so the high-half multiply and the add keep this off the ALU pipe
            W[r] = __umulhi(km & x2 & plus, 0x80000000u) + (km & x0 & zero) * 32768u;
            if (accepting) {
                const uint32_t fnd = km & ((f0 & zero) | (f2 & plus));
                if (fnd && key == 0xffffffffu)
                    key = ((uint32_t)lane << 17) | ((uint32_t)r << 15) | pc |
                          ((uint32_t)(31 - __clz(fnd)) << 10);
            }
        }
    }
    s.pw[level][lane] = make_uint4(W[0], W[1], W[2], W[3]);
    const uint32_t any = W[0] | W[1] | W[2] | W[3];
    const uint32_t m2 = __ballot_sync(TD_FULL, (any & 0x0000ffffu) != 0);
    const uint32_t m0 = __ballot_sync(TD_FULL, (any & 0xffff0000u) != 0);
    if (lane == 0) {
        s.m2[level] = m2;
        s.m0[level] = m0;
    }
    if (accepting) {
        key = __reduce_min_sync(TD_FULL, key);
        if (key != 0xffffffffu) {
            __syncwarp();
            return (int)(key & 0x7fffu);
        }
    }
    __syncwarp();
    return -1;
}

// Next child of `level` in the free order: +2 children first; among them, in
// the plain order (ord = 0), the highest pair slot (the lexicographically
// smallest pair) and its smallest k.  `ord` (td_order_variant) rotates the
// lane priority, reverses the round order and takes the largest k first.
// Returns the move, with bit 15 set for a 0 child, or -1.
__device__ __forceinline__ int td_next_child_rows(td_warp_smem &s, int level, uint32_t ord) {
    const int lane = threadIdx.x & 31;
    const uint32_t m2 = s.m2[level], m0 = s.m0[level];
    if ((m2 | m0) == 0) return -1;
    const bool c2 = m2 != 0;
    const uint32_t lanes = c2 ? m2 : m0;
    const uint32_t rot = ord & 31u;
    // the lane with the largest (lane - rot) mod 32
    const int win = (int)(((31u - (uint32_t)__clz(__funnelshift_r(lanes, lanes, rot))) + rot) & 31u);
    const uint4 Wv = s.pw[level][win];
    const uint32_t cm = c2 ? 0x0000ffffu : 0xffff0000u;
    int r;
    uint32_t w;
    if (ord & 32u) {
        if (Wv.x & cm) { r = 0; w = Wv.x; }
        else if (Wv.y & cm) { r = 1; w = Wv.y; }
        else if (Wv.z & cm) { r = 2; w = Wv.z; }
        else { r = 3; w = Wv.w; }
    } else {
        if (Wv.w & cm) { r = 3; w = Wv.w; }
        else if (Wv.z & cm) { r = 2; w = Wv.z; }
        else if (Wv.y & cm) { r = 1; w = Wv.y; }
        else { r = 0; w = Wv.x; }
    }
    const int b = (ord & 64u) ? 31 - __clz(w & cm) : __ffs(w & cm) - 1;
    const uint32_t nw = w & ~(1u << b);
    const uint32_t pc = reinterpret_cast<const uint16_t *>(&s.pair[win])[r];
    // does the winning lane keep children of this class?
    const uint32_t rest = (r == 0 ? nw : Wv.x) | (r == 1 ? nw : Wv.y) | (r == 2 ? nw : Wv.z) | (r == 3 ? nw : Wv.w);
    if (lane == 0) {
        reinterpret_cast<uint32_t *>(&s.pw[level][win])[r] = nw;
        if (!(rest & cm)) {
            if (c2) s.m2[level] = m2 & ~(1u << win);
            else s.m0[level] = m0 & ~(1u << win);
        }
    }
    __syncwarp();
    const int k = c2 ? b + 1 : b - 15;
    return (int)(pc | ((uint32_t)k << 10) | (c2 ? 0u : 0x8000u));
}

// Free order, the node of `level` just expanded (s.inv is its inverse): takes
// its move that fixes two symbols or three, a +2 child, and returns it, or -1
// where there is none or it is not among the level's children.  Positions x, y,
// z one step of omega apart give that move where their cyclic order is a
// move's; of several, the one of lowest x.  Fewer symbols are left after it, so
// the endgame table is nearer: 2^19 near-reverse S_16 take 41 expansions each
// with it and took 47 without (21.6 -> 19.0 ms), 2^16 mixed ones 11.0 and 12.6
// (1.32 -> 1.21 ms); uniform S_16, which are short, lose what they win (3.50 and
// 3.53 ms).  Only a root search's first attempt uses it: later attempts live on
// other orders (with it in every second one 19.7 ms), and a subtree given away
// is mostly searched to its end.  Where the table does not apply (partial
// sorting, a rate that the bound does not meet) there is nothing to win: the
// batch engine's partial sorting takes the same time with and without it, and
// td_plain_kernel's, whose one attempt is the whole search, 1.71 ms without and
// 1.86 with it (3,001 of n = 8..12).  Called: inlined, it made every search slower.
__device__ __noinline__ int td_take_fixing(td_warp_smem &s, int level, int N) {
    const int x = threadIdx.x & 31;
    int y = x;
    if (x < N) {
        const int p = s.A[level][x == 0 ? N - 1 : x - 1];
        y = s.inv[p + 1 == N ? 0 : p + 1];
    }
    const int z = __shfl_sync(TD_FULL, y, y);
    const uint32_t good = __ballot_sync(TD_FULL, (x < y) + (y < z) + (z < x) == 2);
    if (!good) return -1;
    const int p = __ffs(good) - 1;
    const int q = __shfl_sync(TD_FULL, y, p), u = __shfl_sync(TD_FULL, z, p);
    const int t = p < q ? q < u ? p | q << 5 | u << 10 : u | p << 5 | q << 10 : q | u << 5 | p << 10;
    const ushort4 pq = s.pair[x];
    const uint32_t code = t & 1023, bit = 1u << ((t >> 10) - 1);
    uint4 W = s.pw[level][x];
    bool mine = false;
    if (pq.x == code && (W.x & bit)) { W.x &= ~bit; mine = true; }
    if (pq.y == code && (W.y & bit)) { W.y &= ~bit; mine = true; }
    if (pq.z == code && (W.z & bit)) { W.z &= ~bit; mine = true; }
    if (pq.w == code && (W.w & bit)) { W.w &= ~bit; mine = true; }
    if (mine) {
        s.pw[level][x] = W;
        if (!((W.x | W.y | W.z | W.w) & 0xffffu)) s.m2[level] &= ~(1u << x);
    }
    __syncwarp();
    return __any_sync(TD_FULL, mine) ? t : -1;
}

// Reference order: classifies every child of the node at `level`; fills the
// level's child words and returns the found child's u, or -1.  A node's found
// child is the one of lowest u (the lowest lane of the first 32-chunk,
// sorting_search.cu:585-641); the root's children are accepted when visited.
// Integer issue bounds it.  A lane's pair slots hold one run of consecutive u,
// so at most three shared-memory ORs per lane put 680 children in order.  The
// earlier form read three pair-table entries and a class-table byte per triple
// (22 steps per lane): 16,384 S_12 instances at bound 6 took 12.2 ms, and take
// 7.6 ms with this one.
__device__ __forceinline__ int td_evaluate(td_warp_smem &s, int N, int level, int odd,
                                           uint32_t O, uint32_t F) {
    const int lane = threadIdx.x & 31;
    const int D = level + 1;
    const uint32_t accD = s.acc[D], reachD = s.reach[D];
    const uint32_t f0 = 0u - ((accD >> odd) & 1u), f2 = 0u - ((accD >> (odd + 2)) & 1u);
    const uint32_t x0 = (0u - ((reachD >> odd) & 1u)) & ~f0;
    const uint32_t x2 = (0u - ((reachD >> (odd + 2)) & 1u)) & ~f2;
    const bool accepting = (f0 | f2) != 0;  // warp-uniform
    const int R = td_pair_rounds(N);  // warp-uniform
    const ushort4 pq = s.pair[lane];
    const uint32_t code[TD_MAX_ROUNDS] = {pq.x, pq.y, pq.z, pq.w};
    if (lane < TD_MAX_STEPS) {
        s.cw[level][lane] = 0;
        s.cp[level][lane] = 0;
        if (level == 0) s.root_found[lane] = 0;
    }
    __syncwarp();
    // the lane's children and found children, in order of u from u0
    uint64_t ch = 0, fd = 0, pl = 0;
    int at = 0;
#pragma unroll
    for (int r = 0; r < TD_MAX_ROUNDS; ++r) {
        if (r >= R) break;
        const uint32_t pc = code[r];
        const int i = pc & 31, j = pc >> 5;
        const uint4 ri = s.rows[i], rj = s.rows[j];
        const uint2 fi = s.flg[i], fj = s.flg[j];
        uint32_t plus, zero;
        td_row_classes_x(ri.x, ri.y, ri.z, rj.x, rj.y, rj.z, O, F, fi.x, fj.x, fi.y, fj.y, 31 - j, &plus,
                         &zero);
        const uint32_t km = rj.w;  // k > j
        // k = N-1 comes first: reverse the bits
        ch |= (uint64_t)(__brev(km & ((x2 & plus) | (x0 & zero))) >> (32 - N)) << at;
        if (accepting) fd |= (uint64_t)(__brev(km & ((f2 & plus) | (f0 & zero))) >> (32 - N)) << at;
        if (x0) pl |= (uint64_t)(__brev(km & plus) >> (32 - N)) << at;
        at += N - 1 - j;
    }
    const int u0 = s.u0[lane], w = u0 >> 5, sh = u0 & 31;
    if (level == 0) ch |= fd;
    // ORs the lane's run into the 22 words of an array
    auto put = [&](uint32_t *words, uint64_t run) {
        const uint64_t lo = run << sh;
        const uint32_t hi = sh ? (uint32_t)(run >> (64 - sh)) : 0u;
        if ((uint32_t)lo) atomicOr(&words[w], (uint32_t)lo);
        if (lo >> 32) atomicOr(&words[w + 1], (uint32_t)(lo >> 32));
        if (hi) atomicOr(&words[w + 2], hi);
    };
    if (ch) put(s.cw[level], ch);
    if (x0 && pl) put(s.cp[level], pl);
    if (accepting) {
        if (level == 0) {
            if (fd) put(s.root_found, fd);
        } else {
            const uint32_t key = __reduce_min_sync(TD_FULL, fd ? (uint32_t)(u0 + __ffsll((long long)fd) - 1) : ~0u);
            if (key != ~0u) {
                __syncwarp();
                return (int)key;
            }
        }
    }
    __syncwarp();
    return -1;
}

// Reference order: takes the next child of `level`; returns u or -1.  Chunks
// of 32 are visited from the last one, lanes of a chunk in ascending order (the
// owner's LIFO pop, sorting_search.cu:165-174, 677-686), and the root's
// children in descending order of u.  *accepted is set for a root's child
// that is accepted when visited.
__device__ __forceinline__ int td_next_child(td_warp_smem &s, int level, int *accepted) {
    const int lane = threadIdx.x & 31;
    uint32_t w = lane < TD_MAX_STEPS ? s.cw[level][lane] : 0u;
    const uint32_t some = __ballot_sync(TD_FULL, w != 0);
    *accepted = 0;
    if (!some) return -1;
    const int st = 31 - __clz(some);
    w = __shfl_sync(TD_FULL, w, st);
    const int b = level == 0 ? 31 - __clz(w) : __ffs(w) - 1;
    if (level == 0) *accepted = (int)((s.root_found[st] >> b) & 1u);
    if (lane == 0) s.cw[level][st] = w & ~(1u << b);
    __syncwarp();
    return 32 * st + b;
}

// ---- table of explored states (free order) --------------------------------
//
// Different move orders reach the same state: on near-reverse S_16 about 80%
// of the free-order expansions re-expand a state already expanded at the same
// or a smaller depth.  Whether a node's subtree holds a witness depends only
// on its pinned state L (not on where the caller's array starts: a move is the
// same cycle rotation from any start, so the reachable states do not depend
// on it) and on its depth.  The warps of a launch share one direct-mapped
// table of the states they took up, and a child whose state is in the table
// for the same search at a depth <= the child's is skipped.  This is sound
// also where the entry is another warp's, whose subtree is still being
// searched: whoever records a state takes up each of its children, finds it
// recorded for the same search with at least as much budget, leaves it to the
// endgame table or donates it (the taker then records it or finds it
// recorded).  So, by induction on the length of a state's shortest witness,
// some warp meets the witness of every recorded state; and a search only ends
// without one when every unit of it has ended.
//
// An entry is one 16-byte word, read and written whole (128-bit relaxed
// accesses), so it always names one state exactly:
//   word 0: the state's key (td_tt_key, 57 bits), low 7 bits of the search's
//           number on top
//   word 1: the search's number (the other 51 bits), the side (1 bit: the
//           instance or its inverse), the restart attempt (6 bits: the
//           subtrees of an abandoned attempt were not all searched) and the
//           depth (4 bits)
// A search's number is its launch's epoch and its index there (58 bits), so
// the entries of other launches never match and the table is never cleared.
// Zero words are empty (a recorded state has depth >= 1).
//
// Each warp had a table of its own before (4,096 entries of 8 bytes, 155 MB in
// all): the warps that shared a long search explored the same states again.
// The hardest of 2,048 S_16 instances at their lower bound took 171,000 to
// 258,000 expansions then, against about 14,000 with one table.

// A search starts using the table after this many expansions of a unit: most
// searches of uniform permutations end sooner, and they then never touch it.
// States expanded before are simply not recorded.
#ifndef TD_TT_AFTER
#define TD_TT_AFTER 32
#endif

__device__ __forceinline__ void td_tt_load(const ulonglong2 *p, uint64_t &a, uint64_t &b) {
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(a), "=l"(b)
                 : "l"(p)
                 : "memory");
}

__device__ __forceinline__ void td_tt_store(ulonglong2 *p, uint64_t a, uint64_t b) {
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }"
                 :
                 : "l"(p), "l"(a), "l"(b)
                 : "memory");
}

// The place of a state's entry, and its two words (word 1 without the depth).
__device__ __forceinline__ ulonglong2 *td_tt_entry(const td_search_limits &lim, uint64_t L, uint32_t inst, uint32_t sub,
                                                   uint64_t *w0, uint64_t *w1) {
    const uint64_t id = lim.tt_id + inst;
    *w0 = td_tt_key(L) | (id << 57);
    *w1 = ((id >> 7) << 7) | sub;
    return lim.tt + (((*w0 + *w1 * 0xD6E8FEB86659FD93ull) * 0x9E3779B97F4A7C15ull) >> lim.tt_shift);
}

// Whether the state L (nibbles from N-1 on cleared) is in the table at a depth
// <= lv.
__device__ __forceinline__ bool td_tt_peek(const td_search_limits &lim, uint64_t L, int lv, uint32_t inst, uint32_t sub) {
    uint64_t w0, w1, e0, e1;
    const ulonglong2 *e = td_tt_entry(lim, L, inst, sub, &w0, &w1);
    td_tt_load(e, e0, e1);
    return e0 == w0 && (e1 >> 4) == w1 && (int)(e1 & 15u) <= lv;
}

// Looks up the state of level `lv` (depth lv) in the table and records it
// there; returns whether it was already taken up at a depth <= lv by the
// search `sub` (side << 6 | attempt) of instance `inst` of this launch
// (uniform across the warp).
__device__ __forceinline__ bool td_tt_visit(const td_warp_smem &s, int lv, int N,
                                            uint32_t inst, uint32_t sub) {
    const int m = threadIdx.x & 31;
    const int a = m < N ? s.A[lv][m] : 0xff;
    const int c0 = __ffs(__ballot_sync(TD_FULL, a == 0)) - 1;  // caller position of label 0
    // L[m] = A[(m + 1 + c0) mod N] - 1 for m < N - 1
    int src = m + 1 + c0;
    src -= src >= N ? N : 0;
    const int v = __shfl_sync(TD_FULL, a, m < N - 1 ? src : m) - 1;
    uint32_t lo = 0, hi = 0;
    if (m < N - 1) {
        if (m < 8) lo = (uint32_t)v << (4 * m);
        else hi = (uint32_t)v << (4 * (m - 8));
    }
    lo = __reduce_or_sync(TD_FULL, lo);
    hi = __reduce_or_sync(TD_FULL, hi);
    int hit = 0;
    if (m == 0) {
        uint64_t w0, w1;
        ulonglong2 *e = td_tt_entry(s.lim, (((uint64_t)hi) << 32) | lo, inst, sub, &w0, &w1);
        uint64_t e0, e1;
        td_tt_load(e, e0, e1);
        hit = e0 == w0 && (e1 >> 4) == w1 && (int)(e1 & 15u) <= lv;
        if (!hit) td_tt_store(e, w0, (w1 << 4) | (uint64_t)lv);
    }
    return __shfl_sync(TD_FULL, hit, 0) != 0;
}

#include "td_endgame.cuh"

struct td_dfs_out {
    int status;
    int depth;
    uint16_t found_move;
    uint32_t expansions;
};

// Reserves `want` item slots; returns the first (or -1) and, in `got`, how many
// there are.  Called by one lane.  In the array (the batch engine) a
// fetch-and-add reserves them: slots past the capacity are never written, and
// their tickets wait for the launch to end.  In the ring at most `capacity`
// items are unclaimed, so the count must be checked before it is raised.  The
// pending count covers the items before any taker can finish one (takers wait
// for the ready flag, written later), and so does the batch engine's
// outstanding count.
__device__ __forceinline__ int td_reserve(td_donate_ctx &dc, int want, unsigned long long unit, int *got) {
    int base = -1, n = want;
    if (dc.tickets) {
        if (*(volatile int *)&dc.pool->produced < dc.capacity) {
            base = atomicAdd(&dc.pool->produced, want);
            n = min(want, dc.capacity - base);
            if (n <= 0) base = -1;
        }
        if (base >= 0) atomicAdd(&dc.pool->outstanding, n);
    } else {
        int cur = *(volatile int *)&dc.pool->produced;
        for (;;) {
            if (cur - *(volatile int *)&dc.pool->consumed + want > dc.capacity) break;
            const int prev = atomicCAS(&dc.pool->produced, cur, cur + want);
            if (prev == cur) { base = cur; break; }
            cur = prev;
        }
    }
    if (base >= 0) {
        // the first time, a root search counts itself too
        atomicAdd(&dc.state->pending, (unsigned long long)n * unit + (dc.gave ? 0ull : 1ull));
        dc.gave = 1;
    }
    td_fence();
    *got = base >= 0 ? n : 0;
    return base;
}

// Writes an item into its slot and sets the slot's ready flag.  Called by each
// lane that holds an item.
__device__ __forceinline__ void td_publish(const td_donate_ctx &dc, const td_item &it, int slot) {
    int phys = slot;
    uint32_t tag = dc.epoch;
    if (dc.ring) {
        phys = slot % dc.capacity;
        tag = td_ring_tag(slot);
        if (slot >= dc.capacity) {
            // the slot's previous item (index slot - capacity) is claimed; wait
            // until its taker has read it (bounded).  After an expired wait the
            // slot still belongs to an unread item: it is left alone, and this
            // item's taker gives up at the deadline
            const uint32_t freed = td_ring_tag(slot - dc.capacity) | 0x80000000u;
            for (unsigned spin = 0; *(volatile uint32_t *)&dc.ready[phys] != freed; ++spin) {
                if ((spin & 255u) == 0 && dc.deadline_ns && td_globaltimer() > dc.deadline_ns) {
                    atomicCAS(&dc.pool->error, 0, TD_ERR_TIMEOUT);
                    return;
                }
                __nanosleep(64);
            }
        }
    }
    dc.items[phys] = it;
    td_fence();
    *(volatile uint32_t *)&dc.ready[phys] = tag;
}

// Hands up to `want` (at most 32) remaining children of the shallowest level
// in [d0, level] to the pool as items, one per lane (free move order).  Returns
// the number donated (uniform across the warp).
__device__ __noinline__ int td_donate(td_warp_smem &s, int d0, int level, int N, int want, int attempt) {
    const td_donate_ctx &dc = s.dc;
    const int lane = threadIdx.x & 31;
    int lv = -1;
    for (int l = d0; l <= level && l <= dc.max_level; ++l) {
        if (s.m2[l] | s.m0[l]) { lv = l; break; }
    }
    if (lv < 0) return 0;
    const uint4 Wv = s.pw[lv][lane];
    uint32_t W0 = Wv.x, W1 = Wv.y, W2 = Wv.z, W3 = Wv.w;
    const int cnt = __popc(W0) + __popc(W1) + __popc(W2) + __popc(W3);
    int before = cnt;  // lanes give in lane order
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(TD_FULL, before, o);
        if (lane >= o) before += v;
    }
    const int have = __shfl_sync(TD_FULL, before, 31);
    before -= cnt;
    // leave at least one child to this warp when the level is the current one
    int give = min(min(want, 32), have - (lv == level ? 1 : 0));
    if (give <= 0) return 0;
    int base = -1;
    if (lane == 0) base = td_reserve(s.dc, give, dc.side ? TD_UNIT_INVERSE : 1ull, &give);
    base = __shfl_sync(TD_FULL, base, 0);
    give = __shfl_sync(TD_FULL, give, 0);
    if (base < 0) return 0;  // out of item space: keep the work
    if (lane == 0) {
        atomicAdd(&dc.pool->donations, 1ull);
        atomicAdd(&dc.pool->donated_items, (unsigned long long)give);
    }
    uint64_t Lp;
    int offp;
    td_pack_state(s, lv, N, &Lp, &offp);  // the parent in pinned form
    const ushort4 pq = s.pair[lane];
    // a lane gives its lowest slots first (the ones this warp visits last),
    // and 0-class children (high bits) before +2 children
    const int last = min(give, before + cnt);
    for (; before < last; ++before) {
        uint32_t pc, b;
        if (W0) { pc = pq.x; b = 31 - __clz(W0); W0 &= ~(1u << b); }
        else if (W1) { pc = pq.y; b = 31 - __clz(W1); W1 &= ~(1u << b); }
        else if (W2) { pc = pq.z; b = 31 - __clz(W2); W2 &= ~(1u << b); }
        else { pc = pq.w; b = 31 - __clz(W3); W3 &= ~(1u << b); }
        s.list[before] = (uint16_t)(pc | ((b < 16 ? b + 1 : b - 15) << 10));
    }
    s.pw[lv][lane] = make_uint4(W0, W1, W2, W3);
    const uint32_t any = W0 | W1 | W2 | W3;
    const uint32_t m2 = __ballot_sync(TD_FULL, (any & 0x0000ffffu) != 0);
    const uint32_t m0 = __ballot_sync(TD_FULL, (any & 0xffff0000u) != 0);
    if (lane == 0) {
        s.m2[lv] = m2;
        s.m0[lv] = m0;
    }
    __syncwarp();
    if (lane < give) {
        const uint32_t t = s.list[lane];
        uint64_t nL;
        int noff;
        td_apply_move(Lp, offp, N, t & 31, (t >> 5) & 31, (t >> 10) & 31, &nL, &noff);
        td_item it;
        it.L = nL;
        it.inst = dc.inst;
        it.depth = (uint8_t)((lv + 1) | ((attempt & 7) << 4) | (dc.side << 7));
        it.off = (uint8_t)(noff | ((attempt >> 3) << 5));
#pragma unroll
        for (int d = 0; d < TD_MAX_DEPTH; ++d) it.path[d] = d < lv ? s.path[d] : (d == lv ? (uint16_t)t : 0);
        td_publish(dc, it, base + lane);
    }
    __syncwarp();
    return give;
}

// Queues the inverse of the unit's instance (td_inverse_pinned) as one more
// item, a root of the inverse's side, so that another warp searches it while
// this one goes on; the first witness on either side ends both, and so does the
// instance's side searched to the end without one (found = 2).  Only an
// instance's root search queues its inverse, and once: the race is off for it
// from then on (a second inverse root would share the first one's entries in
// the table of explored states).  In the batch engine items
// are taken once no fresh instance is left, and the inverses queued until then
// come first.  Returns whether it was queued (uniform across the warp).
__device__ __noinline__ int td_spawn_inverse(td_warp_smem &s, int N) {
    const td_donate_ctx &dc = s.dc;
    int ok = 0;
    if ((threadIdx.x & 31) == 0) {
        int got;
        const int slot = td_reserve(s.dc, 1, TD_UNIT_INVERSE, &got);
        if (slot >= 0) {
            td_item it;
            it.L = td_inverse_pinned(s.L[0], N);
            it.inst = dc.inst;
            it.depth = 0x80;
            it.off = 0;
#pragma unroll
            for (int d = 0; d < TD_MAX_DEPTH; ++d) it.path[d] = 0;
            td_publish(dc, it, slot);
            atomicAdd(&dc.pool->races, 1ull);
            s.dc.race = 0;
            ok = 1;
        }
    }
    __syncwarp();
    return __shfl_sync(TD_FULL, ok, 0);
}

// After a unit of the inverse's search found a witness (depth moves: path[0 ..
// depth-2] and found_move), rewrites it as the witness of the instance x in
// the caller's positions: td_witness_from_inverse's steps, one lane per
// position (arrays in registers, block swaps by shuffle, cut points by
// ballot).  Returns 0 if it does not convert (then no witness may be
// recorded).  Uniform across the warp.
__device__ __forceinline__ int td_inverse_result(td_warp_smem &s, const td_instance &x, int k, uint32_t *found_move) {
    const int c = threadIdx.x & 31;
    const int N = x.n_symbols;
    if (k < 1 || k > TD_MAX_DEPTH) return 0;
    // the swap of blocks [i, j) and [j, kk) moves the value at src(c) to c
    auto swap = [&](uint32_t v, uint32_t mv) {
        const int i = mv & 31, j = (mv >> 5) & 31, kk = (mv >> 10) & 31;
        int src = c;
        if (c >= i && c < kk) src = c < i + (kk - j) ? c + (j - i) : c - (kk - j);
        return __shfl_sync(TD_FULL, v, src);
    };
    // lane q holds the inverse's move q, and then the converted move q
    const uint32_t inv = c < k - 1 ? (uint32_t)s.path[c] : (c == k - 1 ? *found_move : 0u);
    __syncwarp();
    // X: the caller's array; S: the identity array after all the inverse's moves
    int p = c + x.offset;
    p -= p >= N ? N : 0;
    uint32_t X = c < N ? (p ? td_nib(x.perm, p - 1) + 1u : 0u) : 0xffu;
    uint32_t S = (uint32_t)c;
    for (int q = 0; q < k; ++q) S = swap(S, __shfl_sync(TD_FULL, inv, q));
    const int prev = c == 0 ? N - 1 : c - 1;
    uint32_t mine = 0;  // lane q: move q of the converted witness
    for (int m = k; m >= 1; --m) {
        const uint32_t mv = __shfl_sync(TD_FULL, inv, m - 1);
        const int i = mv & 31, j = (mv >> 5) & 31, kk = (mv >> 10) & 31;
        if (!(i < j && j < kk && kk < N)) return 0;
        const uint32_t Xp = __shfl_sync(TD_FULL, X, prev);
        // the three cut points of s_m^-1 = (i, i + kk - j, kk) in S, found in X
        // (every lane takes part in every shuffle: they are computed before
        // the comparisons, never inside a short-circuited condition)
        const int g0 = i, g1 = i + kk - j, g2 = kk;
        const uint32_t u0 = __shfl_sync(TD_FULL, S, g0 == 0 ? N - 1 : g0 - 1), v0 = __shfl_sync(TD_FULL, S, g0);
        const uint32_t u1 = __shfl_sync(TD_FULL, S, g1 - 1), v1 = __shfl_sync(TD_FULL, S, g1);
        const uint32_t u2 = __shfl_sync(TD_FULL, S, g2 - 1), v2 = __shfl_sync(TD_FULL, S, g2);
        const bool act = c < N;
        const uint32_t h0 = __ballot_sync(TD_FULL, act & (Xp == u0) & (X == v0));
        const uint32_t h1 = __ballot_sync(TD_FULL, act & (Xp == u1) & (X == v1));
        const uint32_t h2 = __ballot_sync(TD_FULL, act & (Xp == u2) & (X == v2));
        // each cut is one neighbouring pair, so each mask has one bit; their
        // union, taken in ascending order, is the move in the caller's array
        const uint32_t cuts = h0 | h1 | h2;
        if (__popc(h0) != 1 || __popc(h1) != 1 || __popc(h2) != 1 || __popc(cuts) != 3) return 0;
        const int a = __ffs(cuts) - 1;
        const uint32_t rest = cuts & (cuts - 1);
        const int b = __ffs(rest) - 1;
        const int e = 31 - __clz(cuts);
        const uint32_t t = td_pack_move(a, b, e);
        if (c == k - m) mine = t;
        X = swap(X, t);
        S = swap(S, (uint32_t)i | ((uint32_t)(i + kk - j) << 5) | ((uint32_t)kk << 10));  // S_{m-1} = S_m . s_m^-1
    }
    // each lane stores its own move into the path, which it alone read above;
    // the record's writers read it after the barrier
    if (c < k - 1) s.path[c] = (uint16_t)mine;
    *found_move = __shfl_sync(TD_FULL, mine, k - 1);
    __syncwarp();
    return 1;
}

// Whether a witness of instance x (its caller positions: path[0 .. depth-2],
// found_move) is one the instance's own search could return: every move keeps
// the reference's move filter (it touches no symbol that omega fixes, and it
// changes the odd-cycle count by 0 or +2, sorting_search.cu:375-380,
// 240-332), no node before the last passes the acceptance test, and the last
// does.  A witness of the inverse, turned into the instance's positions, keeps
// the filter on the inverse's side but need not on this one: its path passes
// through other states.  Recording only witnesses that pass keeps the verdict
// that of the instance's own filtered search.  Uses the warp's frame (levels
// 0..depth) as scratch; uniform across the warp.
__device__ __forceinline__ bool td_filtered_witness(td_warp_smem &s, const td_instance &x, int k, uint32_t found_move) {
    const int N = x.n_symbols;
    if (k < 1 || k > TD_MAX_DEPTH) return false;
    td_unpack_state(s, 0, x.perm, x.offset, N);
    int odd = 0;
    for (int d = 0;; ++d) {
        uint32_t O, F;
        const int now = td_prepare_rows(s, d, N, O, F);
        if (d > 0) {
            if (now != odd && now != odd + 2) return false;
            const bool accepted = (s.acc[d] >> now) & 1u;
            if (accepted != (d == k)) return false;
            if (d == k) return true;
        }
        odd = now;
        const uint32_t t = d == k - 1 ? found_move : (uint32_t)s.path[d];
        const int i = t & 31, j = (t >> 5) & 31, kk = (t >> 10) & 31;
        if (!(i < j && j < kk && kk < N)) return false;
        if (((F >> i) | (F >> j) | (F >> kk)) & 1u) return false;
        td_apply_bytes(s, d, t, N);
    }
}

// A unit of the inverse's side found a witness of k moves: turns it into one of
// the instance.  Returns its last move; -1 where it does not convert (a failed
// replay), -2 where it leaves the reference's move filter on the instance's
// side (it is dropped: this side then stops, the instance's own search
// decides).
__device__ __noinline__ int td_inverse_witness(td_warp_smem &s, td_instance x, int k, uint32_t found_move) {
    if (!td_inverse_result(s, x, k, &found_move)) return -1;
    return td_filtered_witness(s, x, k, found_move) ? (int)found_move : -2;
}

#include "td_ordered.cuh"

// Depth-first search from the node held at level d0 of `s` (state, path, rate
// masks, pair slots and limits already set).  Leaves
// the frames intact on TD_DFS_BUDGET.  `shared`: a unit of a search that other
// warps may take part in (s.dc says how; in the reference order also s.sp).
//
// The node is expanded at one place of the loop, and what runs rarely is not
// inlined: the loop has to fit the instruction caches.  With three copies of
// the evaluation, two calls of this function per kernel and the rest inlined,
// a warp of the batch engine waited 3.4 to 10.6 cycles per issued instruction
// for its next one, more than for anything else.
template <bool ORDERED>
__device__ __forceinline__ td_dfs_out td_dfs(td_warp_smem &s, int N, int d0, bool shared) {
    const int lane = threadIdx.x & 31;
    const int last_tri = td_tri_base(N) + td_triple_count(N) - 1;  // child u is triple last_tri - u
    td_dfs_out r;
    r.status = TD_DFS_EXHAUSTED;
    r.depth = 0;
    r.found_move = 0;
    r.expansions = 0;
    int level = d0;
    bool solved = false;  // free order: the endgame table has shown the way to a witness
    td_unpack_state(s, d0, s.L[d0], s.off[d0], N);
    uint32_t work = 0;  // nodes expanded here
    int since_check = 0;
    bool due = false;            // the scheduler's counters were read (lane 0)
    int waiting = 0, ended = 0;  // idle warps not yet served by an item; the instance is decided
    int attempt = 0;     // free order: restarts with another child order (td_attempt_budget)
    uint32_t ord = 0, attempt_exp = 0;
    uint32_t attempt_budget = ORDERED ? ~0u : td_attempt_budget(s.lim.restart_base, 0);
    // a unit of a raced instance: the inverse's side, or the instance's side
    // once it queued the inverse
    bool raced = !ORDERED && shared && s.dc.side;
    for (;;) {
        // expand the node at `level`, and let the endgame table decide its
        // children.  A move joins at most three pairs of neighbours, so only a
        // node of at most TD_EG_SYMBOLS + 3 symbols that omega moves has one in
        // the table.
        {
            uint32_t O, F;
            const int odd = td_prepare_rows(s, level, N, O, F);
            const int eg_moves = s.eg_moves;  // 0: the table does not apply
            const int spare = eg_moves - level - ((N - odd) >> 1);
            const bool endgame =
                eg_moves > level + 1 && spare >= 0 && N - __popc(F) <= TD_EG_SYMBOLS + 3;  // warp-uniform
            int found;
            if constexpr (ORDERED) {
                // with two spare moves no child that the table holds is dropped
                if (lane == 0) s.spare[level] = (uint8_t)(endgame && spare < 2 ? spare : 255);
                found = td_evaluate(s, N, level, odd, O, F);
                if (found >= 0) found = td_tri_table[last_tri - found];
            } else {
                if (lane == 0) s.spare[level] = (uint8_t)(endgame ? spare : 255);
                found = td_evaluate_rows(s, N, level, odd, O, F);
            }
            ++work;
            if constexpr (ORDERED) r.expansions = td_add_count(r.expansions, 1u);
            else r.expansions = work;
            if (found >= 0) {
                r.found_move = (uint16_t)found;
                r.depth = level + 1;
                r.status = TD_DFS_FOUND;
                break;
            }
            if constexpr (!ORDERED) {
                ++attempt_exp;
                if (endgame && spare == 0) {
                    const uint4 w = s.pw[level][lane];
                    const unsigned n = __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
                    if (__reduce_add_sync(TD_FULL, n) >= TD_EG_MANY)
                        solved |= td_eg_filter(s, level, N, s.dc.gave && s.lim.tt ? attempt : -1);
                }
            }
        }
        if (td_over_budget(r.expansions, s.lim.max_expansions)) {
            r.status = TD_DFS_BUDGET;
            break;
        }
        if constexpr (!ORDERED) {
            if (attempt_exp >= attempt_budget && !solved) {
                // restart the subtree at d0 with the next child order; the
                // abandoned attempt's states were not explored to the end, so
                // the next attempt's entries have another number
                ++attempt;
                // a root search that may race queues its inverse when it starts
                // attempt dc.race; another warp then searches it alongside
                if (shared && attempt == s.dc.race && !s.dc.side && d0 == 0 && td_spawn_inverse(s, N)) raced = true;
                ord = td_order_variant(attempt);
                attempt_budget = td_attempt_budget(s.lim.restart_base, attempt);
                attempt_exp = 0;
                level = d0;
                continue;
            }
            if (due) {  // the counters were read before the expansion
                due = false;
                const int hungry = __shfl_sync(TD_FULL, waiting, 0);
                if (__shfl_sync(TD_FULL, ended, 0)) {
                    r.status = TD_DFS_ABORTED;
                    break;
                }
                if (hungry > 0 && !s.dc.idle_seen && work >= s.dc.idle_after) {
                    __syncwarp();
                    if (lane == 0) td_serve_idle_warps(s.dc);
                    __syncwarp();
                }
                // a search that has handed out subtrees no longer restarts: the
                // subtrees of an abandoned attempt would go on being searched,
                // and searching in parallel already varies the order.  In a
                // batch, a race that its next restart would have begun begins
                // now (in the serving loop nearly every request would race so:
                // 2,048 requests at their lower bound 7.5 -> 13.7 ms)
                if (hungry > 0 && !solved) {
                    if (s.dc.tickets && s.dc.race == attempt + 1 && attempt_budget != ~0u && td_spawn_inverse(s, N)) raced = true;
                    if (td_donate(s, d0, level, N, min(hungry, s.dc.grain), s.dc.attempt + attempt) > 0)
                        attempt_budget = ~0u;
                }
            }
        }
        if constexpr (ORDERED) {
            if (due) {
                due = false;
                if (__shfl_sync(TD_FULL, waiting, 0) > 0) td_split(s, d0, level, N);
            }
        }
        if ((work & 255u) == 0) {
            int stop = 0;
            if (lane == 0) {
                if (s.lim.deadline_ns && td_globaltimer() > s.lim.deadline_ns) stop = 1;
                // a subtree of a split ordered search: one of lower rank has a witness
                if (s.lim.cutoff && *(volatile const int *)s.lim.cutoff < s.lim.rank) stop = 2;
                if (s.lim.cutoff2 && *(volatile const int *)s.lim.cutoff2 < s.lim.rank2) stop = 2;
            }
            stop = __shfl_sync(TD_FULL, stop, 0);
            if (stop) {
                r.status = stop == 2 ? TD_DFS_ABORTED : TD_DFS_TIMEOUT;
                break;
            }
        }
        // walk to the next node to expand: backtracks, and in free order the
        // children skipped through the tables, change no expansion count, so
        // the checks above run once per expansion
        int walk = 0;  // 1: the subtree is exhausted, 2: a root accepted on visit (ordered), 3: out of budget
        for (bool fresh = !ORDERED && attempt + solved + d0 == 0 && s.eg_moves != 0;; fresh = false) {
            int t = -1;
            if constexpr (ORDERED) {
                const int spare = s.spare[level];
                if (spare != 255) {
                    // the walk of the children dropped here ends without a
                    // witness; a budget that it would exhaust ends it there
                    const uint32_t skipped = td_eg_skip(s, level, N, spare);
                    r.expansions = td_add_count(r.expansions, skipped);
                    if (skipped && td_over_budget(r.expansions, s.lim.max_expansions)) {
                        r.expansions = (uint32_t)s.lim.max_expansions;
                        walk = 3;
                        break;
                    }
                }
                int accepted;
                t = td_next_child(s, level, &accepted);
                if (t >= 0) {
                    t = td_tri_table[last_tri - t];
                    if (accepted) {
                        r.found_move = (uint16_t)t;
                        walk = 2;
                        break;
                    }
                }
            } else {
                if (fresh) t = td_take_fixing(s, level, N);
                if (t < 0) t = td_next_child_rows(s, level, td_level_order(ord, attempt, level));
            }
            if (t < 0) {
                if (level == d0) { walk = 1; break; }
                --level;
                continue;
            }
            if (lane == 0) s.path[level] = (uint16_t)(t & 0x7fff);
            td_apply_bytes(s, level, (uint32_t)t, N);
            if constexpr (!ORDERED) {
                const int spare = s.spare[level];
                if (spare != 255) {
                    // a 0 child has a spare move less than its parent
                    const uint32_t e = td_eg_look(s, level + 1, N, spare == (t >> 15));
                    if (e == 0) {
                        solved = true;
                        break;
                    }
                    if (e != TD_EG_UNKNOWN) continue;
                }
                // taken up already with at least this budget?
                if (!solved && (work >= TD_TT_AFTER || d0 > 0) && s.lim.tt &&
                    td_tt_visit(s, level + 1, N, s.dc.inst, (uint32_t)(s.dc.side << 6) + (uint32_t)(s.dc.attempt + attempt)))
                    continue;
            }
            break;
        }
        if (walk) {
            if (walk == 2) {
                r.depth = level + 1;
                r.status = TD_DFS_FOUND;
            } else if (walk == 3) {
                r.status = TD_DFS_BUDGET;
            }
            break;
        }
        if constexpr (ORDERED) {
            if (shared && r.expansions >= s.lim.split_after && ++since_check >= s.dc.check_every) {
                since_check = 0;
                due = true;
                if (lane == 0) {
                    const unsigned long long pc = *(volatile unsigned long long *)&s.dc.pool->produced;
                    waiting = (int)(pc >> 32) - (int)(uint32_t)pc;
                }
            }
        } else {
            // a raced unit looks for the other side's verdict at least every
            // 16 expansions
            if (shared && ++since_check >= (raced ? min(s.dc.check_every, 16) : s.dc.check_every)) {
                // read now and used after the expansion, which hides the latency
                since_check = 0;
                due = true;
                if (lane == 0) {
                    const unsigned long long pc = *(volatile unsigned long long *)&s.dc.pool->produced;
                    waiting = (int)(pc >> 32) - (int)(uint32_t)pc;
                    // takers holding a ticket past the last item produced; in
                    // the serving loop, idle warps beyond the unclaimed items
                    if (!s.dc.tickets) waiting += *(volatile int *)&s.dc.pool->idle;
                    ended = s.dc.gave ? *(volatile unsigned short *)&s.dc.state->found : 0;
                }
            }
        }
        ++level;
    }
    __syncwarp();
    return r;
}

__device__ __forceinline__ bool td_instance_ok(const td_instance &x) {
    return x.n_symbols <= TD_MAX_N && x.max_moves >= 1 && x.max_moves <= TD_MAX_DEPTH &&
           td_inst_init(x) <= TD_MAX_N;
}

// Loads the warp's pair slots for N, unless they are, and the instance's rate
// masks; places its root at level 0.
__device__ __forceinline__ void td_setup_root(td_warp_smem &s, const td_instance &x) {
    const int lane = threadIdx.x & 31;
    if (s.pairs_n != x.n_symbols) {
        td_load_pairs(s, x.n_symbols);
        if (lane == 0) s.pairs_n = x.n_symbols;
    }
    td_rate_masks(s, x);
    if (lane == 0) {
        s.L[0] = x.perm;
        s.off[0] = x.offset;
    }
    __syncwarp();
}

// Writes words [w0, w1) of a 32-byte result from lanes 0..7.
__device__ __forceinline__ void td_write_result(td_result *out, int status, int depth, uint16_t found_move,
                                                const uint16_t *path, uint32_t expansions, int w0, int w1) {
    const int lane = threadIdx.x & 31;
    uint32_t word = 0;
    if (lane == 0) word = (uint32_t)status;
    else if (lane == 1) word = (uint32_t)depth;
    else if (lane >= 2 && lane < 7) {
        const int m0 = 2 * (lane - 2), m1 = m0 + 1;
        uint32_t lo = 0, hi = 0;
        if (status == TD_FOUND) {
            if (m0 < depth) lo = (m0 == depth - 1) ? found_move : path[m0];
            if (m1 < depth && m1 < TD_MAX_DEPTH) hi = (m1 == depth - 1) ? found_move : path[m1];
        }
        word = lo | (hi << 16);
    } else if (lane == 7) {
        word = expansions;
    }
    if (lane >= w0 && lane < w1) reinterpret_cast<volatile uint32_t *>(out)[lane] = word;
}

// One complete search of instance x by the calling warp (no sharing); returns
// the status it wrote (uniform across the warp).
template <bool ORDERED>
__device__ int td_warp_search(const td_instance &x, td_result *out, td_warp_smem &s) {
    int status = TD_NOT_FOUND, depth = 0;
    uint32_t expansions = 0;
    uint16_t found_move = 0;
    if (!td_instance_ok(x)) {
        status = TD_ERR_ARG;
    } else if (td_triple_count(x.n_symbols) > 0) {
        td_setup_root(s, x);
        const td_dfs_out r = td_dfs<ORDERED>(s, x.n_symbols, 0, false);
        expansions = r.expansions;
        status = td_status_of_dfs(r.status);
        if (status == TD_FOUND) {
            depth = r.depth;
            found_move = r.found_move;
        }
    }
    __syncwarp();
    td_write_result(out, status, depth, found_move, s.path, expansions, 0, 8);
    return status;
}
