// td_endgame.cuh -- the endgame table: which small states are sorted by +2
// moves alone (included by td_kernels.cuh).
//
// A symbol that omega fixes sits right after its predecessor, no move may cut
// there (the move filter, sorting_search.cu:375-380), and so a state behaves
// exactly like the state with its fixed symbols glued to their predecessors:
// the same moves, the same odd-cycle changes, the same missing cycles N - odd.
// The search of a glued state of n' symbols is therefore a constant of the
// engine, and the table holds it for every n' <= 11: entry 0 where the state
// with M = (N - odd) / 2 moves left can be sorted (M moves, each +2), else
// the number of nodes the reference-order walk expands to find that it cannot.
// With a spare move every one of these states can be sorted (the largest
// filtered distance over the table is M + 1; a CPU test rebuilds the table and
// checks it), so one 16-bit word per state decides every bound.
//
// A node looks its children up before it visits them, 32 at a time, one per
// lane: a child that cannot be sorted is dropped without expanding a node of
// its subtree (the reference order adds the entry to its expansion count, so
// the count stays the walk's), and a child that can is taken at once.  The
// index is the Lehmer rank of the glued state: 4,037,912 words, 8 MiB, which
// the L2 keeps; it is filled once per device by td_eg_build_kernel.
//
// Why n' <= 11: in the host emulation of the free order on near-reverse S_16 at
// bound 9 the mean search falls from 80 expansions to 59 with a table of
// n' <= 9, 48 with n' <= 11 and 44 with n' <= 12, whose table would be 12
// times as large; at the lower bound (most of the work then proves that there
// is no witness) from about 3,000 to 1,900, 1,030 and 710.
#pragma once

#ifndef TD_EG_MANY
#define TD_EG_MANY 8            // free order: children from which a node looks them up 32 at a time
#endif
#define TD_EG_UNKNOWN 0x10000u  // td_eg_probe: the child is not in the table

__device__ uint16_t td_eg_table[TD_EG_STATES];

__device__ uint32_t td_eg_bases[TD_EG_SYMBOLS];
__device__ uint32_t td_eg_factorial[TD_EG_SYMBOLS];

// The symbols that omega fixes in the caller's array of `level`: those that
// follow their predecessor (uniform across the warp).
__device__ __forceinline__ uint32_t td_eg_fixed(const td_warp_smem &s, int level, int N) {
    const int c = threadIdx.x & 31;
    uint32_t m = 0;
    if (c < N) {
        const int a = s.A[level][c], b = s.A[level][c == 0 ? N - 1 : c - 1];
        if (a == (b + 1 == N ? 0 : b + 1)) m = 1u << a;
    }
    return __reduce_or_sync(TD_FULL, m);
}

// What the table says of the child that this lane's move `t` makes of the node
// at `level` (pinned state L, off; fixed symbols `fixed`): TD_EG_UNKNOWN (more
// than TD_EG_SYMBOLS symbols left), 0 (sorted within the moves left), or the
// expansions of its walk.  `tight`: the child has no spare move.
__device__ __forceinline__ uint32_t td_eg_probe(const td_warp_smem &s, int level, int N, uint64_t L, int off,
                                                uint32_t fixed, uint32_t t, bool tight) {
    const int i = t & 31, j = (t >> 5) & 31, k = (t >> 10) & 31;
    const uint8_t *A = s.A[level];
    // the three new neighbours (b after a)
    const int a0 = A[i == 0 ? N - 1 : i - 1], b0 = A[j], a1 = A[k - 1], b1 = A[i], a2 = A[j - 1], b2 = A[k];
    if (b0 == (a0 + 1 == N ? 0 : a0 + 1)) fixed |= 1u << b0;
    if (b1 == (a1 + 1 == N ? 0 : a1 + 1)) fixed |= 1u << b1;
    if (b2 == (a2 + 1 == N ? 0 : a2 + 1)) fixed |= 1u << b2;
    const uint32_t kept = ((1u << N) - 1u) & ~fixed;
    const int n = __popc(kept);
    if (n > TD_EG_SYMBOLS) return TD_EG_UNKNOWN;
    if (n == 0 || !tight) return 0;
    uint64_t nL;
    int noff;
    td_apply_move(L, off, N, i, j, k, &nL, &noff);
    return __ldg(&td_eg_table[__ldg(&td_eg_bases[n - 1]) + td_eg_rank(nL, kept)]);
}

// Reference order: lists up to 32 children of `level` still to visit, in
// visiting order, in s.list; returns how many there are in all.
__device__ __forceinline__ int td_eg_list(td_warp_smem &s, int level) {
    const int lane = threadIdx.x & 31;
    const uint32_t w = lane < TD_MAX_STEPS ? s.cw[level][lane] : 0u;
    int from = __popc(w);  // children in this lane's word and those after it
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_down_sync(TD_FULL, from, o);
        if (lane + o < 32) from += v;
    }
    const int all = __shfl_sync(TD_FULL, from, 0);
    int at = from - __popc(w);
    for (uint32_t rest = w; rest && at < 32; ++at) {
        const int b = level == 0 ? 31 - __clz(rest) : __ffs(rest) - 1;
        rest &= ~(1u << b);
        s.list[at] = (uint16_t)(32 * lane + b);
    }
    __syncwarp();
    return all;
}

// Reference order: drops the children of `level` that come before its next
// child to visit and that the table decides, and returns the expansions of
// their walks.  `spare`: the moves that the node can spare (moves left less
// the missing ones).
__device__ __forceinline__ uint32_t td_eg_skip(td_warp_smem &s, int level, int N, int spare) {
    const int lane = threadIdx.x & 31;
    const int last_tri = td_tri_base(N) + td_triple_count(N) - 1;
    const uint32_t fixed = td_eg_fixed(s, level, N);
    uint64_t L;
    int off;
    td_pack_state(s, level, N, &L, &off);
    uint32_t sum = 0;
    for (;;) {
        const int all = td_eg_list(s, level);
        uint32_t e = TD_EG_UNKNOWN;  // lanes past the last child end the run of decided ones
        uint32_t u = 0;
        if (lane < all) {
            u = s.list[lane];
            // a +2 child has the node's spare moves, a 0 child one less
            const bool plus2 = spare == 0 || ((s.cp[level][u >> 5] >> (u & 31)) & 1u);
            e = td_eg_probe(s, level, N, L, off, fixed, td_tri_table[last_tri - (int)u], plus2 ? spare == 0 : spare == 1);
        }
        const uint32_t stop = __ballot_sync(TD_FULL, e == 0 || e == TD_EG_UNKNOWN);
        const bool drop = stop == 0 || lane < __ffs(stop) - 1;
        sum += __reduce_add_sync(TD_FULL, drop ? e : 0u);
        if (drop) atomicAnd(&s.cw[level][u >> 5], ~(1u << (u & 31)));
        __syncwarp();
        if (stop || all <= 32) return sum;
    }
}

// Free order, a node without a spare move (all its children are +2 ones):
// decides the children of `level` by the table.  Where one can be sorted it
// becomes the level's only child (returns true); otherwise only the children
// that the table does not hold stay.  `attempt` >= 0: the search is shared by
// several warps, and of those the ones that the table of explored states holds
// for this attempt are dropped too, 32 looks at once instead of one after the
// other when they are visited (where the others are recorded, as ever).  2,048
// S_16 instances at their lower bound took 2.41 ms without those looks and take
// 2.18 ms, the 250 of S_8..S_16 at lower + 1 0.166 and 0.152 ms; for searches
// that one warp ends alone, whose few repeated states it meets soon, they cost
// as much as they give (2^16 mixed instances 1.72 ms and 1.74 ms), and on nodes
// further from the end they made 2^19 near-reverse ones slower (21.6 and 22.1).
__device__ __noinline__ bool td_eg_filter(td_warp_smem &s, int level, int N, int attempt) {
    const int lane = threadIdx.x & 31;
    const uint32_t fixed = td_eg_fixed(s, level, N);
    uint64_t L;
    int off;
    td_pack_state(s, level, N, &L, &off);
    const uint4 Wv = s.pw[level][lane];
    uint32_t W0 = Wv.x, W1 = Wv.y, W2 = Wv.z, W3 = Wv.w;
    __syncwarp();
    s.pw[level][lane] = make_uint4(0u, 0u, 0u, 0u);
    const ushort4 pq = s.pair[lane];
    bool solved = false;
    for (;;) {
        const int mine = __popc(W0) + __popc(W1) + __popc(W2) + __popc(W3);
        int at = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(TD_FULL, at, o);
            if (lane >= o) at += v;
        }
        const int all = __shfl_sync(TD_FULL, at, 31);
        if (all == 0) break;
        at -= mine;
        for (int q = 0; q < mine && at < 32; ++q, ++at) {
            uint32_t pc, b;
            if (W3) { pc = pq.w; b = __ffs(W3) - 1; W3 &= ~(1u << b); }
            else if (W2) { pc = pq.z; b = __ffs(W2) - 1; W2 &= ~(1u << b); }
            else if (W1) { pc = pq.y; b = __ffs(W1) - 1; W1 &= ~(1u << b); }
            else { pc = pq.x; b = __ffs(W0) - 1; W0 &= ~(1u << b); }
            s.list[at] = (uint16_t)(pc | ((b + 1) << 10));
        }
        __syncwarp();
        uint32_t e = 1, t = 0;
        if (lane < all) {
            t = s.list[lane];
            e = td_eg_probe(s, level, N, L, off, fixed, t, true);
            if (e == TD_EG_UNKNOWN && attempt >= 0) {
                uint64_t nL;
                int noff;
                td_apply_move(L, off, N, t & 31, (t >> 5) & 31, (t >> 10) & 31, &nL, &noff);
                const uint32_t sub = (uint32_t)(s.dc.side << 6) + (uint32_t)(s.dc.attempt + attempt);
                if (td_tt_peek(s.lim, nL & (~0ull >> (64 - 4 * (N - 1))), level + 1, s.dc.inst, sub))
                    e = 1;  // taken up already with at least this budget
            }
        }
        __syncwarp();
        const uint32_t yes = __ballot_sync(TD_FULL, e == 0);
        if (yes) {  // unknown children put back earlier go again
            solved = true;
            s.pw[level][lane] = make_uint4(0u, 0u, 0u, 0u);
            __syncwarp();
        }
        if (yes ? lane == __ffs(yes) - 1 : e == TD_EG_UNKNOWN) {
            // back to its pair's slot (td_pair_code)
            const int i = t & 31, j = (t >> 5) & 31, k = (t >> 10) & 31;
            const int q = (N - 1) * (N - 2) / 2 - 1 - (i * (N - 2) - i * (i - 1) / 2 + (j - i - 1));
            const int R = td_pair_rounds(N);
            atomicOr(reinterpret_cast<uint32_t *>(&s.pw[level][q / R]) + q % R, 1u << (k - 1));
        }
        __syncwarp();
        if (solved) break;
    }
    const uint4 K = s.pw[level][lane];
    const uint32_t any = K.x | K.y | K.z | K.w;
    const uint32_t m2 = __ballot_sync(TD_FULL, (any & 0x0000ffffu) != 0);
    const uint32_t m0 = __ballot_sync(TD_FULL, (any & 0xffff0000u) != 0);
    if (lane == 0) {
        s.m2[level] = m2;
        s.m0[level] = m0;
    }
    __syncwarp();
    return solved;
}

// Free order, one child at a time: what the table says of the state of `level`
// (TD_EG_UNKNOWN, or its entry; 0 without a look at the table when the state
// has a spare move).  Lane m holds the m-th symbol of the array read from
// symbol 0; its digit counts the smaller kept symbols after it, from the bit
// planes of the symbols.  About 60 instructions, as many as a look into the
// table of explored states, which the caller skips for the states found here.
__device__ __forceinline__ uint32_t td_eg_look(const td_warp_smem &s, int level, int N, bool tight) {
    const int m = threadIdx.x & 31;
    const int a = m < N ? s.A[level][m] : 0xff;
    const int c0 = __ffs(__ballot_sync(TD_FULL, a == 0)) - 1;  // caller position of symbol 0
    int src = m + c0;
    src -= src >= N ? N : 0;
    const int v = __shfl_sync(TD_FULL, a, m < N ? src : m);
    const int before = __shfl_sync(TD_FULL, v, m == 0 ? N - 1 : m - 1);
    uint32_t kept = __ballot_sync(TD_FULL, m < N && v != (before + 1 == N ? 0 : before + 1));
    const int n = __popc(kept);
    if (n > TD_EG_SYMBOLS) return TD_EG_UNKNOWN;
    if (n == 0 || !tight) return 0;
    // symbol 0 stands for its block: where it is glued, the block's first
    // symbol is the last one kept
    kept &= (kept & 1u) ? ~1u : ~(0x80000000u >> __clz((int)kept));
    uint32_t lt = 0, eq = kept;
#pragma unroll
    for (int b = 4; b >= 0; --b) {
        const uint32_t plane = __ballot_sync(TD_FULL, (v >> b) & 1);
        const uint32_t mine = 0u - (uint32_t)((v >> b) & 1);
        lt |= eq & ~plane & mine;
        eq &= ~(plane ^ mine);
    }
    uint32_t part = 0;
    if ((kept >> m) & 1u) {
        const int after = __popc(kept & (0xfffffffeu << m));  // symbols after this one, each digit's weight is after!
        part = (uint32_t)__popc(lt & (0xfffffffeu << m)) * __ldg(&td_eg_factorial[after]);
    }
    return __ldg(&td_eg_table[__ldg(&td_eg_bases[n - 1]) + __reduce_add_sync(TD_FULL, part)]);
}

// Fills the table: one warp per state, the states of `missing` moves; their
// +2 children miss one less, so the passes run for 1, 2, ..., 5.  Every pass
// writes final values only.
__global__ void __launch_bounds__(256, 4) td_eg_build_kernel(int missing) {
    extern __shared__ __align__(16) uint8_t td_smem[];
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    td_warp_smem &s = reinterpret_cast<td_warp_smem *>(td_smem)[warp];
    int pairs_n = -1;
    // a cycle of two or more symbols misses at least a third of them
    const uint32_t end = 3 * missing >= TD_EG_SYMBOLS ? TD_EG_STATES : td_eg_base(3 * missing);
    int m = 2;
    for (uint32_t g = blockIdx.x * warps + warp; g < end; g += gridDim.x * warps) {
        while (m + 1 < TD_EG_SYMBOLS && g >= td_eg_base(m + 1)) ++m;
        const int N = m + 1;
        uint32_t r = g - td_eg_base(m), digits[TD_EG_SYMBOLS];
#pragma unroll
        for (int q = 1; q < TD_EG_SYMBOLS; ++q)
            if (q <= m) {
                digits[q] = r % (uint32_t)q;  // the digit of the q-th symbol from the right
                r /= (uint32_t)q;
            }
        uint64_t L = 0;
        uint32_t U = (1u << m) - 1u;
        int at = 0;
#pragma unroll
        for (int q = TD_EG_SYMBOLS - 1; q >= 1; --q)
            if (q <= m) {
                uint32_t v = U;
                for (uint32_t d = digits[q]; d; --d) v &= v - 1u;
                v &= 0u - v;
                U &= ~v;
                L |= (uint64_t)(31 - __clz((int)v)) << (4 * at++);
            }
        for (; at < 16; ++at) L |= (uint64_t)at << (4 * at);
        __syncwarp();
        td_unpack_state(s, 0, L, 0, N);
        if (td_eg_fixed(s, 0, N)) continue;  // not glued: never looked up
        uint32_t O, F;
        const int odd = td_prepare_rows(s, 0, N, O, F);
        if ((N - odd) / 2 != missing) continue;
        if (pairs_n != N) {
            td_load_pairs(s, N);
            pairs_n = N;
        }
        if (lane == 0) {  // every +2 child, and nothing else, is one to visit
            s.acc[1] = 0;
            s.reach[1] = 1u << (odd + 2);
        }
        __syncwarp();
        td_evaluate(s, N, 0, odd, O, F);
        const uint32_t e = 1u + td_eg_skip(s, 0, N, 0);
        const uint32_t left = __ballot_sync(TD_FULL, lane < TD_MAX_STEPS && s.cw[0][lane] != 0);
        if (lane == 0) td_eg_table[g] = left ? 0 : (uint16_t)e;
    }
}
