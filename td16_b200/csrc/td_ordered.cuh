// td_ordered.cuh -- walks of the reference order that several warps share
// (included by td_kernels.cuh; td_ordered_kernel runs it).
//
// The reference's single-queue order is one depth-first walk, so a search that
// runs long is a long serial chain on one warp while the rest of the GPU idles:
// the tail of an ordered batch.  A walk visits a node's children c_0, c_1, ...
// in a fixed order and exhausts each subtree before the next, so the witness it
// meets is the one of the first subtree that holds any, met there exactly as
// that subtree's own walk meets it.  Its remaining children can therefore be
// searched at once, one warp each, and joined in rank order: the witness is the
// found one of lowest rank r, and the walk's expansion count is the sum over
// ranks 0..r, the earlier ones run to exhaustion.  Both equal the one-warp
// walk's, bit for bit.
//
// While warps of the launch wait, a walk gives away the children not yet
// visited of its shallowest level that has any (td_split) and goes on with the
// subtree it is in: that is rank 0 of the new split node, with all that the
// walk has counted so far, and the children given away are ranks 1, 2, ...
// The warp that completes the last record of a node joins them into the record
// that the walk itself had, and so on up (td_split_complete).  Nothing is
// walked twice, and nothing is split while every warp is busy.  A subtree that
// ranks after a found one stops early; its result is never read.  A child of the
// root that is accepted when visited ends the list: no walk goes past it.
// (Without that rule three of four items of 3,001 partial-sorting pairs were
// such subtrees, and their queue kept the walks from being split again: 1.8 to
// 2.1 ms, now 1.2 to 1.7.)
//
// A walk may be split once it has counted `split_after` expansions, those that
// the endgame table spares it included, since they say how long it will be:
// 16,384 S_12 at bound 6 take 0.68 ms, and 0.82 counting the nodes expanded; 512
// S_14 at their lower bound 0.51 and 0.67 ms.
//
// Splitting each root as soon as its walk had run for 64 expansions instead (a
// launch each for the first pass, the listing, the subtrees and the join) took
// 11 to 31 ms for 3,001 partial-sorting pairs, depending on their longest
// subtree, and 33 ms for 256 S_16 at their lower bound; this takes 1.2 to 1.7
// and 3.4 ms.  In one queue the early split loses where most instances have a
// witness (8,192 near-reverse S_13 at bound 7: 18.6 against 6.9 ms): subtrees
// of high rank then run before the ones that cut them off.
#pragma once

#define TD_SPLIT_SKIPPED 2  // status of a subtree whose result is never read

struct __align__(16) td_split_node {  // 48 bytes
    int inst;
    int parent;      // the node whose record this one's result is, -1 = the instance's result
    int rank;        // and the rank there
    int base;        // its first record
    int nkids;       // records: the walk that was split, then the children it gave away
    int remaining;   // records not yet complete
    int cutoff;      // lowest rank with a witness so far
    uint16_t depth;  // depth of the node whose children were given away
    uint16_t path[TD_MAX_DEPTH];
};

// An item: a child given away.
struct __align__(8) td_split_item {
    int node;
    uint16_t rank;
    uint16_t kid;  // the move to it, bit 15: accepted when visited
};

// One record of node k is complete: the warp that completes a node's last one
// joins them in rank order into the record of the walk that was split, and goes
// on with that one's node.  `out`: the instances' results.
__device__ __noinline__ void td_split_complete(const td_split_space &sp, int k) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        int last = 0;
        if (lane == 0) {
            td_fence();
            last = atomicSub(&sp.nodes[k].remaining, 1) == 1;
        }
        if (!__shfl_sync(TD_FULL, last, 0)) return;
        td_fence();
        const td_split_node *nd = &sp.nodes[k];
        const int base = __ldcg(&nd->base), nkids = __ldcg(&nd->nkids), parent = __ldcg(&nd->parent),
                  rank = __ldcg(&nd->rank), inst = __ldcg(&nd->inst);
        uint64_t exp = 0;
        int status = TD_NOT_FOUND, win = -1;
        for (int r0 = 0; r0 < nkids && win < 0; r0 += 32) {
            const uint32_t *it = reinterpret_cast<const uint32_t *>(&sp.records[base + min(r0 + lane, nkids - 1)]);
            const int st = r0 + lane < nkids ? (int)__ldcg(it) : TD_NOT_FOUND;
            const uint32_t e = r0 + lane < nkids ? __ldcg(it + 7) : 0u;
            // the first found one, or one that timed out before any
            const uint32_t ends = __ballot_sync(TD_FULL, st != TD_NOT_FOUND);
            const int first = ends ? __ffs(ends) - 1 : 31;
            uint64_t part = lane <= first ? e : 0u;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(TD_FULL, part, o);
            exp += part;
            if (ends) {
                win = r0 + first;
                status = __shfl_sync(TD_FULL, st, first) == TD_FOUND ? TD_FOUND : TD_ERR_TIMEOUT;
            }
        }
        td_result *to = parent < 0 ? &sp.out[inst] : &sp.records[__ldcg(&sp.nodes[parent].base) + rank];
        uint32_t word = 0;  // the found record's depth and moves, or none
        if (status == TD_FOUND && lane < 8)
            word = __ldcg(reinterpret_cast<const uint32_t *>(&sp.records[base + win]) + lane);
        if (lane == 0) word = (uint32_t)status;
        if (lane == 7) word = exp > 0xffffffffull ? 0xffffffffu : (uint32_t)exp;
        if (lane < 8) reinterpret_cast<volatile uint32_t *>(to)[lane] = word;
        __syncwarp();
        if (parent < 0) return;
        if (lane == 0 && status == TD_FOUND) atomicMin(&sp.nodes[parent].cutoff, rank);
        td_fence();
        __syncwarp();
        k = parent;
    }
}

// Gives away the children not yet visited of the shallowest level in [d0,
// level] that has any (of `level` itself, whose node was just expanded, all but
// the first).  Children that the endgame table decides become records at once,
// and those after one that it knows to be sorted are dropped (the walk never
// gets there).  Where the table decides all of them the level keeps them: they
// rank after the subtree that the walk is in, so they count only if the walk gets
// to them.  (Counted at once they made the expansions of about one in a thousand
// solved near-reverse instances of n = 13..15 too high.)  No deeper level is
// looked at then: of 9,000 nodes made by walks of n = 12..14, in the host
// restatement, one would lie below such a level.
__device__ __noinline__ void td_split(td_warp_smem &s, int d0, int level, int N) {
    const int lane = threadIdx.x & 31;
    const td_split_space &sp = s.sp;
    int lv = d0;
    uint32_t w = 0;
    for (; lv <= level; ++lv) {
        w = lane < TD_MAX_STEPS ? s.cw[lv][lane] : 0u;
        if (__ballot_sync(TD_FULL, w != 0)) break;
    }
    if (lv > level) return;
    const int last_tri = td_tri_base(N) + td_triple_count(N) - 1;
    const int spare = s.spare[lv];  // 255: the table does not apply
    const uint32_t fixed = td_eg_fixed(s, lv, N);
    uint64_t L;
    int off;
    td_pack_state(s, lv, N, &L, &off);
    const int own = lv == level ? 1 : 0;  // children that this walk keeps
    int c = 0, units = 0;
    for (;;) {
        const int all = td_eg_list(s, lv);
        if (all == 0) break;
        uint32_t e = TD_EG_UNKNOWN;
        if (lane < all) {
            const uint32_t u = s.list[lane];
            const uint32_t t = td_tri_table[last_tri - (int)u];
            const uint32_t accepted = lv == 0 ? (s.root_found[u >> 5] >> (u & 31)) & 1u : 0u;
            if (spare != 255) {
                const bool plus2 = spare == 0 || ((s.cp[lv][u >> 5] >> (u & 31)) & 1u);
                e = td_eg_probe(s, lv, N, L, off, fixed, t, plus2 ? spare == 0 : spare == 1);
            }
            if (accepted) e = 0;  // the walk goes no further than this child
            s.kid[c + lane] = (uint16_t)(t | accepted << 15);
            s.kid_e[c + lane] = (uint16_t)(e == TD_EG_UNKNOWN ? 0xffffu : e);
            if (c + lane >= own) atomicAnd(&s.cw[lv][u >> 5], ~(1u << (u & 31)));
        }
        const uint32_t yes = __ballot_sync(TD_FULL, lane < all && e == 0);
        const int got = yes ? __ffs(yes) : min(all, 32);
        const bool mine = lane < got && c + lane >= own;
        units += __popc(__ballot_sync(TD_FULL, mine && (e == 0 || e == TD_EG_UNKNOWN)));
        c += got;
        __syncwarp();
        if (yes) break;
        if (own && c <= 32 && all > 32) {
            // the first child is still listed first: from here on it is passed over
            if (lane == 0) s.cw[lv][s.list[0] >> 5] &= ~(1u << (s.list[0] & 31));
            __syncwarp();
        }
        if (all <= 32) break;
    }
    // what the level keeps: the walk's own child, or none
    uint32_t keep = 0;
    if (own && lane < TD_MAX_STEPS) {
        // the first child in visiting order
        const uint32_t some = __ballot_sync((1u << TD_MAX_STEPS) - 1u, w != 0);
        const int st = 31 - __clz(some);
        if (lane == st) keep = lv == 0 ? 0x80000000u >> __clz(w) : w & (0u - w);
    }
    int first = -1, k = -1, base = -1;
    if (units > 0 && lane == 0) {
        // looked at first, so that the counts pass their limits by no more than
        // one request per warp
        const int most = s.dc.capacity - (c - own + 1);
        // whether warps still wait: others may have served them meanwhile, and
        // every record that nobody waits for is space lost
        const unsigned long long pc = *(volatile unsigned long long *)&s.dc.pool->produced;
        const bool wanted = (int)(pc >> 32) > (int)(uint32_t)pc;
        if (wanted && *(volatile int *)sp.node_count < sp.max_nodes && *(volatile int *)sp.record_count <= most) {
            k = atomicAdd(sp.node_count, 1);
            if (k < sp.max_nodes) {
                base = atomicAdd(sp.record_count, c - own + 1);
                if (base > most) base = -1;
            }
        }
        if (base >= 0) {  // there are no more items than records
            first = atomicAdd(&s.dc.pool->produced, units);
            td_split_node nd;
            nd.inst = s.sp_inst;
            nd.parent = s.sp_node;
            nd.rank = s.sp_rank;
            nd.base = base;
            nd.nkids = c - own + 1;
            nd.remaining = units + 1;
            nd.cutoff = 0x7fffffff;
            nd.depth = (uint16_t)lv;
            for (int q = 0; q < TD_MAX_DEPTH; ++q) nd.path[q] = q < lv ? s.path[q] : 0;
            sp.nodes[k] = nd;
            atomicAdd(&s.dc.pool->outstanding, units);
        }
    }
    base = __shfl_sync(TD_FULL, base, 0);
    if (base < 0) {  // all decided, or no room: the walk keeps its children
        if (lane < TD_MAX_STEPS) s.cw[lv][lane] = w;
        __syncwarp();
        return;
    }
    if (lane < TD_MAX_STEPS) s.cw[lv][lane] = keep;
    __syncwarp();
    first = __shfl_sync(TD_FULL, first, 0);
    k = __shfl_sync(TD_FULL, k, 0);
    // until the join, the instance reads as timed out
    if (s.sp_node < 0 && lane < 8)
        reinterpret_cast<volatile uint32_t *>(&sp.out[s.sp_inst])[lane] = lane == 0 ? (uint32_t)TD_ERR_TIMEOUT : 0u;
    int at = first;
    for (int r0 = own; r0 < c; r0 += 32) {
        const int r = r0 + lane;
        const uint32_t e = r < c ? s.kid_e[r] : 1u;
        const bool unit = e == 0 || e == 0xffffu;
        const uint32_t m = __ballot_sync(TD_FULL, unit);
        if (unit) {
            td_split_item it;
            it.node = k;
            it.rank = (uint16_t)(r - own + 1);
            it.kid = s.kid[r];
            sp.items[at + __popc(m & ((1u << lane) - 1u))] = it;
        } else if (r < c) {  // exhausted
            uint4 *to = reinterpret_cast<uint4 *>(&sp.records[base + r - own + 1]);
            to[0] = make_uint4((uint32_t)TD_NOT_FOUND, 0u, 0u, 0u);
            to[1] = make_uint4(0u, 0u, 0u, e);
        }
        at += __popc(m);
    }
    td_fence();
    __syncwarp();
    td_fence();
    for (int i = first + lane; i < first + units; i += 32) *(volatile uint32_t *)&s.dc.ready[i] = s.dc.epoch;
    __syncwarp();
    if (lane == 0) {
        s.sp_node = k;
        s.sp_rank = 0;
    }
    __syncwarp();
}
