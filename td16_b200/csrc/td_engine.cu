// td_engine.cu -- kernels and host C ABI of the B200 witness-search engine.
//
// Kernels
//   td_plain_kernel       one warp per instance, one launch per batch
//   td_steal_kernel       free order: resident grid; instances by ticket, then
//                         the subtrees that busy warps give away
//   td_ordered_kernel     reference order: the same, with the subtrees joined in
//                         the walk's order (td_ordered.cuh)
//   td_persistent_kernel  reference order, one warp per walk: batches with an
//                         expansion budget or the split off, and the
//                         allocation-free entry
//   td_serve_kernel       requests as they arrive (td_serve.cuh, td_percall.cuh)
//   td_eg_build_kernel    the endgame table, once per device (td_endgame.cuh)
//   td_pairs_*_kernel     pairs to instances and results to triples
//   td_validate_kernel    replays witnesses in pinned form
// Host
//   slots (stream + completion event + device scratch per slot) with the
//   reference's initSlots / searchForSortingSeq semantics, batch entry points,
//   instance preparation and the seeded synthetic generator.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <thread>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "td_kernels.cuh"

#define TD_API extern "C" __attribute__((visibility("default")))

// mirrors include/td16_b200.h
#define TD_OK 0
#define TD_NOT_FOUND_RC 1
#define TD_OVERFLOW 2
#define TD_CUDA_ERROR 3
#define TD_INVALID_ARG 4
#define TD_TIMEOUT 5
#define TD_FLAG_PLAIN 2u
#define TD_FLAG_VERIFY 4u
#define TD_ERR_VERIFY (-6)

struct td_batch_stats {
    uint64_t expansions, found, not_found, errors;
    float kernel_ms;
    uint32_t launches;
    uint64_t donations, donated_items;
    uint64_t races;
};

static_assert(sizeof(td_instance) == 16, "td_instance layout");
static_assert(sizeof(td_result) == 32, "td_result layout");

// ============================================================================
// kernels
// ============================================================================

// The kernels of one batch follow each other at once (launch_after): the next
// one's blocks are placed while its predecessor ends, and wait here until that
// one has ended and its writes are complete.  Returns at once in a kernel
// launched the ordinary way.
__device__ __forceinline__ void td_wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

#define TD_TT_BITS 12  // default of td_configure_table
// 16-byte entries of the table of explored states per resident warp: 2^(bits -
// TD_TT_DOWN), rounded down to a power of two in all.  64 MiB at the default
// for a whole B200: the L2 keeps it.
#ifndef TD_TT_DOWN
#define TD_TT_DOWN 2
#endif
#define TD_TT_INST_BITS 26  // instances per epoch in the table's search numbers
#define TD_RESTART_BASE 16  // default base of the free order's restart budgets (expansions)

// Sets the warp's limits: no tables, no restarts.
__device__ __forceinline__ void td_set_limits(td_warp_smem &s, uint64_t max_exp, uint64_t time_limit_ns) {
    if ((threadIdx.x & 31) == 0) {
        td_search_limits lim;
        lim.max_expansions = td_budget(max_exp);
        lim.split_after = ~0u;
        lim.deadline_ns = time_limit_ns ? td_globaltimer() + time_limit_ns : 0;
        lim.tt = nullptr;
        lim.tt_id = 0;
        lim.tt_shift = 64;
        lim.restart_base = 0;
        lim.cutoff = lim.cutoff2 = nullptr;
        lim.rank = lim.rank2 = 0;
        s.lim = lim;
        s.pairs_n = -1;
    }
    __syncwarp();
}

template <bool ORDERED>
__global__ void __launch_bounds__(256) td_plain_kernel(const td_instance *__restrict__ in,
                                                      td_result *__restrict__ out, int count,
                                                      uint64_t max_exp, uint64_t time_limit_ns) {
    extern __shared__ __align__(16) uint8_t td_smem[];
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5;
    td_warp_smem *ws = reinterpret_cast<td_warp_smem *>(td_smem);
    const int idx = blockIdx.x * warps + warp;
    if (idx >= count) return;
    td_set_limits(ws[warp], max_exp, time_limit_ns);
    const td_instance x = in[idx];
    td_warp_search<ORDERED>(x, &out[idx], ws[warp]);
}

__global__ void __launch_bounds__(256, 4) td_persistent_kernel(const td_instance *__restrict__ in,
                                                           td_result *__restrict__ out, int count,
                                                           int *ticket, int grain, uint64_t max_exp,
                                                           uint64_t time_limit_ns) {
    extern __shared__ __align__(16) uint8_t td_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    td_warp_smem *ws = reinterpret_cast<td_warp_smem *>(td_smem);
    td_set_limits(ws[warp], max_exp, time_limit_ns);
    for (;;) {
        int first = 0;
        if (lane == 0) first = atomicAdd(ticket, grain);
        first = __shfl_sync(TD_FULL, first, 0);
        if (first >= count) break;
        const int last = min(count, first + grain);
        for (int idx = first; idx < last; ++idx) {
            const td_instance x = in[idx];
            td_warp_search<true>(x, &out[idx], ws[warp]);
        }
    }
}

// A launch's epoch (td_epoch_kernel) and when it began.
struct td_epoch {
    uint32_t epoch, pad;
    uint64_t start_ns;
};

// ---- claiming work --------------------------------------------------------------
//
// How the warps of a launch share instances and items (td_steal_kernel,
// td_ordered_kernel).  A warp takes fresh instances by ticket while any are
// left, then one item ticket (fetch-and-add: it never fails) and waits for its
// item: item i belongs to ticket i.  A waiting warp polls only the ready flag
// of its own item, so thousands of them load thousands of different words and
// none that a busy warp needs, and they can poll often.  `outstanding` counts
// the instances in progress plus the items not yet finished: it is raised
// before an instance ticket is taken and before items can be claimed, and
// lowered when a unit ends.  With no instance ticket left and nothing
// outstanding no unit can start again: the warp that brings the count there
// sets `done` and then ~epoch in the flag of every ticket taken.  A warp that
// took its ticket too late for that reads `done` at its first poll and at every
// 16th.  Every wait ends at the launch deadline.
//
// Polling the shared counters instead (five of them, at up to 32 us
// intervals, since shorter ones slowed the busy warps) left the warps idle for
// most of a launch's tail.
struct td_claims {
    td_pool *pool;
    uint32_t *ready;
    uint32_t epoch;
    int count, capacity;
    int my_ticket;  // lane 0: this warp's item ticket, -1 = none
    bool fresh;     // lane 0: instance tickets may be left

    // Wakes the waiting warps of a launch without work.
    __device__ __forceinline__ void wake() {
        const int lane = threadIdx.x & 31;
        int from = 0, taken = 0;
        if (lane == 0) {
            from = *(volatile int *)&pool->produced;
            taken = min(*(volatile int *)&pool->consumed, capacity);
        }
        from = __shfl_sync(TD_FULL, from, 0);
        taken = __shfl_sync(TD_FULL, taken, 0);
        for (int i = from + lane; i < taken; i += 32) *(volatile uint32_t *)&ready[i] = ~epoch;
    }

    // Ends the unit before, if any, and claims the next one: 1 an instance, 2 an
    // item, 0 no work left (uniform across the warp).
    __device__ __forceinline__ int next(td_warp_smem &s, bool first, int *unit_out) {
        const int lane = threadIdx.x & 31;
        unsigned backoff = 64, polls = 0;
        for (;;) {
            int kind = 0, unit = -1;
            if (lane == 0) {
                // both atomics are under way before either result is used
                const int before = first ? 0 : atomicSub(&pool->outstanding, 1);
                first = true;
                if (fresh) {
                    unit = atomicAdd(&pool->inst_ticket, 1);
                    if (unit < count) kind = 1;
                    else fresh = false;
                }
                if (before == 1) {
                    atomicExch(&pool->done, 1);
                    __threadfence();
                    kind = 4;
                }
                if (!kind) {
                    if (my_ticket < 0) {
                        my_ticket = atomicAdd(&pool->consumed, 1);
                        td_serve_idle_warps(s.dc);
                    }
                    const uint32_t flag = my_ticket < capacity ? *(volatile uint32_t *)&ready[my_ticket] : 0u;
                    if (flag == epoch) {
                        kind = 2;
                        unit = my_ticket;
                        my_ticket = -1;
                    } else if (flag == ~epoch) {
                        kind = 3;
                    } else if ((polls++ & 15u) == 0) {
                        if (*(volatile int *)&pool->done) {
                            kind = 3;
                        } else if (s.lim.deadline_ns && td_globaltimer() > s.lim.deadline_ns) {
                            atomicCAS(&pool->error, 0, TD_ERR_TIMEOUT);
                            kind = 3;
                        }
                    }
                }
            }
            kind = __shfl_sync(TD_FULL, kind, 0);
            if (kind == 4) wake();
            if (kind >= 3) return 0;
            if (kind) {
                *unit_out = __shfl_sync(TD_FULL, unit, 0);
                if (kind == 2) td_fence();
                return kind;
            }
            __nanosleep(backoff);
            backoff = min(backoff * 2u, 1024u);
        }
    }
};

#define TD_SPLIT_BUDGET 64          // default expansions of a walk before it may be split (td_configure_split)
#define TD_SPLIT_RECORDS (1 << 20)  // default subtree records per launch

// Resident grid of the reference order: instances by ticket, then the subtrees
// that long walks give away (td_ordered.cuh).
__global__ void __launch_bounds__(256, 4) td_ordered_kernel(const td_instance *__restrict__ in,
                                                        td_result *__restrict__ out, int count, td_pool *pool,
                                                        td_split_space sp, uint32_t *ready, const td_epoch *ep,
                                                        int capacity, int split_after, uint64_t time_limit_ns) {
    extern __shared__ __align__(16) uint8_t td_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    td_warp_smem &s = reinterpret_cast<td_warp_smem *>(td_smem)[warp];
    td_set_limits(s, 0, time_limit_ns);
    td_wait_predecessor();
    if (lane == 0) {
        s.dc.pool = pool;
        s.dc.ready = ready;
        s.dc.epoch = ep->epoch;
        if (time_limit_ns) s.lim.deadline_ns = ep->start_ns + time_limit_ns;
        s.dc.capacity = capacity;
        s.dc.idle_seen = 1;
        s.dc.check_every = 8;
        s.sp = sp;
    }
    __syncwarp();
    td_claims cl;
    cl.pool = pool;
    cl.ready = ready;
    cl.epoch = s.dc.epoch;
    cl.count = count;
    cl.capacity = capacity;
    cl.my_ticket = -1;
    cl.fresh = true;
    for (bool first = true;; first = false) {
        int unit;
        const int kind = cl.next(s, first, &unit);
        if (!kind) return;
        int inst = unit, node = -1, rank = 0, d0 = 0, stop = 0;
        uint32_t kid = 0;
        const td_split_node *nd = nullptr;
        if (kind == 2) {
            const uint2 w = __ldcg(reinterpret_cast<const uint2 *>(&sp.items[unit]));
            node = (int)w.x;
            rank = (int)(w.y & 0xffffu);
            kid = w.y >> 16;
            nd = &sp.nodes[node];
            inst = __ldcg(&nd->inst);
            d0 = (int)__ldcg(&nd->depth) + 1;
        }
        const td_instance x = in[inst];
        const int N = x.n_symbols;
        td_dfs_out r;
        r.status = TD_DFS_EXHAUSTED;
        r.depth = 0;
        r.found_move = 0;
        r.expansions = 0;
        if (lane == 0) {
            s.sp_inst = inst;
            s.sp_node = node;
            s.sp_rank = rank;
            // a first walk is split after split_after expansions, one that was given
            // away sooner
            s.lim.split_after = (uint32_t)(kind == 2 ? split_after / 8 : split_after);
            s.lim.cutoff = s.lim.cutoff2 = nullptr;
        }
        __syncwarp();
        if (td_instance_ok(x) && td_triple_count(N) > 0) {
            td_setup_root(s, x);
            if (kind == 2) {
                // the moves to the subtree
                uint64_t L = x.perm;
                int off = x.offset;
                for (int d = 0; d < d0; ++d) {
                    const uint32_t t = d == d0 - 1 ? kid & 0x7fffu : (uint32_t)__ldcg(&nd->path[d]);
                    td_apply_move(L, off, N, t & 31, (t >> 5) & 31, (t >> 10) & 31, &L, &off);
                    if (lane == 0) s.path[d] = (uint16_t)t;
                }
                if (lane == 0) {
                    s.L[d0] = L;
                    s.off[d0] = (uint8_t)off;
                    // skipped where a lower rank of its node, or of a node further
                    // up, has a witness; the search goes on looking at two of them
                    int k = node, rk = rank;
                    for (int up = 0; k >= 0 && up < 16; ++up) {
                        const td_split_node *q = &sp.nodes[k];
                        if (rk > 0) {
                            if (*(volatile const int *)&q->cutoff < rk) stop = 1;
                            if (!s.lim.cutoff) {
                                s.lim.cutoff = &q->cutoff;
                                s.lim.rank = rk;
                            } else if (!s.lim.cutoff2) {
                                s.lim.cutoff2 = &q->cutoff;
                                s.lim.rank2 = rk;
                            }
                        }
                        rk = __ldcg(&q->rank);
                        k = __ldcg(&q->parent);
                    }
                    // a walk looks at the deadline every 256 nodes, more than
                    // most subtrees have
                    if (!stop && s.lim.deadline_ns && td_globaltimer() > s.lim.deadline_ns) stop = 2;
                }
                stop = __shfl_sync(TD_FULL, stop, 0);
                __syncwarp();
            }
            if (stop) {
                r.status = stop == 2 ? TD_DFS_TIMEOUT : TD_DFS_ABORTED;
            } else if (kid & 0x8000u) {  // accepted when visited: the one-move witness
                r.status = TD_DFS_FOUND;
                r.depth = 1;
                r.found_move = (uint16_t)(kid & 0x7fffu);
            } else {
                r = td_dfs<true>(s, N, d0, true);
            }
        }
        int status = r.status == TD_DFS_ABORTED ? TD_SPLIT_SKIPPED : td_status_of_dfs(r.status);
        if (kind == 1 && !td_instance_ok(x)) status = TD_ERR_ARG;
        __syncwarp();
        node = s.sp_node;  // the walk may have been split
        rank = s.sp_rank;
        td_result *to = node < 0 ? &out[inst] : &sp.records[__ldcg(&sp.nodes[node].base) + rank];
        td_write_result(to, status, r.depth, r.found_move, s.path, r.expansions, 0, 8);
        if (node >= 0) {
            if (lane == 0 && status == TD_FOUND) atomicMin(&sp.nodes[node].cutoff, rank);
            td_fence();
            __syncwarp();
            td_split_complete(s.sp, node);
        }
    }
}

// Records the first error of a search.
__device__ __forceinline__ void td_note_error(td_inst_state *st, int err) {
    atomicCAS(reinterpret_cast<unsigned short *>(&st->error), (unsigned short)0, (unsigned short)err);
}

// HOST_OUT: `out` is host memory mapped into the device (the serving loop), so
// the fences are system-scope; the batch engine's results are device memory,
// where device-scope fences order the same writes at a fraction of the cost.
template <bool HOST_OUT>
__device__ __forceinline__ void td_unit_fence() {
    if (HOST_OUT) __threadfence_system();
    else td_fence();
}

// Ends one unit of a shared search: records a found witness (first finder
// wins), and the unit that finishes the search last writes the final status
// and the summed expansions.  Returns 1 in the warp that finished last.
// `side` 1 marks a unit of the inverse instance's search (td_steal_kernel's
// race; its witness is already in the instance's positions and keeps the
// reference's move filter there).  When the last unit of the instance's own
// side ends with no witness and no error recorded, its whole filtered tree
// was searched: the instance has no witness within the bound, and found = 2
// stops the inverse's side.  The inverse's side never decides "no witness":
// the filter applies to a different tree there.
template <bool HOST_OUT>
__device__ __forceinline__ int td_finish_unit(const td_dfs_out &r, td_inst_state *st, td_result *out,
                                              const uint16_t *path, int side, int gave) {
    const int lane = threadIdx.x & 31;
    if (!gave) {  // a root search by itself: its outcome is the instance's
        const int status = td_status_of_dfs(r.status);
        td_write_result(out, status, status == TD_FOUND ? r.depth : 0, r.found_move, path, r.expansions, 0, 8);
        __syncwarp();
        if (HOST_OUT && lane == 0) __threadfence_system();
        return 1;
    }
    int win = 0, last = 0;
    if (lane == 0) {
        atomicAdd(&st->expansions, r.expansions);
        if (r.status == TD_DFS_FOUND) win = atomicCAS(&st->found, (unsigned short)0, (unsigned short)1) == 0;
        const int err = r.status == TD_DFS_TIMEOUT ? TD_ERR_TIMEOUT : r.status == TD_DFS_BUDGET ? TD_ERR_BUDGET : 0;
        if (err) td_note_error(st, err);
    }
    win = __shfl_sync(TD_FULL, win, 0);
    if (win) td_write_result(out, TD_FOUND, r.depth, r.found_move, path, 0, 0, 7);
    __syncwarp();
    if (lane == 0) {
        td_unit_fence<HOST_OUT>();
        const unsigned long long unit = side ? TD_UNIT_INVERSE : 1ull;
        const unsigned long long before = atomicAdd(&st->pending, 0ull - unit);
        last = before == unit;
        if (last) td_unit_fence<HOST_OUT>();
        else if (!side && (uint32_t)before == 1u && *(volatile unsigned short *)&st->found == 0 &&
                 *(volatile short *)&st->error == 0)
            atomicCAS(&st->found, (unsigned short)0, (unsigned short)2);
    }
    last = __shfl_sync(TD_FULL, last, 0);
    if (last) {
        int found = 0, err = 0;
        unsigned exp = 0;
        if (lane == 0) {
            found = *(volatile unsigned short *)&st->found;
            err = *(volatile short *)&st->error;
            exp = *(volatile unsigned *)&st->expansions;
        }
        found = __shfl_sync(TD_FULL, found, 0);
        err = __shfl_sync(TD_FULL, err, 0);
        exp = __shfl_sync(TD_FULL, exp, 0);
        if (found == 1) td_write_result(out, TD_FOUND, 0, 0, path, exp, 7, 8);
        else td_write_result(out, found == 2 || !err ? TD_NOT_FOUND : err, 0, 0, path, exp, 0, 8);
        __syncwarp();
        // the caller stamps the record as done: the host must see the record
        // (written by lanes 0..7) before the stamp, or it reads the ring
        // slot's record of an earlier request
        if (HOST_OUT && lane == 0) __threadfence_system();
    }
    return last;
}

#define TD_EAGER_UNITS 16  // instances per warp up to which a launch shares its searches from the start

#ifndef TD_STEAL_MIN_BLOCKS
#define TD_STEAL_MIN_BLOCKS 4  // resident blocks of 8 warps per SM the register budget is sized for
#endif
// Resident grid with work donation (free move order).  Warps take fresh
// instances by ticket, then items (td_claims): while item tickets run ahead of
// the items produced, busy warps hand the remaining children of their
// shallowest DFS level to the item array.  Every wait is bounded by the launch
// deadline; the launch ends when no ticket, item or unit is left.
__global__ void __launch_bounds__(256, TD_STEAL_MIN_BLOCKS) td_steal_kernel(const td_instance *__restrict__ in,
                                                      td_result *__restrict__ out, int count, td_pool *pool,
                                                      td_item *items, uint32_t *ready, const td_epoch *ep,
                                                      int capacity, td_inst_state *state, int grain,
                                                      int max_level, int check_every, uint64_t time_limit_ns,
                                                      ulonglong2 *tt, int tt_shift, unsigned epochs,
                                                      uint32_t restart_base, uint64_t max_exp,
                                                      int race) {
    extern __shared__ __align__(16) uint8_t td_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    td_warp_smem *ws = reinterpret_cast<td_warp_smem *>(td_smem);
    td_warp_smem &s = ws[warp];
    // the expansion budget bounds each unit (the root search and each donated
    // subtree); an instance without a witness whose unit ran out reports
    // TD_ERR_BUDGET
    td_set_limits(s, max_exp, time_limit_ns);
    td_wait_predecessor();
    const uint32_t epoch = ep->epoch;  // bumped by td_epoch_kernel before this launch
    if (lane == 0) {
        if (time_limit_ns) s.lim.deadline_ns = ep->start_ns + time_limit_ns;
        // this launch's numbers in the table: its `epochs` epochs, 2^26 searches each
        s.lim.tt_id = (uint64_t)(epoch - epochs + 1u) << TD_TT_INST_BITS;
        s.lim.tt_shift = tt_shift;
        td_donate_ctx dc;
        dc.pool = pool;
        dc.items = items;
        dc.ready = ready;
        dc.epoch = epoch;
        dc.capacity = capacity;
        dc.grain = grain;
        dc.max_level = max_level;
        dc.check_every = check_every > 0 ? check_every : 1;
        dc.ring = 0;
        dc.tickets = 1;
        dc.deadline_ns = s.lim.deadline_ns;
        dc.inst = 0;
        dc.state = nullptr;
        dc.side = 0;
        dc.attempt = 0;
        dc.gave = 0;
        dc.race = 0;
        dc.step = 3;
        dc.idle_after = 0;
        dc.idle_seen = 0;
        s.dc = dc;
        // Few instances per warp: most of the launch is its tail, in which a few
        // long searches are all that is left, and giving subtrees away late
        // costs more than doing it too often.  With up to 16 instances a warp
        // the settings for idle warps hold from the start (only with fewer
        // instances than warps before: 20,011 S_12..S_14 2.13 -> 1.49 ms, 2^16
        // mixed 1.69 -> 1.32, 8,000 S_13 1.16 -> 0.82).  Without them and with
        // them, at 8, 16, 20 and 32 instances a warp: near-reverse S_16 2.22/2.01,
        // 3.32/3.16, 3.90/3.75 and 5.88/5.72 ms, the mix of S_11..S_13 1.28/0.93,
        // 1.78/1.29, 2.15/1.57 and 2.92/2.35, uniform S_16 0.35/0.36, 0.56/0.59,
        // 0.73/0.70 and 1.11/1.10.  So the line is not where the two cross: it
        // was drawn at 10^5 uniform S_16, 21 a warp in 8-warp blocks, where the
        // loads of the idle checks are work that nothing waits for (0.79 ms
        // against 0.75), and uneven batches above it would still gain.
        // An expansion budget bounds each unit, so sharing multiplies it: where it
        // ends before a search's first look at the idle warps, nothing is shared
        // and it bounds the instance (16 expansions each, 4,096 of S_8..S_13:
        // 0.25 ms and 23,000 expansions, shared 0.38 and 62,000).
        if (count <= TD_EAGER_UNITS * (int)(gridDim.x * (blockDim.x >> 5)) &&
            (max_exp == 0 || max_exp > (uint64_t)check_every))
            td_serve_idle_warps(s.dc);
    }
    __syncwarp();
    // Race (`race` = a, 0: off): a root search of a full-sorting instance
    // that starts its restart attempt a queues the instance's inverse
    // (td_spawn_inverse) as an item.  While fresh instances remain every warp
    // is busy, and a second search of an instance would only displace other
    // work; at the end of the launch, where warps idle, it shortens the
    // longest searches.  Most queued inverses belong to instances decided by
    // then and end at once.
    td_claims cl;
    cl.pool = pool;
    cl.ready = ready;
    cl.epoch = epoch;
    cl.count = count;
    cl.capacity = capacity;
    cl.my_ticket = -1;
    cl.fresh = true;
    for (bool first = true;; first = false) {
        int unit;
        const int kind = cl.next(s, first, &unit);
        if (!kind) return;
        // the unit: a fresh instance, a donated subtree or a queued inverse root
        uint32_t idx = (uint32_t)unit;
        int d0 = 0, side = 0, attempt = 0;
        td_item it;
        if (kind == 2) {
            const uint4 *src = reinterpret_cast<const uint4 *>(&items[unit]);
            uint4 *dst = reinterpret_cast<uint4 *>(&it);
            dst[0] = __ldcg(src);  // read through L2: the donor wrote it from another SM
            dst[1] = __ldcg(src + 1);
            idx = it.inst;
            d0 = it.depth & 15;
            side = it.depth >> 7;
            attempt = ((it.depth >> 4) & 7) | ((it.off >> 5) << 3);
        }
        // an item names an instance of this launch and a level of the frame;
        // one that does not is a launch error, never followed
        if (kind == 2 && (idx >= (uint32_t)count || d0 >= TD_MAX_DEPTH || (d0 == 0 && !side))) {
            if (lane == 0) atomicCAS(&pool->error, 0, TD_ERR_VERIFY);
        } else {
            const td_instance x = in[idx];
            td_inst_state *st = &state[idx];
            // other warps see it only through items, published after a fence
            if (kind == 1 && lane == 0) *reinterpret_cast<uint4 *>(st) = make_uint4(0u, 0u, 0u, 0u);
            if (kind == 1 && (!td_instance_ok(x) || td_triple_count(x.n_symbols) == 0)) {
                td_write_result(&out[idx], td_instance_ok(x) ? TD_NOT_FOUND : TD_ERR_ARG, 0, 0, s.path, 0, 0, 8);
            } else {
                int stop = 0;
                if (lane == 0) {
                    if (kind == 2) {
                        // a search looks at the deadline every 256 expansions,
                        // more than most donated subtrees have
                        stop = *(volatile unsigned short *)&st->found != 0;
                        if (!stop && s.lim.deadline_ns && td_globaltimer() > s.lim.deadline_ns) stop = 2;
                    }
                    // a donated subtree is searched once, to the end: restarting
                    // it would only repeat work when it holds no witness; the
                    // root of an inverse instance restarts like any root search
                    s.lim.restart_base = d0 > 0 ? 0u : restart_base;
                    // a unit that may run out of its expansion budget leaves
                    // recorded states unsearched: then only roots use the table
                    s.lim.tt = d0 > 0 && max_exp ? nullptr : tt;
                    s.dc.inst = idx;
                    s.dc.state = st;
                    s.dc.side = side;
                    s.dc.attempt = attempt;
                    s.dc.gave = kind == 2;
                    s.dc.race = kind == 1 && td_inst_full(x) ? race : 0;
                }
                td_setup_root(s, x);
                if (kind == 2) {
                    if (lane == 0) {
                        s.L[d0] = it.L;
                        s.off[d0] = it.off & 31;
                        for (int d = 0; d < d0; ++d) s.path[d] = it.path[d];
                    }
                    __syncwarp();
                    stop = __shfl_sync(TD_FULL, stop, 0);
                    // a donated state that another unit took up needs no second search
                    if (!stop && d0 > 0 && s.lim.tt) {
                        td_unpack_state(s, d0, it.L, it.off & 31, x.n_symbols);
                        stop = td_tt_visit(s, d0, x.n_symbols, idx, (uint32_t)(side << 6 | attempt));
                    }
                } else {
                    stop = 0;
                }
                td_dfs_out r;
                r.status = stop == 2 ? TD_DFS_TIMEOUT : TD_DFS_ABORTED;
                r.depth = 0;
                r.found_move = 0;
                r.expansions = 0;
                if (!stop) r = td_dfs<false>(s, x.n_symbols, d0, true);
                // the unit's names come from shared memory again: registers
                // are what the search is short of
                td_inst_state *us = s.dc.state;
                if (s.dc.side && r.status == TD_DFS_FOUND) {
                    const int t = td_inverse_witness(s, in[s.dc.inst], r.depth, r.found_move);
                    if (t < 0) r.status = TD_DFS_EXHAUSTED;
                    else r.found_move = (uint16_t)t;
                    if (t == -1 && lane == 0) td_note_error(us, TD_ERR_VERIFY);
                }
                td_finish_unit<false>(r, us, &out[s.dc.inst], s.path, s.dc.side, s.dc.gave);
            }
        }
    }
}

// Clears the items' flags and the table (td_epoch_kernel; called, so that the
// kernel, which every launch waits for, stays as short as it is without it).
__device__ __noinline__ void td_clear_tags(uint32_t *ready, int n_ready, ulonglong2 *tt, size_t n_tt) {
    for (int i = 0; i < n_ready; ++i) ready[i] = 0;
    for (size_t i = 0; i < n_tt; ++i) tt[i] = make_ulonglong2(0ull, 0ull);
}

// The first operation of a launch: sets its counters, and its deadline counts
// from here, so that it holds for the growth of the launch's buffers too.
// Advances the launch epoch that tags donated items as written; a launch
// replayed from a CUDA graph therefore never mistakes an item of an earlier
// launch for one of its own.  A launch of more than 2^26 instances takes as
// many epochs as it needs numbers in the table of explored states.  Where the
// epochs start again, the items' flags and the table are cleared (by this one
// thread: it happens once in 2^31 launches).
__global__ void td_epoch_kernel(td_epoch *ep, unsigned epochs, td_pool *pool, int count, int *zeros, int n_zeros,
                                uint32_t *ready, int n_ready, ulonglong2 *tt, size_t n_tt) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    int again;
    ep->epoch = td_next_epoch(ep->epoch, epochs, &again);
    if (again) td_clear_tags(ready, n_ready, tt, n_tt);
    ep->start_ns = td_globaltimer();
    td_pool p;
    memset(&p, 0, sizeof p);
    p.outstanding = count;
    *pool = p;
    for (int i = 0; i < n_zeros; ++i) zeros[i] = 0;
}

// Runs after td_steal_kernel on the same stream.  When a bounded wait of the
// launch gave up (pool->error), some instances may have no result record: one
// never claimed, or one whose donated subtree a taker never received (its
// pending count stays above zero, so no unit wrote the final status).  Those
// get a timeout record, so a caller never reads a stale record of an earlier
// launch.  Without an error every thread returns at once.
__global__ void __launch_bounds__(256) td_finalize_kernel(const td_pool *__restrict__ pool,
                                                          const td_inst_state *__restrict__ state,
                                                          td_result *__restrict__ out, int count) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    td_wait_predecessor();
    if (*(volatile const int *)&pool->error == 0) return;
    const int claimed = min(count, *(volatile const int *)&pool->inst_ticket);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        if (i < claimed && state[i].pending == 0) continue;
        td_result r;
        r.status = TD_ERR_TIMEOUT;
        r.depth = 0;
        for (int m = 0; m < TD_MAX_DEPTH; ++m) r.moves[m] = 0;
        r.reserved = 0;
        r.expansions = i < claimed ? state[i].expansions : 0;
        out[i] = r;
    }
}

// The totals of td_batch_stats, reduced on the device so that the host does
// not walk the result array (2^20 results are 32 MiB of host memory).  Reads
// only the status and expansion words of each record.
struct td_counts {
    unsigned long long expansions, found, not_found, errors;
};

__global__ void __launch_bounds__(256) td_count_kernel(const td_result *__restrict__ res, int count,
                                                       td_counts *__restrict__ c) {
    unsigned long long e = 0;
    uint32_t f = 0, nf = 0, er = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const int st = res[i].status;
        e += res[i].expansions;
        f += st == TD_FOUND;
        nf += st == TD_NOT_FOUND;
        er += st != TD_FOUND && st != TD_NOT_FOUND;
    }
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(TD_FULL, e, o);
    f = __reduce_add_sync(TD_FULL, f);
    nf = __reduce_add_sync(TD_FULL, nf);
    er = __reduce_add_sync(TD_FULL, er);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&c->expansions, e);
        atomicAdd(&c->found, (unsigned long long)f);
        atomicAdd(&c->not_found, (unsigned long long)nf);
        atomicAdd(&c->errors, (unsigned long long)er);
    }
}

// Witness replay in pinned form, the rule of td_witness_ok: every move is an
// in-range position triple i<j<k, there are at most max_moves of them, and the
// last node passes the acceptance test of the instance (satisfies_rate,
// sorting_search.cu:336-346: with full sorting, omega = id).  With full sorting
// this is CertificateValidator's replay (CertificateValidator.java:14-50) in
// pinned form plus the rate test.  The search's move filter is not part of it.
// One thread per instance, 16-byte loads where the buffers allow them.  With full sorting
// the witness holds when the pinned state ends sorted and the last move's depth
// passes the rate test, and the moves are taken from registers in an unrolled
// loop.  (Through td_witness_ok, whose arrays the compiler keeps in local
// memory, 10^6 witnesses of S_16 took 51 us, here 33 us.)  Partial sorting
// counts cycles (td_witness_ok).
__device__ __noinline__ int td_witness_ok_any(td_instance x, td_result r) { return td_witness_ok(x, r); }

__global__ void __launch_bounds__(256) td_validate_kernel(const td_instance *__restrict__ in,
                                                          td_result *__restrict__ res, uint8_t *__restrict__ ok,
                                                          int count, int mark) {
    td_wait_predecessor();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= count) return;
    td_instance x;
    uint4 r0, r1;
    if (((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(res)) & 15u) == 0) {
        const uint4 xw = reinterpret_cast<const uint4 *>(in)[idx];
        r0 = reinterpret_cast<const uint4 *>(res)[2 * (size_t)idx];
        r1 = reinterpret_cast<const uint4 *>(res)[2 * (size_t)idx + 1];
        x.perm = (uint64_t)xw.y << 32 | xw.x;
        x.min_rate = __uint_as_float(xw.z);
        x.n_symbols = (uint8_t)xw.w;
        x.offset = (uint8_t)(xw.w >> 8);
        x.max_moves = (uint8_t)(xw.w >> 16);
        x.packed = (uint8_t)(xw.w >> 24);
    } else {  // the records' own alignment is 8 and 4 bytes
        x = in[idx];
        const uint32_t *r = reinterpret_cast<const uint32_t *>(res) + 8 * (size_t)idx;
        r0 = make_uint4(r[0], r[1], r[2], r[3]);
        r1 = make_uint4(r[4], r[5], r[6], r[7]);
    }
    const int status = (int)r0.x, depth = (int)r0.y;
    const uint32_t moves[5] = {r0.z, r0.w, r1.x, r1.y, r1.z};
    const int N = x.n_symbols;
    int good = status == TD_FOUND && depth >= 1 && depth <= x.max_moves && depth <= TD_MAX_DEPTH && N >= 3 &&
               N <= TD_MAX_N;
    if (good && !td_inst_full(x)) {
        td_result r;
        r.status = status;
        r.depth = depth;
#pragma unroll
        for (int d = 0; d < TD_MAX_DEPTH; ++d) r.moves[d] = (uint16_t)(moves[d >> 1] >> (16 * (d & 1)));
        good = td_witness_ok_any(x, r);
    } else if (good) {
        // the caller's array without label 0, one nibble per label, and label
        // 0's place: a block swap is one of nibbles with the cuts past the 0
        // moved down by one, and needs no rotation (td_apply_move's pinned form
        // does)
        const int n = N - 1;
        const uint64_t mask = ~0ull >> (64 - 4 * n);
        const uint64_t sorted = 0xfedcba9876543210ull;
        int zero = x.offset ? N - x.offset : 0;
        uint64_t L = x.perm & mask;
        if (zero % n) L = ((L << (4 * zero)) | (L >> (4 * (n - zero)))) & mask;
#pragma unroll
        for (int d = 0; d < TD_MAX_DEPTH; ++d) {
            if (d < depth) {
                const uint32_t m = moves[d >> 1] >> (16 * (d & 1));
                const int i = m & 31, j = (m >> 5) & 31, k = (m >> 10) & 31;
                if (!(i < j && j < k && k < N)) { good = 0; break; }
                const int p = i - (zero < i), q = j - (zero < j), r = k - (zero < k);
                zero += zero < i || zero >= k ? 0 : zero < j ? k - j : i - j;
                if (p < q && q < r) {  // else label 0 alone changes places
                    const uint64_t seg = L >> (4 * p);
                    const uint64_t turned = ((seg >> (4 * (q - p))) & (~0ull >> (64 - 4 * (r - q)))) |
                                            (seg << (4 * (r - q)));
                    L ^= ((seg ^ turned) & (~0ull >> (64 - 4 * (r - p)))) << (4 * p);
                }
            }
        }
        if (zero % n) L = (L >> (4 * zero)) | (L << (4 * (n - zero)));
        good = good && ((L ^ sorted) & mask) == 0 && td_accepts(N, td_inst_init(x), x.min_rate, 1, N, depth);
    }
    if (ok) ok[idx] = (uint8_t)good;
    if (mark && status == TD_FOUND && !good) res[idx].status = TD_ERR_VERIFY;
}

// ---- pairs: preparation and results on the device ----------------------------
//
// td_search_pairs hands the caller's arrays over in one copy and takes the
// outputs back in one; the conversions run here.  On the calling thread they
// took 3.5 of the 5.5 ms of a call with 20,011 pairs of n = 12..14.

#define TD_PAIR_SEARCHED (-1000)  // status of a pair that is searched

// The arrays of a call, one after the other (device or pinned host memory).
struct td_pair_arrays {
    int32_t *init, *max_moves;
    float *rate;
    uint8_t *beta, *omega, *n, *full;
    int32_t *status, *depth;
    int16_t *ijk;
};

// One thread per pair: its pinned instance, or its status where there is
// nothing to search (then an instance without moves stands in).
__global__ void __launch_bounds__(128) td_pairs_prepare_kernel(td_pair_arrays a, td_instance *__restrict__ inst,
                                                              int count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    int status = TD_PAIR_SEARCHED;
    td_instance x;
    x.perm = 0;
    x.min_rate = 0.0f;
    x.n_symbols = 0;
    x.offset = 0;
    x.max_moves = 1;
    x.packed = 0;
    const int n = a.n[i], m = a.max_moves[i];
    if (n > TD_MAX_N || m <= 0 || m > TD_MAX_DEPTH) {
        status = TD_INVALID_ARG;
    } else if (td_triple_count(n) == 0) {
        status = TD_NOT_FOUND_RC;
    } else {
        uint8_t b[TD_MAX_N], o[TD_MAX_N];
        for (int q = 0; q < n; ++q) {
            b[q] = a.beta[TD_MAX_N * (size_t)i + q];
            o[q] = a.omega[TD_MAX_N * (size_t)i + q];
        }
        td_instance y;
        if (td_prepare_pair(b, o, n, a.init[i], a.rate[i], m, a.full[i], &y) != 0) status = TD_INVALID_ARG;
        else x = y;
    }
    a.status[i] = status;
    inst[i] = x;
}

// One thread per output triple entry (27 per pair), the first `count` of them
// also for a pair's status and depth.
__global__ void __launch_bounds__(256) td_pairs_unpack_kernel(td_pair_arrays a, const td_result *__restrict__ res,
                                                             int count) {
    const size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= 27 * (size_t)count) return;
    const int i = (int)(at / 27), q = (int)(at % 27);
    const int st = res[i].status, depth = st == TD_FOUND ? res[i].depth : 0;
    // a stand-in instance has no witness
    a.ijk[at] = q / 3 < depth ? (int16_t)((res[i].moves[q / 3] >> (5 * (q % 3))) & 31) : (int16_t)0;
    if (at < (size_t)count) {
        const int s2 = res[at].status;
        a.depth[at] = s2 == TD_FOUND ? res[at].depth : 0;
        if (a.status[at] == TD_PAIR_SEARCHED)
            a.status[at] = s2 == TD_FOUND        ? TD_OK
                           : s2 == TD_NOT_FOUND  ? TD_NOT_FOUND_RC
                           : s2 == TD_ERR_BUDGET ? TD_OVERFLOW
                           : s2 == TD_ERR_TIMEOUT ? TD_TIMEOUT
                                                  : TD_INVALID_ARG;
    }
}

// Integer issue peaks at full occupancy.  Each thread runs `iters` iterations
// of 16 operations over 8 independent chains.  MIX = 0: LOP3 only (ALU pipe
// alone, 16 lanes per SM sub-partition, so at most half a warp instruction per
// clock per sub-partition).  MIX = 1: LOP3 and IMAD alternate (ALU and FMA
// pipes side by side), which can reach one warp instruction per clock per
// sub-partition: the full issue rate.
template <int MIX>
__global__ void __launch_bounds__(256) td_int_peak_kernel(uint32_t *sink, int iters) {
    uint32_t a[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) a[c] = threadIdx.x * 0x9E3779B9u + c * 0x85EBCA6Bu + blockIdx.x;
    const uint32_t m = 0x01000193u | (blockIdx.x << 1);
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                if (MIX && (c & 1))
                    asm volatile("mad.lo.u32 %0, %0, %1, %2;" : "+r"(a[c]) : "r"(m), "r"(a[(c + 3) & 7]));
                else
                    asm volatile("lop3.b32 %0, %0, %1, %2, 0x96;" : "+r"(a[c]) : "r"(a[(c + 1) & 7]), "r"(a[(c + 3) & 7]));
            }
        }
    }
    uint32_t x = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) x ^= a[c];
    if (x == 0x12345678u) sink[blockIdx.x] = x;
}

// ============================================================================
// host side
// ============================================================================

namespace {

struct Slot {
    int device = -1;
    cudaStream_t stream = nullptr;
    cudaEvent_t done = nullptr, t0 = nullptr, t1 = nullptr;
    size_t budget = 0;
    td_instance *d_inst = nullptr;
    td_result *d_res = nullptr;
    td_instance *h_inst = nullptr;
    td_result *h_res = nullptr;
    int *d_ticket = nullptr;
    void *d_batch = nullptr;
    size_t d_batch_bytes = 0;
    // the arrays of td_search_pairs on the device, and the pinned memory
    // (kPairStage bytes) that their copies go through
    uint8_t *d_pairs = nullptr, *h_pairs = nullptr;
    size_t pairs_bytes = 0;
    // donation scratch: pool counters, item array + ready flags, instance state
    td_pool *d_pool = nullptr;
    td_item *d_items = nullptr;
    uint32_t *d_ready = nullptr;
    int item_capacity = 0;
    ulonglong2 *d_tt = nullptr;  // table of explored states
    int tt_log2 = 0, tt_bits = 0;  // log2 of its entries; the setting it was sized for
    td_inst_state *d_state = nullptr;
    size_t state_count = 0;
    td_epoch *d_epoch = nullptr;
    // reference order: the queue's counters, items and flags, the nodes of split
    // walks and the results of their subtrees
    td_pool *d_split_pool = nullptr;  // followed by the node and record counts and the launch epoch
    uint32_t *d_split_ready = nullptr;
    td_split_node *d_nodes = nullptr;
    td_split_item *d_split_items = nullptr;
    td_result *d_split_records = nullptr;
    int split_records = 0;
    // td_batch_stats of host-buffer batches: device totals and their pinned copy
    td_counts *d_counts = nullptr;
    struct HostStats {
        td_counts counts;
        td_pool pool;
    } *h_stats = nullptr;
    int slots_on_device = 1;
    // a batch was captured: buffers that a launch uses stay where they are until
    // the slot goes, and those they outgrew wait in `kept`
    bool captured = false;
    std::vector<void *> kept;
    std::mutex *mu = nullptr;
};

struct DeviceInfo {
    bool ready = false;
    int sms = 0;
    int blocks_per_sm = 0;
    int steal_blocks_per_sm = 0;
};

std::mutex g_mu;
std::vector<Slot> g_slots;
std::vector<DeviceInfo> g_dev;

int g_warps_per_block = 4;
int g_grain = 1;            // instances per ticket (ordered persistent kernel)
// the settings while fresh instances are left; td_serve_idle_warps says what
// they become after that
int g_steal_grain = 4;      // items per donation
int g_split_level = 2;      // donate children of levels <= this
int g_check_every = 64;     // expansions between idle checks
// the same for serving launches, where latency rather than throughput counts
int g_serve_grain = 1;
int g_serve_split_level = 2;
int g_serve_check_every = 32;
int g_tt_bits = TD_TT_BITS;  // log2 entries of the explored-state tables; 0 = no table
uint32_t g_restart_base = TD_RESTART_BASE;  // free-order restart budget base; 0 = no restarts
int g_split_budget = TD_SPLIT_BUDGET;       // reference order: expansions of a walk before a split; 0 = none
int g_split_records = TD_SPLIT_RECORDS;     // reference order: subtree records per launch
int g_race = 8;  // free-order batches: attempt at which a search starts racing its inverse, 0 = off (td_configure_race)

void set_err(char *err, size_t len, const std::string &msg) {
    if (err && len) {
        std::snprintf(err, len, "%s", msg.c_str());
    }
}

std::string cuda_msg(cudaError_t e, const char *file, int line) {
    return std::string(file) + ":" + std::to_string(line) + ": CUDA error " + cudaGetErrorName(e) + " (" +
           cudaGetErrorString(e) + ")";
}

#define TD_CHECK(call)                                                   \
    do {                                                                 \
        cudaError_t e_ = (call);                                         \
        if (e_ != cudaSuccess) {                                         \
            set_err(err, errlen, cuda_msg(e_, __FILE__, __LINE__));      \
            return TD_CUDA_ERROR;                                        \
        }                                                                \
    } while (0)

constexpr size_t TD_SPLIT_HEAD = 256;  // a td_pool, the node and record counts and the epoch
static_assert(sizeof(td_pool) % 8 == 0 && sizeof(td_pool) + 2 * sizeof(int) + sizeof(td_epoch) <= TD_SPLIT_HEAD, "split head");

// Nodes of split walks for `records` subtrees (a split node has more than one
// child nearly always; a walk that finds no node runs whole).
size_t split_nodes(int records) { return (size_t)std::max(1, records / 2); }

constexpr int TD_INSTANCE_WARPS = 4;  // a free-order batch's warps per instance, where the device has them

// log2 of the entries of a table of explored states for `warps` resident warps.
int tt_entries_log2(size_t warps, int bits) {
    int b = 0;
    while (b < 40 && ((size_t)1 << (b + 1)) <= ((warps << bits) >> TD_TT_DOWN)) ++b;
    return std::max(b, 6);
}

size_t smem_bytes(int warps) { return (size_t)warps * sizeof(td_warp_smem); }

std::atomic<uint64_t> g_time_limit_ns{0};

// Launch deadline: td_set_time_limit, else TD16_TIME_LIMIT_S, else 300 s.
uint64_t time_limit_ns() {
    uint64_t v = g_time_limit_ns.load(std::memory_order_relaxed);
    if (v) return v;
    const char *s = std::getenv("TD16_TIME_LIMIT_S");
    double secs = s ? std::atof(s) : 300.0;
    if (!(secs > 0)) secs = 300.0;
    v = (uint64_t)(secs * 1e9);
    g_time_limit_ns.store(v, std::memory_order_relaxed);
    return v;
}

// Loads every kernel of the library on the current device (defined at the
// end of this file).  With lazy module loading a kernel's code would
// otherwise be loaded at its first launch, which may wait for the work
// already on the device, the per-call server's resident launch included.
int preload_kernels(char *err, size_t errlen);

// The launch settings of one launch, read together under g_mu so that a
// concurrent td_configure_* call never hands a launch half of its change.
struct LaunchCfg {
    int warps, grain, steal_grain, split_level, check_every, tt_bits;
    uint32_t restart_base;
    int race;
    int split_budget, split_records;
    int serve_grain, serve_split_level, serve_check_every;
    int sms, steal_blocks_per_sm, blocks_per_sm;  // of the device, for `warps`
};

// Snapshot of the settings and of `device`'s occupancy for them; the device
// must be current and set up (ensure_device).
int launch_cfg(int device, LaunchCfg *c, char *err, size_t errlen) {
    std::lock_guard<std::mutex> g(g_mu);
    c->warps = g_warps_per_block;
    c->grain = g_grain;
    c->steal_grain = g_steal_grain;
    c->split_level = g_split_level;
    c->check_every = g_check_every;
    c->tt_bits = g_tt_bits;
    c->restart_base = g_restart_base;
    c->race = g_race;
    c->split_budget = g_split_budget;
    c->split_records = g_split_records;
    c->serve_grain = g_serve_grain;
    c->serve_split_level = g_serve_split_level;
    c->serve_check_every = g_serve_check_every;
    DeviceInfo &d = g_dev[device];
    const int threads = c->warps * 32;
    if (d.steal_blocks_per_sm == 0) {
        int b = 0;
        TD_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, td_steal_kernel, threads,
                                                               smem_bytes(c->warps)));
        d.steal_blocks_per_sm = std::max(1, b);
    }
    if (d.blocks_per_sm == 0) {
        int b = 0;
        TD_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, td_ordered_kernel, threads,
                                                               smem_bytes(c->warps)));
        d.blocks_per_sm = std::max(1, b);
    }
    c->sms = d.sms;
    c->steal_blocks_per_sm = d.steal_blocks_per_sm;
    c->blocks_per_sm = d.blocks_per_sm;
    return TD_OK;
}

// Fills the tables of the current device, once per device and process: the
// triple and pair-slot tables are uploaded and the endgame table
// (td_endgame.cuh) is built from them in five launches, all on one stream of
// their own, so that they wait for nothing else and each finds what it reads,
// and waited for.  No heap.
constexpr int kTableDevices = 64;
std::mutex g_tables_mu;
bool g_tables_ready[kTableDevices];
uint16_t g_tri[TD_TRI_TABLE];
td_pair_row g_pair_rows[TD_MAX_N + 1][32];

cudaError_t tables_setup(int device, int sms) {
    if (device < 0 || device >= kTableDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> g(g_tables_mu);
    if (g_tables_ready[device]) return cudaSuccess;
    for (int N = 0; N <= TD_MAX_N; ++N) {
        int t = td_tri_base(N);
        for (int i = 0; i < N - 2; ++i)
            for (int j = i + 1; j < N - 1; ++j)
                for (int k = j + 1; k < N; ++k) g_tri[t++] = td_pack_move(i, j, k);
        for (int lane = 0; lane < 32; ++lane) g_pair_rows[N][lane] = td_make_pair_row(N, lane);
    }
    uint32_t bases[TD_EG_SYMBOLS], factorial[TD_EG_SYMBOLS];
    for (int m = 0; m < TD_EG_SYMBOLS; ++m) {
        bases[m] = td_eg_base(m);
        factorial[m] = m ? (uint32_t)m * factorial[m - 1] : 1u;
    }
    cudaStream_t st;
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e != cudaSuccess) return e;
    const size_t smem = smem_bytes(8);
    e = cudaFuncSetAttribute(td_eg_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(td_tri_table, g_tri, sizeof g_tri, 0, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbolAsync(td_pair_table, g_pair_rows, sizeof g_pair_rows, 0, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(td_eg_bases, bases, sizeof bases, 0, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbolAsync(td_eg_factorial, factorial, sizeof factorial, 0, cudaMemcpyHostToDevice, st);
    for (int missing = 1; e == cudaSuccess && missing <= TD_EG_SYMBOLS / 2; ++missing) {
        td_eg_build_kernel<<<4 * sms, 256, smem, st>>>(missing);
        e = cudaGetLastError();
    }
    const cudaError_t done = cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    if (e == cudaSuccess) e = done;
    g_tables_ready[device] = e == cudaSuccess;
    return e;
}

int ensure_device(int device, char *err, size_t errlen) {
    if ((int)g_dev.size() <= device) g_dev.resize(device + 1);
    DeviceInfo &d = g_dev[device];
    if (d.ready) return TD_OK;
    TD_CHECK(cudaSetDevice(device));
    TD_CHECK(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, device));
    const int max_warps = 8;
    const size_t max_smem = smem_bytes(max_warps);
    TD_CHECK(cudaFuncSetAttribute(td_plain_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem));
    TD_CHECK(cudaFuncSetAttribute(td_plain_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem));
    TD_CHECK(cudaFuncSetAttribute(td_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem));
    TD_CHECK(cudaFuncSetAttribute(td_steal_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem));
    TD_CHECK(cudaFuncSetAttribute(td_ordered_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem));
    const int rc = preload_kernels(err, errlen);
    if (rc != TD_OK) return rc;
    TD_CHECK(tables_setup(device, d.sms));
    d.ready = true;
    return TD_OK;
}

void release_slot(Slot &s) {
    if (s.device >= 0) cudaSetDevice(s.device);
    if (s.stream) cudaStreamSynchronize(s.stream);
    if (s.d_inst) cudaFree(s.d_inst);
    if (s.d_res) cudaFree(s.d_res);
    if (s.d_ticket) cudaFree(s.d_ticket);
    if (s.d_batch) cudaFree(s.d_batch);
    if (s.d_pairs) cudaFree(s.d_pairs);
    if (s.h_pairs) cudaFreeHost(s.h_pairs);
    if (s.d_pool) cudaFree(s.d_pool);
    if (s.d_items) cudaFree(s.d_items);
    if (s.d_ready) cudaFree(s.d_ready);
    if (s.d_tt) cudaFree(s.d_tt);
    if (s.d_epoch) cudaFree(s.d_epoch);
    if (s.d_state) cudaFree(s.d_state);
    if (s.d_split_pool) cudaFree(s.d_split_pool);
    if (s.d_split_ready) cudaFree(s.d_split_ready);
    if (s.d_nodes) cudaFree(s.d_nodes);
    if (s.d_split_records) cudaFree(s.d_split_records);
    if (s.d_split_items) cudaFree(s.d_split_items);
    for (void *p : s.kept) cudaFree(p);
    if (s.d_counts) cudaFree(s.d_counts);
    if (s.h_stats) cudaFreeHost(s.h_stats);
    if (s.h_inst) cudaFreeHost(s.h_inst);
    if (s.h_res) cudaFreeHost(s.h_res);
    if (s.done) cudaEventDestroy(s.done);
    if (s.t0) cudaEventDestroy(s.t0);
    if (s.t1) cudaEventDestroy(s.t1);
    if (s.stream) cudaStreamDestroy(s.stream);
    delete s.mu;
    s = Slot{};
}

// the per-call server (td_percall.cuh)
void percall_shutdown();
void percall_park(int device);
int percall_search(int device, const td_instance &x, td_result *out, char *err, size_t errlen);
extern std::atomic<int> g_percall_mode;

void destroy_all() {
    percall_shutdown();
    for (auto &s : g_slots) release_slot(s);
    g_slots.clear();
}

// Launches a kernel that calls td_wait_predecessor right behind the one before it
// on the stream, so that the launches of a batch (epoch, search, finalize,
// replay) overlap: six ordered batches of 4,096 S_10 one after the other take
// 279 us and took 298, 16 instances from host arrays 79 and 85 us.  Every one of
// these kernels waits for its predecessor before it ends, so the last one's end
// is the batch's.
template <typename... P, typename... A>
cudaError_t launch_after(void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Gives a launch buffer that is outgrown back, in stream order (a cudaFree would
// wait for all work on the device, the per-call server's resident launch
// included), or keeps it for the captured launches that hold its address.
template <typename T>
cudaError_t outgrown(Slot &s, T *&p, cudaStream_t stream) {
    cudaError_t e = cudaSuccess;
    if (p && s.captured) s.kept.push_back(p);
    else if (p) e = cudaFreeAsync(p, stream);
    p = nullptr;
    return e;
}

// The size a launch buffer grows to: what is needed, and once old ones are kept
// at least twice the last, so that they hold no more than it does.
size_t grown(const Slot &s, size_t needed, size_t last) { return s.captured ? std::max(needed, 2 * last) : needed; }

// Launch one batch on `stream`.  Instances and results are device pointers.
int launch_batch(Slot &s, int count, const td_instance *d_in, td_result *d_out, unsigned flags,
                 uint64_t max_exp, cudaStream_t stream, char *err, size_t errlen) {
    if (count <= 0) return TD_OK;
    const bool ordered = flags & TD_FLAG_ORDERED;
    LaunchCfg cfg;
    const int rc = launch_cfg(s.device, &cfg, err, errlen);
    if (rc != TD_OK) return rc;
    const int warps = cfg.warps;
    const size_t smem = smem_bytes(warps);
    const int threads = warps * 32;
    if (flags & TD_FLAG_PLAIN) {
        const int blocks = (count + warps - 1) / warps;
        if (ordered) td_plain_kernel<true><<<blocks, threads, smem, stream>>>(d_in, d_out, count, max_exp, time_limit_ns());
        else td_plain_kernel<false><<<blocks, threads, smem, stream>>>(d_in, d_out, count, max_exp, time_limit_ns());
    } else if (!ordered) {
        const unsigned epochs = ((unsigned)(count - 1) >> TD_TT_INST_BITS) + 1u;
        if (s.d_epoch == nullptr) {
            TD_CHECK(cudaMalloc(&s.d_pool, sizeof(td_pool)));
            TD_CHECK(cudaMalloc(&s.d_epoch, sizeof(td_epoch)));
            TD_CHECK(cudaMemsetAsync(s.d_epoch, 0, sizeof(td_epoch), stream));
        }
        td_epoch_kernel<<<1, 1, 0, stream>>>(s.d_epoch, epochs, s.d_pool, count, nullptr, 0, s.d_ready, s.item_capacity,
                                             s.d_tt, s.tt_log2 ? (size_t)1 << s.tt_log2 : 0);
        // item space: the slot budget (the reference's queue budget) less the
        // per-instance state, at 36 bytes per item (record + ready flag)
        if (s.d_items == nullptr) {
            const size_t cap = std::max<size_t>(1024, std::min<size_t>(s.budget / 36, 1u << 26));
            TD_CHECK(cudaMalloc(&s.d_items, cap * sizeof(td_item)));
            TD_CHECK(cudaMalloc(&s.d_ready, cap * sizeof(uint32_t)));
            TD_CHECK(cudaMemsetAsync(s.d_ready, 0, cap * sizeof(uint32_t), stream));
            s.item_capacity = (int)cap;
        }
        if ((size_t)count > s.state_count) {
            const size_t n = grown(s, (size_t)count, s.state_count);
            TD_CHECK(outgrown(s, s.d_state, stream));
            s.state_count = 0;
            TD_CHECK(cudaMallocAsync(&s.d_state, n * sizeof(td_inst_state), stream));
            s.state_count = n;
        }
        // at least the slot's share of the resident grid, so that a small batch
        // (one search from td_search) is spread over that many warps by donation,
        // and TD_INSTANCE_WARPS warps per instance: with one each, the warps
        // whose instance was easy were too few for what the hard ones give away.
        // With 16 slots, 2,048 S_16 at their lower bound took 5.1 ms with one
        // warp each, 2.2 with two and 2.0 with four; 250 of S_8..S_16 0.30, 0.27
        // and 0.22.  It holds for launches side by side too (they end sooner, and
        // make room): from 16 threads 3.8 and 2.2 ms a batch of the former, 0.11
        // and 0.10 ms of the latter.  The whole grid for every batch is no
        // better alone, and slower there (0.25 ms).
        const int resident = cfg.sms * cfg.steal_blocks_per_sm;
        const int share = std::max(1, resident / std::max(1, s.slots_on_device));
        const int64_t wanted = ((int64_t)count * TD_INSTANCE_WARPS + warps - 1) / warps;
        const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(resident, std::max<int64_t>(share, wanted)));
        const int tt_log2 = tt_entries_log2((size_t)resident * warps, cfg.tt_bits);
        if (cfg.tt_bits > 0 && (tt_log2 > s.tt_log2 || (cfg.tt_bits != s.tt_bits && !s.captured))) {
            // sized for the whole resident grid; replaced in stream order after the
            // previous launch (a captured launch keeps it, and then a smaller
            // setting keeps the larger table)
            TD_CHECK(outgrown(s, s.d_tt, stream));
            s.tt_log2 = 0;
            TD_CHECK(cudaMallocAsync(&s.d_tt, sizeof(ulonglong2) << tt_log2, stream));
            TD_CHECK(cudaMemsetAsync(s.d_tt, 0, sizeof(ulonglong2) << tt_log2, stream));  // zero words are empty
            s.tt_log2 = tt_log2;
            s.tt_bits = cfg.tt_bits;
        }
        // the race needs restarts, and an expansion budget per unit would make
        // one side's budget decide the other's; each instance queues its
        // inverse at most once, and at least half the item space is left for
        // donation
        const int race = cfg.restart_base > 0 && max_exp == 0 && count <= s.item_capacity / 2 ? cfg.race : 0;
        TD_CHECK(launch_after(td_steal_kernel, grid, threads, smem_bytes(warps), stream,
            d_in, d_out, count, s.d_pool, s.d_items, s.d_ready, s.d_epoch, s.item_capacity, s.d_state,
            cfg.steal_grain, cfg.split_level, cfg.check_every, time_limit_ns(), cfg.tt_bits > 0 ? s.d_tt : nullptr,
            64 - s.tt_log2, epochs, cfg.restart_base, max_exp, race));
        TD_CHECK(launch_after(td_finalize_kernel, std::max(1, std::min((count + 255) / 256, 2 * cfg.sms)), 256, (size_t)0,
                              stream, s.d_pool, s.d_state, d_out, count));
    } else {
        const int grid_max = cfg.sms * cfg.blocks_per_sm;
        const int grid = std::max(1, std::min(grid_max, (count + warps - 1) / warps));
        if (max_exp == 0 && cfg.split_budget > 0) {
            // stream-ordered buffers; the flags start at zero, epochs at 1
            if (s.d_split_pool == nullptr) {
                TD_CHECK(cudaMallocAsync(&s.d_split_pool, TD_SPLIT_HEAD, stream));
                TD_CHECK(cudaMemsetAsync(s.d_split_pool, 0, TD_SPLIT_HEAD, stream));
            }
            int *node_count = reinterpret_cast<int *>(s.d_split_pool + 1);
            td_epoch *epoch = reinterpret_cast<td_epoch *>(node_count + 2);
            // the node and record counts start at zero in every launch
            td_epoch_kernel<<<1, 1, 0, stream>>>(epoch, 1u, s.d_split_pool, count, node_count, 2, s.d_split_ready,
                                                 s.split_records, nullptr, 0);
            if (cfg.split_records > s.split_records) {
                const size_t n = grown(s, (size_t)cfg.split_records, (size_t)s.split_records);
                TD_CHECK(outgrown(s, s.d_split_ready, stream));
                TD_CHECK(outgrown(s, s.d_nodes, stream));
                TD_CHECK(outgrown(s, s.d_split_items, stream));
                TD_CHECK(outgrown(s, s.d_split_records, stream));
                s.split_records = 0;
                TD_CHECK(cudaMallocAsync(&s.d_split_ready, sizeof(uint32_t) * n, stream));
                TD_CHECK(cudaMallocAsync(&s.d_nodes, sizeof(td_split_node) * split_nodes((int)n), stream));
                TD_CHECK(cudaMallocAsync(&s.d_split_items, sizeof(td_split_item) * n, stream));
                TD_CHECK(cudaMallocAsync(&s.d_split_records, sizeof(td_result) * n, stream));
                TD_CHECK(cudaMemsetAsync(s.d_split_ready, 0, sizeof(uint32_t) * n, stream));
                s.split_records = (int)n;
            }
            td_split_space sp;
            sp.nodes = s.d_nodes;
            sp.node_count = node_count;
            sp.record_count = node_count + 1;
            sp.max_nodes = (int)split_nodes(cfg.split_records);
            sp.items = s.d_split_items;
            sp.records = s.d_split_records;
            sp.out = d_out;
            TD_CHECK(launch_after(td_ordered_kernel, grid_max, threads, smem, stream, d_in, d_out, count, s.d_split_pool, sp,
                                                                  s.d_split_ready, epoch, cfg.split_records,
                                                                  cfg.split_budget, time_limit_ns()));
        } else {
            TD_CHECK(cudaMemsetAsync(s.d_ticket, 0, sizeof(int), stream));
            td_persistent_kernel<<<grid, threads, smem, stream>>>(d_in, d_out, count, s.d_ticket, cfg.grain,
                                                                        max_exp, time_limit_ns());
        }
    }
    TD_CHECK(cudaGetLastError());
    if (flags & TD_FLAG_VERIFY) {
        TD_CHECK(launch_after(td_validate_kernel, (count + 255) / 256, 256, (size_t)0, stream, d_in, d_out,
                              (uint8_t *)nullptr, count, 1));
    }
    return TD_OK;
}

// Device space for the instances and results of a host-buffer batch.
int ensure_batch(Slot &s, size_t count, char *err, size_t errlen) {
    const size_t need = count * (sizeof(td_instance) + sizeof(td_result));
    if (need > s.d_batch_bytes) {  // grows in stream order (no device-wide wait)
        if (s.d_batch) TD_CHECK(cudaFreeAsync(s.d_batch, s.stream));
        s.d_batch = nullptr;
        s.d_batch_bytes = 0;
        TD_CHECK(cudaMallocAsync(&s.d_batch, need, s.stream));
        s.d_batch_bytes = need;
    }
    return TD_OK;
}

// Layout of the arrays of td_search_pairs: the caller's, then the outputs, each
// part from a multiple of 16 bytes.
size_t pairs_in_bytes(size_t c) { return (c * (3 * 4 + 2 * TD_MAX_N + 2) + 15) & ~(size_t)15; }
size_t pairs_out_bytes(size_t c) { return c * (2 * 4 + 27 * sizeof(int16_t)); }

td_pair_arrays pair_arrays(uint8_t *base, size_t c) {
    td_pair_arrays a;
    a.init = (int32_t *)base;
    a.max_moves = a.init + c;
    a.rate = (float *)(a.max_moves + c);
    a.beta = (uint8_t *)(a.rate + c);
    a.omega = a.beta + TD_MAX_N * c;
    a.n = a.omega + TD_MAX_N * c;
    a.full = a.n + c;
    a.status = (int32_t *)(base + pairs_in_bytes(c));
    a.depth = a.status + c;
    a.ijk = (int16_t *)(a.depth + c);
    return a;
}

// Pinned memory of a slot that td_search_pairs' copies go through: allocated at
// the slot's first such call and kept until the slot goes, so that no later call
// pins or frees host memory, which may wait for all work on the device.  65,536
// pairs (the pair consumer's default batch) go in one piece each way.
constexpr size_t kPairStage = 4u << 20;

// A stretch of the arrays of a call and the caller's memory for it.
struct PairPart {
    size_t at, bytes;
    char *host;
};

// Copies what [from, from + bytes) holds of `parts` between the pinned memory,
// which holds that range, and the caller's arrays.
void stage_parts(const PairPart *parts, int count, size_t from, size_t bytes, uint8_t *stage, bool in) {
    for (int i = 0; i < count; ++i) {
        const size_t a = std::max(from, parts[i].at), b = std::min(from + bytes, parts[i].at + parts[i].bytes);
        if (a >= b) continue;
        char *host = parts[i].host + (a - parts[i].at);
        if (in) std::memcpy(stage + (a - from), host, b - a);
        else std::memcpy(host, stage + (a - from), b - a);
    }
}

Slot *get_slot(int slot, char *err, size_t errlen) {
    if (slot < 0 || slot >= (int)g_slots.size() || g_slots[slot].device < 0) {
        set_err(err, errlen, "invalid GPU sorting slot");
        return nullptr;
    }
    return &g_slots[slot];
}

int search_one(int slot, const uint8_t *beta, const uint8_t *omega, int n, int init, float min_rate,
               int max_moves, int full, int16_t *out_ijk, int *out_depth, unsigned flags, char *err,
               size_t errlen) {
    if (out_depth) *out_depth = 0;
    // the reference's order of checks: null arrays, the slot
    // (jni_sorter.cu:59-92), then n, the depth and n < 3
    // (sorting_search.cu:821-827)
    if (!beta || !omega) {
        set_err(err, errlen, "beta and omega must not be null");
        return TD_INVALID_ARG;
    }
    Slot *s;
    {
        std::lock_guard<std::mutex> g(g_mu);
        s = get_slot(slot, err, errlen);
        if (!s) return TD_INVALID_ARG;
    }
    if (n > TD_MAX_N) {
        set_err(err, errlen, "performGpuSortingSearch: n exceeds MAX_N");
        return TD_INVALID_ARG;
    }
    if (max_moves <= 0 || max_moves > TD_MAX_DEPTH) {
        set_err(err, errlen, "performGpuSortingSearch: invalid maximumDepth");
        return TD_INVALID_ARG;
    }
    if (td_triple_count(n) == 0) return TD_NOT_FOUND_RC;
    td_instance x;
    if (td_prepare_pair(beta, omega, n, init, min_rate, max_moves, full, &x) != 0) {
        set_err(err, errlen, "beta/omega are not permutations whose product omega.beta is an n-cycle");
        return TD_INVALID_ARG;
    }
    td_result r;
    if (g_percall_mode.load(std::memory_order_relaxed) == 1) {
        // the device's resident per-call server: no CUDA call per search
        if (flags & TD_FLAG_ORDERED) x.packed |= TD_PACKED_ORDERED;
        const int rc = percall_search(s->device, x, &r, err, errlen);
        if (rc != TD_OK) return rc;
    } else {
        std::lock_guard<std::mutex> g(*s->mu);
        TD_CHECK(cudaSetDevice(s->device));
        *s->h_inst = x;
        TD_CHECK(cudaMemcpyAsync(s->d_inst, s->h_inst, sizeof(td_instance), cudaMemcpyHostToDevice, s->stream));
        // free order: the donation engine over the slot's share of the GPU (as
        // the reference gives each slot SMs x resident blocks / slots queues,
        // sorting_search.cu:740-752); the reference order keeps one warp
        const unsigned how = (flags & TD_FLAG_ORDERED) ? (flags | TD_FLAG_PLAIN) : flags;
        percall_park(s->device);
        int rc = launch_batch(*s, 1, s->d_inst, s->d_res, how, 0, s->stream, err, errlen);
        if (rc != TD_OK) return rc;
        TD_CHECK(cudaMemcpyAsync(s->h_res, s->d_res, sizeof(td_result), cudaMemcpyDeviceToHost, s->stream));
        TD_CHECK(cudaEventRecord(s->done, s->stream));
        TD_CHECK(cudaEventSynchronize(s->done));
        r = *s->h_res;
    }
    if (r.status == TD_FOUND) {
        for (int d = 0; d < r.depth; ++d) {
            out_ijk[3 * d + 0] = (int16_t)(r.moves[d] & 31);
            out_ijk[3 * d + 1] = (int16_t)((r.moves[d] >> 5) & 31);
            out_ijk[3 * d + 2] = (int16_t)((r.moves[d] >> 10) & 31);
        }
        if (out_depth) *out_depth = r.depth;
        return TD_OK;
    }
    if (r.status == TD_NOT_FOUND) return TD_NOT_FOUND_RC;
    if (r.status == TD_ERR_BUDGET) {
        set_err(err, errlen, "GPU sorting search queue overflow");
        return TD_OVERFLOW;
    }
    if (r.status == TD_ERR_TIMEOUT) {
        set_err(err, errlen, "GPU sorting search deadline reached");
        return TD_TIMEOUT;
    }
    set_err(err, errlen, "GPU sorting search rejected its input");
    return TD_INVALID_ARG;
}

// ---- seeded synthetic instances ----------------------------------------------

inline uint64_t splitmix64(uint64_t &s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Lemire's multiply-shift bounded draw on the upper 32 bits, with rejection.
inline uint32_t bounded(uint64_t &s, uint32_t range) {
    uint32_t x = (uint32_t)(splitmix64(s) >> 32);
    uint64_t m = (uint64_t)x * range;
    uint32_t l = (uint32_t)m;
    if (l < range) {
        const uint32_t t = (0u - range) % range;
        while (l < t) {
            x = (uint32_t)(splitmix64(s) >> 32);
            m = (uint64_t)x * range;
            l = (uint32_t)m;
        }
    }
    return (uint32_t)(m >> 32);
}

// lexicographic unranking of r over triples x<y<z of {0..n}
void unrank_triple(int n, uint32_t r, int *x, int *y, int *z) {
    const int M = n + 1;
    for (int a = 0; a < M - 2; ++a) {
        const uint32_t c = (uint32_t)((M - a - 1) * (M - a - 2) / 2);
        if (r < c) {
            for (int b = a + 1; b < M - 1; ++b) {
                const uint32_t cb = (uint32_t)(M - b - 1);
                if (r < cb) {
                    *x = a;
                    *y = b;
                    *z = b + 1 + (int)r;
                    return;
                }
                r -= cb;
            }
        }
        r -= c;
    }
    *x = 0;
    *y = 1;
    *z = 2;
}

}  // namespace

// ============================================================================
// C ABI
// ============================================================================

TD_API int td_init_slots(int total_slots, const int *devices, int device_count, uint64_t budget, char *err,
                         size_t errlen) {
    if (!devices || device_count <= 0) {
        set_err(err, errlen, "devices must contain at least one CUDA device ordinal");
        return TD_INVALID_ARG;
    }
    if (total_slots <= 0) {
        set_err(err, errlen, "totalSlots must be positive");
        return TD_INVALID_ARG;
    }
    if (budget == 0) {
        set_err(err, errlen, "queueBytesBudget must be positive");
        return TD_INVALID_ARG;
    }
    int ndev = 0;
    TD_CHECK(cudaGetDeviceCount(&ndev));
    std::vector<int> per(ndev > 0 ? ndev : 1, 0);
    for (int i = 0; i < device_count; ++i) {
        if (devices[i] < 0 || devices[i] >= ndev) {
            set_err(err, errlen, "devices contains a CUDA device ordinal outside the available range");
            return TD_INVALID_ARG;
        }
        for (int j = 0; j < i; ++j)
            if (devices[j] == devices[i]) {
                set_err(err, errlen, "devices must contain distinct CUDA device ordinals");
                return TD_INVALID_ARG;
            }
    }
    for (int i = 0; i < total_slots; ++i) per[devices[i % device_count]]++;
    std::lock_guard<std::mutex> g(g_mu);
    destroy_all();
    for (int i = 0; i < device_count; ++i) {
        const int dev = devices[i];
        TD_CHECK(cudaSetDevice(dev));
        size_t free_b = 0, total_b = 0;
        TD_CHECK(cudaMemGetInfo(&free_b, &total_b));
        const uint64_t need = budget * (uint64_t)per[dev];
        if (per[dev] > 0 && (budget > UINT64_MAX / (uint64_t)per[dev] || need > free_b)) {
            set_err(err, errlen, "CUDA device " + std::to_string(dev) + " has " + std::to_string(free_b) +
                                     " free bytes, but its search queues require at least " +
                                     std::to_string(need) + " bytes");
            return TD_INVALID_ARG;
        }
        int rc = ensure_device(dev, err, errlen);
        if (rc != TD_OK) return rc;
    }
    g_slots.resize(total_slots);
    for (int i = 0; i < total_slots; ++i) {
        Slot &s = g_slots[i];
        s.device = devices[i % device_count];
        s.budget = budget;
        s.slots_on_device = per[s.device];
        s.mu = new std::mutex();
        cudaError_t e = cudaSetDevice(s.device);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s.done, cudaEventBlockingSync | cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreate(&s.t0);
        if (e == cudaSuccess) e = cudaEventCreate(&s.t1);
        if (e == cudaSuccess) e = cudaMalloc(&s.d_inst, sizeof(td_instance));
        if (e == cudaSuccess) e = cudaMalloc(&s.d_res, sizeof(td_result));
        if (e == cudaSuccess) e = cudaMalloc(&s.d_ticket, sizeof(int));
        if (e == cudaSuccess) e = cudaMallocHost(&s.h_inst, sizeof(td_instance));
        if (e == cudaSuccess) e = cudaMallocHost(&s.h_res, sizeof(td_result));
        if (e != cudaSuccess) {
            set_err(err, errlen, cuda_msg(e, __FILE__, __LINE__));
            destroy_all();
            return TD_CUDA_ERROR;
        }
    }
    return TD_OK;
}

TD_API int td_search(int slot, const uint8_t *beta, const uint8_t *omega, int n, int init, float min_rate,
                     int max_moves, int full, int16_t *out_ijk, int *out_depth, char *err, size_t errlen) {
    return search_one(slot, beta, omega, n, init, min_rate, max_moves, full, out_ijk, out_depth, 0u, err, errlen);
}

TD_API int td_search_ordered(int slot, const uint8_t *beta, const uint8_t *omega, int n, int init,
                             float min_rate, int max_moves, int full, int16_t *out_ijk, int *out_depth,
                             char *err, size_t errlen) {
    return search_one(slot, beta, omega, n, init, min_rate, max_moves, full, out_ijk, out_depth,
                      TD_FLAG_ORDERED, err, errlen);
}

TD_API int td_slot_count(void) {
    std::lock_guard<std::mutex> g(g_mu);
    return (int)g_slots.size();
}

TD_API int td_slot_device(int slot) {
    std::lock_guard<std::mutex> g(g_mu);
    if (slot < 0 || slot >= (int)g_slots.size()) return -1;
    return g_slots[slot].device;
}

TD_API void *td_slot_stream(int slot) {
    std::lock_guard<std::mutex> g(g_mu);
    if (slot < 0 || slot >= (int)g_slots.size()) return nullptr;
    return (void *)g_slots[slot].stream;
}

TD_API int td_destroy(void) {
    std::lock_guard<std::mutex> g(g_mu);
    destroy_all();
    return TD_OK;
}

TD_API int td_configure(int warps_per_block, int grain) {
    if (warps_per_block < 1 || warps_per_block > 8 || grain < 1) return TD_INVALID_ARG;
    std::lock_guard<std::mutex> g(g_mu);
    g_warps_per_block = warps_per_block;
    g_grain = grain;
    for (auto &d : g_dev) d.blocks_per_sm = d.steal_blocks_per_sm = 0;
    return TD_OK;
}

// Sets the deadline of every later launch (seconds > 0); every device wait
// and search ends with a timeout status once it passes.
TD_API int td_set_time_limit(double seconds) {
    if (!(seconds > 0)) return TD_INVALID_ARG;
    g_time_limit_ns.store((uint64_t)(seconds * 1e9), std::memory_order_relaxed);
    return TD_OK;
}

// Work-donation parameters of the free-order engine: items per donation,
// deepest level whose children may be donated, expansions between checks.  They
// hold while every warp has an instance of its own; from the first idle warps
// on, and from the start in launches of few instances per warp,
// td_serve_idle_warps derives sharper ones from them.
TD_API int td_configure_steal(int grain, int split_level, int check_every) {
    if (grain < 1 || split_level < 0 || split_level >= TD_MAX_DEPTH || check_every < 1) return TD_INVALID_ARG;
    std::lock_guard<std::mutex> g(g_mu);
    g_steal_grain = grain;
    g_split_level = split_level;
    g_check_every = check_every;
    return TD_OK;
}

// Size of the table of explored states of later free-order launches:
// 2^(bits - 2) entries of 16 bytes per resident warp (6 <= bits <= 16), rounded
// down to a power of two in all, or 0 to search without it.
TD_API int td_configure_table(int bits) {
    if (bits != 0 && (bits < 6 || bits > 16)) return TD_INVALID_ARG;
    std::lock_guard<std::mutex> g(g_mu);
    g_tt_bits = bits;
    return TD_OK;
}

// Walks of reference-order batches: the expansions after which one may give
// subtrees away (0: never, every walk on one warp) and the subtree records per
// launch (a walk that finds no room goes on whole).  Results do not depend on
// either.
TD_API int td_configure_split(int first_pass_expansions, int records) {
    if (first_pass_expansions < 0 || records < 1 || records > (1 << 24)) return TD_INVALID_ARG;
    std::lock_guard<std::mutex> g(g_mu);
    g_split_budget = first_pass_expansions;
    g_split_records = records;
    return TD_OK;
}

// Restarts of later free-order batch searches: a search that has spent
// base x luby(a) expansions in attempt a starts again with another child order
// (td_attempt_budget, td_order_variant); 0 turns restarts off.  Verdicts do
// not depend on it.
TD_API int td_configure_restart(int base) {
    if (base < 0 || (base > 0 && base < 16)) return TD_INVALID_ARG;
    std::lock_guard<std::mutex> g(g_mu);
    g_restart_base = (uint32_t)base;
    return TD_OK;
}

// Later free-order batches (full sorting) race a search that starts its
// restart attempt `attempt` (1..32; the 32nd is the last, unbounded one)
// against a search of its inverse instance; 0 turns the race off.
TD_API int td_configure_race(int attempt) {
    if (attempt < 0 || attempt > TD_RESTARTS) return TD_INVALID_ARG;
    std::lock_guard<std::mutex> g(g_mu);
    g_race = attempt;
    return TD_OK;
}

// Work distribution of later serving launches (td_serve_open): items per
// donation, deepest level whose children are donated, expansions between
// idle checks.
TD_API int td_configure_serve(int grain, int split_level, int check_every) {
    if (grain < 1 || split_level < 0 || split_level >= TD_MAX_DEPTH || check_every < 1) return TD_INVALID_ARG;
    std::lock_guard<std::mutex> g(g_mu);
    g_serve_grain = grain;
    g_serve_split_level = split_level;
    g_serve_check_every = check_every;
    return TD_OK;
}

TD_API int td_prepare_pairs(int count, const uint8_t *beta, const uint8_t *omega, const uint8_t *n,
                            const int32_t *init, const float *min_rate, const int32_t *max_moves,
                            const uint8_t *full, td_instance *out, int *bad) {
    for (int i = 0; i < count; ++i) {
        if (td_prepare_pair(beta + (size_t)i * TD_MAX_N, omega + (size_t)i * TD_MAX_N, n[i], init[i], min_rate[i],
                            max_moves[i], full[i], &out[i]) != 0) {
            if (bad) *bad = i;
            return TD_INVALID_ARG;
        }
    }
    return TD_OK;
}

TD_API int td_prepare_perms(int count, const int8_t *perms, const uint8_t *n, const int32_t *max_moves,
                            float min_rate, int full, td_instance *out, int *bad) {
    for (int i = 0; i < count; ++i) {
        const int ni = n[i];
        uint8_t beta[TD_MAX_N], omega[TD_MAX_N];
        int init = 0;
        bool okp = ni >= 0 && ni < TD_MAX_N;
        if (okp) {
            uint32_t seen = 0;
            for (int m = 0; m < ni; ++m) {
                const int v = perms[(size_t)i * 16 + m];
                if (v < 0 || v >= ni || (seen >> v) & 1u) okp = false;
                else seen |= 1u << v;
            }
        }
        if (okp) {
            td_perm_to_pair(perms + (size_t)i * 16, ni, beta, omega, &init);
            okp = td_prepare_pair(beta, omega, ni + 1, init, min_rate, max_moves[i], full, &out[i]) == 0;
        }
        if (!okp) {
            if (bad) *bad = i;
            return TD_INVALID_ARG;
        }
    }
    return TD_OK;
}

TD_API int td_synth_perms(uint64_t seed, int count, int n_min, int n_max, int hard_pct, int hard_min, int hard_max,
                          int8_t *perms, uint8_t *n_out) {
    if (n_min < 1 || n_max > 16 || n_min > n_max || hard_min < 0 || hard_max < hard_min) return TD_INVALID_ARG;
    for (int i = 0; i < count; ++i) {
        uint64_t st = seed ^ (uint64_t)i;
        const int n = n_min + (int)bounded(st, (uint32_t)(n_max - n_min + 1));
        int8_t *p = perms + (size_t)i * 16;
        const bool hard = (int)bounded(st, 100) < hard_pct;
        if (hard) {
            for (int m = 0; m < n; ++m) p[m] = (int8_t)(n - 1 - m);
            const int moves = hard_min + (int)bounded(st, (uint32_t)(hard_max - hard_min + 1));
            const uint32_t triples = (uint32_t)((n + 1) * n * (n - 1) / 6);
            for (int mv = 0; mv < moves && triples > 0; ++mv) {
                int x, y, z;
                unrank_triple(n, bounded(st, triples), &x, &y, &z);
                int8_t tmp[16];
                int w = 0;
                for (int q = 0; q < x; ++q) tmp[w++] = p[q];
                for (int q = y; q < z; ++q) tmp[w++] = p[q];
                for (int q = x; q < y; ++q) tmp[w++] = p[q];
                for (int q = z; q < n; ++q) tmp[w++] = p[q];
                std::memcpy(p, tmp, (size_t)n);
            }
        } else {
            for (int m = 0; m < n; ++m) p[m] = (int8_t)m;
            for (int m = n - 1; m > 0; --m) {
                const int j = (int)bounded(st, (uint32_t)(m + 1));
                const int8_t t = p[m];
                p[m] = p[j];
                p[j] = t;
            }
        }
        for (int m = n; m < 16; ++m) p[m] = 0;
        n_out[i] = (uint8_t)n;
    }
    return TD_OK;
}

TD_API int td_search_batch_device(int slot, int count, const td_instance *d_in, td_result *d_out, unsigned flags,
                                  uint64_t max_exp, void *stream, char *err, size_t errlen) {
    Slot *s;
    {
        std::lock_guard<std::mutex> g(g_mu);
        s = get_slot(slot, err, errlen);
        if (!s) return TD_INVALID_ARG;
    }
    if (count < 0 || (count > 0 && (!d_in || !d_out))) {
        set_err(err, errlen, "invalid batch arguments");
        return TD_INVALID_ARG;
    }
    percall_park(s->device);
    std::lock_guard<std::mutex> g(*s->mu);
    TD_CHECK(cudaSetDevice(s->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : s->stream;
    return launch_batch(*s, count, d_in, d_out, flags, max_exp, st, err, errlen);
}

TD_API int td_search_batch(int slot, int count, const td_instance *in, td_result *out, unsigned flags,
                           uint64_t max_exp, td_batch_stats *stats, char *err, size_t errlen) {
    Slot *s;
    {
        std::lock_guard<std::mutex> g(g_mu);
        s = get_slot(slot, err, errlen);
        if (!s) return TD_INVALID_ARG;
    }
    if (count < 0 || (count > 0 && (!in || !out))) {
        set_err(err, errlen, "invalid batch arguments");
        return TD_INVALID_ARG;
    }
    if (count == 0) {
        if (stats) std::memset(stats, 0, sizeof *stats);
        return TD_OK;
    }
    percall_park(s->device);
    std::lock_guard<std::mutex> g(*s->mu);
    TD_CHECK(cudaSetDevice(s->device));
    const int grown = ensure_batch(*s, (size_t)count, err, errlen);
    if (grown != TD_OK) return grown;
    if (stats && !s->d_counts) TD_CHECK(cudaMalloc(&s->d_counts, sizeof(td_counts)));
    if (stats && !s->h_stats) TD_CHECK(cudaMallocHost(&s->h_stats, sizeof(Slot::HostStats)));
    td_instance *d_in = (td_instance *)s->d_batch;
    td_result *d_out = (td_result *)((char *)s->d_batch + (size_t)count * sizeof(td_instance));
    TD_CHECK(cudaMemcpyAsync(d_in, in, (size_t)count * sizeof(td_instance), cudaMemcpyHostToDevice, s->stream));
    TD_CHECK(cudaEventRecord(s->t0, s->stream));
    int rc = launch_batch(*s, count, d_in, d_out, flags, max_exp, s->stream, err, errlen);
    if (rc != TD_OK) return rc;
    TD_CHECK(cudaEventRecord(s->t1, s->stream));
    const bool pooled = !(flags & (TD_FLAG_ORDERED | TD_FLAG_PLAIN)) && s->d_pool;
    if (stats) {
        TD_CHECK(cudaMemsetAsync(s->d_counts, 0, sizeof(td_counts), s->stream));
        const int blocks = std::max(1, std::min((count + 255) / 256, g_dev[s->device].sms * 8));
        td_count_kernel<<<blocks, 256, 0, s->stream>>>(d_out, count, s->d_counts);
        TD_CHECK(cudaGetLastError());
        TD_CHECK(cudaMemcpyAsync(&s->h_stats->counts, s->d_counts, sizeof(td_counts), cudaMemcpyDeviceToHost,
                                 s->stream));
        if (pooled)
            TD_CHECK(cudaMemcpyAsync(&s->h_stats->pool, s->d_pool, sizeof(td_pool), cudaMemcpyDeviceToHost,
                                     s->stream));
    }
    TD_CHECK(cudaMemcpyAsync(out, d_out, (size_t)count * sizeof(td_result), cudaMemcpyDeviceToHost, s->stream));
    TD_CHECK(cudaEventRecord(s->done, s->stream));
    TD_CHECK(cudaEventSynchronize(s->done));
    if (stats) {
        std::memset(stats, 0, sizeof *stats);
        TD_CHECK(cudaEventElapsedTime(&stats->kernel_ms, s->t0, s->t1));
        if (pooled) {
            const td_pool &pool = s->h_stats->pool;
            stats->donations = pool.donations;
            stats->donated_items = pool.donated_items;
            stats->races = pool.races;
            if (pool.error) {
                set_err(err, errlen, "engine launch deadline reached");
                return TD_TIMEOUT;
            }
        }
        const td_counts &c = s->h_stats->counts;
        stats->expansions = c.expansions;
        stats->found = c.found;
        stats->not_found = c.not_found;
        stats->errors = c.errors;
    }
    return TD_OK;
}

// Many reference pairs in one call: the batch form of td_search for a case
// producer that hands over pairs in groups (the enumerator's
// Consumer<CyclicTargetPair>, DirectTwistedBraceletGenerator.java:105-156,
// feeds one pair per call today).  Pair i: beta/omega at stride 17, n[i]
// symbols, init[i], min_rate[i], max_moves[i], full[i].  Outputs per pair:
// status[i] (TD_OK found, TD_NOT_FOUND, or the per-call error class:
// TD_INVALID_ARG, TD_OVERFLOW, TD_TIMEOUT), depth[i] and the position
// triples at out_ijk[27 i ..].  Returns TD_OK when the batch ran (the pair
// statuses say the rest), else the error of the whole call.
TD_API int td_search_pairs(int slot, int count, const uint8_t *beta, const uint8_t *omega, const uint8_t *n,
                           const int32_t *init, const float *min_rate, const int32_t *max_moves,
                           const uint8_t *full, unsigned flags, int32_t *status, int32_t *depth, int16_t *out_ijk,
                           char *err, size_t errlen) {
    if (count < 0 || (count > 0 && (!beta || !omega || !n || !init || !min_rate || !max_moves || !full ||
                                    !status || !depth || !out_ijk))) {
        set_err(err, errlen, "invalid batch arguments");
        return TD_INVALID_ARG;
    }
    Slot *s;
    {
        std::lock_guard<std::mutex> g(g_mu);
        s = get_slot(slot, err, errlen);
        if (!s) return TD_INVALID_ARG;
    }
    if (count == 0) return TD_OK;
    percall_park(s->device);
    std::lock_guard<std::mutex> g(*s->mu);
    TD_CHECK(cudaSetDevice(s->device));
    const size_t c = (size_t)count;
    const size_t in_bytes = pairs_in_bytes(c), bytes = in_bytes + pairs_out_bytes(c);
    if (!s->h_pairs) TD_CHECK(cudaMallocHost(&s->h_pairs, kPairStage));
    if (bytes > s->pairs_bytes) {  // grows in stream order (no device-wide wait)
        if (s->d_pairs) TD_CHECK(cudaFreeAsync(s->d_pairs, s->stream));
        s->d_pairs = nullptr;
        s->pairs_bytes = 0;
        TD_CHECK(cudaMallocAsync(&s->d_pairs, bytes, s->stream));
        s->pairs_bytes = bytes;
    }
    int rc = ensure_batch(*s, c, err, errlen);
    if (rc != TD_OK) return rc;
    td_instance *d_in = (td_instance *)s->d_batch;
    td_result *d_out = (td_result *)((char *)s->d_batch + c * sizeof(td_instance));
    const td_pair_arrays d = pair_arrays(s->d_pairs, c);
    auto part = [&](const void *device, const void *host, size_t n) {
        return PairPart{(size_t)((const uint8_t *)device - s->d_pairs), n, (char *)host};
    };
    const PairPart ins[] = {part(d.init, init, c * sizeof *init),
                            part(d.max_moves, max_moves, c * sizeof *max_moves),
                            part(d.rate, min_rate, c * sizeof *min_rate),
                            part(d.beta, beta, c * TD_MAX_N),
                            part(d.omega, omega, c * TD_MAX_N),
                            part(d.n, n, c),
                            part(d.full, full, c)};
    const PairPart outs[] = {part(d.status, status, c * sizeof *status), part(d.depth, depth, c * sizeof *depth),
                             part(d.ijk, out_ijk, 27 * c * sizeof *out_ijk)};
    for (size_t at = 0; at < in_bytes; at += kPairStage) {
        const size_t m = std::min(kPairStage, in_bytes - at);
        if (at) TD_CHECK(cudaStreamSynchronize(s->stream));  // the piece before has left the pinned memory
        stage_parts(ins, 7, at, m, s->h_pairs, true);
        TD_CHECK(cudaMemcpyAsync(s->d_pairs + at, s->h_pairs, m, cudaMemcpyHostToDevice, s->stream));
    }
    td_pairs_prepare_kernel<<<(count + 127) / 128, 128, 0, s->stream>>>(d, d_in, count);
    TD_CHECK(cudaGetLastError());
    rc = launch_batch(*s, count, d_in, d_out, flags & TD_FLAG_ORDERED, 0, s->stream, err, errlen);
    if (rc != TD_OK) return rc;
    td_pairs_unpack_kernel<<<(unsigned)((27 * c + 255) / 256), 256, 0, s->stream>>>(d, d_out, count);
    TD_CHECK(cudaGetLastError());
    for (size_t at = in_bytes; at < bytes; at += kPairStage) {
        const size_t m = std::min(kPairStage, bytes - at);
        TD_CHECK(cudaMemcpyAsync(s->h_pairs, s->d_pairs + at, m, cudaMemcpyDeviceToHost, s->stream));
        // not the slot's blocking event: a thread that sleeps on it is woken 100
        // to 200 us after the copy (a call of 16 pairs took 0.18 ms, now 0.08)
        TD_CHECK(cudaStreamSynchronize(s->stream));
        stage_parts(outs, 3, at, m, s->h_pairs, false);
    }
    return TD_OK;
}

TD_API int td_validate_batch_device(int count, const td_instance *d_in, const td_result *d_res, uint8_t *d_ok,
                                    void *stream, char *err, size_t errlen) {
    if (count <= 0) return TD_OK;
    const int threads = 256;
    td_validate_kernel<<<(count + threads - 1) / threads, threads, 0, (cudaStream_t)stream>>>(
        d_in, const_cast<td_result *>(d_res), d_ok, count, 0);
    TD_CHECK(cudaGetLastError());
    return TD_OK;
}

TD_API void td_positions_to_symbols(const uint8_t *beta, int n, const int16_t *ijk, int depth, uint8_t *out_abc) {
    uint8_t cur[TD_MAX_N], nxt[TD_MAX_N];
    std::memcpy(cur, beta, (size_t)n);
    for (int d = 0; d < depth; ++d) {
        const int i = ijk[3 * d], j = ijk[3 * d + 1], k = ijk[3 * d + 2];
        out_abc[3 * d] = cur[i];
        out_abc[3 * d + 1] = cur[j];
        out_abc[3 * d + 2] = cur[k];
        int w = 0;
        for (int q = 0; q < i; ++q) nxt[w++] = cur[q];
        for (int q = j; q < k; ++q) nxt[w++] = cur[q];
        for (int q = i; q < j; ++q) nxt[w++] = cur[q];
        for (int q = k; q < n; ++q) nxt[w++] = cur[q];
        std::memcpy(cur, nxt, (size_t)n);
    }
}

namespace {

// Times one form of td_int_peak_kernel on the current device, doubling the
// iteration count until a launch lasts `target_ms`; returns warp instructions
// per second.
template <int MIX>
int time_int_peak(int sms, float target_ms, uint32_t *sink, cudaEvent_t a, cudaEvent_t b, double *rate) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, td_int_peak_kernel<MIX>, 256, 0) != cudaSuccess)
        return -1;
    const int blocks = sms * std::max(1, per_sm);
    int iters = 1024;
    float ms = 0;
    for (int attempt = 0; attempt < 12; ++attempt) {
        td_int_peak_kernel<MIX><<<blocks, 256>>>(sink, iters);  // warm-up at this size
        cudaEventRecord(a);
        td_int_peak_kernel<MIX><<<blocks, 256>>>(sink, iters);
        cudaEventRecord(b);
        if (cudaEventSynchronize(b) != cudaSuccess || cudaEventElapsedTime(&ms, a, b) != cudaSuccess) return -1;
        if (ms >= target_ms) break;
        iters *= 2;
    }
    *rate = (double)blocks * (256 / 32) * (double)iters * 16.0 / (ms * 1e-3);
    return 0;
}

}  // namespace

// Measures the integer issue peaks of `device` in warp instructions per
// second: the full issue rate (LOP3 and IMAD interleaved) and the ALU-pipe
// rate (LOP3 only), each over about `target_ms`.
TD_API int td_int_issue_peak(int device, float target_ms, double *issue_per_s, double *alu_per_s, char *err,
                             size_t errlen) {
    TD_CHECK(cudaSetDevice(device));
    int sms = 0;
    TD_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    uint32_t *sink = nullptr;
    TD_CHECK(cudaMalloc(&sink, sizeof(uint32_t) * sms * 32));
    cudaEvent_t a, b;
    TD_CHECK(cudaEventCreate(&a));
    TD_CHECK(cudaEventCreate(&b));
    double issue = 0, alu = 0;
    const int rc = (time_int_peak<1>(sms, target_ms, sink, a, b, &issue) == 0 &&
                    time_int_peak<0>(sms, target_ms, sink, a, b, &alu) == 0) ? 0 : -1;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(sink);
    TD_CHECK(cudaGetLastError());
    if (rc != 0) {
        set_err(err, errlen, "td_int_issue_peak: a probe launch failed");
        return TD_CUDA_ERROR;
    }
    if (issue_per_s) *issue_per_s = issue;
    if (alu_per_s) *alu_per_s = alu;
    return TD_OK;
}

// ---- batch search without device allocation ----------------------------------
//
// td_search_batch_noalloc is for callers that cannot call cudaMalloc or
// cudaFree: a slot worker that must not stall on the device-wide
// synchronisation those calls can imply while other slots' searches run on
// their own streams, or a host process whose device memory is already held by
// another allocator, so that a new allocation would fail although the caller's
// buffers exist.  The caller passes device buffers for instances and results;
// every other byte the search needs lives in td_noalloc_scratch below and in
// the tables that every search reads (td_eg_table, 8 MiB, is the largest), fixed
// arrays that each GPU loading this library holds until the process exits.
// Limits: TD_NOALLOC_MAX_INSTANCES instances per call and
// TD_NOALLOC_ITEMS donated subtrees in flight (when the item space is full the
// donor keeps the work, so a full item space only costs balance, not results).
// All calls share this one array and it keeps the last call's contents, so
// calls whose launches overlap on the GPU race with each other: serialise
// them (e.g. issue them on one stream).

#define TD_NOALLOC_MAX_INSTANCES 65536
#define TD_NOALLOC_ITEMS 65536
#define TD_NOALLOC_HEAD 256                                             // pool, epoch, ticket
#define TD_NOALLOC_STATE_OFF TD_NOALLOC_HEAD
#define TD_NOALLOC_ITEMS_OFF (TD_NOALLOC_STATE_OFF + TD_NOALLOC_MAX_INSTANCES * 16)
#define TD_NOALLOC_READY_OFF (TD_NOALLOC_ITEMS_OFF + TD_NOALLOC_ITEMS * 32)
#define TD_NOALLOC_BYTES (TD_NOALLOC_READY_OFF + TD_NOALLOC_ITEMS * 4)   // 3.25 MiB + 256 B

static_assert(sizeof(td_pool) + sizeof(td_epoch) + sizeof(int) <= TD_NOALLOC_HEAD, "scratch head");
static_assert(sizeof(td_inst_state) == 16 && sizeof(td_item) == 32, "scratch records");

static __device__ __align__(256) uint8_t td_noalloc_scratch[TD_NOALLOC_BYTES];

namespace {

constexpr int kNoAllocDevices = 64;

// error reporting without heap use
#define TD_CHECK_NA(call)                                                                          \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) {                                                                   \
            if (err && errlen)                                                                     \
                std::snprintf(err, errlen, "%s:%d: CUDA error %s (%s)", __FILE__, __LINE__,         \
                              cudaGetErrorName(e_), cudaGetErrorString(e_));                       \
            return TD_CUDA_ERROR;                                                                  \
        }                                                                                          \
    } while (0)
#define TD_FAIL_NA(...)                                            \
    do {                                                           \
        if (err && errlen) std::snprintf(err, errlen, __VA_ARGS__); \
        return TD_INVALID_ARG;                                     \
    } while (0)

struct NoAllocDevice {
    bool ready;
    uint8_t *scratch;  // device address of td_noalloc_scratch on this device
    int sms;
    int steal_blocks;
    int persistent_blocks;
};

std::mutex g_noalloc_mu;
NoAllocDevice g_noalloc[kNoAllocDevices];

// Once per device, with that device current: takes the scratch array's device
// address and sets the device's tables up (tables_setup).  In host code the
// name td_noalloc_scratch is only a host-side stand-in, never a device address.
int noalloc_setup(int device, char *err, size_t errlen) {
    NoAllocDevice &d = g_noalloc[device];
    if (d.ready) return TD_OK;
    void *ptr = nullptr;
    TD_CHECK_NA(cudaGetSymbolAddress(&ptr, td_noalloc_scratch));
    TD_CHECK_NA(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, device));
    const size_t smem = smem_bytes(4);
    // the limit holds for every launch of a kernel, so it must fit the 8-warp
    // blocks that td_configure allows too
    const int limit = (int)smem_bytes(8);
    TD_CHECK_NA(cudaFuncSetAttribute(td_plain_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
    TD_CHECK_NA(cudaFuncSetAttribute(td_plain_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
    TD_CHECK_NA(cudaFuncSetAttribute(td_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
    TD_CHECK_NA(cudaFuncSetAttribute(td_steal_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
    TD_CHECK_NA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.steal_blocks, td_steal_kernel, 128,
                                                              smem_bytes(4)));
    TD_CHECK_NA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.persistent_blocks, td_persistent_kernel,
                                                              128, smem));
    TD_CHECK_NA(tables_setup(device, d.sms));
    d.scratch = static_cast<uint8_t *>(ptr);
    d.ready = true;
    return TD_OK;
}

}  // namespace

// Batch search on the calling thread's current device that allocates no
// device memory.  d_instances / d_results: caller-owned device buffers of
// `count` records; flags as for td_search_batch_device (TD_FLAG_ORDERED,
// TD_FLAG_PLAIN, TD_FLAG_VERIFY).  Enqueues on `stream` and returns.  The
// first call on a device performs the one-time set-up above unless slots were
// made there before (a symbol-address query, and on a stream of its own the
// table uploads and the five launches that build the endgame table, about 5 ms,
// waited for), so make that first call before any stream capture.  count > 65536
// is rejected.
TD_API int td_search_batch_noalloc(int count, const td_instance *d_instances, td_result *d_results, unsigned flags,
                                   uint64_t max_exp, void *stream, char *err, size_t errlen) {
    if (count < 0 || count > TD_NOALLOC_MAX_INSTANCES)
        TD_FAIL_NA("td_search_batch_noalloc: count %d outside 0..%d (the fixed scratch holds at most %d instances)",
                   count, TD_NOALLOC_MAX_INSTANCES, TD_NOALLOC_MAX_INSTANCES);
    if (count == 0) return TD_OK;
    if (!d_instances || !d_results) TD_FAIL_NA("td_search_batch_noalloc: null instance or result buffer");
    int device = 0;
    TD_CHECK_NA(cudaGetDevice(&device));
    if (device < 0 || device >= kNoAllocDevices)
        TD_FAIL_NA("td_search_batch_noalloc: device ordinal %d out of range", device);
    NoAllocDevice d;
    {
        std::lock_guard<std::mutex> g(g_noalloc_mu);
        const int rc = noalloc_setup(device, err, errlen);
        if (rc != TD_OK) return rc;
        d = g_noalloc[device];
    }
    cudaStream_t st = (cudaStream_t)stream;
    const int warps = 4, threads = 128;
    const size_t smem = smem_bytes(warps);
    const bool ordered = flags & TD_FLAG_ORDERED;
    const uint64_t limit = time_limit_ns();
    td_pool *pool = reinterpret_cast<td_pool *>(d.scratch);
    td_epoch *epoch = reinterpret_cast<td_epoch *>(d.scratch + sizeof(td_pool));
    int *ticket = reinterpret_cast<int *>(d.scratch + sizeof(td_pool) + sizeof(td_epoch));
    td_inst_state *state = reinterpret_cast<td_inst_state *>(d.scratch + TD_NOALLOC_STATE_OFF);
    td_item *items = reinterpret_cast<td_item *>(d.scratch + TD_NOALLOC_ITEMS_OFF);
    uint32_t *ready = reinterpret_cast<uint32_t *>(d.scratch + TD_NOALLOC_READY_OFF);
    const int blocks_needed = (count + warps - 1) / warps;
    if (flags & TD_FLAG_PLAIN) {
        if (ordered)
            td_plain_kernel<true><<<blocks_needed, threads, smem, st>>>(d_instances, d_results, count, max_exp, limit);
        else
            td_plain_kernel<false><<<blocks_needed, threads, smem, st>>>(d_instances, d_results, count, max_exp, limit);
    } else if (ordered) {
        TD_CHECK_NA(cudaMemsetAsync(ticket, 0, sizeof(int), st));
        const int grid = std::max(1, std::min(d.sms * std::max(1, d.persistent_blocks), blocks_needed));
        td_persistent_kernel<<<grid, threads, smem, st>>>(d_instances, d_results, count, ticket, 1, max_exp,
                                                                limit);
    } else {
        // the donation settings, read together (a concurrent td_configure_steal
        // or td_configure_restart writes them under the same lock)
        int grain, split_level, check_every;
        uint32_t restart_base;
        {
            std::lock_guard<std::mutex> g(g_mu);
            grain = g_steal_grain;
            split_level = g_split_level;
            check_every = g_check_every;
            restart_base = g_restart_base;
        }
        // the counters start afresh on every call; items
        // are tagged with a fresh epoch so an earlier call's items never count
        td_epoch_kernel<<<1, 1, 0, st>>>(epoch, 1u, pool, count, nullptr, 0, ready, TD_NOALLOC_ITEMS, nullptr, 0);
        // the whole resident grid (the scratch does not depend on its size):
        // warps without an instance of their own take donated subtrees, so a
        // small batch is spread over the GPU
        const int grid = d.sms * std::max(1, d.steal_blocks);
        td_steal_kernel<<<grid, threads, smem_bytes(warps), st>>>(
            d_instances, d_results, count, pool, items, ready, epoch, TD_NOALLOC_ITEMS, state, grain, split_level,
            check_every, limit, nullptr, 64, 1u, restart_base, max_exp, /*race=*/0);
        TD_CHECK_NA(cudaGetLastError());
        td_finalize_kernel<<<std::max(1, std::min((count + 255) / 256, 2 * d.sms)), 256, 0, st>>>(pool, state,
                                                                                                d_results, count);
    }
    TD_CHECK_NA(cudaGetLastError());
    if (flags & TD_FLAG_VERIFY) {
        td_validate_kernel<<<(count + 255) / 256, 256, 0, st>>>(d_instances, d_results, nullptr, count, 1);
        TD_CHECK_NA(cudaGetLastError());
    }
    return TD_OK;
}

// ---- CUDA graphs -------------------------------------------------------------

namespace {
struct BatchGraph {
    int device;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};
}  // namespace

// Captures one batch launch (search, and the device replay when flags has
// TD_FLAG_VERIFY) over fixed device buffers into a CUDA graph.  Replaying it
// with td_batch_graph_launch costs one graph launch per batch.
TD_API int td_batch_graph_create(int slot, int count, const td_instance *d_in, td_result *d_out, unsigned flags,
                                 uint64_t max_exp, void **out_graph, char *err, size_t errlen) {
    Slot *s;
    {
        std::lock_guard<std::mutex> g(g_mu);
        s = get_slot(slot, err, errlen);
        if (!s) return TD_INVALID_ARG;
    }
    if (!out_graph || count <= 0) {
        set_err(err, errlen, "invalid graph arguments");
        return TD_INVALID_ARG;
    }
    percall_park(s->device);
    std::lock_guard<std::mutex> g(*s->mu);
    TD_CHECK(cudaSetDevice(s->device));
    // one eager launch sizes the slot's scratch outside the capture
    int rc = launch_batch(*s, count, d_in, d_out, flags, max_exp, s->stream, err, errlen);
    if (rc != TD_OK) return rc;
    TD_CHECK(cudaStreamSynchronize(s->stream));
    s->captured = true;
    auto *bg = new BatchGraph();
    bg->device = s->device;
    cudaError_t e = cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        rc = launch_batch(*s, count, d_in, d_out, flags, max_exp, s->stream, err, errlen);
        e = cudaStreamEndCapture(s->stream, &bg->graph);
        if (rc != TD_OK) {
            if (bg->graph) cudaGraphDestroy(bg->graph);
            delete bg;
            return rc;
        }
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&bg->exec, bg->graph, 0);
    if (e != cudaSuccess) {
        if (bg->graph) cudaGraphDestroy(bg->graph);
        delete bg;
        set_err(err, errlen, cuda_msg(e, __FILE__, __LINE__));
        return TD_CUDA_ERROR;
    }
    *out_graph = bg;
    return TD_OK;
}

TD_API int td_batch_graph_launch(void *graph, void *stream, char *err, size_t errlen) {
    auto *bg = static_cast<BatchGraph *>(graph);
    if (!bg) return TD_INVALID_ARG;
    percall_park(bg->device);
    TD_CHECK(cudaSetDevice(bg->device));
    TD_CHECK(cudaGraphLaunch(bg->exec, (cudaStream_t)stream));
    return TD_OK;
}

TD_API int td_batch_graph_destroy(void *graph) {
    auto *bg = static_cast<BatchGraph *>(graph);
    if (!bg) return TD_INVALID_ARG;
    cudaSetDevice(bg->device);
    if (bg->exec) cudaGraphExecDestroy(bg->exec);
    if (bg->graph) cudaGraphDestroy(bg->graph);
    delete bg;
    return TD_OK;
}

#include "td_serve.cuh"
#include "td_percall.cuh"

// defined in td_cert.cu
int td_cert_preload(void);

namespace {

int preload_kernels(char *err, size_t errlen) {
    cudaFuncAttributes a;
    TD_CHECK(cudaFuncGetAttributes(&a, td_plain_kernel<true>));
    TD_CHECK(cudaFuncGetAttributes(&a, td_plain_kernel<false>));
    TD_CHECK(cudaFuncGetAttributes(&a, td_persistent_kernel));
    TD_CHECK(cudaFuncGetAttributes(&a, td_steal_kernel));
    TD_CHECK(cudaFuncGetAttributes(&a, td_ordered_kernel));
    TD_CHECK(cudaFuncGetAttributes(&a, td_epoch_kernel));
    TD_CHECK(cudaFuncGetAttributes(&a, td_eg_build_kernel));
    TD_CHECK(cudaFuncGetAttributes(&a, td_finalize_kernel));
    TD_CHECK(cudaFuncGetAttributes(&a, td_count_kernel));
    TD_CHECK(cudaFuncGetAttributes(&a, td_validate_kernel));
    TD_CHECK(cudaFuncGetAttributes(&a, td_pairs_prepare_kernel));
    TD_CHECK(cudaFuncGetAttributes(&a, td_pairs_unpack_kernel));
    TD_CHECK(cudaFuncGetAttributes(&a, td_int_peak_kernel<0>));
    TD_CHECK(cudaFuncGetAttributes(&a, td_int_peak_kernel<1>));
    TD_CHECK(cudaFuncGetAttributes(&a, td_serve_kernel<TD_SERVE_FREE>));
    TD_CHECK(cudaFuncGetAttributes(&a, td_serve_kernel<TD_SERVE_ORDERED>));
    TD_CHECK(cudaFuncGetAttributes(&a, td_serve_kernel<TD_SERVE_PER_REQUEST>));
    TD_CHECK((cudaError_t)td_cert_preload());
    return TD_OK;
}

}  // namespace
