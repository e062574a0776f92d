// gdp_batch.cu -- the batched engine: many problems (instances) or many
// bound vectors of one problem (branch-and-bound nodes) propagated together
// in one persistent cooperative launch.
//
// Each batch member ("unit") is a DevProblem: its own bounds, change bitmap,
// marks and round flags, over its own layout (instances) or a layout shared
// with the other units (nodes). Every unit follows exactly the Jacobi rounds
// it would follow alone -- units never read each other's bounds -- so its
// bounds, round count and infeasibility verdict equal those of a
// single-problem propagation. What the batch adds is scheduling:
//   * one work list per round across all units: (unit, slice/tile) entries
//     queued when a changed variable marks a row, plus full sweeps (a
//     virtual range over a unit's work items) for units whose last round
//     tightened many bounds;
//   * a unit leaves the loop the round it converges or turns infeasible, so
//     short and long propagations share the launch without waiting rounds;
//   * nodes start from the marks of the variables whose bounds differ from a
//     certified fixpoint of the same problem (every other row is at its
//     fixpoint already and would find nothing).
// The round loop runs in one cooperative kernel (grid barriers between the
// phases, bounded waits) and the whole device part of a call is built once as a
// CUDA graph and replayed.
//
// Reference: the reference propagates one problem per call
// (include/interface.h:10-251); its GPU round loop is
// src/propagators/GPU_propagator.cuh:160-255.
#include "gdp_batch.h"

#include <algorithm>
#include <chrono>
#include <cstring>

#include "gdp_learned.cuh"
#include "gdp_sequence.h"
#include "gdp_sweep.h"

namespace gdp {

namespace {

// Finds the unit whose half-open range [base[u], base[u+1]) holds x.
__device__ __forceinline__ int find_unit(const int *base, int n_units, int x) {
    int lo = 0, hi = n_units;  // base[lo] <= x < base[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(base + mid) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void push_entry(const BatchDev &B, int par, int u, int item) {
    const unsigned idx = atomicAdd(B.tail + par, 1u);
    if (idx >= B.cap_entries) {
        atomicExch(B.error, (int)kErrQueueOverflow);
        return;
    }
    B.entries[(size_t)par * B.cap_entries + idx] = ((unsigned long long)(unsigned)u << 32) | (unsigned)item;
}

__device__ __forceinline__ void push_tile(unsigned long long *q, unsigned *tail, unsigned cap, int *error, int u,
                                          int t) {
    const unsigned idx = atomicAdd(tail, 1u);
    if (idx >= cap) {
        atomicExch(error, (int)kErrQueueOverflow);
        return;
    }
    q[idx] = ((unsigned long long)(unsigned)u << 32) | (unsigned)t;
}

// The rows of the changed variables of a warp (lane l's variable if `on`, its
// index entries [k0, k1)) of unit u are marked and queued for round `stamp`:
// variable by variable, 32 entries at a time (a thread that walks its
// variables' rows alone makes up to four dependent trips to L2 for each). A
// slice is queued once per round, a split row with all its tiles; the queue
// slots of a step's slices are reserved together. Learned units: SELL rows
// turn dirty instead of marked (learned_mark_position).
template <bool kLearned>
__device__ __forceinline__ void push_rows(const BatchDev &B, const DevProblem &Pu, int u, bool on, int k0, int k1,
                                          int stamp, int lane) {
    const int par = stamp & 1;
    unsigned long long *ent = B.entries + (size_t)par * B.cap_entries;
    const unsigned long long unit = (unsigned long long)(unsigned)u << 32;
    const bool lrn = kLearned && Pu.learned == 1;
    for (unsigned vars = __ballot_sync(kFull, on && k0 < k1); vars; vars &= vars - 1) {
        const int src = __ffs(vars) - 1;
        const int e0 = __shfl_sync(kFull, k0, src), e1 = __shfl_sync(kFull, k1, src);
        for (int e = e0; e < e1; e += 32) {
            bool fresh = false;
            int slice = 0;
            if (e + lane < e1) {
                const int p = __ldg(&Pu.var_ent[e + lane].pos);
                if (p < Pu.n_srows) {
                    slice = __ldg(Pu.pos_slice + p);
                    if (lrn) {
                        atomicAdd(Pu.dcount + p, 1);
                        if (Pu.dirty[p] == 0) atomicCAS(Pu.dirty + p, 0, stamp);
                    } else {
                        Pu.mark[p] = stamp;
                    }
                    fresh = __ldcg(Pu.slice_stamp + slice) != stamp &&
                            atomicExch(Pu.slice_stamp + slice, stamp) != stamp;
                } else if (atomicExch(Pu.mark + p, stamp) != stamp) {
                    const int row = p - Pu.n_srows;
                    const int t0 = __ldg(Pu.lrow_tile0 + row), nt = __ldg(Pu.lrow_tile0 + row + 1) - t0;
                    const unsigned at = atomicAdd(B.tail + par, (unsigned)nt);
                    if ((unsigned long long)at + nt > B.cap_entries) atomicExch(B.error, (int)kErrQueueOverflow);
                    else
                        for (int t = 0; t < nt; t++) ent[at + t] = unit | (unsigned)(-(t0 + t) - 1);
                }
            }
            const unsigned bal = __ballot_sync(kFull, fresh);
            if (!bal) continue;
            unsigned at = 0;
            if (lane == 0) at = atomicAdd(B.tail + par, (unsigned)__popc(bal));
            at = __shfl_sync(kFull, at, 0);
            if ((unsigned long long)at + __popc(bal) > B.cap_entries) {
                if (lane == 0) atomicExch(B.error, (int)kErrQueueOverflow);
            } else if (fresh) {
                ent[at + __popc(bal & ((1u << lane) - 1u))] = unit | (unsigned)slice;
            }
        }
    }
}

// A warp's copy of the unit it works on, in shared memory: the fields are
// pointers and sizes that do not change during the launch, and every access
// through a unit in global memory is one more dependent load (from L2 after
// each barrier). Turning to unit u, statistics gathered for another one go to
// its flags.
struct UnitCache {
    alignas(16) unsigned char raw[sizeof(DevProblem)];
};
__device__ __forceinline__ const DevProblem &unit_of(const BatchDev &B, UnitCache &c, WarpSmem &ws, int &unit, int u,
                                                     int lane) {
    static_assert(sizeof(DevProblem) % 8 == 0 && alignof(DevProblem) <= 16, "copied by 8-byte words");
    if (unit != u) {
        if (unit >= 0) stats_flush(*reinterpret_cast<const DevProblem *>(c.raw), ws, lane);
        __syncwarp();
        const unsigned long long *src = reinterpret_cast<const unsigned long long *>(B.units + u);
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(c.raw);
        for (int i = lane; i < (int)(sizeof(DevProblem) / 8); i += 32) dst[i] = __ldg(src + i);
        __syncwarp();
        unit = u;
    }
    return *reinterpret_cast<const DevProblem *>(c.raw);
}

// One warp builds the list of units swept in full in the next round, in unit
// order, with the prefix of their work-item counts, while the rest of its CTA
// commits (with the whole CTA on the list first, a round of few changes waited
// for it: 8 chain MIPs 31.8 ms, 31.4 so).
template <class Pred>
__device__ void build_full_sweep_list(const BatchDev &B, int lane, Pred &&pred) {
    int units = 0, before = 0;  // listed so far, their items
    for (int u0 = 0; u0 < B.n_units; u0 += 32) {
        const int u = u0 + lane;
        const bool f = u < B.n_units && pred(u);
        const int items = f ? B.units[u].n_items : 0;
        const unsigned listed = __ballot_sync(kFull, f);
        int upto = items;  // inclusive scan
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(kFull, upto, off);
            if (lane >= off) upto += v;
        }
        if (f) {
            const int k = units + __popc(listed & ((1u << lane) - 1u));
            B.fs_unit[k] = u;
            B.fs_prefix[k] = before + upto - items;
        }
        units += __popc(listed);
        before += __shfl_sync(kFull, upto, 31);
    }
    if (lane == 0) {
        B.fs_prefix[units] = before;
        B.n_fs[0] = units;
    }
}

// The kind of round r + 1 of learned unit Pu after round r.
__device__ __forceinline__ int unit_next_kind(const DevProblem &Pu, int r) {
    const RoundFlags &fr = Pu.flags[1 + (r & 1)];
    return learned_next_kind(fr.kind, fr.tight, fr.rows_deferred, Pu.n_srows, Pu.use_marking);
}
// A learned unit is finished after round r when it turned infeasible or a
// FULL or FLUSH round changed nothing (its certification).
__device__ __forceinline__ bool unit_certified(const DevProblem &Pu, int r) {
    const RoundFlags &fr = Pu.flags[1 + (r & 1)];
    return learned_certifies(fr.kind, fr.tight);
}

// Round bookkeeping of unit u after round r (every phase of r is complete).
__device__ __forceinline__ void close_round(const BatchDev &B, int u, int r) {
    RoundFlags &f0 = B.units[u].flags[0];
    if (f0.done) return;
    f0.rounds = r;
    if (B.units[u].learned == 1) {
        const bool cert = unit_certified(B.units[u], r);
        if (B.units[u].flags[1 + (r & 1)].kind == kRoundFull) f0.full_rounds += 1;
        if (f0.infeasible || cert || r >= B.max_rounds) {
            f0.done = 1;
            f0.change = (f0.infeasible || cert) ? B.units[u].flags[1 + (r & 1)].change : 1;
        }
        return;
    }
    const int ch = B.units[u].flags[1 + (r & 1)].change;
    if (f0.infeasible) {
        f0.done = 1;
        f0.change = ch;
    } else if (!ch || r >= B.max_rounds) {
        f0.done = 1;
        f0.change = ch;
    }
}

__device__ __forceinline__ bool unit_next_marked(const DevProblem &Pu, int r) {
    return next_round_marked(Pu, Pu.flags[1 + (r & 1)].tight);
}

}  // namespace

namespace {

// ---- the persistent round loop ----------------------------------------------
// Round r (par = r & 1):
//   A  work list of round r: full-sweep items (virtual range over fs_unit),
//      then queued entries[par]; split tiles of multi-tile rows go to cq.
//   B  cq: row screens of multi-tile rows; tiles needing the exact pass go to xq.
//   C  xq (only if not empty): exact partials combined, candidates, a tile's in
//      quarters on four warps (24 mixed instances 10.4 -> 9.9 ms, 64 nodes of 50,000
//      rows 12.13 -> 11.76).
//   F  commit changed variables of every unit; mark and queue rows for r + 1
//      (units staying on marked rounds), full-sweep list for r + 1.
// After F every CTA reads the same next-round work size and leaves together.
// kLearned: units with a model (learned == 1) run learned rounds (gdp_learned.cu)
// -- each unit its own sequence of FULL / LEARNED / FLUSH rounds, the kind of
// round r in flags[1 + (r & 1)].kind; a slice whose marked rows the model
// deferred is queued again for the next round, and a unit ends only with a FULL
// round that changes nothing, exactly as in its single-problem learned run.
// kCtas per SM: 3 (80 registers), or 2 (128) for batches with little work in a
// round (Batch::size_grid) and for learned ones (32 chain MIPs, 3.3M rows: 189 ms
// with 3, 182 with 2).
template <bool kLearned, int kCtas>
__global__ void __launch_bounds__(kCtaThreads, kCtas) k_batch_loop(BatchDev B) {
    WarpSmem *ws = warp_smem();
    __shared__ LearnSmem ls[kLearned ? kWarpsPerCta : 1];
    const int lane = threadIdx.x & 31;
    WarpSmem &mine = ws[threadIdx.x >> 5];
    __shared__ UnitCache units[kWarpsPerCta];
    UnitCache &cache = units[threadIdx.x >> 5];
    LearnSmem &L = ls[kLearned ? (threadIdx.x >> 5) : 0];
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gthreads = gridDim.x * blockDim.x;
    int last = 0;
    unsigned target = 0;  // grid barrier
    int unit = -1;        // unit in the warp's cache, which its statistics belong to
    stats_zero(mine, lane);
    // the round's work: units in the full sweep, their items, queued entries
    int nfs = *((volatile int *)B.n_fs), fs_items = *((volatile int *)(B.fs_prefix + nfs));
    int n_entries = (int)min(*((volatile unsigned *)(B.tail + 1)), B.cap_entries);
    for (int r = 1; r <= B.max_rounds; r++) {
        const int par = r & 1;
        unsigned *ctr = B.ctr + 4 * par;
        // close round r - 1 for every unit (its flags are final); the entry
        // queue of round r - 1 (parity par ^ 1) was emptied in its phase B and
        // fills for round r + 1 (phase A: slices with deferred rows, phase F)
        if (r > 1)
            for (int u = gtid; u < B.n_units; u += gthreads) close_round(B, u, r - 1);
        // ---- A
        {
            const unsigned long long *ent = B.entries + (size_t)par * B.cap_entries;
            const int n_work = fs_items + n_entries;
            WarpCursor<false> cur;
            cur.start(ctr + 0, 1, grid_warps(), n_work);
            for (;;) {
                const int i = cur.next(lane);
                if (i >= n_work) break;
                int u, it;
                bool marked;
                if (i < fs_items) {
                    const SweepItem at = sweep_item(B.fs_prefix, nfs, fs_items, i);
                    u = B.fs_unit[at.unit];
                    it = __ldg(B.units[u].items + at.item);
                    marked = false;
                } else {
                    const unsigned long long e = ent[i - fs_items];
                    u = (int)(e >> 32);
                    it = (int)(unsigned)e;
                    marked = true;
                }
                const DevProblem &Pu = unit_of(B, cache, mine, unit, u, lane);
                const bool due = *((volatile int *)&Pu.flags[0].infeasible) == 0;
                int *change = &Pu.flags[1 + par].change;
                unsigned *tight = &Pu.flags[1 + par].tight;
                if (kLearned && Pu.learned == 1) {
                    if (!due) continue;
                    const int kind = Pu.flags[1 + par].kind;
                    if (it >= 0) {
                        if (lane == 0) L.marked = 0;
                        __syncwarp();
                        const bool deferred = sell_slice_learned<0>(Pu, it, lane, r, kind, change, tight, mine, L);
                        if (lane == 0) {
                            if (L.marked) atomicAdd(&Pu.flags[1 + par].rows_deferred, L.marked);
                            if (deferred && r < B.max_rounds && atomicExch(Pu.slice_stamp + it, r + 1) != r + 1)
                                push_entry(B, par ^ 1, u, it);
                        }
                    } else if (split_partial<0>(Pu, -it - 1, lane, r, kind != kRoundFull, change, tight, mine) &&
                               lane == 0) {
                        push_tile(B.cq, B.tail + 2, B.cap_tiles, B.error, u, -it - 1);
                    }
                } else if (it >= 0) {
                    sell_slice<0, false>(Pu, it, lane, r, marked, change, tight, mine, 0, 0, 1, due);
                } else if (due && split_partial<0>(Pu, -it - 1, lane, r, marked, change, tight, mine) && lane == 0) {
                    push_tile(B.cq, B.tail + 2, B.cap_tiles, B.error, u, -it - 1);
                }
            }
        }
        if (!grid_barrier(B.barrier, B.error, B.spin_limit, target)) return;
        // ---- B (plus the resets for round r + 1: its slots were last used in r - 1)
        if (gtid == 0) {
            unsigned *nctr = B.ctr + 4 * (par ^ 1);
            nctr[0] = 0u; nctr[1] = 0u; nctr[2] = 0u; nctr[3] = 0u;
            B.tail[par] = 0u;  // round r's entry queue is consumed; it fills again in round r + 1
        }
        for (int u = gtid; u < B.n_units; u += gthreads) {
            RoundFlags &fn = B.units[u].flags[1 + (par ^ 1)];
            fn.change = 0; fn.tight = 0u; fn.exact = 0;
            fn.rows_deferred = 0ULL;  // learned units: marked rows met in the round
        }
        const int n_cq = (int)min(*((volatile unsigned *)(B.tail + 2)), B.cap_tiles);
        if (n_cq) {
            WarpCursor<false> cur;
            cur.start(ctr + 1, 1, grid_warps(), n_cq);
            for (;;) {
                const int i = cur.next(lane);
                if (i >= n_cq) break;
                const unsigned long long e = B.cq[i];
                const int u = (int)(e >> 32), t = (int)(unsigned)e;
                const DevProblem &Pu = unit_of(B, cache, mine, unit, u, lane);
                if (split_cand<0>(Pu, t, lane, r, false, &Pu.flags[1 + par].exact, mine) && lane == 0)
                    push_tile(B.xq, B.tail + 3, B.cap_tiles, B.error, u, t);
            }
            if (!grid_barrier(B.barrier, B.error, B.spin_limit, target)) return;
            // ---- C
            const int n_xq = (int)min(*((volatile unsigned *)(B.tail + 3)), B.cap_tiles);
            if (n_xq) {
                WarpCursor<false> curx;
                const int parts = n_xq <= INT_MAX / kTileParts ? kTileParts : 1;
                curx.start(ctr + 2, 1, grid_warps(), parts * n_xq);
                for (;;) {
                    const int i = curx.next(lane);
                    if (i >= parts * n_xq) break;
                    const unsigned long long e = B.xq[i / parts];
                    const int u = (int)(e >> 32), t = (int)(unsigned)e;
                    const DevProblem &Pu = unit_of(B, cache, mine, unit, u, lane);
                    split_exact<0>(Pu, t, lane, r, &Pu.flags[1 + par].change, &Pu.flags[1 + par].tight, mine,
                                   i % parts, parts);
                }
                if (!grid_barrier(B.barrier, B.error, B.spin_limit, target)) return;
            }
        }
        // ---- F (a row recorded infeasible in round r turns into the unit's
        // verdict here, where the variable rule sets it)
        for (int u = gtid; u < B.n_units; u += gthreads)
            if (B.units[u].flags[0].infeasible_row != INT_MAX) B.units[u].flags[0].infeasible = 1;
        const bool more = r < B.max_rounds;
        if (blockIdx.x == 0) {
            if (more && threadIdx.x < 32)
                build_full_sweep_list(B, lane, [&](int u) {
                    const DevProblem &Pu = B.units[u];
                    if (kLearned && Pu.learned == 1)
                        return !Pu.flags[0].done && !Pu.flags[0].infeasible && !unit_certified(Pu, r) &&
                               unit_next_kind(Pu, r) == kRoundFull;
                    return !Pu.flags[0].done && Pu.flags[1 + par].change && !unit_next_marked(Pu, r);
                });
            else if (!more && threadIdx.x == 0) {
                B.n_fs[0] = 0;
                B.fs_prefix[0] = 0;
            }
            if (threadIdx.x == 0) { B.tail[2] = 0u; B.tail[3] = 0u; }
            if (kLearned) {  // learned units that need round r + 1 even without queued work
                __shared__ int s_pend;
                if (threadIdx.x == 0) s_pend = 0;
                __syncthreads();
                for (int u = threadIdx.x; u < B.n_units; u += blockDim.x) {
                    const DevProblem &Pu = B.units[u];
                    if (Pu.learned == 1 && more && !Pu.flags[0].done && !Pu.flags[0].infeasible &&
                        !unit_certified(Pu, r))
                        atomicAdd(&s_pend, 1);
                }
                __syncthreads();
                if (threadIdx.x == 0) B.n_pending[0] = s_pend;
            }
        }
        if (kLearned)
            for (int u = gtid; u < B.n_units; u += gthreads)
                if (B.units[u].learned == 1) B.units[u].flags[1 + (par ^ 1)].kind = unit_next_kind(B.units[u], r);
        // the units' bitmaps are one array of words: a warp reads a few of them
        // at a time, commits a word's 32 variables with a lane each and pushes
        // their rows together
        {
            const int nw = grid_warps();
            int gw = 1;  // words of a claim: about four claims per warp, at most 32 words
            while (gw < 32 && 8LL * gw * nw <= B.total_words) gw <<= 1;
            const int groups = (B.total_words + gw - 1) / gw;
            WarpCursor<false> cur;
            cur.start(ctr + 3, 1, nw, groups);
            for (;;) {
                const int grp = cur.next(lane);
                if (grp >= groups) break;
                const int w0 = grp * gw;
                unsigned my = 0u;
                if (lane < gw && w0 + lane < B.total_words) {
                    my = __ldcg(B.chg + w0 + lane);
                    if (my) B.chg[w0 + lane] = 0u;
                }
                for (unsigned words = __ballot_sync(kFull, my != 0u); words; words &= words - 1) {
                    const int q = __ffs(words) - 1;
                    const unsigned bits = __shfl_sync(kFull, my, q);
                    const int u = find_unit(B.wbase, B.n_units, w0 + q);
                    const DevProblem &Pu = unit_of(B, cache, mine, unit, u, lane);
                    const bool on = (bits >> lane) & 1u;
                    const int j = (w0 + q - __ldg(B.wbase + u)) * 32 + lane;
                    int k0 = 0, k1 = 0;
                    double2 b = make_double2(0.0, 0.0);
                    if (on) {
                        b = Pu.bnd_nxt[j];
                        k0 = __ldg(Pu.var_ptr + j);
                        k1 = __ldg(Pu.var_ptr + j + 1);
                    }
                    if (lane == 0) atomicAdd(&Pu.flags[0].changed_vars, (unsigned long long)__popc(bits));
                    const bool lrn = kLearned && Pu.learned == 1;
                    const bool push = more && (lrn ? (!unit_certified(Pu, r) && unit_next_kind(Pu, r) != kRoundFull)
                                                   : unit_next_marked(Pu, r));
                    if (on) {
                        Pu.bnd[j] = b;
                        store_bnd32<0>(Pu, j, b, r);
                        if (var_infeasible(b.x, b.y)) {
                            Pu.flags[0].infeasible = 1;
                            atomicMin(&Pu.flags[0].infeasible_var, j);
                        }
                    }
                    if (push) push_rows<kLearned>(B, Pu, u, on, k0, k1, r + 1, lane);
                }
            }
        }
        if (!grid_barrier(B.barrier, B.error, B.spin_limit, target)) return;
        last = r;
        nfs = *((volatile int *)B.n_fs);
        n_entries = (int)min(*((volatile unsigned *)(B.tail + (par ^ 1))), B.cap_entries);
        fs_items = *((volatile int *)(B.fs_prefix + nfs));
        const int next = fs_items + n_entries;
        const int pending = kLearned ? *((volatile int *)B.n_pending) : 0;
        if (!more || (next == 0 && pending == 0)) break;
    }
    if (unit >= 0) stats_flush(*reinterpret_cast<const DevProblem *>(cache.raw), mine, lane);
    for (int u = gtid; u < B.n_units; u += gthreads) close_round(B, u, last);
    if (gtid == 0) B.rounds_out[0] = last;
}

// Initial state of every unit: interleaved bounds, cleared bitmaps and marks,
// the round-0 infeasibility check.
__global__ void __launch_bounds__(256) k_batch_init(BatchDev B, const double *lb, const double *ub,
                                                     const long long *var_base) {
    const int u = blockIdx.y;
    const DevProblem &Pu = B.units[u];
    const long long vb = var_base[u];
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < Pu.n; j += gridDim.x * blockDim.x) {
        const double2 b = make_double2(lb[vb + j], ub[vb + j]);
        Pu.bnd[j] = b;
        Pu.bnd_nxt[j] = b;
        store_bnd32<0>(Pu, j, b, 0);
        if (var_infeasible(b.x, b.y)) {
            Pu.flags[0].infeasible = 1;
            atomicMin(&Pu.flags[0].infeasible_var, j);
        }
    }
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < Pu.n_chg_words; w += gridDim.x * blockDim.x)
        Pu.chg[w] = 0u;
    const int npos = Pu.n_srows + Pu.n_lrows;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += gridDim.x * blockDim.x) Pu.mark[p] = 0;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < Pu.n_slices; s += gridDim.x * blockDim.x)
        Pu.slice_stamp[s] = 0;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < Pu.n_lrows; r += gridDim.x * blockDim.x)
        Pu.row_exact[r] = 0;
    if (Pu.learned == 1)
        for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < Pu.n_srows; p += gridDim.x * blockDim.x) {
            Pu.dirty[p] = 0;
            Pu.dcount[p] = 0;
            Pu.last_proc[p] = 0;
            Pu.last_tight[p] = 0;
            Pu.rstat[p] = make_float2(0.f, 0.f);
            Pu.rinfo[p] = 0u;
        }
}

// Round-1 marks of units started from a certified fixpoint `ref` of their
// problem: the rows of every variable whose bounds differ from it.
__global__ void __launch_bounds__(256) k_batch_seed_marks(BatchDev B, const double2 *ref, const int *seed_mode) {
    const int u = blockIdx.y;
    const DevProblem &Pu = B.units[u];
    if (seed_mode[u] != 1 || Pu.flags[0].infeasible) return;
    const int lane = threadIdx.x & 31;
    for (int j0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); j0 < Pu.n; j0 += gridDim.x * blockDim.x) {
        const int j = j0 + lane;
        bool on = false;
        int k0 = 0, k1 = 0;
        if (j < Pu.n) {
            const double2 a = Pu.bnd[j], b = ref[j];
            on = dbits(a.x) != dbits(b.x) || dbits(a.y) != dbits(b.y);
            if (on) {
                k0 = __ldg(Pu.var_ptr + j);
                k1 = __ldg(Pu.var_ptr + j + 1);
            }
        }
        push_rows<false>(B, Pu, u, on, k0, k1, 1, lane);
    }
}

// Round-1 full-sweep list (units with seed_mode 0) and round-0 bookkeeping.
__global__ void __launch_bounds__(kCtaThreads) k_batch_plan(BatchDev B, const int *seed_mode) {
    for (int u = threadIdx.x; u < B.n_units; u += blockDim.x) {
        RoundFlags &f0 = B.units[u].flags[0];
        if (f0.infeasible) {  // infeasible before any round
            f0.done = 1;
            f0.rounds = 0;
        }
    }
    __syncthreads();
    if (threadIdx.x < 32)
        build_full_sweep_list(B, threadIdx.x, [&](int u) { return seed_mode[u] == 0 && !B.units[u].flags[0].infeasible; });
}

__global__ void __launch_bounds__(256) k_batch_fini(BatchDev B, double *lb, double *ub, const long long *var_base) {
    const int u = blockIdx.y;
    const DevProblem &Pu = B.units[u];
    const long long vb = var_base[u];
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < Pu.n; j += gridDim.x * blockDim.x) {
        const double2 b = Pu.bnd[j];
        lb[vb + j] = b.x;
        ub[vb + j] = b.y;
    }
}

}  // namespace

// ---- launchers --------------------------------------------------------------
namespace {
const void *batch_loop(bool learned, bool little) {
    if (learned) return (const void *)k_batch_loop<true, 2>;
    return little ? (const void *)k_batch_loop<false, 2> : (const void *)k_batch_loop<false, 3>;
}
}  // namespace

int batch_occupancy(int *blocks_per_sm, bool learned, bool little) {
    const void *k = batch_loop(learned, little);
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCtaSmem);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k, kCtaThreads, kCtaSmem);
}

int launch_batch(const BatchDev &B, int grid, const double *lb, const double *ub, double *lb_out,
                 double *ub_out, const long long *var_base, int max_unit_n, const double2 *ref,
                 const int *seed_mode, bool learned, bool little, Sequence &seq) {
    const dim3 vgrid((unsigned)std::max(1, std::min((max_unit_n + 255) / 256, 64)), (unsigned)B.n_units);
    BatchDev Bc = B;
    void *init[] = {&Bc, &lb, &ub, &var_base}, *seed[] = {&Bc, &ref, &seed_mode}, *plan[] = {&Bc, &seed_mode},
         *loop[] = {&Bc}, *fini[] = {&Bc, &lb_out, &ub_out, &var_base};
    cudaError_t e = seq.kernel((const void *)k_batch_init, vgrid, 256, init, 0);
    if (e == cudaSuccess && ref) e = seq.kernel((const void *)k_batch_seed_marks, vgrid, 256, seed, 0);
    if (e == cudaSuccess) e = seq.kernel((const void *)k_batch_plan, 1, kCtaThreads, plan, 0);
    if (e == cudaSuccess) e = seq.kernel(batch_loop(learned, little), grid, kCtaThreads, loop, kCtaSmem, true);
    if (e == cudaSuccess) e = seq.kernel((const void *)k_batch_fini, vgrid, 256, fini, 0);
    return (int)e;
}

}  // namespace gdp
