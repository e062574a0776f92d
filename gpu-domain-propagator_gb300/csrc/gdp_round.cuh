// gdp_round.cuh -- the device side of one Jacobi propagation round, shared
// by the single-problem kernels (gdp_round.cu) and the batched engine
// (gdp_batch.cu).
//
// A round reads the round-start bounds (cur), writes every tightening into nxt
// with an FP64 min/max atomic and flags the variable in a bitmap; the finalize
// phase copies flagged variables nxt -> cur, applies the infeasibility rule
// and marks the rows of changed variables for the next round. The result does
// not depend on scheduling: each row's sums run in a fixed order from the
// snapshot and min/max commute.
//
// GB300's FP64 pipe (about 1.75 lane-ops per clock per SM) is the scarce
// resource, so the kernels spend it only on rows that an FP32 interval screen
// could not prove skippable, and there on the arithmetic of gdp_exact.cuh.
// Classification against the +-1e20 infinity thresholds is integer work on the
// bit patterns.
//
// Reference: the round body of GPUAtomicDomainPropagation
// (src/kernels/atomic_kernel.cuh:9-450) and of the megakernel
// (src/kernels/atomic_megakernel.cuh:14-490), re-planned for a snapshot
// schedule; math from src/propagation_methods.cuh:78-276.
#pragma once

#include <climits>
#include <cuda_runtime.h>

#include "gdp_device.cuh"
#include "gdp_exact.cuh"
#include "gdp_internal.h"

namespace gdp {
namespace {

// Phase timers, compiled only into a library built with -DGDP_PHASE_TIMERS
// (build.py --phase-timers): the megakernel stamps %globaltimer at the start of
// each round and after each of its grid barriers, every warp adds the time it
// spends in each phase, and the exact pass of SELL rows adds its two passes'
// warp time by lane-group size. In the plain build timer_now() is 0 and the
// recording calls are empty.
constexpr int kTimerRounds = 1024;  // rounds recorded (later rounds are not)
constexpr int kTimerSlots = 8;      // per round: 5 stamps + 3 work counters; 5 phase busy sums
constexpr int kTimerPass = 16;      // 2 passes x lane-group sizes 1..32, then one-lane row work
#ifdef GDP_PHASE_TIMERS
__device__ unsigned long long g_timer_wall[kTimerRounds * kTimerSlots];
__device__ unsigned long long g_timer_busy[kTimerRounds * kTimerSlots];
__device__ unsigned long long g_timer_pass[kTimerPass];
__device__ __forceinline__ unsigned long long timer_now() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// warp time of the exact pass's pass 1 [t0, t1) and pass 2 [t1, now)
__device__ __forceinline__ void timer_pass(int lane, int lg, unsigned long long t0, unsigned long long t1) {
    if (lane == 0) {
        const unsigned long long t2 = timer_now();
        atomicAdd(&g_timer_pass[2 * lg], t1 - t0);
        atomicAdd(&g_timer_pass[2 * lg + 1], t2 - t1);
    }
}
// items of one-lane rows: their elements (slot 12) against 32 x the longest
// row (slot 13), the lane utilisation of the sums
__device__ __forceinline__ void timer_lanes(int lane, int lg, int len) {
    if (lg != 0) return;
    const int sum = __reduce_add_sync(0xffffffffu, len), mx = __reduce_max_sync(0xffffffffu, len);
    if (lane == 0) {
        atomicAdd(&g_timer_pass[12], (unsigned long long)sum);
        atomicAdd(&g_timer_pass[13], 32ull * (unsigned long long)mx);
    }
}
#else
__device__ __forceinline__ unsigned long long timer_now() { return 0ull; }
__device__ __forceinline__ void timer_pass(int, int, unsigned long long, unsigned long long) {}
__device__ __forceinline__ void timer_lanes(int, int, int) {}
#endif

__device__ __forceinline__ void mark_changed(const DevProblem &P, int j) {
    atomicOr(P.chg + (j >> 5), 1u << (j & 31));
}

// Bounds are written by the finalize phase of the same megakernel launch, so
// they are read with coherent loads (never the read-only path).
__device__ __forceinline__ double2 load_bnd(const DevProblem &P, int j) { return P.bnd[j]; }
// The layout of bnd32 is fixed per kernel: kRec = 1, the stamped 16-byte
// records (BndScr) of single-problem contexts -- the round loops of the
// megakernel, the phase kernels and learned marking; kRec = 0, the 8-byte
// copies of batch members.
// Variable j's screen copy of its bounds.
template <int kRec>
__device__ __forceinline__ float2 load_bnd32(const DevProblem &P, int j) {
    return P.bnd32[kRec ? 2 * (long long)j : j];
}
// The screen copy of variable j's bounds, with chg set when the variable was
// committed at the end of the round before `round` (one 16-byte load of the
// stamped record; copies without stamps leave chg alone).
template <int kRec>
__device__ __forceinline__ float2 load_bnd32_chg(const DevProblem &P, int j, int round, int &chg) {
    if (!kRec) return P.bnd32[j];
    const float4 v = reinterpret_cast<const float4 *>(P.bnd32)[j];
    chg |= __float_as_int(v.z) == round - 1 ? 1 : 0;
    return make_float2(v.x, v.y);
}
// Screen of a lane's `cnt` elements, `stride` apart from col / a32: kScreenStep
// gathers at a time, with the next step's indices and coefficients in flight.
// Written out because the compiler keeps the streaming loads in program order:
// in a plain unrolled loop an element's loads stay behind the gather of the
// element before it, and every element costs the lane two memory latencies (a
// slice of 1,024 elements: 25 us on 60,001 rows, the whole phase's length).
// 2M rows 29.3 -> 26.8 ms, 300,000 7.77 -> 6.44, 20,000 2.88 -> 2.54. Steps of
// 4 without the loads ahead: 27.6, 6.54, 2.59; of 8: 27.1, 6.46, 2.69 and 7%
// more for node batches.
constexpr int kScreenStep = 4;
template <int kRec, int kStride>
__device__ __forceinline__ void screen_elements(const DevProblem &P, const int *col, const float *a32, int cnt,
                                                int round, Scr &c, int &chg) {
    int j[kScreenStep];
    float a[kScreenStep];
    auto load = [&](int i0) {
#pragma unroll
        for (int i = 0; i < kScreenStep; i++) {
            j[i] = i0 + i < cnt ? __ldcs(col + kStride * (i0 + i)) : -1;
            a[i] = i0 + i < cnt ? __ldcs(a32 + kStride * (i0 + i)) : 0.0f;
        }
    };
    load(0);
    for (int i0 = 0; i0 < cnt; i0 += kScreenStep) {
        float2 b[kScreenStep];
        float ai[kScreenStep];
        bool on[kScreenStep];
#pragma unroll
        for (int i = 0; i < kScreenStep; i++) {
            on[i] = j[i] >= 0;
            ai[i] = a[i];
            b[i] = on[i] ? load_bnd32_chg<kRec>(P, j[i], round, chg) : make_float2(0.0f, 0.0f);
        }
        load(i0 + kScreenStep);
#pragma unroll
        for (int i = 0; i < kScreenStep; i++)
            if (on[i]) scr_add(c, ai[i], b[i]);
    }
}
// Stores variable j's screen copy of bounds b committed at the end of `round`.
template <int kRec>
__device__ __forceinline__ void store_bnd32(const DevProblem &P, int j, double2 b, int round) {
    const float2 f = bnd_screen(b);
    if (kRec) reinterpret_cast<float4 *>(P.bnd32)[j] = make_float4(f.x, f.y, __int_as_float(round), 0.0f);
    else P.bnd32[j] = f;
}
// Whether a row the screen cannot skip takes the exact pass in `round`: a row
// none of whose variables changed at the end of the previous round (chg == 0)
// was last processed with the same bounds, so its activities and candidates
// are those of that processing -- applied then, or not EPS-better than bounds
// that have not moved since -- and it can neither tighten a bound nor turn
// infeasible. Round 1 processes every row. Valid where every row with a
// changed variable is processed in the next round (full sweeps and exact
// marking): not under learned deferral, and only with stamped records.
template <int kRec>
__device__ __forceinline__ bool row_due(const DevProblem &P, int round, int chg) {
    return chg != 0 || round <= 1 || !kRec || P.learned != 0;
}

// Elements, bounds and targets of the exact pass (gdp_exact.cuh): the
// row-contiguous copy of the SELL rows, or the split rows.
struct CtxTarget {
    static constexpr bool kAligned = true;  // one-lane rows (gdp_internal.h)
    static constexpr bool kNan = false;
    const DevProblem &P;
    const int *col;
    const double *val;
    const double2 *bnd;
    __device__ __forceinline__ CtxTarget(const DevProblem &p, const int *c, const double *v)
        : P(p), col(c), val(v), bnd(p.bnd) {}
    __device__ __forceinline__ bool cont(int j) const { return __ldg(P.is_cont + j) != 0; }
    __device__ __forceinline__ void apply(int j, double v, bool lower) const {
        if (lower) atomic_max_f64(&P.bnd_nxt[j].x, v);
        else atomic_min_f64(&P.bnd_nxt[j].y, v);
        mark_changed(P, j);
    }
};
__device__ __forceinline__ CtxTarget sell_target(const DevProblem &P) { return CtxTarget(P, P.xcol, P.xval); }
__device__ __forceinline__ CtxTarget split_target(const DevProblem &P) { return CtxTarget(P, P.lcol, P.lval); }

// Warp-aggregated round bookkeeping: change flag and tightening count.
__device__ __forceinline__ void report_tight(int tight, int lane, int *change, unsigned *tight_ctr) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) tight += __shfl_down_sync(kFull, tight, off);
    if (lane == 0 && tight) {
        *change = 1;
        atomicAdd(tight_ctr, (unsigned)tight);
    }
}

// ---- SELL-g rows: one warp per slice, g lanes per row ----------------------
struct WarpSmem {
    ExactSmem xs;
    unsigned char own[32];     // lanes whose rows take the exact pass in place
    int row_tight[kItemRows];  // learned marking: tightenings of the item's rows
    // work statistics of this warp, written by lane 0 and flushed to the
    // round flags once per launch (batch members: per item): same-address
    // atomics from every warp serialise in L2
    unsigned long long st_rows, st_nnz, st_exact, st_div, st_xrows, st_go, st_seq, st_drift, st_drift_nnz;
};

constexpr size_t kCtaSmem = sizeof(WarpSmem) * kWarpsPerCta;
// The CTA's warps' shared memory (dynamic: above the 48 KB of static arrays).
__device__ __forceinline__ WarpSmem *warp_smem() {
    extern __shared__ __align__(16) unsigned char warp_smem_raw[];
    return reinterpret_cast<WarpSmem *>(warp_smem_raw);
}

__device__ __forceinline__ void stats_zero(WarpSmem &ws, int lane) {
    if (lane == 0) {
        ws.st_rows = 0; ws.st_nnz = 0; ws.st_exact = 0; ws.st_div = 0;
        ws.st_xrows = 0; ws.st_go = 0; ws.st_seq = 0; ws.st_drift = 0; ws.st_drift_nnz = 0;
    }
}
__device__ __forceinline__ void stats_flush(const DevProblem &P, WarpSmem &ws, int lane) {
    if (lane == 0) {
        if (ws.st_rows) atomicAdd(&P.flags[0].rows_proc, ws.st_rows);
        if (ws.st_nnz) atomicAdd(&P.flags[0].nnz_proc, ws.st_nnz);
        if (ws.st_exact) atomicAdd(&P.flags[0].nnz_exact, ws.st_exact);
        if (ws.st_div) atomicAdd(&P.flags[0].divisions, ws.st_div);
        if (ws.st_xrows) atomicAdd(&P.flags[0].rows_exact, ws.st_xrows);
        if (ws.st_go) atomicAdd(&P.flags[0].rows_go, ws.st_go);
        if (ws.st_seq) atomicAdd(&P.flags[0].rows_seqmax, ws.st_seq);
        if (ws.st_drift) atomicAdd(&P.flags[0].rows_drift, ws.st_drift);
        if (ws.st_drift_nnz) atomicAdd(&P.flags[0].nnz_drift, ws.st_drift_nnz);
        ws.st_rows = 0; ws.st_nnz = 0; ws.st_exact = 0; ws.st_div = 0;
        ws.st_xrows = 0; ws.st_go = 0; ws.st_seq = 0; ws.st_drift = 0; ws.st_drift_nnz = 0;
    }
}

// A row whose activities exclude [lhs, rhs] (row_infeasible): only its index is
// recorded here; the finalize step of the round turns it into the verdict, so
// that every driver completes the round as the oracle does.
__device__ __forceinline__ void record_row_infeasible(const DevProblem &P, int pos) {
    atomicMin(&P.flags[0].infeasible_row, __ldg(P.pos_row + pos));
}

// ---- the reference's sequential EPS-max, for rows row_go_from_max leaves open
// First maximum (order key, index) of d_k = fl(|a_k| fl(ub - lb)) over the
// elements [0, e) of a row stored contiguously at (col, val), with the
// leading 0.0 at index -1; NaN terms never count. All 32 lanes call it and
// every lane returns the result (a butterfly of an associative selection).
__device__ __forceinline__ void row_first_max(const double2 *bnd, const int *col, const double *val, int e,
                                              int lane, long long &km, int &p) {
    Acc s;
    acc_init(s);
    for (int k = lane; k < e; k += 32) {
        const double2 b = bnd[__ldg(col + k)];
        acc_add_delta(s, dmul(fabs(__ldg(val + k)), dsub(b.y, b.x)), k);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const long long ok = __shfl_xor_sync(kFull, s.km, off);
        const int op = __shfl_xor_sync(kFull, s.p, off);
        acc_take_max(s, ok, op);
    }
    km = s.km;
    p = s.p;
}

// The reference's sequential EPS-max of the row's elements [0, len)
// (computeActivities, src/propagation_methods.cuh:188-190), given the first
// maximum (km, p) of [0, len). Over a prefix [0, E) with first maximum (M, q),
// m(E) = fl(M - m(q)) > EPS ? M : m(q) (row_go_from_max), and m(E) = M outright
// when the first maximum M' of [0, q) has fl(M - M') > EPS; m = 0 when the
// maximum is the leading 0.0. The prefix maxima are warp passes; their values
// wait in a stack of one level per lane. A chain deeper than 32 levels (values
// each within EPS of the next) ends with a serial scan. All 32 lanes call it.
__device__ __noinline__ double seq_eps_max(const double2 *bnd, const int *col, const double *val, int len,
                                           long long km, int p, int lane) {
    double stack = 0.0;
    int depth = 0, E = len;
    double x = 0.0;
    for (;;) {
        if (p < 0) {
            x = 0.0;
            break;
        }
        const double M = __longlong_as_double(km);
        if (depth == 32) {
            double m = 0.0;
            if (lane == 0)
                for (int k = 0; k < E; k++) {
                    const double2 b = bnd[__ldg(col + k)];
                    const double d = dmul(fabs(__ldg(val + k)), dsub(b.y, b.x));
                    if (eps_gt(d, m)) m = d;
                }
            x = __shfl_sync(kFull, m, 0);
            break;
        }
        if (lane == depth) stack = M;
        depth++;
        long long km2;
        int p2;
        row_first_max(bnd, col, val, p, lane, km2, p2);
        if (p2 >= 0 && eps_gt(M, __longlong_as_double(km2))) {
            depth--;  // m(E) = M
            x = M;
            break;
        }
        E = p;
        km = km2;
        p = p2;
    }
    for (int i = depth - 1; i >= 0; i--) {
        const double Mi = __shfl_sync(kFull, stack, i);
        if (eps_gt(Mi, x)) x = Mi;
    }
    return x;
}

// The grid's warps.
__device__ __forceinline__ int grid_warps() { return (int)((gridDim.x * blockDim.x) >> 5); }
// This warp's index with consecutive indices on different CTAs: the first
// items of a heaviest-first list go to different SMs.
__device__ __forceinline__ int grid_warp_striped() { return (int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x); }

// Warp-level work claims over items 0 .. n - 1, `step` at a time: the first
// claim is the warp's own number (no atomic: 3,648 warps that all begin with
// one on the same address wait 4.7 us for it), further ones come from a
// counter. kAhead: the next claim is in flight while the current item is
// processed -- for items of similar cost; an item claimed ahead cannot be
// taken by an idle warp.
template <bool kAhead>
struct WarpCursor {
    unsigned *ctr;
    int step, first, base;
    bool more;      // the grid's first claims do not cover the items
    unsigned pre;   // kAhead, lane 0: the claim in flight
    __device__ __forceinline__ void start(unsigned *c, int stp, int warps, int n, bool from_last = false) {
        ctr = c;
        step = stp;
        first = (from_last ? warps - 1 - grid_warp_striped() : grid_warp_striped()) * stp;
        base = warps * stp;
        more = n > base;
        pre = 0;
    }
    __device__ __forceinline__ int next(int lane) {
        int i = first;
        if (first >= 0) {
            first = -1;
        } else if (more) {
            if (!kAhead && lane == 0) pre = atomicAdd(ctr, (unsigned)step);
            i = base + (int)__shfl_sync(kFull, pre, 0);
        } else {
            i = INT_MAX;
        }
        if (kAhead && more && lane == 0) pre = atomicAdd(ctr, (unsigned)step);
        return i;
    }
};

// Learned marking: scores and per-row outcomes of one slice (the features
// of the slice's rows live in the storage of the division queue, which is empty until the
// exact pass).
struct LearnSmem {
    float z[32];
    unsigned char tight[32];
    unsigned char go[32];
    unsigned long long marked;  // marked SELL rows met by this warp in the current phase
};

// Combines the partial screens of a group of g lanes (g a power of two,
// warp-uniform) into its first lane: shuffle tree with offsets g/2, ..., 1.
__device__ __forceinline__ void scr_group_reduce(Scr &c, int g) {
    for (int off = g >> 1; off > 0; off >>= 1) {
        Scr o;
        o.mn = __shfl_down_sync(kFull, c.mn, off);
        o.mx = __shfl_down_sync(kFull, c.mx, off);
        o.S = __shfl_down_sync(kFull, c.S, off);
        o.U = __shfl_down_sync(kFull, c.U, off);
        o.minf = __shfl_down_sync(kFull, c.minf, off);
        o.maxf = __shfl_down_sync(kFull, c.maxf, off);
        scr_combine(c, o);
    }
}

// Adds the warp's row and non-zero counts to the round statistics.
__device__ __forceinline__ void count_work(WarpSmem &ws, int lane, int rows, int nnz, int nnz_exact) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        rows += __shfl_down_sync(kFull, rows, off);
        nnz += __shfl_down_sync(kFull, nnz, off);
        nnz_exact += __shfl_down_sync(kFull, nnz_exact, off);
    }
    if (lane == 0) {
        ws.st_rows += (unsigned long long)rows;
        ws.st_nnz += (unsigned long long)nnz;
        ws.st_exact += (unsigned long long)nnz_exact;
    }
}

// Rows of an exact item whose chains get 2^lh lanes each: 32 / 2^lh / g rows of
// g = 2^lg lanes, at least one (with fewer lanes per chain then).
__device__ __forceinline__ int item_rows(int lh, int lg) { return max(32 >> (lh + lg), 1); }

// Exact pass of one item of SELL rows (lane r holds row r, its position in
// pos), up to 2^lc lanes per chain: sums, row test, row-side infeasibility,
// candidates into the division queue Q. Returns whether this
// lane's row passed its test. Rows whose test only the sequential EPS-max
// decides (the largest |a| (ub - lb) exceeds the slack by EPS to 2.00001e-9)
// compute it with the whole warp, row by row.
__device__ __noinline__ bool exact_item(const DevProblem &P, const CtxTarget &T, WarpSmem &ws, ExactQueue &Q,
                                           int lc, int lg, const ExactRow &R, int pos, int lane,
                                           int *row_tight = nullptr) {
    const unsigned long long t0 = timer_now();
    timer_lanes(lane, lg, R.in ? R.len : 0);
    int cand;
    const int lh = min(lc, 5 - lg);
    const ExactSums X = lh == 0 ? exact_sums(T, ws.xs, R, lg, lane, cand)
                                : exact_sums_spread(T, ws.xs, R, lg, lh, lane, cand);
    double s = 0.0, t = 0.0, mn = 0.0;
    int dec = 0;
    if (R.in) {
        bool bad;
        dec = exact_decide(R, X, s, t, mn, bad);
        if (bad) record_row_infeasible(P, pos);
    }
    unsigned amb = __ballot_sync(kFull, dec == 2);
    const unsigned rows = __ballot_sync(kFull, R.in);
    if (lane == 0) {
        ws.st_xrows += __popc(rows);
        if (lg > 0) ws.st_seq += __popc(amb);  // one-lane rows are summed in the reference's order anyway
    }
    for (; amb; amb &= amb - 1) {
        const int q = __ffs(amb) - 1;
        const int qb = __shfl_sync(kFull, R.base, q), ql = __shfl_sync(kFull, R.len, q);
        const double m = seq_eps_max(P.bnd, T.col + qb, T.val + qb, ql, __shfl_sync(kFull, X.km, q),
                                     __shfl_sync(kFull, X.p, q), lane);
        if (lane == q) dec = eps_le(m, mn) ? 0 : 1;
    }
    const bool go = R.in && dec == 1;
    const unsigned bg = __ballot_sync(kFull, go);
    if (lane == 0) ws.st_go += __popc(bg);
    const unsigned long long t1 = timer_now();
    exact_candidates(T, ws.xs, Q, R, X, go, s, t, cand, lane, row_tight);
    timer_pass(lane, lg, t0, t1);
    return go;
}

// Ends a warp's exact work: the queued divisions, the tightening count and
// the division count.
__device__ __forceinline__ void exact_finish(const CtxTarget &T, WarpSmem &ws, ExactQueue &Q, int lane, int *change,
                                             unsigned *tight_ctr) {
    exact_drain(T, ws.xs, Q, true, lane);
    report_tight(Q.tight, lane, change, tight_ctr);
    if (lane == 0) ws.st_div += (unsigned long long)Q.pushed;
    Q.tight = 0;
    Q.pushed = 0;
}

// The rows of a slice that take the exact pass, in place: `exact` is set in
// the leader lane of each (rl << lg), which holds the row's position, length,
// sides and screen results. tight / go (learned marking; may be null) receive
// the outcome of the row in slice slot rl.
__device__ __forceinline__ void exact_slice(const DevProblem &P, WarpSmem &ws, int lg, bool exact, int pos, int base,
                                            int len, float slack_lo, int minf, int maxf, double lhs, double rhs,
                                            int lane, int *change, unsigned *tight_ctr,
                                            unsigned char *tight = nullptr, unsigned char *go = nullptr) {
    const unsigned rows = __ballot_sync(kFull, exact);
    if (!rows) return;
    // all of the rows in one item, with as many lanes per chain as they leave. Two
    // items of two lanes per chain take the same FP64 instructions, but a second
    // pass of loads, row tests and candidates, and the code to run through items
    // costs the caller registers (2,000 rows 0.368 -> 0.341 ms, 64 nodes of 50,000
    // rows 13.2 -> 12.15, 24 mixed instances 11.5 -> 10.5).
    const int n = __popc(rows);
    int lh = 0;
    while (lh + lg < 5 && item_rows(lh + 1, lg) >= n) lh++;
    __syncwarp();
    if (exact) ws.own[__popc(rows & ((1u << lane) - 1u))] = (unsigned char)lane;
    __syncwarp();
    const CtxTarget T = sell_target(P);
    ExactQueue Q{0, 0, 0};
    ExactRow R;
    R.in = lane < n;
    const int own = R.in ? ws.own[lane] : 0;
    const int p = __shfl_sync(kFull, pos, own);
    R.base = __shfl_sync(kFull, base, own);
    R.len = __shfl_sync(kFull, len, own);
    R.slack_lo = __shfl_sync(kFull, slack_lo, own);
    R.minf = __shfl_sync(kFull, minf, own);
    R.maxf = __shfl_sync(kFull, maxf, own);
    R.lhs = __shfl_sync(kFull, lhs, own);
    R.rhs = __shfl_sync(kFull, rhs, own);
    if (tight) {
        ws.row_tight[lane] = 0;
        __syncwarp();
    }
    const bool passed = exact_item(P, T, ws, Q, lh, lg, R, p, lane, tight ? ws.row_tight : nullptr);
    if (tight) {
        exact_drain(T, ws.xs, Q, true, lane, ws.row_tight);
        if (R.in) {
            tight[own >> lg] = ws.row_tight[lane] > 0;
            go[own >> lg] = passed;
        }
        __syncwarp();
    }
    exact_finish(T, ws, Q, lane, change, tight_ctr);
}

// A row's infinity counts (the screen's are exact), up to 3 each.
__device__ __forceinline__ int pack_inf(const Scr &c) { return min(c.minf, 3) | min(c.maxf, 3) << 2; }

// One SELL-g slice per warp: 32/g rows, g lanes per row. Lane l serves row
// l >> lg and its elements sub, sub+g, ... (sub = l & (g-1)), stored
// column-major (step i of lane l at slice_ptr[slice] + 32 i + l).
// The FP32 screen runs here; rows it cannot skip are queued for the exact-rows
// phase (kDefer) or take the exact pass in place (batch members, and contexts of
// nothing but one-lane rows with at most three slices per warp, or with up to four
// warps per slice: `part` of `parts`).
template <int kRec, bool kDefer>
__device__ __forceinline__ void sell_slice(const DevProblem &P, int slice, int lane, int round, bool marked,
                                           int *change, unsigned *tight_ctr, WarpSmem &ws, int par = 0, int part = 0,
                                           int parts = 1, bool due = true) {
    const int lg = __ldg(P.slice_lg + slice);
    const int g = 1 << lg;
    const int row0 = __ldg(P.slice_row0 + slice);
    const int nrows = __ldg(P.slice_row0 + slice + 1) - row0;
    const int rl = lane >> lg, sub = lane & (g - 1);
    const int r = row0 + rl;
    // what a row needs is loaded in one go: the chain of a lone slice's dependent
    // loads is a small round's length (8 chain MIPs, 1,992 rounds: 33.5 -> 31.6 ms,
    // 2,000 rows 0.295 -> 0.29)
    const long long base = __ldg(P.slice_ptr + slice) + lane;
    const int row_len = rl < nrows ? __ldg(P.srow_len + r) : 0;
    const bool act = rl < nrows && (!marked || P.mark[r] == round) && due;
    if (!__any_sync(kFull, act)) return;
    const int len = act ? row_len : 0;
    const int cnt = len > sub ? (len - sub + g - 1) >> lg : 0;  // my elements
    const bool leader = act && sub == 0;
    const int xbase = leader ? __ldg(P.xptr + r) : 0;  // used at the end

    // FP32 screen
    bool exact = false;
    const double lhs = leader ? __ldg(P.srow_lhs + r) : 0.0, rhs = leader ? __ldg(P.srow_rhs + r) : 0.0;
    float slack_lo = 0.0f;  // the screen's lower bound of its slacks, leaders of exact rows
    Scr c;
    scr_init(c);
    {
        const int *col = P.sell_col + base;
        const float *val = P.sell_a32 + base;
        int chg = 0;
        screen_elements<kRec, 32>(P, col, val, cnt, round, c, chg);
        if (g > 1) {
            scr_group_reduce(c, g);
            for (int off = g >> 1; off > 0; off >>= 1) chg |= __shfl_xor_sync(kFull, chg, off);
        }
        if (leader) {
            exact = !scr_skips(c, len, lhs, rhs) && row_due<kRec>(P, round, chg);
            if (exact) {
                float hi;
                scr_slack(c, len, lhs, rhs, slack_lo, hi);
            }
        }
    }
    if (!kDefer && parts > 1) {  // my share of the exact rows
        const unsigned rows = __ballot_sync(kFull, exact);
        exact = exact && __popc(rows & ((1u << lane) - 1u)) % parts == part;
    }
    const bool counted = leader && part == 0;
    count_work(ws, lane, counted ? 1 : 0, counted ? len : 0, (leader && exact) ? len : 0);
    if (kDefer) {
        const unsigned bal = __ballot_sync(kFull, exact);
        if (!bal) return;
        unsigned first = 0;
        if (lane == 0) first = atomicAdd(P.xctr + 16 * par + lg, (unsigned)__popc(bal));
        first = __shfl_sync(kFull, first, 0);
        if (exact) P.xrow[P.cls_begin[lg] + first + __popc(bal & ((1u << lane) - 1u))] = XRow{xbase, r, len, slack_lo, pack_inf(c)};
        return;
    }
    exact_slice(P, ws, lg, exact, r, xbase, len, slack_lo, c.minf, c.maxf, lhs, rhs, lane, change, tight_ctr);
}

// K slices of one-lane rows (g = 1) screened together in the deferred-exact
// mode: lane l screens row l of each slice, so the K rows' column, coefficient
// and bound loads are in flight at the same time (a slice of short rows holds
// only 64..128 non-zeros: alone, its chain of dependent loads leaves the warp
// waiting), and the exact rows of all K slices are queued with one counter
// update. Decisions and queue contents equal those of K sell_slice calls.
template <int K, int kRec>
__device__ __forceinline__ void sell_slices_g1(const DevProblem &P, const int (&sl)[K], int lane, int round,
                                               bool marked, WarpSmem &ws, int par) {
    int r[K], len[K];
    long long base[K];
    double lhs[K], rhs[K];
    bool act[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int row0 = __ldg(P.slice_row0 + sl[k]);
        r[k] = row0 + lane;
        act[k] = lane < __ldg(P.slice_row0 + sl[k] + 1) - row0;
        base[k] = __ldg(P.slice_ptr + sl[k]) + lane;
    }
    if (marked) {
#pragma unroll
        for (int k = 0; k < K; k++)
            if (act[k]) act[k] = P.mark[r[k]] == round;
    }
    int mx = 0, xbase[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        len[k] = act[k] ? __ldg(P.srow_len + r[k]) : 0;
        xbase[k] = act[k] ? __ldg(P.xptr + r[k]) : 0;
        mx = max(mx, len[k]);
    }
    Scr c[K];
    int chg[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        scr_init(c[k]);
        chg[k] = 0;
    }
    constexpr int S = 2;  // elements per row and step: 2 K index loads, then their gathers
    for (int i0 = 0; i0 < mx; i0 += S) {
        int j[K][S];
        float a[K][S];
        float2 b[K][S];
#pragma unroll
        for (int i = 0; i < S; i++)
#pragma unroll
            for (int k = 0; k < K; k++) {
                const bool on = i0 + i < len[k];
                j[k][i] = on ? __ldcs(P.sell_col + base[k] + 32 * (i0 + i)) : -1;
                a[k][i] = on ? __ldcs(P.sell_a32 + base[k] + 32 * (i0 + i)) : 0.0f;
            }
#pragma unroll
        for (int i = 0; i < S; i++)
#pragma unroll
            for (int k = 0; k < K; k++)
                b[k][i] = j[k][i] >= 0 ? load_bnd32_chg<kRec>(P, j[k][i], round, chg[k]) : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < S; i++)
#pragma unroll
            for (int k = 0; k < K; k++)
                if (j[k][i] >= 0) scr_add(c[k], a[k][i], b[k][i]);
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
        lhs[k] = 0.0;
        rhs[k] = 0.0;
        if (act[k]) {
            lhs[k] = __ldg(P.srow_lhs + r[k]);
            rhs[k] = __ldg(P.srow_rhs + r[k]);
        }
    }
    bool exact[K];
    float slo[K];
    int rows = 0, nnz = 0, nnz_exact = 0, total = 0;
    unsigned bal[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        exact[k] = act[k] && !scr_skips(c[k], len[k], lhs[k], rhs[k]) && row_due<kRec>(P, round, chg[k]);
        slo[k] = 0.0f;
        if (exact[k]) {
            float hi;
            scr_slack(c[k], len[k], lhs[k], rhs[k], slo[k], hi);
        }
        rows += act[k] ? 1 : 0;
        nnz += len[k];
        nnz_exact += exact[k] ? len[k] : 0;
        bal[k] = __ballot_sync(kFull, exact[k]);
        total += __popc(bal[k]);
    }
    count_work(ws, lane, rows, nnz, nnz_exact);
    if (!total) return;
    unsigned first = 0;
    if (lane == 0) first = atomicAdd(P.xctr + 16 * par, (unsigned)total);
    first = __shfl_sync(kFull, first, 0) + (unsigned)P.cls_begin[0];
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int k = 0; k < K; k++) {
        if (exact[k]) P.xrow[first + __popc(bal[k] & lt)] = XRow{xbase[k], r[k], len[k], slo[k], pack_inf(c[k])};
        first += __popc(bal[k]);
    }
}

// Exact-rows phase: the rows the screen queued, in items of 32 / g rows per
// warp, or of fewer rows with more lanes per chain (up to 8: a row's sums then
// take a quarter of the FP64 instructions) as long as the grid has a warp for
// each item. The items of all classes are one list, widest class first; a warp
// takes one by its own number and claims further ones from a counter only when
// there are more items than warps. The first warps come from the tiles of the
// candidate phase: with tiles for up to half of the warps the widest items go to
// the last ones (the same warps had the tiles and the widest items before: 5,000
// rows 1.45 -> 1.35 ms, 20,000 rows 2.28 -> 2.10, 60,001 rows 3.57 -> 3.52); with
// tiles for all of them the order is a coin toss (150,000 rows 4.08, 4.24 from the
// last).
__device__ __forceinline__ void exact_rows_phase(const DevProblem &P, int par, int *change, unsigned *tight_ctr,
                                                 WarpSmem &ws, int lane) {
    const int nw = grid_warps();
    // lane 5 - lg: the class's rows and items, with the items of the wider classes before it
    const int rows = lane < 6 ? (int)*((volatile unsigned *)(P.xctr + 16 * par + 5 - lane)) : 0;
    int lh = 3, items, upto, total;
    for (;; lh--) {
        const int per = lane < 6 ? item_rows(lh, 5 - lane) : 1;
        items = (rows + per - 1) / per;
        upto = items;  // inclusive prefix
#pragma unroll
        for (int off = 1; off < 8; off <<= 1) {
            const int v = __shfl_up_sync(kFull, upto, off);
            if (lane >= off) upto += v;
        }
        total = __shfl_sync(kFull, upto, 5);
        if (lh == 0 || total <= nw) break;
    }
    const CtxTarget T = sell_target(P);
    ExactQueue Q{0, 0, 0};
    WarpCursor<false> cur;
    cur.start(P.xctr + 16 * par + 8, 1, nw, total, 2 * P.n_mtiles <= nw);
    for (;;) {
        const int it = cur.next(lane);
        if (it >= total) break;
        const int cl = __ffs(__ballot_sync(kFull, lane < 6 && it < upto)) - 1;
        const int lg = 5 - cl, per = item_rows(lh, lg);
        const int k0 = (it - (__shfl_sync(kFull, upto, cl) - __shfl_sync(kFull, items, cl))) * per;
        const int n = min(per, __shfl_sync(kFull, rows, cl) - k0);
        ExactRow R;
        R.in = lane < n;
        R.base = 0; R.len = 0; R.slack_lo = 0.0f; R.minf = 0; R.maxf = 0; R.lhs = 0.0; R.rhs = 0.0;
        int pos = 0;
        if (R.in) {
            const XRow x = P.xrow[P.cls_begin[lg] + k0 + lane];
            pos = x.pos;
            R.base = (int)x.base;
            R.len = x.len;
            R.slack_lo = x.slack_lo;
            R.minf = x.inf & 3;
            R.maxf = x.inf >> 2;
            R.lhs = __ldg(P.srow_lhs + pos);
            R.rhs = __ldg(P.srow_rhs + pos);
        }
        exact_item(P, T, ws, Q, lh, lg, R, pos, lane);
    }
    exact_finish(T, ws, Q, lane, change, tight_ctr);
}

// ---- split rows: one warp per tile ----------------------------------------
// Drift bound (single-problem plain rounds; marked rounds use it): a split row
// the screen skipped with certified margin m (scr_margin) stays skippable while
// the bound D of how far its slack has fallen since -- finalize adds |a|
// (lb' - lb + ub - ub') rounded up for every tightening of one of its
// variables, infinite when an infinite bound becomes finite -- satisfies
// D (1 + 2^-22) <= m: the factor covers D's own rounding (an FP64 sum of
// rounded-up terms, up to 2^28 of them) and |a| against its FP32 copy. Such a
// row tightens nothing and is feasible, exactly as its screen would decide.
// Its work is counted as screened, so the statistics equal a full screen's.
template <int kRec>
__device__ __forceinline__ bool drift_active(const DevProblem &P) {
    return kRec != 0 && P.learned == 0 && P.lrow_margin != nullptr;
}
__device__ __forceinline__ bool drift_skips(const DevProblem &P, int row) {
    const double m = P.lrow_margin[row];
    if (!(m >= 0.0)) return false;
    return __dmul_ru(P.lrow_drift[row], 1.0 + 0x1p-22) <= m;  // false for NaN and inf drifts
}
// A screen of split row `row` refreshes its certificate (one writer per row).
__device__ __forceinline__ void drift_reset(const DevProblem &P, int row, const Scr &c, int n, double lhs,
                                            double rhs) {
    P.lrow_margin[row] = scr_margin(c, n, lhs, rhs);
    P.lrow_drift[row] = 0.0;
}
__device__ __forceinline__ void acc_shfl_reduce(Acc &s) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        Acc o;
        o.minact = __shfl_down_sync(kFull, s.minact, off);
        o.maxact = __shfl_down_sync(kFull, s.maxact, off);
        o.minf = __shfl_down_sync(kFull, s.minf, off);
        o.maxf = __shfl_down_sync(kFull, s.maxf, off);
        o.km = __shfl_down_sync(kFull, s.km, off);
        o.p = __shfl_down_sync(kFull, s.p, off);
        acc_combine(s, o);
    }
}

// The reference's row test (row_go_from_max, seq_eps_max where it cannot
// decide) and the candidates of split row `row` over the element range
// [b, e) of one tile, from the row's complete activities and first maximum
// held by lane 0. Elements whose FP32 upper bound of |a| (ub - lb) does not
// exceed the smaller slack are no candidates; the others form the FP64
// product. The row's first tile also checks it for row-side infeasibility.
template <int kRec>
__device__ __noinline__ void split_row_candidates(const DevProblem &P, int row, int b, int e, const Acc &s0,
                                                     int lane, int *change, unsigned *tight_ctr, WarpSmem &ws) {
    const int t0 = __ldg(P.lrow_tile0 + row);
    const int rb = __ldg(P.tile_begin + t0);
    ExactRow R;
    R.in = lane == 0;
    R.base = b;
    R.len = e - b;
    R.slack_lo = 0.0f;
    R.minf = s0.minf;
    R.maxf = s0.maxf;
    R.lhs = __ldg(P.lrow_lhs + row);
    R.rhs = __ldg(P.lrow_rhs + row);
    ExactSums X{s0.minact, s0.maxact, s0.km, s0.p};
    double s = 0.0, t = 0.0, mn = 0.0;
    int go = 0;
    if (lane == 0) {
        bool bad;
        go = exact_decide(R, X, s, t, mn, bad);
        if (b == rb && bad) record_row_infeasible(P, P.n_srows + row);
    }
    go = __shfl_sync(kFull, go, 0);
    if (go == 2) {  // every tile of the row reaches the same m
        const int re = __ldg(P.tile_end + __ldg(P.lrow_tile0 + row + 1) - 1);
        const double m = seq_eps_max(P.bnd, P.lcol + rb, P.lval + rb, re - rb, __shfl_sync(kFull, s0.km, 0),
                                     __shfl_sync(kFull, s0.p, 0), lane);
        if (lane == 0) {
            go = eps_le(m, mn) ? 0 : 1;
            if (b == rb) ws.st_seq++;
        }
        go = __shfl_sync(kFull, go, 0);
    }
    if (!go) return;
    const CtxTarget T = split_target(P);
    ExactQueue Q{0, 0, 0};
    exact_candidates(T, ws.xs, Q, R, X, lane == 0, s, t, 0, lane);  // the row's constants, in slot 0
    const float cut = __shfl_sync(kFull, f32_dn(dbits(mn)), 0);  // below both slacks
    constexpr int kSteps = 4;
    for (int k0 = b + lane; k0 - lane < e; k0 += 32 * kSteps) {
        int j[kSteps];
        float a[kSteps];
        float2 bb[kSteps];
#pragma unroll
        for (int i = 0; i < kSteps; i++) {
            const int k = k0 + 32 * i;
            j[i] = k < e ? __ldg(P.lcol + k) : -1;
            a[i] = k < e ? __ldg(P.la32 + k) : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kSteps; i++) bb[i] = j[i] >= 0 ? load_bnd32<kRec>(P, j[i]) : make_float2(0.0f, 0.0f);
        unsigned todo = 0u;  // my elements that may be candidates
#pragma unroll
        for (int i = 0; i < kSteps; i++)
            if (j[i] >= 0 && !(delta_upper32(a[i], bb[i]) <= cut)) todo |= 1u << i;
#pragma unroll 1
        for (int i = 0; i < kSteps; i++) {
            const bool on = (todo >> i) & 1u;
            if (!__any_sync(kFull, on)) continue;
            exact_push(T, ws.xs, Q, on, k0 + 32 * i, 0, lane, nullptr);
        }
    }
    exact_finish(T, ws, Q, lane, change, tight_ctr);
}

__device__ __forceinline__ void scr_shfl_reduce(Scr &c) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        Scr o;
        o.mn = __shfl_down_sync(kFull, c.mn, off);
        o.mx = __shfl_down_sync(kFull, c.mx, off);
        o.S = __shfl_down_sync(kFull, c.S, off);
        o.U = __shfl_down_sync(kFull, c.U, off);
        o.minf = __shfl_down_sync(kFull, c.minf, off);
        o.maxf = __shfl_down_sync(kFull, c.maxf, off);
        scr_combine(c, o);
    }
}

// Exact FP64 partial of the element range [b, e) of a split row whose first
// element is rb: lane l sums elements l, l+32, ... in order, shuffle tree
// across lanes, with the first maximum of |a| (ub - lb) (indices from rb);
// lane 0 holds the result.
__device__ __forceinline__ Acc tile_exact(const DevProblem &P, int b, int e, int rb, int lane) {
    Acc s;
    acc_init(s);
#pragma unroll 4
    for (int k = b + lane; k < e; k += 32) {
        const int j = __ldg(P.lcol + k);
        const double a = __ldg(P.lval + k);
        const double2 bb = load_bnd(P, j);
        acc_add_terms(s, a, bb.x, bb.y);
        acc_add_delta(s, dmul(fabs(a), dsub(bb.y, bb.x)), k - rb);
    }
    acc_shfl_reduce(s);
    return s;
}

// Activity phase, split-row tile t: the FP32 screen of the tile. A row that
// fits in one tile is finished here (screen decision, exact pass, candidates);
// tiles of longer rows store their screen partial for the candidate phase
// (returns true for those).
template <int kRec>
__device__ __forceinline__ bool split_partial(const DevProblem &P, int t, int lane, int round, bool marked,
                                              int *change, unsigned *tight_ctr, WarpSmem &ws) {
    const int row = __ldg(P.tile_row + t);
    if (marked && P.mark[P.n_srows + row] != round) return false;
    const int b = __ldg(P.tile_begin + t), e = __ldg(P.tile_end + t);
    const int t0 = __ldg(P.lrow_tile0 + row);
    const bool single = __ldg(P.lrow_tile0 + row + 1) - t0 == 1;
    if (marked && drift_active<kRec>(P) && drift_skips(P, row)) {  // the same values for every lane
        if (lane == 0) {
            ws.st_nnz += (unsigned long long)(e - b);
            ws.st_drift_nnz += (unsigned long long)(e - b);
            if (t == t0) {
                ws.st_rows += 1ULL;
                ws.st_drift += 1ULL;
            }
            if (!single) P.lrow_skip[row] = round;  // the candidate phase skips the row too
        }
        return false;
    }
    Scr c;
    scr_init(c);
    int chg = 0;
    screen_elements<kRec, 32>(P, P.lcol + b + lane, P.la32 + b + lane, e > b + lane ? (e - b - lane + 31) / 32 : 0, round,
                              c, chg);
    scr_shfl_reduce(c);
    chg = __any_sync(kFull, chg) ? 1 : 0;
    int exact = 0;
    if (lane == 0) {
        ws.st_nnz += (unsigned long long)(e - b);
        if (t == t0) ws.st_rows += 1ULL;
        if (single) {
            const double lhs = __ldg(P.lrow_lhs + row), rhs = __ldg(P.lrow_rhs + row);
            exact = !scr_skips(c, e - b, lhs, rhs) && row_due<kRec>(P, round, chg);
            if (drift_active<kRec>(P)) drift_reset(P, row, c, e - b, lhs, rhs);
            if (exact) ws.st_exact += (unsigned long long)(e - b);
        } else {
            TileScr ts;
            ts.mn = c.mn; ts.mx = c.mx; ts.S = c.S; ts.U = c.U; ts.minf = c.minf; ts.maxf = c.maxf;
            ts.chg = chg;
            ts.pad = 0;
            P.tile_scr[t] = ts;
        }
    }
    if (!single) return true;
    if (!__shfl_sync(kFull, exact, 0)) return false;
    const Acc s = tile_exact(P, b, e, b, lane);
    split_row_candidates<kRec>(P, row, b, e, s, lane, change, tight_ctr, ws);
    return false;
}

// Candidate phase, tile t of a multi-tile row: the row's screen (the tile
// partials combined by all lanes in a fixed order, so every tile of the row
// reaches the same decision); a row the screen cannot skip gets this tile's
// exact FP64 partial, and its first tile flags the row for the exact phase
// (returns true when the tile computed its exact partial).
template <int kRec>
__device__ __forceinline__ bool split_cand(const DevProblem &P, int t, int lane, int round, bool marked,
                                           int *exact_ctr, WarpSmem &ws) {
    const int row = __ldg(P.tile_row + t);
    if (marked && P.mark[P.n_srows + row] != round) return false;
    if (drift_active<kRec>(P) && P.lrow_skip[row] == round) return false;  // skipped on its drift bound
    const int t0 = __ldg(P.lrow_tile0 + row), t1 = __ldg(P.lrow_tile0 + row + 1);
    Scr c;
    scr_init(c);
    int chg = 0;
    for (int u = t0 + lane; u < t1; u += 32) {
        const TileScr p = P.tile_scr[u];
        Scr o;
        o.mn = p.mn; o.mx = p.mx; o.S = p.S; o.U = p.U; o.minf = p.minf; o.maxf = p.maxf;
        scr_combine(c, o);
        chg |= p.chg;
    }
    scr_shfl_reduce(c);
    chg = __any_sync(kFull, chg) ? 1 : 0;
    int exact = 0;
    if (lane == 0) {
        const int n_row = __ldg(P.tile_end + t1 - 1) - __ldg(P.tile_begin + t0);
        const double lhs = __ldg(P.lrow_lhs + row), rhs = __ldg(P.lrow_rhs + row);
        exact = !scr_skips(c, n_row, lhs, rhs) && row_due<kRec>(P, round, chg);
        if (drift_active<kRec>(P) && t == t0) drift_reset(P, row, c, n_row, lhs, rhs);
    }
    if (!__shfl_sync(kFull, exact, 0)) return false;
    const int b = __ldg(P.tile_begin + t), e = __ldg(P.tile_end + t);
    const Acc s = tile_exact(P, b, e, __ldg(P.tile_begin + t0), lane);
    if (lane == 0) {
        TilePart tp;
        tp.minact = s.minact; tp.maxact = s.maxact; tp.km = s.km; tp.minf = s.minf; tp.maxf = s.maxf;
        tp.p = s.p;
        tp.pad = 0;
        P.tile_part[t] = tp;
        ws.st_exact += (unsigned long long)(e - b);
        if (t == t0) {
            P.row_exact[row] = round;
            atomicAdd(exact_ctr, 1);
        }
    }
    return true;
}

constexpr int kTileParts = 4;  // candidates of a tile in quarters: a long tile is no phase's long pole
// Exact phase, tile t of a multi-tile row flagged this round: the row's exact
// partials combined in tile order, then the decision and this tile's candidates.
template <int kRec>
__device__ __forceinline__ void split_exact(const DevProblem &P, int t, int lane, int round, int *change,
                                            unsigned *tight_ctr, WarpSmem &ws, int part = 0, int parts = 1) {
    const int row = __ldg(P.tile_row + t);
    if (P.row_exact[row] != round) return;
    // lanes load 32 partials at a time; lane 0 folds them in tile order
    const int t0 = __ldg(P.lrow_tile0 + row), t1 = __ldg(P.lrow_tile0 + row + 1);
    Acc s;
    acc_init(s);
    for (int b = t0; b < t1; b += 32) {
        TilePart tp = {0.0, 0.0, 0, 0, 0, -1, 0};
        if (b + lane < t1) tp = P.tile_part[b + lane];
        const int cnt = min(32, t1 - b);
        for (int i = 0; i < cnt; i++) {
            Acc o;
            o.minact = __shfl_sync(kFull, tp.minact, i);
            o.maxact = __shfl_sync(kFull, tp.maxact, i);
            o.minf = __shfl_sync(kFull, tp.minf, i);
            o.maxf = __shfl_sync(kFull, tp.maxf, i);
            o.km = __shfl_sync(kFull, tp.km, i);
            o.p = __shfl_sync(kFull, tp.p, i);
            if (lane == 0) {
                if (b + i == t0) s = o;
                else acc_combine(s, o);
            }
        }
    }
    // this item's part of the tile: parts of whole warp steps
    const int tb = __ldg(P.tile_begin + t), te = __ldg(P.tile_end + t);
    const int step = ((te - tb + parts - 1) / parts + 31) & ~31;
    const int pb = min(te, tb + part * step), pe = min(te, pb + step);
    if (pb < pe) split_row_candidates<kRec>(P, row, pb, pe, s, lane, change, tight_ctr, ws);
}

// Adds the warp's committed-change counts to the round flags, one atomic per warp.
// Every lane of the warp calls it, from wherever its loop left it.
__device__ __forceinline__ void flush_changed(const DevProblem &P, unsigned long long changed) {
    __syncwarp();
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) changed += __shfl_down_sync(kFull, changed, off);
    if ((threadIdx.x & 31) == 0 && changed) atomicAdd(&P.flags[0].changed_vars, changed);
}

// Commit changed variables nxt -> cur, apply the infeasibility rules (a row
// recorded infeasible in this round, a variable whose bounds cross), mark the
// rows of changed variables for the next round, clear the bitmap.
// One warp per word of the bitmap: lane l commits variable 32 w + l, then the
// warp pushes the marks of each changed variable's rows together, 32 per step,
// with the first steps of four variables in flight: what bounds it is the
// latency of the index entries, most of which come from HBM (2M rows, 72 rounds:
// 29.88 -> 29.42 ms against one variable after the other; a thread walking its word's variables and their rows alone
// leaves the commit of a round with many changes to a few long serial chains).
// tid / nthreads: a grid of whole warps.
__device__ __forceinline__ void finalize_words(const DevProblem &P, int round, bool push_marks, int tid,
                                               int nthreads) {
    const int lane = tid & 31;
    unsigned long long changed = 0;
    auto push = [&](int2 e, double dj) {  // e: {pos, acoef}
        P.mark[e.x] = round + 1;
        // a split row's slack moves by at most |a| (lb' - lb + ub - ub')
        if (e.x >= P.n_srows && P.lrow_drift)
            atomicAdd(P.lrow_drift + (e.x - P.n_srows), __dmul_ru((double)__int_as_float(e.y), dj));
    };
    if (tid == 0 && *((volatile int *)&P.flags[0].infeasible_row) != INT_MAX) P.flags[0].infeasible = 1;
    for (int w = tid >> 5; w < P.n_chg_words; w += nthreads >> 5) {
        const unsigned bits = __ldcg(P.chg + w);
        if (!bits) continue;  // warp-uniform
        double delta = 0.0;  // upper bound of (lb' - lb) + (ub - ub') of my variable
        int p0 = 0, p1 = 0;  // its rows
        if ((bits >> lane) & 1u) {
            const int j = w * 32 + lane;
            const double2 b = __ldcg(P.bnd_nxt + j);
            const double2 o = P.bnd[j];
            if (push_marks) {
                p0 = __ldg(P.var_ptr + j);
                p1 = __ldg(P.var_ptr + j + 1);
                delta = (neginf_bits(dbits(o.x)) || posinf_bits(dbits(o.y)))
                                ? __longlong_as_double(0x7FF0000000000000LL)  // an infinite bound became finite
                                : __dadd_ru(__dsub_ru(b.x, o.x), __dsub_ru(o.y, b.y));
            }
            P.bnd[j] = b;
            store_bnd32<1>(P, j, b, round);
            if (var_infeasible(b.x, b.y)) {
                P.flags[0].infeasible = 1;
                atomicMin(&P.flags[0].infeasible_var, j);
            }
        }
        __syncwarp();
        if (lane == 0) {
            P.chg[w] = 0u;
            changed += __popc(bits);
        }
        constexpr int kVars = 4;
        for (unsigned rem = __ballot_sync(kFull, p0 < p1); rem;) {
            int q[kVars], q1[kVars];
            double dj[kVars];
            int2 e[kVars];
#pragma unroll
            for (int i = 0; i < kVars; i++) {
                const int bit = rem ? __ffs(rem) - 1 : 0;
                q[i] = __shfl_sync(kFull, p0, bit) + lane;
                q1[i] = __shfl_sync(kFull, p1, bit);
                dj[i] = __shfl_sync(kFull, delta, bit);
                if (!rem) q1[i] = 0;
                rem &= rem - 1;
                if (q[i] < q1[i]) e[i] = __ldg(reinterpret_cast<const int2 *>(P.var_ent) + q[i]);
            }
#pragma unroll
            for (int i = 0; i < kVars; i++) {
                if (q[i] < q1[i]) push(e[i], dj[i]);
                for (int p = q[i] + 32; p < q1[i]; p += 32)
                    push(__ldg(reinterpret_cast<const int2 *>(P.var_ent) + p), dj[i]);
            }
        }
    }
    flush_changed(P, changed);
}

// ---- work distribution ----------------------------------------------------
template <bool kDefer>
__device__ __forceinline__ void activity_item(const DevProblem &P, int it, int lane, int round, bool marked,
                                              int *change, unsigned *tight_ctr, WarpSmem &ws, int par, int part = 0,
                                              int parts = 1) {
    if (it >= 0) sell_slice<1, kDefer>(P, it, lane, round, marked, change, tight_ctr, ws, par, part, parts);
    else split_partial<1>(P, -it - 1, lane, round, marked, change, tight_ctr, ws);
}

// Items are claimed one, two or three at a time: from 8 items per warp on in
// pairs, from 32 on in threes (two items on one warp are twice its latency, but
// the light end of the heaviest-first order, slices of one-lane rows, is screened
// as a group with all its loads in flight). One at a time against pairs, 300,000
// rows (6.6 items per warp): 5.6 against 6.1 ms; 600,000 (13): 10.4 against 10.2;
// pairs against threes, 1M rows (22): 15.6 and 15.6; 2M rows (44): 27.4 against
// 26.8. Other claims run item by item.
template <int K>
__device__ __forceinline__ bool screen_group(const DevProblem &P, const int (&it)[3], int lane, int round, bool marked,
                                             WarpSmem &ws, int par) {
    int sl[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        if (it[k] < 0 || __ldg(P.slice_lg + it[k]) != 0) return false;
        sl[k] = it[k];
    }
    sell_slices_g1<K, 1>(P, sl, lane, round, marked, ws, par);
    return true;
}
template <bool kDefer>
__device__ __forceinline__ void activity_phase(const DevProblem &P, int round, bool marked, unsigned *ctr,
                                               int *change, unsigned *tight_ctr, WarpSmem &ws, int lane,
                                               int par = 0) {
    const int nw = grid_warps();
    if (!kDefer && P.parts > 1) {  // a warp for each part of each slice
        const int i = grid_warp_striped();
        if (i < P.n_items * P.parts)
            activity_item<kDefer>(P, __ldg(P.items + i / P.parts), lane, round, marked, change, tight_ctr, ws, par,
                                  i % P.parts, P.parts);
        return;
    }
    const int take = P.n_items >= 32 * nw ? 3 : P.n_items >= 8 * nw ? 2 : 1;  // items of a claim
    WarpCursor<true> cur;
    cur.start(ctr, take, nw, P.n_items);
    for (;;) {
        const int i = cur.next(lane);
        if (i >= P.n_items) break;
        int it[3];
#pragma unroll
        for (int k = 0; k < 3; k++) it[k] = k < take && i + k < P.n_items ? __ldg(P.items + i + k) : -1;
        if (kDefer && i + take <= P.n_items) {
            if (take == 3 && screen_group<3>(P, it, lane, round, marked, ws, par)) continue;
            if (take == 2 && screen_group<2>(P, it, lane, round, marked, ws, par)) continue;
        }
#pragma unroll 1
        for (int k = 0; k < take && i + k < P.n_items; k++)
            activity_item<kDefer>(P, it[k], lane, round, marked, change, tight_ctr, ws, par);
    }
}

// Candidate phase over the tiles of multi-tile rows: warp w takes the tiles
// w, w + W, ... (W warps), one per lane per step, and runs those whose row is
// due (every tile in an unmarked round, the tiles of marked rows otherwise).
// The tiles hold at most split_tile non-zeros each and the deferred exact rows
// that follow in the same phase are claimed dynamically, so a static
// assignment costs no balance and saves a contended claim per tile.
__device__ __forceinline__ void candidate_phase(const DevProblem &P, int round, bool marked, int *exact_ctr,
                                                WarpSmem &ws, int lane) {
    const int nw = grid_warps();
    for (int i0 = grid_warp_striped(); i0 < P.n_mtiles; i0 += 32 * nw) {
        const int i = i0 + lane * nw;
        int t = 0;
        bool live = false;
        if (i < P.n_mtiles) {
            t = __ldg(P.mtiles + i);
            live = !marked || P.mark[P.n_srows + __ldg(P.tile_row + t)] == round;
        }
        for (unsigned bal = __ballot_sync(kFull, live); bal; bal &= bal - 1)
            split_cand<1>(P, __shfl_sync(kFull, t, __ffs(bal) - 1), lane, round, false, exact_ctr, ws);
    }
}

// Exact phase over the tiles of the multi-tile rows flagged this round, with
// the same static assignment as the candidate phase, each tile's candidates in
// quarters (a warp per quarter): the row test is the same for every quarter,
// and a tile's 1,024 candidate tests and divisions on one warp were the
// phase's long pole while the rest of the grid waited at its barrier.
__device__ __forceinline__ void exact_phase(const DevProblem &P, int round, int *change, unsigned *tight_ctr,
                                            WarpSmem &ws, int lane) {
    const int nw = grid_warps();
    const int n_items = P.n_mtiles * kTileParts;
    for (int i0 = grid_warp_striped(); i0 < n_items; i0 += 32 * nw) {
        const int i = i0 + lane * nw;
        int t = 0;
        bool live = false;
        if (i < n_items) {
            t = __ldg(P.mtiles + i / kTileParts);
            live = P.row_exact[__ldg(P.tile_row + t)] == round;
        }
        for (unsigned bal = __ballot_sync(kFull, live); bal; bal &= bal - 1) {
            const int src = __ffs(bal) - 1;
            split_exact<1>(P, __shfl_sync(kFull, t, src), lane, round, change, tight_ctr, ws,
                           (i0 + src * nw) % kTileParts, kTileParts);
        }
    }
}

// Whether the activity phase of this round's parity queued exact rows.
__device__ __forceinline__ bool exact_rows_queued(const DevProblem &P, int par) {
    unsigned n = 0;
#pragma unroll
    for (int lg = 0; lg < 6; lg++) n |= *((volatile unsigned *)(P.xctr + 16 * par + lg));
    return n != 0;
}

// Whether the round after one with `tight` tightenings runs on marked rows.
__device__ __forceinline__ bool next_round_marked(const DevProblem &P, unsigned tight) {
    return P.use_marking == 2 || (P.use_marking == 1 && tight < P.mark_threshold);
}

// Grid barrier with a bounded wait. bar counts arrivals and only grows (zero
// at launch); `target` is the caller's copy of the count that the next barrier
// completes at. Thread 0 of each CTA arrives with one release add and polls
// the count itself: no last arriver resets it and raises a second word, which
// cost a round trip more (456 CTAs: 1.6 us a barrier instead of 2.9; 152: 1.2
// instead of 2.5; 8: 0.7 instead of 1.6). The polls are relaxed loads and one
// fence follows them: an acquire load per poll invalidates the L1 that the
// SM's other CTAs still work with. Counts are compared modulo 2^32.
// Any CTA that waits longer than `limit` clock64 cycles (or sees another
// CTA's error) records kErrBarrierTimeout and every CTA leaves the round loop
// at its next barrier. The default limit is 4e9 cycles, about 2 s at 2 GHz.
// A single CTA needs no fence and keeps its L1 (100 rows: 0.23 -> 0.16 ms):
// __syncthreads makes what any of its threads wrote, by atomics or plain stores,
// what all of them read afterwards, by plain loads too (the change bitmap of the
// allocation-free loop, the drift bounds of split rows).
__device__ __forceinline__ bool grid_barrier(unsigned *bar, int *error, long long limit, unsigned &target) {
    __syncthreads();
    if (gridDim.x == 1) return *((volatile int *)error) == kErrNone;
    int ok = 1;
    target += gridDim.x;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        const long long t0 = clock64();
        for (int polls = 1;; polls++) {
            unsigned count;
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(count) : "l"(bar) : "memory");
            if ((int)(count - target) >= 0) break;
            if (clock64() - t0 > limit) {
                atomicExch(error, (int)kErrBarrierTimeout);
                ok = 0;
                break;
            }
            if (polls % 16 == 0 && *((volatile int *)error) != kErrNone) {
                ok = 0;
                break;
            }
            __nanosleep(20);
        }
        __threadfence();
        if (*((volatile int *)error) != kErrNone) ok = 0;
    }
    return __syncthreads_and(ok) != 0;
}

}  // namespace
}  // namespace gdp
