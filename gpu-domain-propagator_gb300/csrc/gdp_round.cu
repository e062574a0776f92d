// gdp_round.cu -- one Jacobi propagation round on sm_103a, as phase kernels
// (GPU_LOOP driver) and as a persistent cooperative megakernel that runs every
// round in one launch (MEGAKERNEL driver) or one round per launch (CPU_LOOP).
// The round's device functions live in gdp_round.cuh.
#include <algorithm>
#include <cstddef>

#include "gdp_round.cuh"
#include "gdp_sequence.h"

namespace gdp {

namespace {

// Shared memory of 16 warps (and 1 KB the system keeps per CTA) as a share of
// the 228 KB per SM, in percent.
constexpr int kCarveout = (int)((16 * sizeof(WarpSmem) + 6 * 1024) * 100 / (228 * 1024) + 1);

// ---- phase kernels (GPU_LOOP) -----------------------------------
// The screen alone needs few registers: 32 warps per SM. The exact passes take
// 16 with 128 registers, as in the megakernel (60,001 rows: 4.9 ms with 4 CTAs of
// 64 registers for all three, 4.0 with these).
__global__ void __launch_bounds__(kCtaThreads, 4) k_activity(const __grid_constant__ DevProblem P) {
    WarpSmem *ws = warp_smem();
    const int round = P.flags[0].rounds;
    if (P.flags[0].infeasible) return;
    stats_zero(ws[threadIdx.x >> 5], threadIdx.x & 31);
    activity_phase<true>(P, round, P.flags[0].mark_cur != 0, P.queue + 0, &P.flags[0].change, &P.flags[0].tight,
                   ws[threadIdx.x >> 5], threadIdx.x & 31);
    stats_flush(P, ws[threadIdx.x >> 5], threadIdx.x & 31);
}

__global__ void __launch_bounds__(kCtaThreads, 2) k_candidates(const __grid_constant__ DevProblem P) {
    WarpSmem *ws = warp_smem();
    const int round = P.flags[0].rounds;
    if (P.flags[0].infeasible) return;
    // the multi-tile rows' tiles (1,024 non-zeros each) first, the deferred
    // exact rows (at most split_tile non-zeros, mostly short) after them: the
    // heavy items do not end up as the phase's tail
    stats_zero(ws[threadIdx.x >> 5], threadIdx.x & 31);
    candidate_phase(P, round, P.flags[0].mark_cur != 0, &P.flags[0].exact, ws[threadIdx.x >> 5], threadIdx.x & 31);
    if (exact_rows_queued(P, 0))
        exact_rows_phase(P, 0, &P.flags[0].change, &P.flags[0].tight, ws[threadIdx.x >> 5], threadIdx.x & 31);
    stats_flush(P, ws[threadIdx.x >> 5], threadIdx.x & 31);
}

__global__ void __launch_bounds__(kCtaThreads, 2) k_exact(const __grid_constant__ DevProblem P) {
    WarpSmem *ws = warp_smem();
    const int round = P.flags[0].rounds;
    if (P.flags[0].infeasible || P.flags[0].exact == 0) return;
    stats_zero(ws[threadIdx.x >> 5], threadIdx.x & 31);
    exact_phase(P, round, &P.flags[0].change, &P.flags[0].tight, ws[threadIdx.x >> 5], threadIdx.x & 31);
    stats_flush(P, ws[threadIdx.x >> 5], threadIdx.x & 31);
}

// Starts a round: counts it, takes the mode that the finished round's
// tightenings chose, clears the change flag, tightening count and work
// counters. One thread.
__device__ __forceinline__ void begin_round(const DevProblem &P) {
    const int r = P.flags[0].rounds;
    P.flags[0].mark_cur = r > 0 && next_round_marked(P, P.flags[0].tight);
    P.flags[0].change = 0;
    P.flags[0].tight = 0u;
    P.flags[0].exact = 0;
    P.flags[0].rounds = r + 1;
    for (int i = 0; i < 4; i++) P.queue[i] = 0u;
    for (int i = 0; i < 16; i++) P.xctr[i] = 0u;
}

__global__ void k_round_begin(DevProblem P) {
    if (!P.flags[0].infeasible) begin_round(P);
}

// Every thread derives the same next-round mode from the final tightening
// count. The last CTA to finish (queue[3] counts them) decides whether the
// graph's WHILE node runs another round, and starts it: two single-thread
// kernels less per round (about 3 us of a 28 us round on 2,000 rows).
__global__ void __launch_bounds__(256) k_finalize(DevProblem P, cudaGraphConditionalHandle h) {
    const bool push = next_round_marked(P, P.flags[0].tight);
    finalize_words(P, P.flags[0].rounds, push, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(P.queue + 3, 1u) != gridDim.x - 1) return;
    __threadfence();
    volatile RoundFlags *f = P.flags;
    const bool more = f->change && !f->infeasible && f->rounds < P.max_rounds;
    if (more) begin_round(P);
    cudaGraphSetConditional(h, more ? 1u : 0u);
}

// The initial bounds' infeasibility check.
__device__ __forceinline__ void check_bounds(const DevProblem &P) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < P.n; j += gridDim.x * blockDim.x) {
        const double2 b = P.bnd[j];
        if (var_infeasible(b.x, b.y)) {
            P.flags[0].infeasible = 1;
            atomicMin(&P.flags[0].infeasible_var, j);
        }
    }
}
__global__ void __launch_bounds__(256) k_check_bounds(DevProblem P) { check_bounds(P); }

// Everything that a propagation starts from: round state, bounds in the three
// forms the rounds read, cleared bitmap, marks and drift bounds. lb / ub may
// be host memory that the device reaches directly. A single CTA checks the
// bounds itself.
__global__ void __launch_bounds__(1024) k_start(DevProblem P, const double *lb, const double *ub) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    int *state = reinterpret_cast<int *>(P.flags);
    for (int i = tid; i < (int)(3 * sizeof(RoundFlags) / sizeof(int)); i += nt)
        state[i] = i == (int)(offsetof(RoundFlags, infeasible_var) / sizeof(int)) ||
                                   i == (int)(offsetof(RoundFlags, infeasible_row) / sizeof(int))
                           ? INT_MAX
                           : 0;
    if (tid < 8) P.queue[tid] = 0u;
    if (tid < 32) P.xctr[tid] = 0u;
    if (tid < 2) P.barrier[tid] = 0u;
    for (int w = tid; w < P.n_chg_words; w += nt) P.chg[w] = 0u;
    for (int r = tid; r < P.n_lrows; r += nt) {
        P.row_exact[r] = 0;
        P.lrow_margin[r] = -1.0;  // no drift bound carried over from an earlier propagation
        P.lrow_drift[r] = 0.0;
        P.lrow_skip[r] = 0;
    }
    if (P.use_marking)
        for (int p = tid; p < P.n_srows + P.n_lrows; p += nt) P.mark[p] = 0;
    for (int j = tid; j < P.n; j += nt) {
        const double2 b = make_double2(lb[j], ub[j]);
        P.bnd[j] = b;
        P.bnd_nxt[j] = b;
        store_bnd32<1>(P, j, b, 0);
    }
    if (gridDim.x == 1) {
        __syncthreads();
        check_bounds(P);
    }
}

// The result, unless the rounds ended with a device error. lb / ub may be host
// memory that the device reaches directly.
__global__ void __launch_bounds__(256) k_finish(DevProblem P, double *lb, double *ub) {
    if (P.flags[0].error != kErrNone) return;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < P.n; j += gridDim.x * blockDim.x) {
        const double2 b = P.bnd[j];
        lb[j] = b.x;
        ub[j] = b.y;
    }
}

// ---- megakernel -----------------------------------------------------------
#ifdef GDP_PHASE_TIMERS
// Stamp k of round r by one thread (0: round start, 1: after phase A's
// barrier, 2: after B's, 3: after C's, 4: after F's, with the cumulative
// processed rows, non-zeros and exact non-zeros in slots 5-7).
__device__ __forceinline__ void timer_stamp(const DevProblem &P, int round, int k) {
    if (blockIdx.x != 0 || threadIdx.x != 0 || round >= kTimerRounds) return;
    unsigned long long *w = g_timer_wall + round * kTimerSlots;
    w[k] = timer_now();
    if (k == 4) {
        w[5] = *((volatile unsigned long long *)&P.flags[0].rows_proc);
        w[6] = *((volatile unsigned long long *)&P.flags[0].nnz_proc);
        w[7] = *((volatile unsigned long long *)&P.flags[0].nnz_exact);
    }
}
// adds the warp's time in phase k of round r since t0 (0: A, 1: B multi-tile
// rows, 2: B deferred exact rows, 3: C, 4: F), and keeps the longest single
// warp's time of the phase group in slot 5 (A), 6 (B) or 7 (C and F)
__device__ __forceinline__ void timer_busy(const DevProblem &P, WarpSmem &ws, int lane, int round, int k,
                                           unsigned long long t0) {
    stats_flush(P, ws, lane);  // the stamps read the work counters round by round
    if (lane == 0 && round < kTimerRounds) {
        const unsigned long long dt = timer_now() - t0;
        atomicAdd(&g_timer_busy[round * kTimerSlots + k], dt);
        atomicMax(&g_timer_busy[round * kTimerSlots + (k == 0 ? 5 : k <= 2 ? 6 : 7)], dt);
    }
}
#else
__device__ __forceinline__ void timer_stamp(const DevProblem &, int, int) {}
__device__ __forceinline__ void timer_busy(const DevProblem &, WarpSmem &, int, int, int, unsigned long long) {}
#endif

// Round loop on the device. flags[0] holds the sticky state; flags[1 + (round
// & 1)] the per-round change flag, tightening and exact-row counts, and
// queue[4 * (round & 1) + phase] the per-round work counters, double-buffered
// so that nothing a CTA may still read is cleared: the next round's slots are cleared after the current
// round's first barrier, which every CTA passes only after finishing the
// previous round.
// W warps per CTA; with 16 / W resident CTAs per SM every instance holds 16
// warps per SM with 128 registers each. 24 warps with 80 registers spill around
// the exact pass, and six warps share an SM quarter's FP64 unit instead of four:
// 60,001 rows 4.29 -> 3.62 ms with 16, 300,000 6.45 -> 6.07, 2,000 0.333 -> 0.314,
// 2M rows 27.0 either way (12 warps: 3.5, 6.3, 0.31 and 31.5).
// A launch runs the rounds first .. last, or fewer when one changes nothing or
// turns infeasible; a launch after that one does nothing (flags[0].done), so
// that a host loop may queue a round before it knows whether the round is
// needed. Between launches barrier[1] keeps the barrier count and the round's
// tightenings the next round's mode. mail (may be null): host memory that
// receives {the round, whether another one follows}.
// kInPlace (P.in_place): a problem of one-lane rows only, with at most three slices
// per warp: the screen's warp takes its rows through the exact pass at once,
// which saves the queue, a phase and a barrier. With wide rows in the problem their
// items would follow one another on one warp (2,000 power-law rows: 1.86 -> 2.34
// ms), and they are deferred.
template <int W, bool kInPlace>
__global__ void __launch_bounds__(32 * W, 16 / W) k_megakernel(const __grid_constant__ DevProblem P, int first,
                                                               int last, int *mail) {
    WarpSmem *ws = warp_smem();
    const int lane = threadIdx.x & 31;
    WarpSmem &mine = ws[threadIdx.x >> 5];
    int *err = &P.flags[0].error;
    if (P.flags[0].done || P.flags[0].error != kErrNone) return;
    int last_change = 0, infeasible = P.flags[0].infeasible;
    unsigned target = P.barrier[1];  // grid barrier
    stats_zero(mine, lane);
    // round 1 processes every row
    bool marked = first > 1 && next_round_marked(P, P.flags[1 + ((first - 1) & 1)].tight);
    if (infeasible == 0) {
        for (int round = first; round <= last; round++) {
            const int par = round & 1;
            int *change = &P.flags[1 + par].change;
            unsigned *tight = &P.flags[1 + par].tight;
            int *exact = &P.flags[1 + par].exact;
            unsigned *q = P.queue + 4 * par;
            timer_stamp(P, round, 0);
            unsigned long long t0 = timer_now();
            activity_phase<!kInPlace>(P, round, marked, q + 0, change, tight, mine, lane, par);
            timer_busy(P, mine, lane, round, 0, t0);
            if (!grid_barrier(P.barrier, err, P.spin_limit, target)) return;
            timer_stamp(P, round, 1);
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                P.flags[1 + (par ^ 1)].change = 0;
                P.flags[1 + (par ^ 1)].tight = 0u;
                P.flags[1 + (par ^ 1)].exact = 0;
                P.queue[4 * (par ^ 1) + 0] = 0u;
                P.queue[4 * (par ^ 1) + 1] = 0u;
                P.queue[4 * (par ^ 1) + 2] = 0u;
                if (P.xctr)
                    for (int i = 0; i < 16; i++) P.xctr[16 * (par ^ 1) + i] = 0u;
            }
            const bool xrows = !kInPlace && exact_rows_queued(P, par);
            if (!kInPlace && (xrows || P.n_mtiles)) {
                t0 = timer_now();
                if (P.n_mtiles) candidate_phase(P, round, marked, exact, mine, lane);  // heavy items first
                timer_busy(P, mine, lane, round, 1, t0);
                t0 = timer_now();
                if (xrows) exact_rows_phase(P, par, change, tight, mine, lane);
                timer_busy(P, mine, lane, round, 2, t0);
                if (!grid_barrier(P.barrier, err, P.spin_limit, target)) return;
                timer_stamp(P, round, 2);
                if (P.n_mtiles && *((volatile int *)exact)) {
                    t0 = timer_now();
                    exact_phase(P, round, change, tight, mine, lane);
                    timer_busy(P, mine, lane, round, 3, t0);
                    if (!grid_barrier(P.barrier, err, P.spin_limit, target)) return;
                    timer_stamp(P, round, 3);
                }
            }
            marked = next_round_marked(P, *((volatile unsigned *)tight));
            t0 = timer_now();
            finalize_words(P, round, marked, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
            timer_busy(P, mine, lane, round, 4, t0);
            if (blockIdx.x == 0 && threadIdx.x == 0) P.flags[0].rounds = round;
            if (!grid_barrier(P.barrier, err, P.spin_limit, target)) return;
            timer_stamp(P, round, 4);
            last_change = *((volatile int *)change);
            infeasible = *((volatile int *)&P.flags[0].infeasible);
            if (!last_change || infeasible) break;
        }
    }
    stats_flush(P, mine, lane);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const bool more = last_change && !infeasible;
        P.flags[0].change = last_change;
        P.flags[0].done = more ? 0 : 1;
        P.barrier[1] = target;
        if (mail) {
            *((volatile int *)mail + 1) = more ? 1 : 0;
            __threadfence_system();
            *((volatile int *)mail) = P.flags[0].rounds;
        }
    }
}

}  // namespace

// ---- phase timers ---------------------------------------------------------

int phase_timers_clear() {
#ifdef GDP_PHASE_TIMERS
    static const unsigned long long zero[kTimerRounds * kTimerSlots] = {};
    cudaError_t e = cudaMemcpyToSymbol(g_timer_wall, zero, sizeof(zero));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_timer_busy, zero, sizeof(zero));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_timer_pass, zero, sizeof(unsigned long long) * kTimerPass);
    return (int)e;
#else
    return -1;
#endif
}

int phase_timers_read(unsigned long long *wall, unsigned long long *busy, unsigned long long *pass, int rounds) {
#ifdef GDP_PHASE_TIMERS
    const size_t k = sizeof(unsigned long long) * kTimerSlots * (size_t)std::min(std::max(rounds, 0), kTimerRounds);
    cudaError_t e = cudaSuccess;
    if (wall) e = cudaMemcpyFromSymbol(wall, g_timer_wall, k);
    if (busy && e == cudaSuccess) e = cudaMemcpyFromSymbol(busy, g_timer_busy, k);
    if (pass && e == cudaSuccess) e = cudaMemcpyFromSymbol(pass, g_timer_pass, sizeof(unsigned long long) * kTimerPass);
    return (int)e;
#else
    (void)wall, (void)busy, (void)pass, (void)rounds;
    return -1;
#endif
}

// ---- launchers ------------------------------------------------------------

int launch_start(const DevProblem &P, const double *lb, const double *ub, int blocks, cudaStream_t s) {
    if (blocks <= 32) {  // up to 8,192 variables or rows: one CTA, one launch
        k_start<<<1, 1024, 0, s>>>(P, lb, ub);
        return (int)cudaGetLastError();
    }
    k_start<<<blocks, 256, 0, s>>>(P, lb, ub);
    k_check_bounds<<<blocks, 256, 0, s>>>(P);
    return (int)cudaGetLastError();
}

int launch_finish(const DevProblem &P, double *lb, double *ub, int blocks, cudaStream_t s) {
    k_finish<<<blocks, 256, 0, s>>>(P, lb, ub);
    return (int)cudaGetLastError();
}

int launch_round_begin(const DevProblem &P, cudaStream_t s) {
    k_round_begin<<<1, 1, 0, s>>>(P);
    return (int)cudaGetLastError();
}

int add_round(const DevProblem &P, unsigned long long handle, int act_blocks, int cand_blocks, int vec_blocks,
              Sequence &seq) {
    DevProblem Pc = P;
    cudaGraphConditionalHandle h = (cudaGraphConditionalHandle)handle;
    void *args[] = {&Pc, &h};
    cudaError_t e = cudaSuccess;
    if (P.n_items) e = seq.kernel((const void *)k_activity, act_blocks, kCtaThreads, args, kCtaSmem);
    if (e == cudaSuccess) e = seq.kernel((const void *)k_candidates, cand_blocks, kCtaThreads, args, kCtaSmem);
    if (e == cudaSuccess && P.n_mtiles) e = seq.kernel((const void *)k_exact, cand_blocks, kCtaThreads, args, kCtaSmem);
    if (e == cudaSuccess) e = seq.kernel((const void *)k_finalize, vec_blocks, 256, args, 0);
    return (int)e;
}

namespace {
const void *megakernel_of(int cta_warps, bool in_place) {
    switch (cta_warps) {
        case 4: return in_place ? (const void *)k_megakernel<4, true> : (const void *)k_megakernel<4, false>;
        case 16: return in_place ? (const void *)k_megakernel<16, true> : (const void *)k_megakernel<16, false>;
        default: return in_place ? (const void *)k_megakernel<8, true> : (const void *)k_megakernel<8, false>;
    }
}
}  // namespace

int phase_occupancy(int *act, int *cand, int *mega, int cta_warps, bool in_place) {
    const void *mk = megakernel_of(cta_warps, in_place);
    const size_t mega_smem = sizeof(WarpSmem) * (size_t)cta_warps;
    cudaError_t e = cudaFuncSetAttribute(mk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mega_smem);
    for (const void *k : {(const void *)k_activity, (const void *)k_candidates, (const void *)k_exact})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCtaSmem);
    // a carveout that just holds 16 warps' shared memory, the rest of the
    // 256 KB per SM serving as L1 for the element streams
    if (e == cudaSuccess) e = cudaFuncSetAttribute(mk, cudaFuncAttributePreferredSharedMemoryCarveout, kCarveout);
    if (e != cudaSuccess) return (int)e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(act, k_activity, kCtaThreads, kCtaSmem);
    if (e != cudaSuccess) return (int)e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(cand, k_exact, kCtaThreads, kCtaSmem);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(mega, mk, 32 * cta_warps, mega_smem);
}

int launch_megakernel(const DevProblem &P, int first, int last, int *mail, int grid, int cta_warps, cudaStream_t s) {
    DevProblem Pc = P;
    void *args[] = {&Pc, &first, &last, &mail};
    return (int)cudaLaunchCooperativeKernel(megakernel_of(cta_warps, P.in_place != 0), dim3(grid), dim3(32 * cta_warps), args,
                                            sizeof(WarpSmem) * (size_t)cta_warps, s);
}

}  // namespace gdp
