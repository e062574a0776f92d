// gdp_exact.cuh -- the exact FP64 pass of the rows that the FP32 screen cannot
// skip: activities, the reference's row test, candidates and their divisions,
// for a few rows per warp.
//
// What bounds it: the FP64 pipe. A dependent FP64 add takes 71 cycles, and a
// warp's next FP64 instruction starts 68 to 76 cycles after its last one even
// when it does not depend on it (measured: one FP64 unit per SM quarter, 0.44
// lanes per clock), so an FP64 instruction costs the same with one active lane
// as with 32, and the number of FP64 instructions in a row's path is its
// latency. One lane walking a row of 32 elements executes 8 of them per
// element (two products, two sums, |a| (ub - lb), the EPS-max): 256
// instructions, 9.4 us, whether the warp's other lanes have rows or not.
//
// Here the rows of a warp are one flat list of elements. 32 lanes form the
// products of 32 consecutive elements, whichever rows they belong to, and
// stage them in shared memory (5 FP64 instructions per 32 elements); then one
// lane per row, lane of the row's summation order and side (minimum and
// maximum activity in different lanes) adds them up in that order: one FP64
// add per step for both sides of 16 / g rows. The additions and their order
// are those of one lane (g = 1) or g lanes per row, so every bit is the same.
// The first maximum of |a| (ub - lb) is found by integer compares beside the
// adds. 16 rows of L elements take 3.5 L FP64 instructions instead of 8 L (and
// 32 rows 7 L instead of 8 L).
//
// Elements whose |a| (ub - lb) exceeds the screen's lower bound of both slacks
// -- the only ones that can yield a candidate -- are collected while they are
// staged, so the candidate tests run on full warps over a few elements per row
// instead of visiting the rows again; divisions wait in a queue that carries
// their numerators and outlives the rows, and run 32 at a time.
#pragma once

#include "gdp_device.cuh"

namespace gdp {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kStage = 128;     // elements staged at a time
constexpr int kItemRows = 16;   // most rows of a warp's item (g = 1; 16 / g rows of g lanes)
constexpr int kCandCap = 96;    // collected elements; rows that yield more are read again
constexpr int kDivCap = 96;     // >= 31 pending + 64 pushed per step

// A queued division: numerator, element, and code: bit 0 the side (0 upper
// bound, 1 lower), bit 1 whether the variable's other bound is added, bits 2..
// the row's slot.
struct DivEntry {
    double num;
    int k;
    unsigned code;
};

struct ExactSmem {
    double t[2][kStage];  // minimum / maximum activity terms
    double d[kStage];     // |a| (ub - lb)
    DivEntry div[kDivCap];
    double cand_d[kCandCap];
    int cand_k[kCandCap];
    unsigned char cand_s[kCandCap];  // row slot, bit 7: a > 0
    double slack[kItemRows], nsur[kItemRows];  // rhs - minact, maxact - lhs
    long long cut[kItemRows];  // order key that |a| (ub - lb) must exceed
    int src[kItemRows];        // element index of the row's flat index 0
    unsigned info[kItemRows];  // bits 0, 1: usable sides; 2, 3: minf; 4, 5: maxf; 6: candidates wanted
};

// The rows of an item: lane r < n holds row r (in is set for those lanes).
struct ExactRow {
    bool in;
    int base, len;    // first element, elements
    float slack_lo;   // the screen's lower bound of both slacks
    int minf, maxf;   // infinite contributions (the screen counts them exactly)
    double lhs, rhs;
};

// What a row's sums gave, in the lane that holds the row.
struct ExactSums {
    double minact, maxact;
    long long km;  // first maximum of |a| (ub - lb): order key and element (-1: the leading 0.0)
    int p;
};

struct ExactQueue {
    int cnt;     // divisions pending (warp-uniform)
    int pushed;  // divisions queued so far (warp-uniform)
    int tight;   // bounds tightened by this lane
};

// Flat list of the item's rows: lane r's row has the flat indices pre .. pre + len - 1.
struct FlatRows {
    int pre, len, total;
};
__device__ __forceinline__ FlatRows flat_rows(const ExactRow &R, int lane) {
    FlatRows F;
    F.len = R.in ? R.len : 0;
    int inc = F.len;
#pragma unroll
    for (int off = 1; off < kItemRows; off <<= 1) {
        const int v = __shfl_up_sync(kFull, inc, off);
        if (lane >= off) inc += v;
    }
    F.total = __shfl_sync(kFull, inc, kItemRows - 1);
    F.pre = inc - F.len;
    return F;
}
// The slot of the row that owns flat element f0 + lane (rows of the list are
// not empty, so their first elements are distinct).
__device__ __forceinline__ int flat_slot(const FlatRows &F, int f0, int lane) {
    const int s = F.pre - f0;
    const unsigned starts = __reduce_or_sync(kFull, (F.len && s >= 0 && s < 32) ? 1u << s : 0u);
    const int before = __popc(__ballot_sync(kFull, F.len && s < 0));
    return before + __popc(starts & (kFull >> (31 - lane))) - 1;
}

// The terms of one element as computeActivities forms them
// (src/propagation_methods.cuh:188-214); an infinite contribution is left out
// of its sum (adding +0.0 changes no sum that starts at +0.0).
__device__ __forceinline__ void exact_terms(double a, double2 b, double &tmin, double &tmax, double &d) {
    const long long ab = dbits(a);
    const bool pos = gt_eps_bits(ab), lneg = neginf_bits(dbits(b.x)), upos = posinf_bits(dbits(b.y));
    const bool gt0 = gt0_bits(ab);
    tmin = (pos ? lneg : upos) ? 0.0 : dmul(a, gt0 ? b.x : b.y);
    tmax = (pos ? upos : lneg) ? 0.0 : dmul(a, gt0 ? b.y : b.x);
    d = dmul(fabs(a), dsub(b.y, b.x));
}

// Runs queued divisions 32 at a time (all of them with `all`): the candidate
// of tightenVarUpperBound / tightenVarLowerBound (src/propagation_methods.cuh:
// 78-134), applied if it is EPS-better than the round-start bound. T gives the
// elements, the bounds and the targets; row_tight (may be null) counts the
// tightenings by row slot.
template <class T>
__device__ __forceinline__ void exact_drain(const T &t, ExactSmem &xs, ExactQueue &Q, bool all, int lane,
                                            int *row_tight = nullptr) {
    while (Q.cnt >= 32 || (all && Q.cnt > 0)) {
        const int take = min(Q.cnt, 32);
        if (lane < take) {
            const DivEntry q = xs.div[lane];
            const int j = __ldg(t.col + q.k);
            const double a = __ldg(t.val + q.k);
            const double2 b = t.bnd[j];
            const bool lower = q.code & 1u;
            double nb = ddiv(q.num, a);
            if (q.code & 2u) nb = dadd(nb, lower ? b.y : b.x);
            if (!t.cont(j)) nb = lower ? eps_ceil(nb) : eps_floor(nb);
            if (lower ? eps_gt(nb, b.x) : eps_lt(nb, b.y)) {
                t.apply(j, nb, lower);
                Q.tight++;
                if (row_tight) atomicAdd(row_tight + (q.code >> 2), 1);
            }
        }
        __syncwarp();
        const int rest = Q.cnt - take;
        DivEntry mv[2];
#pragma unroll
        for (int i = 0; i < 2; i++)
            if (lane + 32 * i < rest) mv[i] = xs.div[take + lane + 32 * i];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 2; i++)
            if (lane + 32 * i < rest) xs.div[lane + 32 * i] = mv[i];
        __syncwarp();
        Q.cnt = rest;
    }
}

// Queues the divisions of one element per lane (tightenVariable, src/
// propagation_methods.cuh:223-276): element k with |a| (ub - lb) = d of the row
// in slot `slot`; pos: a > 0. Lanes without an element pass on = false.
template <class T>
__device__ __forceinline__ void exact_push(const T &t, ExactSmem &xs, ExactQueue &Q, bool on, int k, int slot,
                                           bool pos, double d, int lane, int *row_tight) {
    int sides = 0;
    unsigned info = 0;
    double s = 0.0, u = 0.0;
    if (on) {
        info = xs.info[slot];
        s = xs.slack[slot];
        u = xs.nsur[slot];
        const bool rs = (info & 1u) && eps_gt_fast(d, s);
        const bool ls = (info & 2u) && eps_gt_fast(d, u);
        const int minf = (info >> 2) & 3, maxf = (info >> 4) & 3;
        const int nu = pos ? minf : maxf, nl = pos ? maxf : minf;
        bool uo = (pos ? rs : ls) && nu <= 1, lo = (pos ? ls : rs) && nl <= 1;
        if ((uo && nu == 1) || (lo && nl == 1)) {  // the only infinite contribution must be this variable's
            const double2 b = t.bnd[__ldg(t.col + k)];
            uo = uo && (nu == 0 || neginf_bits(dbits(b.x)));
            lo = lo && (nl == 0 || posinf_bits(dbits(b.y)));
        }
        sides = (uo ? 1 : 0) | (lo ? 2 : 0);
    }
    const unsigned bu = __ballot_sync(kFull, sides & 1), bl = __ballot_sync(kFull, sides & 2);
    if (!(bu | bl)) return;
    const unsigned lt = (1u << lane) - 1u;
    // lhs - maxact is -(maxact - lhs) (round-to-nearest is symmetric), +0.0 when they are equal
    const double surplus = __longlong_as_double((dbits(u) << 1) ? dbits(u) ^ (1LL << 63) : 0LL);
    if (sides & 1)
        xs.div[Q.cnt + __popc(bu & lt)] =
                DivEntry{pos ? s : surplus, k, (unsigned)slot << 2 | ((pos ? info >> 2 : info >> 4) & 3u ? 0u : 2u)};
    if (sides & 2)
        xs.div[Q.cnt + __popc(bu) + __popc(bl & lt)] = DivEntry{
                pos ? surplus : s, k, (unsigned)slot << 2 | ((pos ? info >> 4 : info >> 2) & 3u ? 0u : 2u) | 1u};
    __syncwarp();
    Q.cnt += __popc(bu) + __popc(bl);
    Q.pushed += __popc(bu) + __popc(bl);
    exact_drain(t, xs, Q, false, lane, row_tight);
}

// Activities and first maximum of the item's rows, g = 2^lg lanes per row in
// the summation order (16 / g rows; one row for g = 32). Collects the elements
// above the rows' cuts; cand receives their number (more than kCandCap: the
// list is not complete).
template <class T>
__device__ __forceinline__ ExactSums exact_sums(const T &t, ExactSmem &xs, const ExactRow &R, const FlatRows &F,
                                                int lg, int lane, int &cand) {
    const int g = 1 << lg;
    __syncwarp();
    if (R.in) {
        xs.src[lane] = R.base - F.pre;
        xs.cut[lane] = order_key(dbits(R.slack_lo == R.slack_lo ? (double)R.slack_lo : -1e308));
    }
    __syncwarp();
    // this lane's part of the adds: side, row slot and lane of the row
    const int side = lg < 5 ? lane >> 4 : 0;
    const int slot = lg < 5 ? (lane & 15) >> lg : 0;
    const int sub = lane & (g - 1);
    const int rpre = __shfl_sync(kFull, F.pre, slot), rlen = __shfl_sync(kFull, F.len, slot);
    double acc = 0.0, acc2 = 0.0;  // acc2: maximum activity of a 32-lane row
    long long km = 0;
    int p = -1, e = sub;
    cand = 0;
    for (int w0 = 0; w0 < F.total; w0 += kStage) {
        constexpr int kSteps = kStage / 32;
        int k[kSteps], slots[kSteps], j[kSteps];
        double a[kSteps];
        double2 b[kSteps];
#pragma unroll
        for (int i = 0; i < kSteps; i++) {
            slots[i] = flat_slot(F, w0 + 32 * i, lane);
            const int f = w0 + 32 * i + lane;
            k[i] = f < F.total ? xs.src[slots[i]] + f : -1;
            j[i] = k[i] >= 0 ? __ldg(t.col + k[i]) : 0;
            a[i] = k[i] >= 0 ? __ldg(t.val + k[i]) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < kSteps; i++) b[i] = k[i] >= 0 ? t.bnd[j[i]] : make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < kSteps; i++) {
            if (w0 + 32 * i >= F.total) break;  // warp-uniform
            double d;
            exact_terms(a[i], b[i], xs.t[0][32 * i + lane], xs.t[1][32 * i + lane], d);
            xs.d[32 * i + lane] = d;
            const long long db = dbits(d);
            const bool keep = k[i] >= 0 && (order_key(db) > xs.cut[slots[i]] ||
                                            (db & 0x7FF0000000000000LL) == 0x7FF0000000000000LL);
            const unsigned bal = __ballot_sync(kFull, keep);
            const int at = cand + __popc(bal & ((1u << lane) - 1u));
            if (keep && at < kCandCap) {
                xs.cand_d[at] = d;
                xs.cand_k[at] = k[i];
                xs.cand_s[at] = (unsigned char)(slots[i] | (gt0_bits(dbits(a[i])) ? 128 : 0));
            }
            cand += __popc(bal);
        }
        __syncwarp();
        const int end = min(rlen, w0 + kStage - rpre);  // elements of my row staged so far
        const int at = rpre - w0;  // staged index of my row's element 0
#pragma unroll 4
        for (; e < end; e += g) {
            acc = dadd(acc, xs.t[side][at + e]);
            if (lg == 5) acc2 = dadd(acc2, xs.t[1][at + e]);
            const long long kd = order_key(dbits(xs.d[at + e]));
            if (kd > km && kd <= kKeyPosInf) {
                km = kd;
                p = e;
            }
        }
        __syncwarp();
    }
    for (int off = g >> 1; off > 0; off >>= 1) {
        acc = dadd(acc, __shfl_down_sync(kFull, acc, off));
        if (lg == 5) acc2 = dadd(acc2, __shfl_down_sync(kFull, acc2, off));
        const long long ok = __shfl_down_sync(kFull, km, off);
        const int op = __shfl_down_sync(kFull, p, off);
        if (ok > km || (ok == km && op < p)) {
            km = ok;
            p = op;
        }
    }
    // back to the lanes that hold the rows
    const int lead = R.in ? lane << lg : 0;
    ExactSums s;
    s.minact = __shfl_sync(kFull, acc, lead);
    const double hi = __shfl_sync(kFull, acc, (lead + 16) & 31), hi32 = __shfl_sync(kFull, acc2, 0);
    s.maxact = lg < 5 ? hi : hi32;
    s.km = __shfl_sync(kFull, km, lead);
    s.p = __shfl_sync(kFull, p, lead);
    return s;
}

// The row test of the rows from their sums: s and t are rhs - minact and
// maxact - lhs. 0: skip, 1: process, 2: only the sequential EPS-max decides
// (row_go_from_max). bad: the row is infeasible (row_infeasible).
__device__ __forceinline__ int exact_decide(const ExactRow &R, const ExactSums &S, double &s, double &t, double &mn,
                                            bool &bad) {
    s = dsub(R.rhs, S.minact);
    t = dsub(S.maxact, R.lhs);
    mn = (t < s) ? t : s;
    // a row with both slacks >= 0 is feasible
    bad = (dbits(s) < 0 || dbits(t) < 0) && row_infeasible(S.minact, S.maxact, R.minf, R.maxf, R.lhs, R.rhs);
    return row_go_from_max(R.minf, R.maxf, __longlong_as_double(S.km), mn);
}

// Candidates of the rows with go set (lanes that hold rows), from their
// slacks s and t; cand: the collected elements.
template <class T>
__device__ __forceinline__ void exact_candidates(const T &t, ExactSmem &xs, ExactQueue &Q, const ExactRow &R,
                                                 const FlatRows &F, const ExactSums &S, bool go, double s, double u,
                                                 int cand, int lane, int *row_tight = nullptr) {
    if (!__any_sync(kFull, go)) return;
    if (R.in) {
        const bool rhs_ok = !posinf_bits(dbits(R.rhs)) && !neginf_bits(dbits(S.minact));
        const bool lhs_ok = !neginf_bits(dbits(R.lhs)) && !posinf_bits(dbits(S.maxact));
        xs.slack[lane] = s;
        xs.nsur[lane] = u;
        xs.info[lane] = (rhs_ok ? 1u : 0u) | (lhs_ok ? 2u : 0u) | (unsigned)min(R.minf, 3) << 2 |
                        (unsigned)min(R.maxf, 3) << 4 | (go ? 64u : 0u);
    }
    __syncwarp();
    if (cand <= kCandCap) {
        for (int i0 = 0; i0 < cand; i0 += 32) {
            const int i = i0 + lane;
            const bool on = i < cand && (xs.info[xs.cand_s[i] & 127] & 64u);
            const int c = on ? xs.cand_s[i] : 0;
            exact_push(t, xs, Q, on, on ? xs.cand_k[i] : 0, c & 127, c & 128, on ? xs.cand_d[i] : 0.0, lane,
                       row_tight);
        }
    } else {  // more than the list holds: every element of the rows again
        for (int f0 = 0; f0 < F.total; f0 += 32) {
            const int slot = flat_slot(F, f0, lane), f = f0 + lane;
            const bool on = f < F.total && (xs.info[slot] & 64u);
            int k = 0;
            bool pos = false;
            double d = 0.0;
            if (on) {
                k = xs.src[slot] + f;
                const double a = __ldg(t.val + k);
                const double2 b = t.bnd[__ldg(t.col + k)];
                pos = gt0_bits(dbits(a));
                d = dmul(fabs(a), dsub(b.y, b.x));
            }
            exact_push(t, xs, Q, on, k, slot, pos, d, lane, row_tight);
        }
    }
}

}  // namespace
}  // namespace gdp
