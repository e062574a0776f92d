// gdp_exact.cuh -- the exact FP64 pass of the rows that the FP32 screen cannot
// skip: activities, the reference's row test, candidates and their divisions,
// for a few rows per warp (an item).
//
// What bounds it: the FP64 pipe. A dependent FP64 add takes 71 cycles, and a
// warp's next FP64 instruction starts 68 to 76 cycles after its last one even
// when it does not depend on it (measured: one FP64 unit per SM quarter, 0.44
// lanes per clock), so an FP64 instruction costs the same with one active lane
// as with 32, and the number of FP64 instructions in a row's path is its
// latency. So
//   * per element 4 products and 2 additions are FP64 (no conversion, no
//     compare, no subtraction for the EPS-max: the first maximum of
//     |a| (ub - lb) is found by integer compares and decides the row test
//     (row_go_from_max) unless it lies in a band of 1e-9);
//   * elements whose |a| (ub - lb) exceeds the screen's lower bound of both
//     slacks -- the only ones that can yield a candidate -- are collected on
//     the way, and the candidate tests run on full warps over those alone
//     instead of visiting the rows again;
//   * divisions wait in a queue that carries their numerators and outlives the
//     rows, and run 32 at a time.
#pragma once

#include "gdp_device.cuh"

namespace gdp {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kItemRows = 32;   // most rows of an item
constexpr int kCandCap = 96;    // collected elements; rows that yield more are read again
constexpr int kDivCap = 64;     // >= 31 pending + 32 pushed per side

// A queued division: numerator, element, and code: bit 0 the side (0 upper
// bound, 1 lower), bit 1 whether the variable's other bound is added, bits 2..
// the row's slot.
struct DivEntry {
    double num;
    int k;
    unsigned code;
};

struct ExactSmem {
    DivEntry div[kDivCap];
    double slack[kItemRows], nsur[kItemRows];  // rhs - minact, maxact - lhs
    int cand_k[kCandCap];
    int src[kItemRows];                 // element index of the row's flat index 0
    unsigned char cand_s[kCandCap];     // row slot
    unsigned char info[kItemRows];      // bits 0, 1: usable sides; 2, 3: minf; 4, 5: maxf; 6: candidates wanted; 7: lhs is -0.0
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
    for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(kFull, inc, off);
        if (lane >= off) inc += v;
    }
    F.total = __shfl_sync(kFull, inc, 31);
    F.pre = inc - F.len;
    return F;
}
// The slot of the row that owns flat element f0 + lane (rows of the list are
// not empty, so their first elements are distinct; slots are lanes 0, 1, ...).
__device__ __forceinline__ int flat_slot(const FlatRows &F, int f0, int lane) {
    const int s = F.pre - f0;
    const unsigned starts = __reduce_or_sync(kFull, (F.len && s >= 0 && s < 32) ? 1u << s : 0u);
    const int before = __popc(__ballot_sync(kFull, F.len && s < 0));
    return before + __popc(starts & (kFull >> (31 - lane))) - 1;
}

// The terms of one element as computeActivities forms them
// (src/propagation_methods.cuh:188-214); an infinite contribution is left out
// of its sum (adding +0.0 changes no sum that starts at +0.0).
// kNan: a NaN bound is no infinity (T::kNan).
template <bool kNan>
__device__ __forceinline__ void exact_terms(double a, double2 b, double &tmin, double &tmax, double &d) {
    const long long ab = dbits(a);
    const bool pos = gt_eps_bits(ab), lneg = neg_inf<kNan>(b.x), upos = pos_inf<kNan>(b.y);
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
            if (!t.cont(j)) nb = eps_round(nb, lower);
            if (eps_better(nb, lower ? b.x : b.y, lower)) {
                t.apply(j, nb, lower);
                Q.tight++;
                if (row_tight) atomicAdd(row_tight + (q.code >> 2), 1);
            }
        }
        __syncwarp();
        Q.cnt -= take;  // at most 31 are left: they do not overlap the ones that ran
        if (lane < Q.cnt) xs.div[lane] = xs.div[take + lane];
        __syncwarp();
    }
}

// Queues the divisions of one element per lane (tightenVariable, src/
// propagation_methods.cuh:223-276): element k with |a| (ub - lb) = d of the row
// in slot `slot`. Lanes without an element pass on = false.
template <class T>
__device__ __forceinline__ void exact_push(const T &t, ExactSmem &xs, ExactQueue &Q, bool on, int k, int slot,
                                           int lane, int *row_tight) {
    bool uo = false, lo = false, pos = false;
    unsigned info = 0;
    double s = 0.0, u = 0.0;
    if (on) {
        const double a = __ldg(t.val + k);
        const double2 b = t.bnd[__ldg(t.col + k)];
        const double d = dmul(fabs(a), dsub(b.y, b.x));
        pos = gt0_bits(dbits(a));
        info = xs.info[slot];
        s = xs.slack[slot];
        u = xs.nsur[slot];
        const bool rs = (info & 1u) && eps_gt_fast(d, s);
        const bool ls = (info & 2u) && eps_gt_fast(d, u);
        const int minf = (info >> 2) & 3, maxf = (info >> 4) & 3;
        const int nu = pos ? minf : maxf, nl = pos ? maxf : minf;
        // a side with one infinite contribution is usable if it is this variable's
        uo = (pos ? rs : ls) && (nu == 0 || (nu == 1 && neg_inf<T::kNan>(b.x)));
        lo = (pos ? ls : rs) && (nl == 0 || (nl == 1 && pos_inf<T::kNan>(b.y)));
    }
    const unsigned bu = __ballot_sync(kFull, uo), bl = __ballot_sync(kFull, lo);
    const unsigned lt = (1u << lane) - 1u;
    // lhs - maxact is -(maxact - lhs) (round-to-nearest is symmetric); when they are equal
    // it is +0.0, or -0.0 if lhs is (a sum that starts at +0.0 never is)
    const double surplus = __longlong_as_double((dbits(u) << 1) ? dbits(u) ^ (1LL << 63)
                                                                : (long long)((unsigned long long)(info & 128u) << 56));
    if (bu) {
        if (uo)
            xs.div[Q.cnt + __popc(bu & lt)] =
                    DivEntry{pos ? s : surplus, k, (unsigned)slot << 2 | ((info >> (pos ? 2 : 4)) & 3u ? 0u : 2u)};
        __syncwarp();
        Q.cnt += __popc(bu);
        Q.pushed += __popc(bu);
        exact_drain(t, xs, Q, false, lane, row_tight);
    }
    if (bl) {
        if (lo)
            xs.div[Q.cnt + __popc(bl & lt)] = DivEntry{
                    pos ? surplus : s, k, (unsigned)slot << 2 | ((info >> (pos ? 4 : 2)) & 3u ? 0u : 2u) | 1u};
        __syncwarp();
        Q.cnt += __popc(bl);
        Q.pushed += __popc(bl);
        exact_drain(t, xs, Q, false, lane, row_tight);
    }
}

// The order key that |a| (ub - lb) must exceed to be collected.
__device__ __forceinline__ long long candidate_cut(float slack_lo) {
    return order_key(dbits(slack_lo == slack_lo ? (double)slack_lo : -1e308));
}
// Collects the lanes' elements with keep set: element k of the row in `slot`.
// cand counts them all; the list holds the first kCandCap.
__device__ __forceinline__ void collect(ExactSmem &xs, int &cand, bool keep, int k, int slot, int lane) {
    const unsigned bal = __ballot_sync(kFull, keep);
    const int at = cand + __popc(bal & ((1u << lane) - 1u));
    if (keep && at < kCandCap) {
        xs.cand_k[at] = k;
        xs.cand_s[at] = (unsigned char)slot;
    }
    cand += __popc(bal);
}

// First maximum by integer compares: the larger key, of equal ones the earlier
// element.
__device__ __forceinline__ void take_first_max(long long &km, int &p, long long ok, int op) {
    if (ok > km || (ok == km && op < p)) {
        km = ok;
        p = op;
    }
}

// Activities and first maximum of the item's rows. A chain is one of the
// g = 2^lg lanes in the row's summation order; H = 2^lh lanes work on a chain,
// so an item has 32 / H chains (32 / H / g rows). The additions and their order
// are those of the contract whatever H is (an element beyond the row's end adds
// +0.0, which changes no sum that starts at +0.0).
//
// H = 1: a lane forms its chain's terms and adds up both sides: 6 FP64
// instructions per step of the chains. For rounds with many rows.
// T::kAligned: rows start on 16-byte boundaries and are padded to them, so
// four columns and four coefficients of a one-lane row are three loads.
template <class T>
__device__ __forceinline__ ExactSums exact_sums(const T &t, ExactSmem &xs, const ExactRow &R, int lg, int lane,
                                                int &cand) {
    constexpr int kU = 4;
    const int g = 1 << lg;
    const int slot = lane >> lg, sub = lane & (g - 1);
    const int base = __shfl_sync(kFull, R.base, slot) + sub;
    const int len = __shfl_sync(kFull, R.in ? R.len : 0, slot);
    const long long cut = candidate_cut(__shfl_sync(kFull, R.slack_lo, slot));
    const int steps = len > sub ? (len - sub + g - 1) >> lg : 0;
    const int most = __reduce_max_sync(kFull, steps);
    double acc = 0.0, acc2 = 0.0;
    long long km = 0;
    int p = -1;
    cand = 0;
    __syncwarp();  // the list is free
    for (int s0 = 0; s0 < most; s0 += kU) {
        int j[kU];
        double a[kU];
        double2 b[kU];
        if (T::kAligned && lg == 0) {
            if (s0 < steps) {
                const int4 c4 = __ldg(reinterpret_cast<const int4 *>(t.col + base + s0));
                const double2 v0 = __ldg(reinterpret_cast<const double2 *>(t.val + base + s0));
                const double2 v1 = __ldg(reinterpret_cast<const double2 *>(t.val + base + s0 + 2));
                j[0] = c4.x; j[1] = c4.y; j[2] = c4.z; j[3] = c4.w;
                a[0] = v0.x; a[1] = v0.y; a[2] = v1.x; a[3] = v1.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < kU; i++)
                if (s0 + i < steps) {
                    j[i] = __ldg(t.col + base + ((s0 + i) << lg));
                    a[i] = __ldg(t.val + base + ((s0 + i) << lg));
                }
        }
#pragma unroll
        for (int i = 0; i < kU; i++)
            if (s0 + i < steps) b[i] = t.bnd[j[i]];
        unsigned keep = 0u;
#pragma unroll
        for (int i = 0; i < kU; i++)
            if (s0 + i < steps) {
                double tmin, tmax, d;
                exact_terms<T::kNan>(a[i], b[i], tmin, tmax, d);
                acc = dadd(acc, tmin);
                acc2 = dadd(acc2, tmax);
                const long long db = dbits(d), kd = order_key(db);
                if (kd > km && kd <= kKeyPosInf) {
                    km = kd;
                    p = sub + ((s0 + i) << lg);
                }
                if (kd > cut || (db & 0x7FF0000000000000LL) == 0x7FF0000000000000LL) keep |= 1u << i;
            }
        if (__any_sync(kFull, keep)) {
#pragma unroll
            for (int i = 0; i < kU; i++) collect(xs, cand, (keep >> i) & 1u, base + ((s0 + i) << lg), slot, lane);
        }
    }
    for (int off = g >> 1; off > 0; off >>= 1) {
        acc = dadd(acc, __shfl_down_sync(kFull, acc, off));
        acc2 = dadd(acc2, __shfl_down_sync(kFull, acc2, off));
        const long long ok = __shfl_down_sync(kFull, km, off);
        take_first_max(km, p, ok, __shfl_down_sync(kFull, p, off));
    }
    // back to the lanes that hold the rows
    const int lead = R.in ? lane << lg : 0;
    ExactSums s;
    s.minact = __shfl_sync(kFull, acc, lead);
    s.maxact = __shfl_sync(kFull, acc2, lead);
    s.km = __shfl_sync(kFull, km, lead);
    s.p = __shfl_sync(kFull, p, lead);
    return s;
}

// H = 2^lh >= 2 lanes per chain: they form the terms of H consecutive steps
// together (4 FP64 instructions), then the even lanes add up the minimum and
// the odd lanes the maximum activity (H adds, terms by shuffles): 4 / H + 1 per
// step. The same rate as H = 1 at H = 2 and a shorter path: a 32-element row
// takes 96 FP64 instructions at H = 2, 48 at H = 8, 192 at H = 1. For rounds
// with few rows.
template <class T>
__device__ __forceinline__ ExactSums exact_sums_spread(const T &t, ExactSmem &xs, const ExactRow &R, int lg, int lh,
                                                       int lane, int &cand) {
    constexpr int kU = 4;
    const int g = 1 << lg, H = 1 << lh;
    const int chain = lane >> lh, h = lane & (H - 1), first = lane - h;
    const int slot = chain >> lg, sub = chain & (g - 1);
    const int base = __shfl_sync(kFull, R.base, slot) + sub;
    const int len = __shfl_sync(kFull, R.in ? R.len : 0, slot);
    const long long cut = candidate_cut(__shfl_sync(kFull, R.slack_lo, slot));
    const int steps = len > sub ? (len - sub + g - 1) >> lg : 0;
    const int most = __reduce_max_sync(kFull, steps);
    double acc = 0.0;
    long long km = 0;
    int p = -1;
    cand = 0;
    __syncwarp();  // the list is free
    for (int s0 = 0; s0 < most; s0 += kU * H) {
        int j[kU];
        double a[kU];
        double2 b[kU];
#pragma unroll
        for (int i = 0; i < kU; i++) {
            const int q = s0 + i * H + h;
            j[i] = q < steps ? __ldg(t.col + base + (q << lg)) : -1;
            a[i] = q < steps ? __ldg(t.val + base + (q << lg)) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < kU; i++) b[i] = j[i] >= 0 ? t.bnd[j[i]] : make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < kU; i++) {
            const int q0 = s0 + i * H;
            if (q0 >= most) break;  // warp-uniform
            double tmin = 0.0, tmax = 0.0;
            bool keep = false;
            if (j[i] >= 0) {
                double d;
                exact_terms<T::kNan>(a[i], b[i], tmin, tmax, d);
                const long long db = dbits(d), kd = order_key(db);
                if (kd > km && kd <= kKeyPosInf) {
                    km = kd;
                    p = sub + ((q0 + h) << lg);
                }
                keep = kd > cut || (db & 0x7FF0000000000000LL) == 0x7FF0000000000000LL;
            }
            const int adds = min(H, most - q0);
            for (int q = 0; q < adds; q++) {
                const double lo = __shfl_sync(kFull, tmin, first + q), hi = __shfl_sync(kFull, tmax, first + q);
                acc = dadd(acc, (h & 1) ? hi : lo);
            }
            if (__any_sync(kFull, keep)) collect(xs, cand, keep, base + ((q0 + h) << lg), slot, lane);
        }
    }
    for (int off = 1; off < H; off <<= 1) {
        const long long ok = __shfl_xor_sync(kFull, km, off);
        take_first_max(km, p, ok, __shfl_xor_sync(kFull, p, off));
    }
    for (int off = g >> 1; off > 0; off >>= 1) {
        acc = dadd(acc, __shfl_down_sync(kFull, acc, off << lh));
        const long long ok = __shfl_down_sync(kFull, km, off << lh);
        take_first_max(km, p, ok, __shfl_down_sync(kFull, p, off << lh));
    }
    const int lead = R.in ? lane << (lg + lh) : 0;
    ExactSums s;
    s.minact = __shfl_sync(kFull, acc, lead);
    s.maxact = __shfl_sync(kFull, acc, lead + 1);
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
    const long long ks = order_key(dbits(s)), kt = order_key(dbits(t));
    mn = kt < ks && !nan_bits(dbits(s)) && !nan_bits(dbits(t)) ? t : s;  // t < s ? t : s
    // a row with both slacks >= 0 is feasible
    bad = (dbits(s) < 0 || dbits(t) < 0) && row_infeasible(S.minact, S.maxact, R.minf, R.maxf, R.lhs, R.rhs);
    return row_go_from_max(R.minf, R.maxf, __longlong_as_double(S.km), mn);
}

// Candidates of the rows with go set (lanes that hold rows), from their
// slacks s and u; cand: the collected elements.
template <class T>
__device__ __forceinline__ void exact_candidates(const T &t, ExactSmem &xs, ExactQueue &Q, const ExactRow &R,
                                                 const ExactSums &S, bool go, double s, double u, int cand, int lane,
                                                 int *row_tight = nullptr) {
    if (!__any_sync(kFull, go)) return;
    if (R.in) {
        const bool rhs_ok = !pos_inf<T::kNan>(R.rhs) && !neg_inf<T::kNan>(S.minact);
        const bool lhs_ok = !neg_inf<T::kNan>(R.lhs) && !pos_inf<T::kNan>(S.maxact);
        xs.slack[lane] = s;
        xs.nsur[lane] = u;
        xs.info[lane] = (unsigned char)((rhs_ok ? 1 : 0) | (lhs_ok ? 2 : 0) | min(R.minf, 3) << 2 |
                                        min(R.maxf, 3) << 4 | (go ? 64 : 0) |
                                        (dbits(R.lhs) == (long long)(1ULL << 63) ? 128 : 0));
    }
    __syncwarp();
    if (cand <= kCandCap) {
        for (int i0 = 0; i0 < cand; i0 += 32) {
            const int i = i0 + lane;
            const int slot = i < cand ? xs.cand_s[i] : 0;
            const bool on = i < cand && (xs.info[slot] & 64);
            exact_push(t, xs, Q, on, on ? xs.cand_k[i] : 0, slot, lane, row_tight);
        }
    } else {  // more than the list holds: every element of the rows again
        const FlatRows F = flat_rows(R, lane);
        if (R.in) xs.src[lane] = R.base - F.pre;
        __syncwarp();
        for (int f0 = 0; f0 < F.total; f0 += 32) {
            const int slot = max(flat_slot(F, f0, lane), 0), f = f0 + lane;
            const bool on = f < F.total && (xs.info[slot] & 64);
            exact_push(t, xs, Q, on, on ? xs.src[slot] + f : 0, slot, lane, row_tight);
        }
    }
}

}  // namespace
}  // namespace gdp
