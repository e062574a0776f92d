// gdp_noalloc.cu -- propagation entry point that allocates no memory.
//
// Some callers cannot call cudaMalloc: a branch-and-bound solver or a
// framework whose device memory is owned by its own pool (PyTorch's caching
// allocator, a solver's arena) and that propagates thousands of nodes in a
// loop, where cudaMalloc/cudaFree would synchronize the device and fragment
// the pool. gdp_propagate_noalloc serves them: the caller passes the problem
// and the bounds already in device memory, and the working memory the round
// loop needs (round-start bounds, changed-variable bitmaps, the list of long
// rows, round state) lives in one file-scope device array of fixed size,
// kNoallocMaxVars variables.
//
// That array exists once per GPU that loads this library and stays resident
// until the process exits. Every call shares it and it keeps the last call's
// contents, so each call re-initialises it; two calls that overlap on the GPU
// (different streams or threads at the same time) race on it and must be
// serialized by the caller.
//
// The CSR is checked on the device before any round (row pointers, column
// range, variable types, finite coefficients), so a bad index is reported as
// an error instead of turning into an out-of-range access.
//
// Every row's sums run left to right with the reference's row test (the
// reference's cpu_omp round function, bit for bit), so results equal those of
// the context path for every row up to the context's thread_row_max.
//
// How the rounds run. One cooperative launch runs every round. The caller's
// CSR is used as it is (no layout), so the rows come in any order and of any
// length, and what bounds a round is latency: a row read by one thread costs
// two dependent loads per element, 8 ms a round for a row of 15,000
// non-zeros. So
//   * a warp takes 32 consecutive rows. The elements of the rows of up to 32
//     non-zeros are read as one flat list, 128 at a time, whatever rows they
//     belong to; a longer row is read by the whole warp; a row longer than
//     kLongRow by a whole CTA, before the warps take their rows;
//   * every row is first screened with the FP32 enclosure of gdp_device.cuh,
//     on copies rounded in registers (integer work: conversions would use the
//     FP64 pipe). A row that the screen skips, or none of whose variables
//     changed in the round before, tightens nothing and is feasible;
//   * the rows that are left take the exact pass of gdp_exact.cuh, left to
//     right; the products of a row longer than kLongRow are formed by a whole
//     CTA, and two lanes add them up (71 cycles per element);
//   * after a round with fewer than n / 16 changed variables a row is looked
//     up in the bitmap first and its bounds are read only if a bit is set.
// On 100,000-row power-law MIPs (2.2M non-zeros, rows of up to 20,000, 56 to 73
// rounds, four seeds) a call takes 11 to 22 ms instead of 650 to 830 ms (one
// thread per row, three launches and a synchronisation per round).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <climits>
#include <cstring>
#include <mutex>
#include <string>

#include "gdp_context.h"
#include "gdp_device.cuh"
#include "gdp_round.cuh"

namespace gdp {
namespace {

constexpr int kNoallocMaxVars = 1 << 20;
constexpr int kNoallocWords = kNoallocMaxVars / 32;
// Rows longer than this are read by a whole CTA (a warp takes 8 us for 1,024
// elements, about the time of a chunk of 32 short rows).
constexpr int kLongRow = 1024;
// Capacity of the list of long rows; a problem with more of them (over 67M
// non-zeros) has every row read by a warp.
constexpr unsigned kLongCap = 1 << 16;
constexpr int kNaWarps = 8;
constexpr int kNaThreads = 32 * kNaWarps;

// Round state: flags.* as in the context path; per-round values by parity.
struct NaState {
    RoundFlags flags;
    unsigned barrier[2];
    int bad[4];  // first offending index per input check (INT_MAX: none), see k_noalloc_prepare
    unsigned n_long;
    unsigned claim[2];    // rows claimed in chunks of 32, beyond the first chunk of each warp
    unsigned changed[2];  // variables committed in the round
    int tight[2];         // some row tightened a bound in the round
};

constexpr size_t kStateBytes = 512;
static_assert(sizeof(NaState) <= kStateBytes, "round state fits its reserve");
constexpr size_t kNoallocBytes = sizeof(double2) * (size_t)kNoallocMaxVars +
                                 2 * sizeof(unsigned) * (size_t)kNoallocWords + sizeof(int) * (size_t)kLongCap +
                                 kStateBytes;

// [cur: kNoallocMaxVars bound pairs][two bitmaps][long rows][state]
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocBytes];

struct NoallocView {
    double2 *cur;      // round-start bounds; the caller's arrays receive the round's atomics
    unsigned *chg[2];  // variables changed in the round, by round parity
    int *longs;        // rows longer than kLongRow
    NaState *st;
};

NoallocView view_of(unsigned char *base) {
    NoallocView v;
    v.cur = reinterpret_cast<double2 *>(base);
    v.chg[0] = reinterpret_cast<unsigned *>(v.cur + kNoallocMaxVars);
    v.chg[1] = v.chg[0] + kNoallocWords;
    v.longs = reinterpret_cast<int *>(v.chg[1] + kNoallocWords);
    v.st = reinterpret_cast<NaState *>(v.longs + kLongCap);
    return v;
}

// Device address of the scratch array and the cooperative grid, looked up once
// per device (the host symbol g_noalloc_scratch is only a stand-in for it in
// host code).
std::mutex g_setup_mutex;
unsigned char *g_scratch_addr[64] = {nullptr};
int g_grid[64] = {0};

struct Csr {
    int m, n;
    const int *col, *row_ptr, *vartype;
    const double *val, *lhs, *rhs;
    double *lb, *ub;
};

__global__ void k_noalloc_init(NoallocView S, int words) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    for (int w = tid; w < words; w += nt) {
        S.chg[0][w] = 0u;
        S.chg[1][w] = 0u;
    }
    if (tid == 0) {
        NaState s = {};
        s.flags.infeasible_var = INT_MAX;
        s.flags.infeasible_row = INT_MAX;
        for (int i = 0; i < 4; i++) s.bad[i] = INT_MAX;
        *S.st = s;
    }
}

// Input checks of the device CSR, each reading only in-range entries of the
// arrays it checks: bad[0] the first row i with row_ptr[i + 1] < row_ptr[i]
// (-1: row_ptr[0] != 0 or row_ptr[m] != nnz), bad[1] the first non-zero whose
// column is outside [0, n), bad[2] the first variable whose type is not 0, 1
// or 3, bad[3] the first non-finite coefficient. Beside them the round-start
// bounds, the check of the input bounds and the list of long rows.
__global__ void __launch_bounds__(256) k_noalloc_prepare(Csr A, int nnz, NoallocView S) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    NaState *st = S.st;
    if (tid == 0 && (A.row_ptr[0] != 0 || A.row_ptr[A.m] != nnz)) atomicMin(st->bad + 0, -1);
    for (unsigned i = tid; i < (unsigned)A.m; i += nt) {
        const int b = A.row_ptr[i], e = A.row_ptr[i + 1];
        if (e < b) atomicMin(st->bad + 0, (int)i);
        else if ((long long)e - b > kLongRow) {
            const unsigned at = atomicAdd(&st->n_long, 1u);
            if (at < kLongCap) S.longs[at] = (int)i;
        }
    }
    for (unsigned k = tid; k < (unsigned)nnz; k += nt) {
        const int j = A.col[k];
        if (j < 0 || j >= A.n) atomicMin(st->bad + 1, (int)k);
        if (!isfinite(A.val[k])) atomicMin(st->bad + 3, (int)k);
    }
    for (int j = tid; j < A.n; j += nt) {
        const int t = A.vartype[j];
        if (t != 0 && t != 1 && t != 3) atomicMin(st->bad + 2, j);
        const double2 b = make_double2(A.lb[j], A.ub[j]);
        S.cur[j] = b;
        if (var_infeasible(b.x, b.y)) {
            st->flags.infeasible = 1;
            atomicMin(&st->flags.infeasible_var, j);
        }
    }
}

// ---- FP32 screen copies formed in registers ------------------------------------
// Round-to-nearest float of a double whose magnitude lies in [2^-126, 2^127),
// by integer arithmetic.
__device__ __forceinline__ float f32_rn_bits(long long b) {
    const unsigned long long mag = (unsigned long long)b & 0x7FFFFFFFFFFFFFFFULL;
    const unsigned r = (unsigned)((mag + 0x0FFFFFFFULL + ((mag >> 29) & 1ULL)) >> 29) - (896u << 23);
    return __uint_as_float(r | ((unsigned)((unsigned long long)b >> 32) & 0x80000000u));
}
// coef_screen in integer arithmetic.
__device__ __forceinline__ float coef_screen_bits(double a) {
    const long long b = dbits(a);
    const unsigned long long mag = (unsigned long long)b & 0x7FFFFFFFFFFFFFFFULL;
    const unsigned sign = (unsigned)((unsigned long long)b >> 32) & 0x80000000u;
    if (mag == 0) return __uint_as_float(sign);
    if (b > 0 && b <= kBitsEps) return __uint_as_float(0x7FC00000u);
    if (mag > 0x4270000000000000ULL) return __uint_as_float(sign | 0x7F800000u);   // above 2^40
    if (mag < 0x3C30000000000000ULL) return __uint_as_float(sign | 0x7FC00000u);   // below 2^-60
    return f32_rn_bits(b);
}
// bnd_screen in integer arithmetic; a non-zero bound below 2^-126 in magnitude
// is NaN (its row takes the exact pass).
__device__ __forceinline__ float bound_screen_bits(long long b, bool infinite, float inf) {
    const unsigned long long mag = (unsigned long long)b & 0x7FFFFFFFFFFFFFFFULL;
    if (infinite) return inf;
    if (mag == 0) return 0.0f;
    if (mag > (unsigned long long)kBits2p100 || mag < 0x3810000000000000ULL) return __uint_as_float(0x7FC00000u);
    return f32_rn_bits(b);
}
__device__ __forceinline__ float2 bnd_screen_bits(double2 v) {
    const long long l = dbits(v.x), u = dbits(v.y);
    return make_float2(bound_screen_bits(l, neg_inf<true>(v.x), -kF32Inf),
                       bound_screen_bits(u, pos_inf<true>(v.y), kF32Inf));
}

__device__ __forceinline__ bool bit_of(const unsigned *map, int j) { return (map[j >> 5] >> (j & 31)) & 1u; }

// ---- shared memory of a warp ------------------------------------------------------
// The chunk's screen stages its copies where the exact pass stages its terms.
constexpr int kStage = 64;   // elements the exact pass stages at a time
constexpr int kNaRows = 16;  // rows of an item of the exact pass
struct NaWarp {
    ExactSmem xs;
    double t[2][kStage];  // minimum / maximum activity terms
    double d[kStage];     // |a| (ub - lb)
    int src[32];
    unsigned char own[32];  // lanes of the rows that take the exact pass
    unsigned long long rows, nnz;  // rows that this warp swept and their non-zeros, kept by lane 0
};
constexpr int kScreenStage = 128;  // elements the screen stages at a time
__device__ __forceinline__ float2 *stage_b(NaWarp &ws) { return reinterpret_cast<float2 *>(ws.t[0]); }
__device__ __forceinline__ float *stage_a(NaWarp &ws) { return reinterpret_cast<float *>(ws.d); }
static_assert(sizeof(float2) * kScreenStage <= sizeof(NaWarp::t) && sizeof(float) * kScreenStage <= sizeof(NaWarp::d),
              "the copies fit the staging area");

// A flat list over the chunk's rows: the lanes with `in` set hold rows of `len`
// elements whose first is at CSR index b and at flat index pre; ws.src[rank]
// holds b - pre of the rank-th row of the list.
struct Flat {
    bool in;
    int pre, len, total;
};
__device__ __forceinline__ Flat flat_of(NaWarp &ws, bool in, int b, int len, int lane) {
    Flat F;
    F.in = in && len > 0;
    F.len = F.in ? len : 0;
    int inc = F.len;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(kFull, inc, off);
        if (lane >= off) inc += v;
    }
    F.total = __shfl_sync(kFull, inc, 31);
    F.pre = inc - F.len;
    const unsigned mask = __ballot_sync(kFull, F.in);
    __syncwarp();
    if (F.in) ws.src[__popc(mask & ((1u << lane) - 1u))] = b - F.pre;
    __syncwarp();
    return F;
}
// The rank of the row (among the list's rows) that owns flat element f0 + lane.
__device__ __forceinline__ int flat_rank(const Flat &F, int f0, int lane) {
    const int d = F.pre - f0;
    const unsigned starts = __reduce_or_sync(kFull, (F.in && d >= 0 && d < 32) ? 1u << d : 0u);
    const int before = __popc(__ballot_sync(kFull, F.in && d < 0));
    return before + __popc(starts & (kFull >> (31 - lane))) - 1;
}
// The bits of a 32-element step at f0 that belong to this lane's row.
__device__ __forceinline__ unsigned flat_range(const Flat &F, int f0) {
    const int lo = max(F.pre - f0, 0), hi = min(F.pre + F.len - f0, 32);
    if (!F.in || hi <= lo) return 0u;
    return (kFull >> (32 - (hi - lo))) << lo;
}

constexpr size_t kNaSmem = sizeof(NaWarp) * kNaWarps;

// Elements, bounds and targets of the exact pass: candidates go to the
// caller's arrays.
struct NaTarget {
    static constexpr bool kNan = true;
    const int *col;
    const double *val;
    const double2 *bnd;
    const int *vartype;
    double *lb, *ub;
    unsigned *chg;
    __device__ __forceinline__ bool cont(int j) const { return __ldg(vartype + j) == 3; }
    __device__ __forceinline__ void apply(int j, double v, bool lower) const {
        if (lower) atomic_max_f64(lb + j, v);
        else atomic_min_f64(ub + j, v);
        atomicOr(chg + (j >> 5), 1u << (j & 31));
    }
};

// Left-to-right activities and first maximum of an item of up to kNaRows rows.
// The rows are one flat list of elements, kStage staged at a time: 32 lanes
// form the products of 32 consecutive elements, whichever rows they belong
// to, then lane 2 r adds up row r's minimum activity and lane 2 r + 1 its
// maximum activity, so a long row costs one FP64 add per element.
__device__ __forceinline__ ExactSums flat_sums(const NaTarget &t, NaWarp &ws, const ExactRow &R, int lane, int &cand) {
    ExactSmem &xs = ws.xs;
    const FlatRows F = flat_rows(R, lane);
    __syncwarp();
    if (R.in) xs.src[lane] = R.base - F.pre;
    __syncwarp();
    const int side = lane & 1, mine = lane >> 1;
    const int rpre = __shfl_sync(kFull, F.pre, mine), rlen = __shfl_sync(kFull, F.len, mine);
    const long long my_cut = candidate_cut(R.slack_lo);
    double acc = 0.0;
    long long km = 0;
    int p = -1, e = 0;
    cand = 0;
    constexpr int kSteps = kStage / 32;
    int k[kSteps], slots[kSteps], j[kSteps];
    double a[kSteps];
    auto load = [&](int w0) {  // element indices, columns and coefficients of a window
#pragma unroll
        for (int i = 0; i < kSteps; i++) {
            slots[i] = flat_slot(F, w0 + 32 * i, lane);
            const int f = w0 + 32 * i + lane;
            k[i] = f < F.total ? xs.src[slots[i]] + f : -1;
            j[i] = k[i] >= 0 ? __ldg(t.col + k[i]) : 0;
            a[i] = k[i] >= 0 ? __ldg(t.val + k[i]) : 0.0;
        }
    };
    load(0);
    for (int w0 = 0; w0 < F.total; w0 += kStage) {
        double2 b[kSteps];
#pragma unroll
        for (int i = 0; i < kSteps; i++) b[i] = k[i] >= 0 ? t.bnd[j[i]] : make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < kSteps; i++) {
            if (w0 + 32 * i >= F.total) break;  // warp-uniform
            double d;
            exact_terms<NaTarget::kNan>(a[i], b[i], ws.t[0][32 * i + lane], ws.t[1][32 * i + lane], d);
            ws.d[32 * i + lane] = d;
            const long long db = dbits(d);
            const long long cut = __shfl_sync(kFull, my_cut, max(slots[i], 0));
            const bool keep = k[i] >= 0 && (order_key(db) > cut ||
                                            (db & 0x7FF0000000000000LL) == 0x7FF0000000000000LL);
            collect(xs, cand, keep, k[i], slots[i], lane);
        }
        if (w0 + kStage < F.total) load(w0 + kStage);  // in flight while this window is added up
        __syncwarp();
        const int end = min(rlen, w0 + kStage - rpre);  // elements of my row staged so far
        const int at = rpre - w0;  // staged index of my row's element 0
#pragma unroll 4
        for (; e < end; e++) {
            acc = dadd(acc, ws.t[side][at + e]);
            const long long kd = order_key(dbits(ws.d[at + e]));
            if (kd > km && kd <= kKeyPosInf) {
                km = kd;
                p = e;
            }
        }
        __syncwarp();
    }
    ExactSums s;
    const int lead = R.in ? 2 * lane : 0;
    s.minact = __shfl_sync(kFull, acc, lead);
    s.maxact = __shfl_sync(kFull, acc, lead + 1);
    s.km = __shfl_sync(kFull, km, lead);
    s.p = __shfl_sync(kFull, p, lead);
    return s;
}

// The exact pass of the rows of `rows` (lanes; each holds its row's CSR start
// b, length and the screen's results), kNaRows at a time.
__device__ __forceinline__ void exact_rows(const Csr &A, const NoallocView &S, const NaTarget &T, NaWarp &ws,
                                           ExactQueue &Q, unsigned rows, int row0, int b, int len, float slack_lo,
                                           int minf, int maxf, int lane) {
    const int n = __popc(rows);
    __syncwarp();
    if ((rows >> lane) & 1u) ws.own[__popc(rows & ((1u << lane) - 1u))] = (unsigned char)lane;
    __syncwarp();
    for (int i0 = 0; i0 < n; i0 += kNaRows) {
        ExactRow R;
        R.in = lane < kNaRows && i0 + lane < n;
        const int own = R.in ? ws.own[i0 + lane] : 0;
        R.base = __shfl_sync(kFull, b, own);
        R.len = __shfl_sync(kFull, len, own);
        R.slack_lo = __shfl_sync(kFull, slack_lo, own);
        R.minf = __shfl_sync(kFull, minf, own);
        R.maxf = __shfl_sync(kFull, maxf, own);
        R.lhs = R.in ? __ldg(A.lhs + row0 + own) : 0.0;
        R.rhs = R.in ? __ldg(A.rhs + row0 + own) : 0.0;
        int cand;
        const ExactSums X = flat_sums(T, ws, R, lane, cand);
        double s = 0.0, t = 0.0, mn = 0.0;
        int dec = 0;
        if (R.in) {
            bool bad;
            dec = exact_decide(R, X, s, t, mn, bad);
            if (bad) atomicMin(&S.st->flags.infeasible_row, row0 + own);
        }
        for (unsigned amb = __ballot_sync(kFull, dec == 2); amb; amb &= amb - 1) {
            const int q = __ffs(amb) - 1;
            const int qb = __shfl_sync(kFull, R.base, q), ql = __shfl_sync(kFull, R.len, q);
            const double m = seq_eps_max(T.bnd, A.col + qb, A.val + qb, ql, __shfl_sync(kFull, X.km, q),
                                         __shfl_sync(kFull, X.p, q), lane);
            if (lane == q) dec = eps_le(m, mn) ? 0 : 1;
        }
        exact_candidates(T, ws.xs, Q, R, X, R.in && dec == 1, s, t, cand, lane);
    }
}

// FP32 screen of the elements first, first + step, ... of the row of len
// elements at CSR index b (step: a warp's lanes or a CTA's threads), four
// loads of each kind in flight. Offsets are unsigned: no overflow below 2^32.
__device__ __forceinline__ void screen_strided(const Csr &A, const NoallocView &S, const unsigned *prev, int b, int len,
                                               int first, int step, Scr &c, int &hit) {
    for (unsigned o = first; o < (unsigned)len; o += 4 * step) {
        int j[4];
        double a[4];
        double2 bb[4];
        bool ok[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            ok[i] = o + i * step < (unsigned)len;
            j[i] = ok[i] ? __ldg(A.col + b + (o + i * step)) : 0;
            a[i] = ok[i] ? __ldg(A.val + b + (o + i * step)) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            bb[i] = ok[i] ? S.cur[j[i]] : make_double2(0.0, 0.0);
            if (ok[i] && bit_of(prev, j[i])) hit = 1;
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (ok[i]) scr_add(c, coef_screen_bits(a[i]), bnd_screen_bits(bb[i]));
    }
}
// Whether a variable of the elements changed in the round before.
__device__ __forceinline__ int hit_strided(const Csr &A, const unsigned *prev, int b, int len, int first, int step) {
    int hit = 0;
#pragma unroll 4
    for (unsigned o = first; o < (unsigned)len; o += step) hit |= bit_of(prev, __ldg(A.col + b + o)) ? 1 : 0;
    return hit;
}

// ---- a chunk of 32 rows, one warp -----------------------------------------------------
__device__ __forceinline__ void na_chunk(const Csr &A, const NoallocView &S, const NaTarget &T, const unsigned *prev,
                                         NaWarp &ws, ExactQueue &Q, int row0, int round, bool sparse, int long_len,
                                         int lane) {
    int b = 0, len = 0;
    if (lane < A.m - row0) {
        b = __ldg(A.row_ptr + row0 + lane);
        len = __ldg(A.row_ptr + row0 + lane + 1) - b;
    }
    bool small = len >= 1 && len <= 32;
    if (sparse) {  // keep the short rows with a changed variable
        const Flat F = flat_of(ws, small, b, len, lane);
        unsigned any = 0u;
#pragma unroll 4
        for (int f0 = 0; f0 < F.total; f0 += 32) {
            const int rank = flat_rank(F, f0, lane);
            const bool ok = f0 + lane < F.total;
            const bool hit = ok && bit_of(prev, __ldg(A.col + ws.src[rank] + f0 + lane));
            any |= __ballot_sync(kFull, hit) & flat_range(F, f0);
        }
        small = any != 0u;
    }
    Scr c;
    scr_init(c);
    unsigned hits = 0u;
    const Flat F = flat_of(ws, small, b, len, lane);
    for (int w0 = 0; w0 < F.total; w0 += kScreenStage) {
        int j[kScreenStage / 32];
        double a[kScreenStage / 32];
        double2 bb[kScreenStage / 32];
        bool ok[kScreenStage / 32], hit[kScreenStage / 32];
#pragma unroll
        for (int i = 0; i < kScreenStage / 32; i++) {
            const int f0 = w0 + 32 * i;
            const int rank = flat_rank(F, f0, lane);
            ok[i] = f0 + lane < F.total;
            const int k = ok[i] ? ws.src[rank] + f0 + lane : 0;
            j[i] = ok[i] ? __ldg(A.col + k) : 0;
            a[i] = ok[i] ? __ldg(A.val + k) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < kScreenStage / 32; i++) {
            bb[i] = ok[i] ? S.cur[j[i]] : make_double2(0.0, 0.0);
            hit[i] = ok[i] && bit_of(prev, j[i]);
        }
#pragma unroll
        for (int i = 0; i < kScreenStage / 32; i++) {
            hits |= __ballot_sync(kFull, hit[i]) & flat_range(F, w0 + 32 * i);
            stage_a(ws)[32 * i + lane] = coef_screen_bits(a[i]);
            stage_b(ws)[32 * i + lane] = bnd_screen_bits(bb[i]);
        }
        __syncwarp();
        const int lo = max(F.pre - w0, 0), hi = F.in ? min(F.pre + F.len - w0, kScreenStage) : 0;
        for (int i = lo; i < hi; i++) scr_add(c, stage_a(ws)[i], stage_b(ws)[i]);
        __syncwarp();
    }
    // the chunk's longer rows, one after another by the whole warp
    bool mid = len > 32 && len <= long_len;
    for (unsigned rem = __ballot_sync(kFull, mid); rem; rem &= rem - 1) {
        const int src = __ffs(rem) - 1;
        const int rb = __shfl_sync(kFull, b, src), rn = __shfl_sync(kFull, len, src);
        if (sparse && !__any_sync(kFull, hit_strided(A, prev, rb, rn, lane, 32))) {
            if (lane == src) mid = false;
            continue;
        }
        Scr r;
        scr_init(r);
        int hit = 0;
        screen_strided(A, S, prev, rb, rn, lane, 32, r, hit);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            Scr o;
            o.mn = __shfl_xor_sync(kFull, r.mn, off);
            o.mx = __shfl_xor_sync(kFull, r.mx, off);
            o.S = __shfl_xor_sync(kFull, r.S, off);
            o.U = __shfl_xor_sync(kFull, r.U, off);
            o.minf = __shfl_xor_sync(kFull, r.minf, off);
            o.maxf = __shfl_xor_sync(kFull, r.maxf, off);
            scr_combine(r, o);
        }
        hit = __any_sync(kFull, hit);
        if (lane == src) {
            c = r;
            hits = hit ? 1u : 0u;
        }
    }
    const unsigned swept = __ballot_sync(kFull, small || mid);
    const int swept_nnz = __reduce_add_sync(kFull, small || mid ? len : 0);
    if (lane == 0) {
        ws.rows += (unsigned)__popc(swept);
        ws.nnz += (unsigned)swept_nnz;
    }
    // round 1 takes every row; later a row without a changed variable was last
    // processed with these bounds and finds nothing
    bool exact = false;
    float slack_lo = 0.0f, hi;
    if ((small || mid) && (hits != 0u || round == 1)) {
        const double lhs = __ldg(A.lhs + row0 + lane), rhs = __ldg(A.rhs + row0 + lane);
        exact = !scr_skips(c, len, lhs, rhs);
        if (exact) scr_slack(c, len, lhs, rhs, slack_lo, hi);
    }
    const unsigned rows = __ballot_sync(kFull, exact);
    if (rows) exact_rows(A, S, T, ws, Q, rows, row0, b, len, slack_lo, c.minf, c.maxf, lane);
}

// ---- a long row, one CTA ----------------------------------------------------------------
struct NaBlock {
    Scr part[kNaWarps];
    long long km[kNaWarps];
    int p[kNaWarps];
    int hit[kNaWarps];
    int decision;
    ExactSums sums;
    double s, t;
};
__device__ __forceinline__ void na_long_row(const Csr &A, const NoallocView &S, const NaTarget &T,
                                            const unsigned *prev, NaWarp *wss, NaBlock &bs, ExactQueue &Q, int row,
                                            int round, bool sparse, int lane) {
    const int wid = threadIdx.x >> 5;
    const int b = __ldg(A.row_ptr + row);
    const unsigned len = (unsigned)(__ldg(A.row_ptr + row + 1) - b);
    if (sparse && !__syncthreads_or(hit_strided(A, prev, b, len, threadIdx.x, kNaThreads))) return;
    if (threadIdx.x == 0) {
        wss[0].rows += 1;
        wss[0].nnz += len;
    }
    Scr c;
    scr_init(c);
    int hit = 0;
    screen_strided(A, S, prev, b, len, threadIdx.x, kNaThreads, c, hit);
    scr_shfl_reduce(c);
    hit = __any_sync(kFull, hit);
    if (lane == 0) {
        bs.part[wid] = c;
        bs.hit[wid] = hit;
    }
    __syncthreads();
    ExactRow R;  // the row, in every thread (thread 0 decides)
    R.in = threadIdx.x == 0;
    R.base = b;
    R.len = (int)len;
    R.lhs = __ldg(A.lhs + row);
    R.rhs = __ldg(A.rhs + row);
    Scr r = bs.part[0];
    hit = bs.hit[0];
    for (int w = 1; w < kNaWarps; w++) {
        scr_combine(r, bs.part[w]);
        hit |= bs.hit[w];
    }
    R.minf = r.minf;
    R.maxf = r.maxf;
    if (!((hit || round == 1) && !scr_skips(r, (int)len, R.lhs, R.rhs))) {  // the same for every thread
        __syncthreads();
        return;
    }
    // products by every warp, kStage elements each; then one lane per side adds
    // them up in order, the first maximum of |a| (ub - lb) beside them
    double acc = 0.0;
    long long km = 0;
    int p = -1;
    for (unsigned w0 = 0; w0 < len; w0 += kNaWarps * kStage) {
        const unsigned base = w0 + wid * kStage;
        int j[kStage / 32];
        double a[kStage / 32];
        double2 bb[kStage / 32];
#pragma unroll
        for (int i = 0; i < kStage / 32; i++) {
            const unsigned o = base + 32 * i + lane;
            j[i] = o < len ? __ldg(A.col + b + o) : -1;
            a[i] = o < len ? __ldg(A.val + b + o) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < kStage / 32; i++) bb[i] = j[i] >= 0 ? T.bnd[j[i]] : make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < kStage / 32; i++)
            if (j[i] >= 0) {
                double d;
                exact_terms<NaTarget::kNan>(a[i], bb[i], wss[wid].t[0][32 * i + lane], wss[wid].t[1][32 * i + lane], d);
                const long long kd = order_key(dbits(d));
                if (kd > km && kd <= kKeyPosInf) {
                    km = kd;
                    p = (int)(base + 32 * i + lane);
                }
            }
        __syncthreads();
        if (threadIdx.x < 2)
            for (int w = 0; w < kNaWarps && w0 + w * kStage < len; w++) {
                const int n = (int)min(len - w0 - w * kStage, (unsigned)kStage);
#pragma unroll 8
                for (int i = 0; i < n; i++) acc = dadd(acc, wss[w].t[lane][i]);
            }
        __syncthreads();
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const long long ok = __shfl_xor_sync(kFull, km, off);
        const int op = __shfl_xor_sync(kFull, p, off);
        if (ok > km || (ok == km && op < p)) {
            km = ok;
            p = op;
        }
    }
    if (lane == 0) {
        bs.km[wid] = km;
        bs.p[wid] = p;
    }
    __syncthreads();
    if (wid == 0) {
        ExactSums X;
        X.minact = __shfl_sync(kFull, acc, 0);
        X.maxact = __shfl_sync(kFull, acc, 1);
        X.km = bs.km[0];
        X.p = bs.p[0];
        for (int w = 1; w < kNaWarps; w++)
            if (bs.km[w] > X.km || (bs.km[w] == X.km && bs.p[w] < X.p)) {
                X.km = bs.km[w];
                X.p = bs.p[w];
            }
        double s, t, mn;
        bool bad;
        int dec = exact_decide(R, X, s, t, mn, bad);
        if (dec == 2)
            dec = eps_le(seq_eps_max(T.bnd, A.col + b, A.val + b, (int)len, X.km, X.p, lane), mn) ? 0 : 1;
        if (lane == 0) {
            if (bad) atomicMin(&S.st->flags.infeasible_row, row);
            bs.decision = dec;
            bs.sums = X;
            bs.s = s;
            bs.t = t;
        }
    }
    __syncthreads();
    if (bs.decision == 1) {
        // the row in slot 0 of every warp; each warp tests its share of the elements
        ExactSmem &xs = wss[wid].xs;
        R.in = lane == 0;
        exact_candidates(T, xs, Q, R, bs.sums, lane == 0, bs.s, bs.t, 0, lane);  // the row's constants alone
        for (unsigned o0 = 32 * wid; o0 < len; o0 += kNaThreads) {
            const unsigned o = o0 + lane;
            exact_push(T, xs, Q, o < len, o < len ? (int)(b + o) : 0, 0, lane, nullptr);
        }
    }
    __syncthreads();  // bs and the staging areas are free for the next row
}

// ---- every round in one cooperative launch ------------------------------------------------
// Warps are numbered across the CTAs, so that consecutive chunks go to
// different SMs; each starts with the chunk of its number and claims further
// ones from a counter. Two CTAs per SM hold the 128 registers without a spill:
// 13.0 ms against 14.6 ms at three (100,000 power-law rows), 1.95 against
// 2.43 ms on 300,000 rows of 2 to 16.
__global__ void __launch_bounds__(kNaThreads, 2) k_noalloc_rounds(Csr A, NoallocView S, int words, int max_rounds) {
    extern __shared__ __align__(16) unsigned char na_smem[];  // kNaWarps NaWarp
    __shared__ NaBlock bs;
    NaWarp *wss = reinterpret_cast<NaWarp *>(na_smem);
    NaState *st = S.st;
    if (st->bad[0] != INT_MAX || st->bad[1] != INT_MAX || st->bad[2] != INT_MAX || st->bad[3] != INT_MAX ||
        st->flags.infeasible)
        return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    NaWarp &ws = wss[wid];
    const int warp = wid * gridDim.x + blockIdx.x, nwarps = gridDim.x * kNaWarps;
    const int chunks = (A.m - 1) / 32 + 1;
    const int n_long = st->n_long <= kLongCap ? (int)st->n_long : 0;
    const int long_len = n_long == (int)st->n_long ? kLongRow : INT_MAX;
    int last_tight = 0;
    unsigned target = 0;  // grid barrier
    if (lane == 0) ws.rows = ws.nnz = 0;
    for (int round = 1; round <= max_rounds; round++) {
        const int par = round & 1;
        const unsigned *prev = S.chg[par ^ 1];
        unsigned *chg = S.chg[par];
        const bool sparse = round > 1 && *((volatile unsigned *)&st->changed[par ^ 1]) < (unsigned)max(1, A.n / 16);
        const NaTarget T{A.col, A.val, S.cur, A.vartype, A.lb, A.ub, chg};
        ExactQueue Q{0, 0, 0};
        for (int l = blockIdx.x; l < n_long; l += gridDim.x)
            na_long_row(A, S, T, prev, wss, bs, Q, S.longs[l], round, sparse, lane);
        for (int ch = warp; ch < chunks;) {
            na_chunk(A, S, T, prev, ws, Q, 32 * ch, round, sparse, long_len, lane);
            if (nwarps >= chunks) break;
            unsigned next = 0;
            if (lane == 0) next = atomicAdd(&st->claim[par], 1u);
            ch = nwarps + (int)__shfl_sync(kFull, next, 0);
        }
        exact_drain(T, ws.xs, Q, true, lane);
        if (__any_sync(kFull, Q.tight) && lane == 0) st->tight[par] = 1;
        if (!grid_barrier(st->barrier, &st->flags.error, kLongSpinLimit, target)) return;
        // commit: the caller's arrays hold the round's result
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            st->claim[par ^ 1] = 0u;
            st->changed[par ^ 1] = 0u;
            st->tight[par ^ 1] = 0;
            st->flags.rounds = round;
            if (*((volatile int *)&st->flags.infeasible_row) != INT_MAX) st->flags.infeasible = 1;
        }
        int changed = 0;
        for (int w = warp; w < words; w += nwarps) {
            const unsigned bits = __ldcg(chg + w);
            if (lane == 0 && __ldcg(prev + w)) S.chg[par ^ 1][w] = 0u;
            if (!bits) continue;
            changed += __popc(bits);
            if ((bits >> lane) & 1u) {
                const int j = 32 * w + lane;
                const double2 v = make_double2(__ldcg(A.lb + j), __ldcg(A.ub + j));
                S.cur[j] = v;
                if (var_infeasible(v.x, v.y)) {
                    st->flags.infeasible = 1;
                    atomicMin(&st->flags.infeasible_var, j);
                }
            }
        }
        if (lane == 0 && changed) {
            atomicAdd(&st->changed[par], (unsigned)changed);
            atomicAdd(&st->flags.changed_vars, (unsigned long long)changed);
        }
        if (!grid_barrier(st->barrier, &st->flags.error, kLongSpinLimit, target)) return;
        last_tight = *((volatile int *)&st->tight[par]);
        if (!last_tight || *((volatile int *)&st->flags.infeasible)) break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) st->flags.change = last_tight;
    if (lane == 0 && ws.rows) {
        atomicAdd(&st->flags.rows_proc, ws.rows);
        atomicAdd(&st->flags.nnz_proc, ws.nnz);
    }
}

#define NA_CUDA(expr)                                                                   \
    do {                                                                                \
        cudaError_t e_ = (expr);                                                        \
        if (e_ != cudaSuccess) {                                                        \
            set_error(std::string(#expr) + " failed: " + cudaGetErrorString(e_));       \
            return GDP_ERROR;                                                           \
        }                                                                               \
    } while (0)

GDP_RETCODE setup_for_current_device(unsigned char **out, int *grid) {
    int dev = 0;
    NA_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) { set_error("device ordinal out of range"); return GDP_ERROR; }
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_scratch_addr[dev]) {
        void *p = nullptr;
        int bps = 0, sms = 0;
        NA_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        NA_CUDA(cudaFuncSetAttribute(k_noalloc_rounds, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNaSmem));
        NA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_noalloc_rounds, kNaThreads, kNaSmem));
        NA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        g_grid[dev] = std::max(1, bps) * sms;
        g_scratch_addr[dev] = static_cast<unsigned char *>(p);
    }
    *out = g_scratch_addr[dev];
    *grid = g_grid[dev];
    return GDP_OKAY;
}

}  // namespace

GDP_RETCODE propagate_noalloc(int m, int n, int nnz, const int *d_col, const int *d_row_ptr,
                              const double *d_val, const double *d_lhs, const double *d_rhs,
                              double *d_lb, double *d_ub, const int *d_vartype, int max_rounds,
                              cudaStream_t s, gdp_stats *st) {
    const auto t0 = std::chrono::steady_clock::now();
    if (st) *st = gdp_stats{};
    if (m < 0 || n < 0 || nnz < 0) { set_error("negative problem size"); return GDP_ERROR; }
    if (n > kNoallocMaxVars) {
        set_error("gdp_propagate_noalloc supports at most " + std::to_string(kNoallocMaxVars) +
                  " variables (its fixed device scratch); got " + std::to_string(n));
        return GDP_ERROR;
    }
    if (m == 0 || n == 0 || nnz == 0) {
        if (st) { st->converged = 1; st->infeasible_var = -1; st->infeasible_row = -1; }
        return GDP_OKAY;
    }
    if (!d_col || !d_row_ptr || !d_val || !d_lhs || !d_rhs || !d_lb || !d_ub || !d_vartype) {
        set_error("null device pointer");
        return GDP_ERROR;
    }
    if (max_rounds <= 0) max_rounds = GDP_MAX_NUM_ROUNDS;
    unsigned char *base = nullptr;
    int grid = 0;
    if (setup_for_current_device(&base, &grid) != GDP_OKAY) return GDP_ERROR;
    NoallocView S = view_of(base);
    Csr A{m, n, d_col, d_row_ptr, d_vartype, d_val, d_lhs, d_rhs, d_lb, d_ub};
    int words = (n + 31) / 32;
    // the input checks run before the rounds, which start only if they passed:
    // nothing indexes with the caller's CSR until then
    k_noalloc_init<<<std::min((words + 255) / 256, 64), 256, 0, s>>>(S, words);
    NA_CUDA(cudaGetLastError());
    const int big = std::max(std::max(m, n), nnz);
    k_noalloc_prepare<<<std::min((big - 1) / 256 + 1, 2048), 256, 0, s>>>(A, nnz, S);
    NA_CUDA(cudaGetLastError());
    // few CTAs for few rows: one warp per chunk of 32 rows, a CTA per 1,024
    // variables to commit, a CTA per kLongRow non-zeros that may be long rows
    const int want = std::max(std::max((m - 1) / (32 * kNaWarps) + 1, (n + 1023) / 1024),
                              (nnz - 1) / kLongRow + 1);
    grid = std::max(1, std::min(grid, want));
    void *args[] = {&A, &S, &words, &max_rounds};
    NA_CUDA(cudaLaunchCooperativeKernel((const void *)k_noalloc_rounds, dim3(grid), dim3(kNaThreads), args, kNaSmem, s));
    NaState h;
    NA_CUDA(cudaMemcpyAsync(&h, S.st, sizeof(h), cudaMemcpyDeviceToHost, s));
    NA_CUDA(cudaStreamSynchronize(s));
    const int *bad = h.bad;
    if (bad[0] != INT_MAX) {
        set_error(bad[0] < 0 ? std::string("csr_row_ptrs must start at 0 and end at nnz")
                             : "csr_row_ptrs is not monotone (row " + std::to_string(bad[0]) + ")");
        return GDP_ERROR;
    }
    if (bad[1] != INT_MAX) {
        set_error("column index out of range at non-zero " + std::to_string(bad[1]));
        return GDP_ERROR;
    }
    if (bad[2] != INT_MAX) {
        set_error("vartype must be 0, 1 or 3 (variable " + std::to_string(bad[2]) + ")");
        return GDP_ERROR;
    }
    if (bad[3] != INT_MAX) {
        set_error("non-finite coefficient at non-zero " + std::to_string(bad[3]));
        return GDP_ERROR;
    }
    const RoundFlags &f = h.flags;
    if (f.error != kErrNone) {
        set_error("device error " + std::to_string(f.error) + " (grid barrier wait exceeded its limit)");
        if (st) st->device_error = f.error;
        return GDP_ERROR;
    }
    if (st) {
        st->rounds = f.rounds;
        st->infeasible = f.infeasible;
        st->infeasible_var = (f.infeasible && f.infeasible_var != INT_MAX) ? f.infeasible_var : -1;
        st->infeasible_row = (f.infeasible && f.infeasible_row != INT_MAX) ? f.infeasible_row : -1;
        st->converged = (f.infeasible || !f.change) ? 1 : 0;
        st->kernel_launches = 3;
        st->changed_vars = f.changed_vars;
        st->rows_processed = (long long)f.rows_proc;
        st->nnz_processed = (long long)f.nnz_proc;
        st->bytes_algorithmic = 12.0 * (double)f.nnz_proc + 20.0 * (double)f.rows_proc + 36.0 * n * (double)f.rounds;
        st->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
    return GDP_OKAY;
}

}  // namespace gdp

#pragma GCC visibility push(default)
extern "C" GDP_RETCODE gdp_propagate_noalloc(int n_cons, int n_vars, int nnz, const int *d_csr_col_indices,
                                             const int *d_csr_row_ptrs, const double *d_csr_vals,
                                             const double *d_lhss, const double *d_rhss, double *d_lbs,
                                             double *d_ubs, const int *d_vartypes, int max_rounds,
                                             void *stream, gdp_stats *stats) {
    return gdp::guarded([&]() -> GDP_RETCODE {
        return gdp::propagate_noalloc(n_cons, n_vars, nnz, d_csr_col_indices, d_csr_row_ptrs, d_csr_vals,
                                      d_lhss, d_rhss, d_lbs, d_ubs, d_vartypes, max_rounds,
                                      static_cast<cudaStream_t>(stream), stats);
    });
}
#pragma GCC visibility pop
