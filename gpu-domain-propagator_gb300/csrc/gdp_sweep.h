// gdp_sweep.h -- the order in which a batch's full sweep claims its work items.
// Device code that the CPU tests compile by itself as plain C++.
#pragma once

#ifdef __CUDACC__
#define GDP_SWEEP_FN __host__ __device__ __noinline__
#else
#define GDP_SWEEP_FN inline
#endif

namespace gdp {
namespace {

// Work item i of the full sweep: every unit's items are ordered heaviest first,
// and one unit after the other would leave the last unit's heavy items to the
// end of the phase. So the claims run through the units kSweepParts times, an
// equal part of each unit's list at a time: part s of unit k holds as many items
// as [prefix[k], prefix[k + 1]) holds numbers = s mod kSweepParts, which makes
// the parts' prefixes functions of the units'. 24 mixed instances of up to 60,000 rows: 12.42 -> 11.53
// ms (of 77 us of screening a round, 29 were the wait for the last items). Not
// inlined: that cost every other batch 2%.
constexpr int kSweepParts = 8;
struct alignas(8) SweepItem {
    int unit, item;  // the unit's place in the sweep's list, its work item
};
GDP_SWEEP_FN SweepItem sweep_item(const int *prefix, int nfs, int total, int i) {
    constexpr int K = kSweepParts;
    const int q = total / K, rem = total % K;
    const int s = i < rem * (q + 1) ? i / (q + 1) : rem + (i - rem * (q + 1)) / q;
    i -= s * q + (s < rem ? s : rem);  // within part s
    auto below = [&](int x) { return (x + K - 1 - s) / K; };                  // numbers under x that are s mod K
    auto before = [&](int x) { return x / K * s + (s < x % K ? s : x % K); };  // ... that are less than s mod K
    int lo = 0, hi = nfs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (below(prefix[mid]) <= i) lo = mid;
        else hi = mid - 1;
    }
    const int p0 = prefix[lo], p1 = prefix[lo + 1];
    return SweepItem{lo, before(p1) - before(p0) + i - below(p0)};
}

}  // namespace
}  // namespace gdp
