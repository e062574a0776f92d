// gdp_pages.h -- host pages that the GPU is about to write. Plain C++: the CPU
// tests compile it by itself.
#pragma once

#include <cstddef>

namespace gdp {

constexpr size_t kPageBytes = 4096;

// Touches every page of [p, p + bytes), `threads` host threads at most: the GPU's
// first write to a page that nothing has touched yet is a fault of many
// microseconds. The bytes keep their values, so a call that fails afterwards
// leaves the array as it was. bytes > 0.
inline void touch_pages(void *p, size_t bytes, int threads) {
    char *c = static_cast<char *>(p);
    // one write access that changes nothing; storing zeros took the same time (1M
    // logits into a new array: 0.43 ms either way)
    auto touch = [&](size_t at) { __atomic_fetch_or(c + at, (char)0, __ATOMIC_RELAXED); };
    const long long pages = (long long)((bytes + kPageBytes - 1) / kPageBytes);
#pragma omp parallel for schedule(static) num_threads(threads) if (threads > 1)
    for (long long i = 0; i < pages; i++) touch(kPageBytes * (size_t)i);
    touch(bytes - 1);  // an array that does not start on a page has one more
}

}  // namespace gdp
