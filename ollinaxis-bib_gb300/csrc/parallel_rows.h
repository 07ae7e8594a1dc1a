// Rows of a host array, shared out among host threads.
#pragma once
#include <algorithm>
#include <cstddef>
#include <thread>
#include <vector>

namespace ollin {

// f(j) for the rows lo <= j < hi, on several host threads where there are
// points enough (the initial data take about 50 ns a point in exp, log and
// pow).  Rows are independent, so the values do not depend on the threads.  f
// does not throw.
template <typename F>
void parallel_rows(int lo, int hi, std::size_t points, const F& f) {
    const std::size_t most = std::min<std::size_t>(16, std::max(1u, std::thread::hardware_concurrency()));
    const int n = (int)std::min<std::size_t>(most, points / 32768 + 1);
    auto part = [&](int k) {
        for (int j = lo + (int)((long)(hi - lo) * k / n); j < lo + (int)((long)(hi - lo) * (k + 1) / n); ++j) f(j);
    };
    std::vector<std::thread> threads;
    int k = 1;
    try {
        threads.reserve(n);
        for (; k < n; ++k) threads.emplace_back(part, k);
    } catch (...) {
        // no more threads, or no memory for them, to be had: the rest of the
        // rows here.  (Anything thrown past the threads already running would
        // end the process.)
    }
    part(0);
    for (; k < n; ++k) part(k);
    for (std::thread& t : threads) t.join();
}

}  // namespace ollin
