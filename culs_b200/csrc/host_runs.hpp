// Host work on contiguous runs of a batch's graphs, one thread a run.
#pragma once
#include <algorithm>
#include <cstdint>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace culs {

// Threads worth using for n graphs of `total` weight in all, `grain` being the
// weight that is worth one (starting one costs about 15 us).
inline int host_threads(int64_t total, int64_t grain, int n) {
    const unsigned hw = std::thread::hardware_concurrency();
    return (int)std::max<int64_t>(1, std::min({(int64_t)(hw ? hw : 1u), (int64_t)32, (int64_t)n, total / grain}));
}

// Graphs [0, n) in at most `parts` contiguous runs of about equal weight:
// the runs' starts and the end.
template <class W>
std::vector<int> split_runs(int n, int parts, W weight) {
    int64_t total = 0, acc = 0;
    for (int g = 0; g < n; g++) total += weight(g);
    std::vector<int> cut{0};
    for (int g = 0; g < n; g++) {
        acc += weight(g);
        if ((int)cut.size() < parts && acc * parts >= total * (int64_t)cut.size() && g + 1 < n) cut.push_back(g + 1);
    }
    cut.push_back(n);
    return cut;
}

// Calls fn(run) for every run: run 0 on the caller's thread, and so the runs
// for which no thread can be started; every other run on a new thread, where
// begin() comes first (it sets the current CUDA device, which a new thread
// does not inherit).  Both return an error code, 0 for none, and begin's ends
// its run.  Once every thread has been joined, the lowest failed run's code is
// returned, or an exception of any run is rethrown.
template <class Thread = std::thread, class Begin, class F>
int run_parallel(int runs, Begin begin, F fn) {
    std::exception_ptr err;
    std::mutex mu;
    std::vector<int> code((size_t)std::max(runs, 1), 0);
    auto call = [&](int r, bool fresh) {
        try {
            if (fresh) code[r] = begin();
            if (!code[r]) code[r] = fn(r);
        } catch (...) {
            std::lock_guard<std::mutex> lk(mu);
            if (!err) err = std::current_exception();
        }
    };
    std::vector<Thread> th;
    th.reserve((size_t)std::max(runs, 1));
    int started = 1;
    try {
        for (; started < runs; started++) th.emplace_back(call, started, true);
    } catch (...) {  // no more threads: the rest of the runs stay here
    }
    if (runs > 0) call(0, false);
    for (int r = started; r < runs; r++) call(r, false);
    for (auto &t : th) t.join();
    if (err) std::rethrow_exception(err);
    for (int c : code)
        if (c) return c;
    return 0;
}

}  // namespace culs
