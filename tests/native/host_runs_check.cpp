// Checks the host worker runs of the transfers (culs_b200/csrc/host_runs.hpp)
// on the CPU: every graph in one run, an error code of any run reaches the
// caller, a new thread's set-up comes before its run and its failure ends it,
// an exception is rethrown after every thread has been joined, and runs for
// which no thread starts stay on the caller's.  Built and run by
// tests/test_host_runs.py.
#include <atomic>
#include <cstdio>
#include <numeric>
#include <stdexcept>
#include <system_error>

#include "host_runs.hpp"

using namespace culs;

static int g_bad = 0;
#define CHECK(c)                                                \
    do {                                                        \
        if (!(c)) {                                             \
            printf("FAIL %s:%d: %s\n", __FILE__, __LINE__, #c); \
            g_bad++;                                            \
        }                                                       \
    } while (0)

static thread_local int t_device = 0;  // what a new thread finds
static std::atomic<int> g_alive{0};

// a thread of which only so many can be started
struct FewThreads {
    static inline int left = 0;
    std::thread t;
    template <class F, class... A>
    explicit FewThreads(F &&f, A &&...a) {
        if (left-- <= 0) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
        t = std::thread(std::forward<F>(f), std::forward<A>(a)...);
    }
    FewThreads(FewThreads &&) = default;
    void join() { t.join(); }
};

int main() {
    for (int n : {1, 2, 3, 7, 100})
        for (int parts : {1, 2, 5, 200}) {
            const std::vector<int> cut = split_runs(n, parts, [](int g) { return (int64_t)(g % 3 ? 1 : 50); });
            CHECK(cut.front() == 0 && cut.back() == n && (int)cut.size() - 1 <= std::min(n, parts));
            for (size_t i = 1; i < cut.size(); i++) CHECK(cut[i - 1] < cut[i]);
        }
    CHECK(host_threads(0, 1, 10) == 1 && host_threads(1 << 30, 1 << 20, 1) == 1 && host_threads(1 << 30, 1, 1000) <= 32);
    t_device = 3;  // the caller's
    for (int runs : {0, 1, 2, 9}) {
        auto device = [] { return t_device = 3, 0; };
        std::vector<int> seen(runs + 1, 0);
        CHECK(run_parallel(runs, device, [&](int r) { return seen[r] += t_device == 3, 0; }) == 0);
        CHECK(std::accumulate(seen.begin(), seen.end(), 0) == runs);
        // any run's error, the lowest run's first
        for (int bad = 0; bad < runs; bad++) {
            CHECK(run_parallel(runs, device, [&](int r) { return r == bad ? 700 + r : 0; }) == 700 + bad);
            CHECK(run_parallel(runs, device, [&](int r) { return r >= bad ? 700 + r : 0; }) == 700 + bad);
        }
        // a device that cannot be set
        std::atomic<int> ran{0};
        CHECK(run_parallel(runs, [] { return 101; }, [&](int) { return ran++, 0; }) == (runs > 1 ? 101 : 0));
        CHECK(ran == std::min(runs, 1));
        // exceptions wait for the others
        for (int bad = 0; bad < runs; bad++) {
            bool caught = false;
            try {
                run_parallel(runs, device, [&](int r) -> int {
                    g_alive++;
                    if (r == bad) {
                        g_alive--;
                        throw std::runtime_error("run");
                    }
                    std::this_thread::sleep_for(std::chrono::milliseconds(5));
                    g_alive--;
                    return 0;
                });
            } catch (const std::runtime_error &) {
                caught = true;
            }
            CHECK(caught && g_alive == 0);
        }
        // no threads, or too few
        for (int left : {0, 1, 3, 100}) {
            FewThreads::left = left;
            std::vector<int> done(runs + 1, 0);
            const int rc = run_parallel<FewThreads>(runs, device, [&](int r) { return done[r] += t_device == 3, r == 8 ? 9 : 0; });
            CHECK(rc == (runs == 9 ? 9 : 0));
            CHECK(std::accumulate(done.begin(), done.end(), 0) == runs);
        }
    }
    printf("bad %d\n", g_bad);
    return g_bad != 0;
}
