// Check of the host thread pool (loki_b200/csrc/lk_host.hpp): every item once,
// and an exception of any item rethrown to the caller instead of ending the
// process; and the number of threads the table builders' work gets. Prints "ok" or the first failure.
#include <cstdio>
#include <new>
#include <stdexcept>
#include <string>

#include "lk_host.hpp"

int main() {
    for (const uint64_t n : {0ull, 1ull, 7ull, 1000ull}) {
        std::vector<std::atomic<int>> seen(n);
        lk::parallel_for<int>(n, 1 << 20, [&](uint64_t i, int&) { ++seen[i]; });
        for (const auto& s : seen) {
            if (s != 1) {
                std::printf("an item ran %d times of %llu items\n", s.load(), static_cast<unsigned long long>(n));
                return 1;
            }
        }
    }
    for (const uint64_t bad : {0ull, 3ull, 999ull}) {
        bool caught = false;
        try {
            lk::parallel_for<int>(1000, 1 << 20, [&](uint64_t i, int&) {
                if (i == bad) {
                    throw std::bad_alloc();
                }
            });
        } catch (const std::bad_alloc&) {
            caught = true;
        }
        if (!caught) {
            std::printf("item %llu: exception lost\n", static_cast<unsigned long long>(bad));
            return 1;
        }
    }
    // 400 frequencies of 1,024 samples at a bin a sample: every sample is
    // evaluated, which is work for all the threads there are (up to 8 here)
    const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
    const uint64_t each = lk::fold_run_evaluations({0.5, 10.0}, 1e-3, 100, 1024);
    if (each != 1024 || lk::host_threads(400, each) < std::min(cores, 8u)) {
        std::printf("%u threads for 400 x %llu evaluations\n", lk::host_threads(400, each),
                    static_cast<unsigned long long>(each));
        return 1;
    }
    std::printf("ok\n");
    return 0;
}
