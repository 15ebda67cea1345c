// Check of the host thread pool (loki_b200/csrc/lk_host.hpp): every item once,
// and an exception of any item rethrown to the caller instead of ending the
// process. Prints "ok" or the first failure.
#include <cstdio>
#include <new>
#include <stdexcept>
#include <string>

#include "lk_host.hpp"

int main() {
    for (const uint64_t n : {0ull, 1ull, 7ull, 1000ull}) {
        std::vector<std::atomic<int>> seen(n);
        lk::parallel_for(n, 1 << 20, [&](uint64_t i) { ++seen[i]; });
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
            lk::parallel_for(1000, 1 << 20, [&](uint64_t i) {
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
    std::printf("ok\n");
    return 0;
}
