// Host thread pool of the plan-time table builders (no device code).
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace lk {

// Host threads for n items of `each` units of work: about one per 2^16 units,
// at most 32.
inline unsigned host_threads(uint64_t n, uint64_t each) {
    const uint64_t want = n * (each + 1) / 65536 + 1;
    return static_cast<unsigned>(
        std::min<uint64_t>({want, std::max<uint64_t>(n, 1), 32, std::max(1u, std::thread::hardware_concurrency())}));
}

// fn(i) for i < n on host threads. The first exception of any fn ends the loop
// and is rethrown here; threads that cannot be started leave their share to
// the others.
template <class F>
void parallel_for(uint64_t n, uint64_t each, F&& fn) {
    const unsigned nthreads = host_threads(n, each);
    std::atomic<uint64_t> next{0};
    std::exception_ptr error;
    std::mutex error_lock;
    auto work = [&] {
        try {
            for (uint64_t i = next++; i < n; i = next++) {
                fn(i);
            }
        } catch (...) {
            next = n;
            const std::lock_guard<std::mutex> g(error_lock);
            if (!error) {
                error = std::current_exception();
            }
        }
    };
    std::vector<std::thread> pool;
    try {
        pool.reserve(nthreads);
        for (unsigned t = 1; t < nthreads; ++t) {
            pool.emplace_back(work);
        }
    } catch (const std::exception&) {
    }
    work();
    for (auto& t : pool) {
        t.join();
    }
    if (error) {
        std::rethrow_exception(error);
    }
}

}  // namespace lk
