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

// Host threads for n items of `each` units of work: one per 32,768 units, about
// 200 us of the table builders' work against up to as much for starting a thread,
// at most 32.
inline unsigned host_threads(uint64_t n, uint64_t each) {
    const uint64_t want = n * (each + 1) / 32768 + 1;
    return static_cast<unsigned>(
        std::min<uint64_t>({want, std::max<uint64_t>(n, 1), 32, std::max(1u, std::thread::hardware_concurrency())}));
}

// Phase-bin evaluations that finding the runs of a frequency takes, by the
// fastest of freqs: two a run from two samples a bin on, else one a sample.
inline uint64_t fold_run_evaluations(const std::vector<double>& freqs, double tsamp, uint64_t nbins,
                                     uint64_t segment_len) {
    double most = 0.0;
    for (const double f : freqs) {
        const double step = f * tsamp * static_cast<double>(nbins);  // bins per sample
        most = std::max(most, step < 0.5 ? 2.0 * step : 1.0);
    }
    return static_cast<uint64_t>(most * static_cast<double>(segment_len));
}

// fn(i, state) for i < n on host threads, each with a State of its own. The first exception of any fn ends the loop
// and is rethrown here; threads that cannot be started leave their share to
// the others.
template <class State, class F>
void parallel_for(uint64_t n, uint64_t each, F&& fn) {
    const unsigned nthreads = host_threads(n, each);
    std::atomic<uint64_t> next{0};
    std::exception_ptr error;
    std::mutex error_lock;
    auto work = [&] {
        try {
            State state{};
            for (uint64_t i = next++; i < n; i = next++) {
                fn(i, state);
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
