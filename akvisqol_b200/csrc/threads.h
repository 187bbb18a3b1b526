// Short-lived helper threads of a call.
#pragma once

#include <cstddef>
#include <exception>
#include <thread>
#include <vector>

namespace vqb {

// work(t), t < n, at once: t = 0 on the calling thread, the others on threads
// of their own as far as those can be started (a process may be out of
// threads or memory). So work takes its items from a queue, and whoever runs
// finishes them. Returns when all have ended, with the first exception of any.
template <class F>
void run_threads(size_t n, F &&work) {
    std::vector<std::exception_ptr> errs(n > 0 ? n : 1);
    auto guarded = [&](size_t t) {
        try {
            work(t);
        } catch (...) {
            errs[t] = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(errs.size());  // (no exception between a thread's start and its place here)
    try {
        for (size_t t = 1; t < n; ++t) pool.emplace_back(guarded, t);
    } catch (const std::exception &) {
        // the threads that did start share the items with this one
    }
    guarded(0);
    for (auto &t : pool) t.join();
    for (const auto &e : errs)
        if (e) std::rethrow_exception(e);
}

}  // namespace vqb
