// Work shared out over host threads.
#pragma once
#include <algorithm>
#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace nsg {

// Run f() on `threads` threads, the caller's among them, or on as many as the
// system grants (f takes its items from a shared counter, so fewer threads only
// take longer).  Returns when all are done; the first exception of any f() is
// thrown then.
template <class F>
void on_threads(size_t threads, F&& f) {
    std::exception_ptr err;
    std::mutex lock;
    auto guarded = [&]() noexcept {
        try {
            f();
        } catch (...) {
            const std::lock_guard<std::mutex> hold(lock);
            if (!err) err = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(threads);
    try {
        while (pool.size() + 1 < threads) pool.emplace_back(guarded);
    } catch (const std::system_error&) {  // no more threads to be had
    }
    guarded();
    for (auto& t : pool) t.join();
    if (err) std::rethrow_exception(err);
}

}  // namespace nsg
