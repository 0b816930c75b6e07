// Host work spread over the machine's cores.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace e8g {

// fn(order[i]) for every i, in this order, on up to a thread per core (this one among them). An exception
// of a call is thrown again here once every thread has stopped; threads that cannot be started are
// done without.
template <class F> void for_each_on_cores(std::vector<uint32_t> const &order, F &&fn) {
    const uint32_t n = static_cast<uint32_t>(order.size());
    std::atomic<uint32_t> next{0};
    std::mutex lock;
    std::exception_ptr error;
    auto work = [&] {
        for (uint32_t i; (i = next.fetch_add(1)) < n;) {
            try {
                fn(order[i]);
            } catch (...) {
                std::lock_guard<std::mutex> hold(lock);
                if (!error)
                    error = std::current_exception();
                next = n;
            }
        }
    };
    const uint32_t most = std::min<uint32_t>(n, std::max(1u, std::thread::hardware_concurrency()));
    std::vector<std::thread> threads;
    threads.reserve(most);
    try {
        while (threads.size() + 1 < most)
            threads.emplace_back(work);
    } catch (...) { // std::system_error, or std::bad_alloc for a thread's state
    }
    work();
    for (std::thread &t : threads)
        t.join();
    if (error)
        std::rethrow_exception(error);
}

} // namespace e8g
