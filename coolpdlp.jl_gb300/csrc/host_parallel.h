// host_parallel.h -- loops over host threads (plain C++: also built by the tests).
#pragma once

#include <algorithm>
#include <cstdint>
#include <exception>
#include <thread>
#include <vector>

namespace cpdlp {

// f(k) for k in [0, count) on up to 16 host threads, each a contiguous block of k
// (f must not depend on which thread runs it).  What f throws reaches the caller
// when all threads have ended; a thread that cannot be started leaves its block
// to this one.
template <class F>
void parallel_for(int64_t count, F&& f) {
    const int64_t hw = std::max<int64_t>(1, std::min<int64_t>(16, std::thread::hardware_concurrency()));
    const int64_t nt = std::min<int64_t>(hw, std::max<int64_t>(1, count / 64));
    std::vector<std::exception_ptr> err((size_t)nt);
    auto block = [&](int64_t t) {
        try {
            for (int64_t k = count * t / nt; k < count * (t + 1) / nt; k++) f(k);
        } catch (...) {
            err[(size_t)t] = std::current_exception();
        }
    };
    std::vector<std::thread> th;
    th.reserve((size_t)nt);
    for (int64_t t = 1; t < nt; t++) {
        try {
            th.emplace_back(block, t);
        } catch (...) {
            block(t);
        }
    }
    block(0);
    for (auto& x : th) x.join();
    for (auto& e : err)
        if (e) std::rethrow_exception(e);
}

}  // namespace cpdlp
