// A host-thread loop for the set-up code.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

namespace bsg {

// fn(i) for every i in [0, n), on up to 32 host threads taking chunks of
// `chunk` indices from a shared counter.  Callers write only to locations
// that index i owns, so the result does not depend on the schedule.
// max_threads 1 runs inline: small systems (and the many systems of a batch,
// which are already set up on parallel host threads) skip the thread start-up.
template <typename F>
void parallel_for(int64_t n, int64_t chunk, F fn, int max_threads = 32) {
    const int64_t nchunks = (n + chunk - 1) / chunk;
    const unsigned hw = std::max(1u, std::min((unsigned)std::max(1, max_threads), std::thread::hardware_concurrency()));
    const int nt = (int)std::min<int64_t>((int64_t)hw, nchunks);
    if (nt <= 1) {
        for (int64_t i = 0; i < n; ++i) fn(i);
        return;
    }
    std::atomic<int64_t> next{0};
    std::atomic<bool> oom{false};
    auto work = [&]() {
        try {
            for (;;) {
                const int64_t c = next.fetch_add(1);
                if (c >= nchunks || oom) return;
                const int64_t i1 = std::min(n, (c + 1) * chunk);
                for (int64_t i = c * chunk; i < i1; ++i) fn(i);
            }
        } catch (const std::bad_alloc &) {
            oom = true;   // reported to the caller below as an allocation failure
        }
    };
    // fewer threads where the system gives no more: the chunks go round all the same
    std::vector<std::thread> th;
    th.reserve((size_t)nt);
    try {
        for (int k = 1; k < nt; ++k) th.emplace_back(work);
    } catch (const std::system_error &) {
    }
    work();
    for (auto &x : th) x.join();
    if (oom) throw std::bad_alloc();
}

}  // namespace bsg
