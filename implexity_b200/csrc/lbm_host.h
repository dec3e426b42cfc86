// lbm_host.h -- host threads of the runtime.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <memory>
#include <thread>

namespace lbm {

// fn(begin, end) over [0, n), in chunks that helper threads share with the
// calling one where the work is worth it.  The caller takes chunks itself and
// waits only for chunks in progress: a helper that is not scheduled in time
// (the caller's own thread pool may still spin on every core) finds nothing
// left and leaves without touching fn.
template <typename F>
void parallel_range(int64_t n, F&& fn) {
    constexpr int64_t CHUNK = 1 << 16;
    struct Job {
        std::atomic<int64_t> next{0}, done{0};
    };
    const int64_t chunks = (n + CHUNK - 1) / CHUNK;
    const auto take = [n, chunks](Job& job, F& f) {
        for (int64_t c; (c = job.next.fetch_add(1)) < chunks; job.done.fetch_add(1)) f(c * CHUNK, std::min(n, (c + 1) * CHUNK));
    };
    if (chunks < 4) {
        if (n > 0) fn((int64_t)0, n);
        return;
    }
    const auto job = std::make_shared<Job>();
    const int64_t helpers = std::min<int64_t>({7, (int64_t)std::thread::hardware_concurrency() - 1, chunks / 2 - 1});
    for (int64_t k = 0; k < helpers; ++k) {
        // whatever stops a helper from starting (no more threads, no memory for its
        // state): nothing may unwind past fn while the earlier ones run it
        try {
            std::thread([job, take, &fn] { take(*job, fn); }).detach();
        } catch (...) {
            break;
        }
    }
    take(*job, fn);
    while (job->done.load() < chunks) std::this_thread::yield();
}

}  // namespace lbm
