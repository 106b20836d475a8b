// Host threads of one call (the staged copies).
#pragma once

#include <exception>
#include <thread>

namespace gcu {

constexpr unsigned kMaxWorkers = 8;

// Runs work(t) on the calling thread (t = 0) and on up to workers - 1 others
// (kMaxWorkers at most). Fewer where a thread cannot be started, for want of
// threads or of memory: an exception that left this function would end the
// process with the threads that are running, so the work has to be handed out
// as it is asked for.
template <class Work>
void run_workers(unsigned workers, const Work& work) {
    std::thread pool[kMaxWorkers];
    for (unsigned t = 1; t < workers && t < kMaxWorkers; ++t) {
        try {
            pool[t] = std::thread([&work, t] { work(t); });
        } catch (const std::exception&) {
            break;
        }
    }
    work(0);
    for (auto& t : pool)
        if (t.joinable()) t.join();
}

}  // namespace gcu
