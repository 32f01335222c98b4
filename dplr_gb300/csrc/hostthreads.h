// hostthreads.h -- host threads of a call behind a C entry point.
#pragma once

#include <exception>
#include <thread>
#include <vector>

namespace dg {

// work() on up to `count` threads, the caller's among them, and waits for them.
// work takes its share from a common counter, so fewer threads do the same: where
// the system gives none (an exception here would end the process, the entry
// points being C), the caller's runs alone.
template <class F> void run_on_threads(unsigned count, F &work)
{
    std::vector<std::thread> th;
    try {
        th.reserve(count);
        for (unsigned t = 1; t < count; ++t) th.emplace_back([&work]() { work(); });
    } catch (const std::exception &) {
    }
    work();
    for (std::thread &t : th) t.join();
}

}  // namespace dg
