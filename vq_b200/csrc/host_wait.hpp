// host_wait.hpp -- a wait of the host with an end: what does not come within the limit is named in an error.
#pragma once
#include <chrono>
#include <cstdint>
#include <string>

#include "backend.hpp"

namespace vqb {

// Far above any call that works (the longest queue measured in front of a small result, ten levels of a tree over 1M rows, is 15 ms; a
// caller's stream may hold work of its own), and short enough for whoever looks for the reason of a stop.
constexpr double HOST_WAIT_SECONDS = 600.0;

// Calls poll() until it returns true; what() says what it was waiting for.  The clock is read every 4096th time: a poll is a fraction
// of a microsecond.
template <typename Poll, typename What> void wait_until(Poll &&poll, What &&what, double limit_s = HOST_WAIT_SECONDS)
{
    const auto t0 = std::chrono::steady_clock::now();
    for (uint64_t i = 1; !poll(); ++i) {
        if (i % 4096 != 0) continue;
        const double waited = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        if (waited > limit_s)
            throw Error(100, "gave up after " + std::to_string((long)(waited + 0.5)) + " s of waiting for " + what());
    }
}

} // namespace vqb
