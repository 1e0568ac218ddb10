// A step's logits from the device to the caller's buffer, through a pinned one (host code; `Dev` is what does it: see fl_lib.cu).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstring>

namespace fl {

constexpr size_t kLogitsParts = 16;      // at most

// Returns when the n floats are in `host`.  From 4 MiB on the caller's pages are brought in while the device still computes (new ones cost a
// fault each) and the transfer goes in parts, each copied on while the next arrives.  64 rows of 32000 logits behind a device step of 0.6 ms,
// whole call: 1.25 -> 1.15 ms (copying with helper threads: no faster here, they wake up late).
// Nothing in `host` changes before the step is known to be good: bringing a page in leaves its contents, and the first part is copied on when
// its transfer -- and with it every kernel of the step -- is over and dev.check() has passed.
//   dev.begin(parts)   dev.fetch(p, at, count): part p, enqueued   dev.wait(p): until part p is in `pinned`   dev.check(): throws for a failed step
template <typename Dev>
void deliver_logits(Dev& dev, const float* pinned, float* host, size_t n) {
    constexpr size_t kPart = 512 * 1024;        // floats
    const size_t parts = std::max<size_t>(1, std::min(kLogitsParts, n / kPart));
    auto at = [&](size_t p) { return n * p / parts; };
    dev.begin((int)parts);
    for (size_t p = 0; p < parts; ++p) dev.fetch((int)p, at(p), at(p + 1) - at(p));
    if (parts > 1)
        for (size_t i = 0; i < n * sizeof(float); i += 4096) __atomic_fetch_or(reinterpret_cast<unsigned char*>(host) + i, 0, __ATOMIC_RELAXED);
    for (size_t p = 0; p < parts; ++p) {
        dev.wait((int)p);
        if (p == 0) dev.check();
        std::memcpy(host + at(p), pinned + at(p), (at(p + 1) - at(p)) * sizeof(float));
    }
}

}  // namespace fl
