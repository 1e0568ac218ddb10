// Buffers that are taken anew when a call is larger than all before it (host code).
#pragma once
#include <cstddef>

namespace fl {

// `take` allocates the buffers for `want`; their size counts as had only once all of them are there.  An allocation that fails leaves 0: some
// buffers are gone then, and the next call takes every one again.
template <typename F>
void grow(size_t& cap, size_t want, F&& take) {
    if (want <= cap) return;
    cap = 0;
    take();
    cap = want;
}

}  // namespace fl
