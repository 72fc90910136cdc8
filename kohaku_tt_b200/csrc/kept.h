// Host code without CUDA.
#pragma once
#include <atomic>

namespace ktt {

// A number >= 0 that is asked for once and kept in `slot` (zero before). `ask` returns it, or a negative number if it
// could not be had: that is not kept, and the next caller asks again.
template <typename Ask>
int kept(std::atomic<int>& slot, Ask ask) {
    const int known = slot.load(std::memory_order_relaxed);
    if (known != 0) return known - 1;
    const int got = ask();
    if (got >= 0) slot.store(got + 1, std::memory_order_relaxed);
    return got;
}

}  // namespace ktt
