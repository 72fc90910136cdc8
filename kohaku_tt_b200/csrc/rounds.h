// Host code without CUDA.
#pragma once
#include <cstdint>

namespace ktt {

constexpr int kMostLevels = 64;

// The time at which the last of `machines` is done, when each item goes to the first free one: `cost[i]`
// us of `count[i]` items, the longest first. Machines that are done at the same time are one group: a level adds
// one at most, so that up to 2 * kMostLevels levels have room.
inline float makespan(const float* cost, const int64_t* count, int levels, int64_t machines) {
    constexpr int kRoom = 2 * kMostLevels + 2;
    float at[kRoom];
    int64_t of[kRoom];
    int n = 1, first = 0;
    at[0] = 0.f;
    of[0] = machines;
    for (int i = 0; i < levels; ++i) {
        for (int64_t left = count[i]; left > 0;) {
            const int64_t take = left < of[first] ? left : of[first];
            const float done = at[first] + cost[i];
            left -= take;
            of[first] -= take;
            if (of[first] == 0) ++first;
            int j = n;   // (mostly the last)
            while (j > first && at[j - 1] > done) --j;
            if (j > first && at[j - 1] == done) {
                of[j - 1] += take;
                continue;
            }
            if (n == kRoom) {   // make room at the front
                for (int k = first; k < n; ++k) {
                    at[k - first] = at[k];
                    of[k - first] = of[k];
                }
                n -= first;
                j -= first;
                first = 0;
            }
            for (int k = n; k > j; --k) {
                at[k] = at[k - 1];
                of[k] = of[k - 1];
            }
            at[j] = done;
            of[j] = take;
            ++n;
        }
    }
    return at[n - 1];
}

}  // namespace ktt
