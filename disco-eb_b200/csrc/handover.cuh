// Hand-over of steps between the warps of a block through counters in shared memory (device only).
#pragma once

#include "stepper.cuh"

namespace dscb {

// Bounded wait of one warp on a shared-memory counter: lane 0 polls until *flag >= target (or
// the block's abort flag is set, or the poll budget runs out, after which it sets the abort
// flag itself); returns true when the target was reached.  No wait can last forever.
constexpr long long kMaxPolls = 1LL << 24;  // ~2 s with the back-off below; a step takes < 1 ms
__device__ inline long long poll_budget(const DiscoebControl& c) { return c.max_polls > 0 ? (long long)c.max_polls : kMaxPolls; }
__device__ inline bool wait_at_least(const WarpTeam& tm, volatile int* flag, int target, volatile int* abort_flag,
                              long long max_polls)
{
    int ok = 0;
    if (tm.leader()) {
        long long polls = 0;
        while (true) {
            if (*flag >= target) { ok = 1; break; }
            if (*abort_flag) break;
            if (++polls > max_polls) { *abort_flag = 1; break; }
            __nanosleep(100);
        }
        __threadfence_block();
    }
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

}  // namespace dscb
