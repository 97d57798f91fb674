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

// A mode's status once its forward solve has ended with `st` (the whole warp): the steps still in the
// slots (`total` published over `slots` of them, each taken `takers` times) are waited for, because a
// tangent that gave up on them would leave NaN behind a forward that finished.  Where several blocks
// share a mode (status then holds 0 before the launch), the highest code of any of them stays.
__device__ inline void report_status(const WarpTeam& tm, int st, int total, int slots, int takers,
                                     volatile int* consumed, volatile int* abort_flag, long long max_polls, bool shared,
                                     int32_t* status)
{
    bool taken = true;
    for (int sl = 0; sl < slots; ++sl)
        taken = taken && wait_at_least(tm, consumed + sl, takers * ((total + slots - 1 - sl) / slots), abort_flag,
                                       max_polls);
    if (st == DISCOEB_OK && !taken) st = DISCOEB_ABORTED;
    if (tm.leader()) {
        if (shared) atomicMax(status, st);
        else *status = st;
    }
}

}  // namespace dscb
