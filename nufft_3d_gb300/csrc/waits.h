// The turns of a bounded wait.  Plain C++, so that the bookkeeping can be
// checked without a stalled device.
#pragma once

#ifdef __CUDACC__
#define NUFFT_HD __host__ __device__ __forceinline__
#else
#define NUFFT_HD inline
#endif

namespace nufft3d {

enum WaitTurn { kWaitOn, kWaitReport, kWaitGiveUp };

struct BoundedWait {
    int failed = 0;     // polls that found nothing
    bool told = false;  // the report has been made
};

// Before the next poll: report a wait (once) after `polls` failed polls and
// give it up after `limit`.  Who gives up reports as well: with polls >= limit
// there was no report before.
NUFFT_HD WaitTurn wait_turn(BoundedWait &w, int polls, int limit)
{
    if (w.failed >= limit) return kWaitGiveUp;
    if (w.told || w.failed < polls) return kWaitOn;
    w.told = true;
    return kWaitReport;
}

}  // namespace nufft3d
