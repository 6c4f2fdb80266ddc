// The time a polling wait has spent, in clocks, without the time the GPU ran
// something else.
//
// The clock goes on while a kernel is switched out (another process's time
// slice, a debugger), so a difference of two readings alone would let a proof
// time out because it lost the GPU. A gap between two looks at the barrier
// therefore counts kWaitStep clocks (half a millisecond) at most: 2^11 of them
// reach the longest limit, while a wait that runs is over within microseconds of
// its time slice.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define WAIT_CLOCK_FN __host__ __device__ __forceinline__
#else
#define WAIT_CLOCK_FN inline
#endif

constexpr uint32_t kWaitStep = 1u << 20;

struct WaitClock {
  uint32_t last = 0, spent = 0;
  bool started = false;
  // At a look that found nothing, the clock's low word being `now`: true once
  // more than `limit` (at most 2^31) clocks were spent since the first.
  WAIT_CLOCK_FN bool passed(uint32_t now, uint32_t limit) {
    const uint32_t step = now - last;
    if (started) spent += step < kWaitStep ? step : kWaitStep;
    started = true;
    last = now;
    return spent > limit;
  }
};
