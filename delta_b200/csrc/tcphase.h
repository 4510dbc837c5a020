// tcphase.h -- which phase of an mbarrier its waiter has to wait for, when one thread commits
// work to it and waits for each commit before the next.  Host and device: the order of the
// phases is tested on the CPU against a model of the mbarrier.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define DELTA_HD __host__ __device__ __forceinline__
#else
#define DELTA_HD inline
#endif

namespace delta {

// A wait for a phase returns once that phase has completed, and a wait for the parity of the
// phase before the open one returns at once.  So the parity changes only when a wait has
// succeeded: after one that ran out, the commit it waited for is still to come, and the wait
// that makes sure of it (drain) has to ask for the same phase again.  No commit may be added
// in between: with two outstanding, both could arrive before the waiter looks, and the phase
// it asks for would be open again.
struct TcPhase {
  uint32_t parity = 0;  // of the phase that the commit in flight, or the next one, completes
  bool late = false;    // the last wait ran out

  // wait(parity): a bounded wait, true if that phase has completed
  template <class Wait>
  DELTA_HD bool wait(Wait &&bounded_wait) {
    late = !bounded_wait(parity);
    if (!late) parity ^= 1u;
    return !late;
  }
  // Whatever was committed has completed: true at once if the last wait succeeded, else after
  // one more bounded wait for the same phase.
  template <class Wait>
  DELTA_HD bool drain(Wait &&bounded_wait) {
    return !late || wait(bounded_wait);
  }
};

// What a kernel writes to its error flag when a wait ran out: the work had ended by the time
// the kernel freed its TMEM, or had not.
constexpr int kTcLate = 1, kTcLost = 2;

}  // namespace delta
