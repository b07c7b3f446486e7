// tlq_mg_wait.cuh -- when a relax gives up waiting for a neighbouring plane
// (tlq_gravity.cu).
#pragma once

namespace tlq {

// After a second, or after so many polls: polls alone took 2^24 of them, and
// one costs from 0.4 us (a progress counter) to the time of two 128-bit
// loads, a second and more.  TLQ_MG_WAIT_LIMIT in the environment of
// tlq_create overrides the polls (a short limit lets a test make the wait run
// out and check the error status).
constexpr unsigned MG_WAIT_NS = 1000000000u;
constexpr long long MG_WAIT_LIMIT = 1LL << 24;

// One wait: out(c) after each poll that found nothing, until it says that the
// wait is over (another block gave up, the polls or the time ran out).  The
// clock is read every 256 polls, from the 256th on: most waits end before
// that, and a read is as long as a poll.  32-bit words: the clock's differences
// are taken every 256 polls, far below its 4.3 s, and the time runs out
// before 2^32 polls.
struct MgWait {
  unsigned polls = 0, since = 0;
  template <class Ctl>
  __device__ __forceinline__ bool out(const Ctl* c) {
    if (*(const volatile int*)&c->abort || (long long)++polls > c->wait_limit) return true;
    if (polls & 255u) return false;
    unsigned now;
    asm volatile("mov.u32 %0, %globaltimer_lo;" : "=r"(now));
    if (polls == 256u) since = now;
    return now - since > MG_WAIT_NS;
  }
};

}  // namespace tlq
