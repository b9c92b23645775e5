// The waits of the persistent solve's shared-memory rings (gmres_persistent.cu), for the device and,
// in tests, the host.  A launch that breaks has to end: every wait has a time limit and gives up
// early once the launch is marked as failing.
//
// Env is one thread's view of a wait: done() (the phase is complete), now() (ns), failing() (the
// launch is marked), fail() (mark it) and, of a warp's lanes, all(p) (true when p is for every lane).
#pragma once

#ifdef __CUDACC__
#define CFDV_WAIT_HD __host__ __device__ __forceinline__
#else
#define CFDV_WAIT_HD inline
#endif

namespace cfdv {

constexpr unsigned long long kWaitNs = 2000000000ull;  // 2 s: far above any wait of a sound launch

// one thread: false when the launch is failing (with `heed`) or the time is up (marked then)
template <class Env>
CFDV_WAIT_HD bool wait_thread(Env& w, bool heed = true) {
  if (w.done()) return true;
  const unsigned long long t0 = w.now();
  for (unsigned polls = 1;; polls++) {
    if (w.done()) return true;
    if ((polls & 63u) == 0) {
      if (heed && w.failing()) return false;
      if (w.now() - t0 > kWaitNs) {
        w.fail();
        return false;
      }
    }
  }
}

// the lanes of a warp together: one answer for all of them.  Each lane sees the mark and the clock
// at its own polls; a lane that left alone would keep the others waiting at the next warp-wide
// instruction while it waits for them at the block's barrier.
template <class Env>
CFDV_WAIT_HD bool wait_warp(Env& w) {
  return w.all(wait_thread(w));
}

// a bulk copy that has been issued: it lands whether or not the launch is failing, and a block must
// not end before that, since the copy writes its shared memory
template <class Env>
CFDV_WAIT_HD bool wait_landed(Env& w) {
  return wait_thread(w, false);
}

}  // namespace cfdv
