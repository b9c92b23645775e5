// Test-only CPU build of the ring waits (cfdv_b200/csrc/bounded_wait.h): 32 threads are the lanes of
// a warp, each with its own clock and its own view of the phase and of the failure mark.  Used only
// by tests/test_bounded_wait.py.
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

#include "../../cfdv_b200/csrc/bounded_wait.h"

namespace {
struct Vote {  // all 32 lanes meet here, as in a warp vote
  std::mutex m;
  std::condition_variable cv;
  int here = 0;
  bool every = true;
  bool operator()(bool p) {
    std::unique_lock<std::mutex> l(m);
    every = every && p;
    if (++here == 32) cv.notify_all();
    cv.wait(l, [&] { return here == 32; });
    return every;
  }
};
struct Lane {
  long done_at, failing_at;  // the poll from which this lane sees them (-1: never)
  unsigned long long ns_per_poll, t = 0;
  Vote* vote;
  long polls = 0;
  int marked = 0;
  bool done() {
    t += ns_per_poll;
    return done_at >= 0 && polls++ >= done_at;
  }
  unsigned long long now() const { return t; }
  bool failing() const { return failing_at >= 0 && polls >= failing_at; }
  void fail() { marked = 1; }
  bool all(bool p) { return (*vote)(p); }
};
}  // namespace

// kind 0: wait_thread, 1: wait_warp, 2: wait_landed; per lane the answer and whether it marked the launch
extern "C" void emu_wait(int kind, const long* done_at, const long* failing_at, unsigned long long ns_per_poll,
                         int* answer, int* marked) {
  Vote vote;
  std::vector<std::thread> th;
  for (int l = 0; l < 32; l++)
    th.emplace_back([&, l] {
      Lane w{done_at[l], failing_at[l], ns_per_poll, 0, &vote};
      answer[l] = kind == 0 ? cfdv::wait_thread(w) : kind == 1 ? cfdv::wait_warp(w) : cfdv::wait_landed(w);
      marked[l] = w.marked;
    });
  for (auto& t : th) t.join();
}
