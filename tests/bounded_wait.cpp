// Host driver for tests/test_bounded_wait.py: the waits of a kernel's roles
// (amca3d_gb300/csrc/bounded_wait.h) with the 32 lanes of a warp as threads
// and a vote that every lane takes part in. Prints a line per scenario: name,
// rounds, rounds with two verdicts, rounds with a wrong one.
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>

#include "../amca3d_gb300/csrc/bounded_wait.h"

namespace {

constexpr int kLanes = 32;

// __all_sync: every lane hands in its vote and gets whether all were true.
struct Vote {
  std::mutex m;
  std::condition_variable cv;
  int arrived = 0, round = 0;
  bool all = true, verdict = true;
  bool operator()(bool ok) {
    std::unique_lock<std::mutex> l(m);
    all = all && ok;
    const int mine = round;
    if (++arrived == kLanes) {
      verdict = all;
      all = true;
      arrived = 0;
      ++round;
      cv.notify_all();
    } else {
      cv.wait(l, [&] { return round != mine; });
    }
    return verdict;
  }
};

unsigned long long now_ns() {
  return (unsigned long long)std::chrono::duration_cast<std::chrono::nanoseconds>(
             std::chrono::steady_clock::now().time_since_epoch())
      .count();
}

// done(lane): what lane sees of the barrier, `late` lanes only after a while.
enum Scenario { kDone, kAbortBeforeSome, kRunsOutForSome, kRunsOutForAll };

void run(const char *name, Scenario s, int rounds) {
  long split = 0, wrong = 0;
  for (int r = 0; r < rounds; ++r) {
    Vote vote;
    volatile int abort = s == kAbortBeforeSome ? 1 : 0;
    std::vector<int> verdict(kLanes);
    std::vector<std::thread> lanes;
    for (int lane = 0; lane < kLanes; ++lane)
      lanes.emplace_back([&, lane] {
        int looks = 0;
        // the barrier completes for the lanes that look late enough, or never
        const bool sees = s == kDone || ((s == kAbortBeforeSome || s == kRunsOutForSome) && lane % 3 != r % 3);
        verdict[lane] = amca::wait_or_abort_together([&] { return sees && ++looks > lane % 2; }, now_ns, 200000ull, &abort,
                                                     [&](bool ok) { return vote(ok); });
      });
    for (auto &t : lanes) t.join();
    bool same = true;
    for (int v : verdict) same = same && v == verdict[0];
    split += !same;
    wrong += same && verdict[0] != (s == kDone);
    wrong += s != kDone && !abort;
  }
  std::printf("%s %d %ld %ld\n", name, rounds, split, wrong);
}

}  // namespace

int main() {
  run("done", kDone, 20);
  run("abort_before_some", kAbortBeforeSome, 60);
  run("runs_out_for_some", kRunsOutForSome, 60);
  run("runs_out_for_all", kRunsOutForAll, 20);
  return 0;
}
