// Host driver for tests/test_velocity_share.py: the sharing of host-velocity
// requests (amca3d_gb300/csrc/velocity_share.h) with helpers that join late
// and are held at the points where the protocol reads its request word.
// Every entry of a request has to be evaluated exactly once, and before the
// request counts as answered. Usage: velocity_share <scenario> <rounds>;
// prints "<requests> <wrong> <unanswered>".
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include "../amca3d_gb300/csrc/velocity_share.h"

namespace {

using Clock = std::chrono::steady_clock;
constexpr int kCap = 512;

struct Bench {
  amca::VelocityShare share;
  std::atomic<unsigned> published{0};  // the request whose entries the launching thread evaluates
  unsigned T[kCap] = {};
  std::atomic<unsigned> v[kCap], evals[kCap];
  long requests = 0, wrong = 0, unanswered = 0;

  void eval(unsigned i) {
    v[i].store(T[i] * 3u + 1u, std::memory_order_relaxed);
    evals[i].fetch_add(1u, std::memory_order_relaxed);
  }
  // One request; false where it stayed unanswered for `limit`.
  bool request(unsigned seq, unsigned n, std::chrono::milliseconds limit = std::chrono::milliseconds(2000)) {
    for (unsigned i = 0; i < n; ++i) {
      T[i] = seq * 1000u + i;
      v[i].store(0u);
      evals[i].store(0u);
    }
    const auto end = Clock::now() + limit;
    const bool answered = share.serve(
        seq, n,
        [&](unsigned i) {
          published.store(seq);
          eval(i);
        },
        [&] { return Clock::now() > end; });
    ++requests;
    bool ok = true;
    for (unsigned i = 0; i < n; ++i) ok = ok && v[i].load() == T[i] * 3u + 1u && evals[i].load() == 1u;
    unanswered += !answered;
    wrong += answered && !ok;
    return answered;
  }
  // until the launching thread is at a request after `seq`, or half a second
  void await_request_after(unsigned seq) const {
    const auto end = Clock::now() + std::chrono::milliseconds(500);
    while (published.load() <= seq && Clock::now() < end) std::this_thread::yield();
  }
  void print() const { std::printf("%ld %ld %ld\n", requests, wrong, unanswered); }
};

// A helper that joins while requests are shared by others is held after its
// first two loads of the word, before it is counted and with a request in hand
// that was shared without it, each time until the next request is out; with
// `slow` the other helper's entries come late, so that a request counted off
// in its place is answered without them.
void late(int rounds, bool slow) {
  Bench total;
  for (int k = 0; k < rounds; ++k) {
    Bench b;
    std::thread first([&] {
      b.share.help([&](unsigned i) {
        if (slow && i == 1) std::this_thread::sleep_for(std::chrono::milliseconds(1));
        b.eval(i);
      });
    });
    std::thread second;
    bool up = true;
    for (unsigned seq = 1; seq <= 60 && up; ++seq) {
      if (seq == 10)
        second = std::thread([&] {
          int loads = 0;
          b.share.help([&](unsigned i) { b.eval(i); },
                       [&] {
                         if (++loads <= 2) b.await_request_after(b.published.load());
                       });
        });
      up = b.request(seq, 200);
    }
    b.share.stop();
    first.join();
    if (second.joinable()) second.join();
    total.requests += b.requests;
    total.wrong += b.wrong;
    total.unanswered += b.unanswered;
  }
  total.print();
}

// Seven helpers start one after another, each descheduled now and then, beside
// back-to-back requests of 1 to 300 entries.
void staggered(int rounds) {
  Bench total;
  for (int k = 0; k < rounds; ++k) {
    Bench b;
    std::vector<std::thread> helpers;
    std::thread starter([&] {
      for (int h = 0; h < 7; ++h) {
        helpers.emplace_back([&, h] {
          unsigned x = 12345u + 77u * (unsigned)h + 1000u * (unsigned)k;
          auto now_and_then = [&](unsigned of, int us) {
            x = x * 1664525u + 1013904223u;
            if ((x >> 8) % of == 0) std::this_thread::sleep_for(std::chrono::microseconds(us));
          };
          b.share.help(
              [&](unsigned i) {
                now_and_then(4000, 50);
                b.eval(i);
              },
              [&] { now_and_then(5, 120); });
        });
        std::this_thread::sleep_for(std::chrono::microseconds(400));
      }
    });
    bool up = true;
    for (unsigned seq = 1; seq <= 400 && up; ++seq) up = b.request(seq, 1u + seq * 37u % 300u);
    starter.join();
    b.share.stop();
    for (auto &t : helpers) t.join();
    total.requests += b.requests;
    total.wrong += b.wrong;
    total.unanswered += b.unanswered;
  }
  total.print();
}

// A helper that does not come back in time: serve ends when nobody waits for the answer any more.
void abandoned() {
  Bench b;
  std::atomic<bool> go{false};
  std::thread helper([&] {
    b.share.help([&](unsigned) {
      while (!go.load()) std::this_thread::sleep_for(std::chrono::milliseconds(1));
    });
  });
  bool answered = true;  // (the first requests may be made before the helper has joined)
  for (unsigned seq = 1; seq <= 2000 && answered; ++seq) {
    answered = b.request(seq, 64, std::chrono::milliseconds(20));
    std::this_thread::sleep_for(std::chrono::microseconds(100));
  }
  go.store(true);
  b.share.stop();
  helper.join();
  b.print();
}

}  // namespace

int main(int argc, char **argv) {
  const char *s = argc > 1 ? argv[1] : "late";
  const int rounds = argc > 2 ? std::atoi(argv[2]) : 10;
  if (!std::strcmp(s, "late")) late(rounds, false);
  else if (!std::strcmp(s, "late_beside_slow")) late(rounds, true);
  else if (!std::strcmp(s, "staggered")) staggered(rounds);
  else abandoned();
  return 0;
}
