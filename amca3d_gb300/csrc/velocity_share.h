// velocity_share.h — one request for host velocities, evaluated by the thread
// that launched the kernel together with helpers that come to life beside it.
// Host code without CUDA, so that the protocol is tested by itself.
//
// A request is published as one word: its number, the threads that share it
// and its entry count. A helper that has read a word knows from that word
// alone whether it takes part, so it evaluates and counts off each request at
// most once, however long it was descheduled before or after the load, and
// whether or not it was counted when the request was made. (With the number
// and the threads in words of their own, a helper stopped between the two
// loads took up the next request twice: its second count made the launching
// thread wait for ever, or answer before another helper had written its part.)
#pragma once

#include <atomic>
#include <cstdint>
#include <thread>

namespace amca {

class VelocityShare {
 public:
  static constexpr unsigned kSharedFrom = 64;      // entries from which a request is worth sharing
  static constexpr unsigned kMaxThreads = 255;     // that a request's word can name
  static constexpr unsigned kMaxEntries = 0xffffffu;

  // Launching thread: request number `seq` (never the one before) of n entries.
  // It evaluates entries 0, use, 2 use, ... by eval(i), helper w entries w, w +
  // use, ...; true once all are done. ended() is asked from time to time while
  // a helper is still at it: where it says that nobody waits for the answer any
  // more, serve returns false without one.
  template <class Eval, class Ended>
  bool serve(uint32_t seq, unsigned n, Eval eval, Ended ended) {
    unsigned use = 1;
    if (n >= kSharedFrom) use += helpers_.load(std::memory_order_acquire);
    if (use > 1) {
      left_.store(use - 1, std::memory_order_relaxed);
      request_.store((uint64_t)seq << 32 | (uint64_t)use << 24 | n, std::memory_order_release);
    }
    for (unsigned i = 0; i < n; i += use) eval(i);
    if (use > 1)
      for (unsigned spin = 1; left_.load(std::memory_order_acquire) != 0; ++spin)
        if (spin % 4096u == 0 && ended()) return false;
    return true;
  }

  // A helper, until stop(): evaluates its share of the requests made since it
  // came to life, spinning (yielding when idle for long) on the request word.
  // seen() follows the first load of the word and every load of a new one (tests
  // hold a thread there).
  template <class Eval, class Seen>
  void help(Eval eval, Seen seen) {
    uint64_t last = request_.load(std::memory_order_acquire);
    seen();
    const unsigned w = 1u + helpers_.fetch_add(1u, std::memory_order_acq_rel);
    for (unsigned idle = 0; !stop_.load(std::memory_order_acquire);) {
      const uint64_t r = request_.load(std::memory_order_acquire);
      if (r == last) {
        if (++idle > 4096) std::this_thread::yield();
        continue;
      }
      seen();
      last = r;
      idle = 0;
      const unsigned use = (unsigned)(r >> 24) & 0xffu, n = (unsigned)r & 0xffffffu;
      if (w >= use) continue;  // made before this helper counted
      for (unsigned i = w; i < n; i += use) eval(i);
      left_.fetch_sub(1, std::memory_order_acq_rel);
    }
  }
  template <class Eval>
  void help(Eval eval) {
    help(eval, [] {});
  }
  void stop() { stop_.store(true, std::memory_order_release); }

 private:
  std::atomic<uint64_t> request_{0};
  std::atomic<unsigned> left_{0};     // helpers still evaluating the request
  std::atomic<unsigned> helpers_{0};  // helpers alive
  std::atomic<bool> stop_{false};
};

}  // namespace amca
