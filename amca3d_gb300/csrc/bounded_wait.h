// bounded_wait.h — waits of the roles of a block, each with a limit and all of
// them ended by the first that runs out. Device code; plain C++ for a test that
// runs lanes as threads.
#pragma once

#ifdef __CUDACC__
#define AMCA_WAIT __device__ __forceinline__
#else
#define AMCA_WAIT inline
#endif

namespace amca {

// Waits until done() holds, for at most `limit` by the clock now(). False when
// the wait ran out, which sets *abort, or found *abort set.
template <class Done, class Now>
AMCA_WAIT bool wait_or_abort(Done done, Now now, unsigned long long limit, volatile int *abort) {
  if (done()) return true;
  const unsigned long long t0 = now();
  while (!done()) {
    if (*abort) return false;
    if (now() - t0 > limit) {
      *abort = 1;
      return false;
    }
  }
  return true;
}

// The same for lanes that go on together: `all` is their vote, so every lane
// gets one verdict, true where every lane's wait ended with done(). Lane by
// lane, one may find the barrier complete where the next finds the abort; the
// first would go on to instructions of the whole warp that the other has left.
template <class Done, class Now, class All>
AMCA_WAIT bool wait_or_abort_together(Done done, Now now, unsigned long long limit, volatile int *abort, All all) {
  return all(wait_or_abort(done, now, limit, abort));
}

}  // namespace amca
