// Host build of the server's side-stream set (era-bellman-cuda_b200/csrc/fork_set.h)
// for tests/test_fork_set.py: creation that fails after a given number.
#include "fork_set.h"

extern "C" {
// creates for `chains` with `streams` streams and `events` events to be had;
// out: streams held, events held; returns bit k set when k chains are served (k < 32)
unsigned fork_create(unsigned chains, unsigned streams, unsigned events, unsigned *out) {
  msm_b200::fork_set<int, int> forks;
  auto make = [](unsigned &left) {
    return [&left](int &handle) {
      handle = (int)left;
      return left > 0 ? (left--, true) : false;
    };
  };
  forks.create(chains, make(streams), make(events));
  out[0] = (unsigned)forks.streams.size();
  out[1] = (unsigned)forks.events.size();
  unsigned served = 0;
  for (unsigned k = 0; k < 32; k++)
    served |= (unsigned)forks.serves(k) << k;
  return served;
}
}
