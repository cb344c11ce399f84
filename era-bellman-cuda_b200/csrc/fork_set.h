// Side streams for the parts of a group that can run side by side, and the
// events that fork and join them.  They are an option: what could not be
// created is done without.  Free of CUDA calls (the caller passes the functions
// that create), so that the CPU tests make creation fail
// (tests/native/fork_check.cpp).
#pragma once

#include <cstddef>
#include <vector>

namespace msm_b200 {

template <class STREAM, class EVENT> struct fork_set {
  std::vector<STREAM> streams;
  std::vector<EVENT> events; // one to fork, then one per stream to join

  // Creates streams and events for `chains` chains, or as many as can be had:
  // make_stream(STREAM &) and make_event(EVENT &) return false when they fail.
  template <class MAKE_STREAM, class MAKE_EVENT> void create(size_t chains, MAKE_STREAM make_stream, MAKE_EVENT make_event) {
    STREAM stream{};
    while (streams.size() < chains && make_stream(stream))
      streams.push_back(stream);
    EVENT event{};
    while (events.size() < chains + 1 && make_event(event))
      events.push_back(event);
  }

  // Whether `chains` chains can run on side streams; one alone has nothing to run beside.
  bool serves(size_t chains) const { return chains > 1 && streams.size() >= chains && events.size() > chains; }
};

} // namespace msm_b200
