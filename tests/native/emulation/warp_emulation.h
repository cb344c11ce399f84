// Runs device code of the library on the host: every thread of one cluster is
// a fiber of the calling thread, and the warp, block and cluster intrinsics
// that the code uses exchange values between fibers.  A fiber runs until it
// waits in an intrinsic; an intrinsic returns once all threads it belongs to
// have called the same one (a warp's calls name all 32 lanes).  Threads that
// call different intrinsics, or wait for one that has returned, end the
// process with a message.  Fibers are resumed in ascending or descending
// order; it is not a race detector beyond that.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#include <ucontext.h>

namespace emulation {

// a meeting point of `size` threads, used over and over
struct meeting {
  unsigned size = 0, arrived = 0, generation = 0;
  const char *what = nullptr;
};

struct warp_state {
  meeting at;
  uint64_t slot[2][32]; // by the generation's parity: a lane is at most one call ahead
};

struct fiber {
  ucontext_t context;
  std::vector<char> stack;
  unsigned block = 0, thread = 0;
  const meeting *waits = nullptr;
  unsigned generation = 0;
  bool done = false;
};

struct cluster_state {
  unsigned blocks = 0, threads = 0;
  std::vector<fiber> fibers;
  std::vector<warp_state> warps;
  std::vector<meeting> block_meetings;
  meeting cluster_meeting;
  ucontext_t scheduler;
  fiber *current = nullptr;
  std::function<void(unsigned)> body;
};

inline cluster_state *running = nullptr;

[[noreturn]] inline void fail(const char *message, const char *what) {
  const fiber *f = running->current;
  std::fprintf(stderr, "block %u thread %u: %s (%s)\n", f ? f->block : 0, f ? f->thread : 0, message, what ? what : "");
  std::exit(3);
}

// returns the generation in which the threads met
inline unsigned meet(meeting &m, const char *what) {
  fiber &f = *running->current;
  if (m.arrived == 0)
    m.what = what;
  else if (std::strcmp(m.what, what) != 0)
    fail("threads meet in different calls", what);
  const unsigned generation = m.generation;
  if (++m.arrived == m.size) {
    m.arrived = 0;
    m.generation++;
    return generation;
  }
  f.waits = &m;
  f.generation = generation;
  swapcontext(&f.context, &running->scheduler);
  return generation;
}

inline warp_state &warp() {
  const fiber &f = *running->current;
  return running->warps[(f.block * running->threads + f.thread) / 32];
}
inline unsigned lane() { return running->current->thread & 31; }

template <class T> uint64_t to_word(T v) {
  static_assert(sizeof(T) <= 8, "one slot");
  uint64_t w = 0;
  std::memcpy(&w, &v, sizeof(T));
  return w;
}
template <class T> T of_word(uint64_t w) {
  T v;
  std::memcpy(&v, &w, sizeof(T));
  return v;
}

// every lane's value, once all lanes have given theirs
template <class T> const uint64_t *exchange(unsigned mask, T v, const char *what) {
  if (mask != 0xffffffffu)
    fail("not the whole warp", what);
  warp_state &w = warp();
  uint64_t *slots = w.slot[w.at.generation & 1];
  slots[lane()] = to_word(v);
  meet(w.at, what);
  return slots;
}

inline void fiber_main() {
  cluster_state &c = *running;
  c.body(c.current->block);
  c.current->done = true;
  swapcontext(&c.current->context, &c.scheduler);
}

// body(block) for every thread of a cluster
inline void run(unsigned blocks, unsigned threads, bool descending, std::function<void(unsigned)> body) {
  cluster_state c;
  c.blocks = blocks;
  c.threads = threads;
  c.body = std::move(body);
  c.fibers.resize((size_t)blocks * threads);
  c.warps.resize((size_t)blocks * threads / 32);
  c.block_meetings.resize(blocks);
  for (auto &w : c.warps)
    w.at.size = 32;
  for (auto &m : c.block_meetings)
    m.size = threads;
  c.cluster_meeting.size = blocks * threads;
  running = &c;
  for (unsigned k = 0; k < blocks * threads; k++) {
    fiber &f = c.fibers[k];
    f.block = k / threads;
    f.thread = k % threads;
    f.stack.resize(128 << 10);
    getcontext(&f.context);
    f.context.uc_stack.ss_sp = f.stack.data();
    f.context.uc_stack.ss_size = f.stack.size();
    f.context.uc_link = nullptr;
    makecontext(&f.context, fiber_main, 0);
  }
  for (bool all_done = false; !all_done;) {
    bool progress = false;
    all_done = true;
    // a warp's fibers until all of them wait for another warp or are done
    for (unsigned n = 0; n < c.warps.size(); n++) {
      const unsigned w = descending ? (unsigned)c.warps.size() - 1 - n : n;
      for (bool again = true; again;) {
        again = false;
        for (unsigned l = 0; l < 32; l++) {
          fiber &f = c.fibers[w * 32 + (descending ? 31 - l : l)];
          if (f.done || (f.waits && f.waits->generation == f.generation))
            continue;
          f.waits = nullptr;
          c.current = &f;
          swapcontext(&c.scheduler, &f.context);
          c.current = nullptr;
          again = progress = true;
        }
      }
      for (unsigned l = 0; l < 32; l++)
        all_done = all_done && c.fibers[w * 32 + l].done;
    }
    if (!progress && !all_done) {
      for (fiber &f : c.fibers)
        if (!f.done) {
          c.current = &f;
          fail("waits for threads that do not come", f.waits->what);
        }
    }
  }
  running = nullptr;
}

inline uint3 thread_index() { return {running->current->thread, 0, 0}; }

} // namespace emulation

#define threadIdx (emulation::thread_index())

template <class T> T __shfl_sync(unsigned mask, T v, unsigned src) { return emulation::of_word<T>(emulation::exchange(mask, v, "shfl")[src & 31]); }
template <class T> T __shfl_xor_sync(unsigned mask, T v, unsigned x) {
  return emulation::of_word<T>(emulation::exchange(mask, v, "shfl_xor")[emulation::lane() ^ x]);
}
template <class T> T __shfl_up_sync(unsigned mask, T v, unsigned d) {
  const uint64_t *all = emulation::exchange(mask, v, "shfl_up");
  return emulation::of_word<T>(all[emulation::lane() >= d ? emulation::lane() - d : emulation::lane()]);
}
inline unsigned __ballot_sync(unsigned mask, bool v) {
  const uint64_t *all = emulation::exchange(mask, v, "ballot");
  unsigned r = 0;
  for (int k = 0; k < 32; k++)
    r |= (unsigned)(all[k] != 0) << k;
  return r;
}
inline bool __any_sync(unsigned mask, bool v) { return __ballot_sync(mask, v) != 0; }
inline bool __all_sync(unsigned mask, bool v) { return __ballot_sync(mask, v) == 0xffffffffu; }
inline uint32_t __reduce_and_sync(unsigned mask, uint32_t v) {
  const uint64_t *all = emulation::exchange(mask, v, "reduce_and");
  uint32_t r = 0xffffffffu;
  for (int k = 0; k < 32; k++)
    r &= (uint32_t)all[k];
  return r;
}
inline void __syncwarp() { emulation::exchange(0xffffffffu, 0, "syncwarp"); }
inline void __syncthreads() { emulation::meet(emulation::running->block_meetings[emulation::running->current->block], "syncthreads"); }

template <class T, class U> auto min(T a, U b) { return a < b ? a : b; }
