// The end of the bucket reduction, one block per window: the levels of
// reduce_level_kernel whose few additions leave most of the GPU idle anyway,
// one after another in shared memory, then the window's results.
#pragma once

#include "msm_group4.cuh"

namespace msm_b200 {

// Levels `level`..log_g - 1 of window w (see reduce_level_kernel), whose tree
// and streams of E = G >> level entries are in global memory.  Every addition
// takes a group of four lanes; operands are read before a barrier and sums
// written after it, in place (job i of a stream writes entry i, which no later
// job of that stream reads).  Then OUT(sum) may read sum(s), the sum of stream
// s.  The whole block calls.
template <class OUT>
__device__ __forceinline__ void reduce_tail(const xyzz *__restrict__ tree, const xyzz *__restrict__ streams, unsigned w, unsigned log_g, unsigned level,
                                            OUT out) {
  extern __shared__ uint4 tail_memory[];
  xyzz *const sh = reinterpret_cast<xyzz *>(tail_memory);
  const unsigned t = threadIdx.x, role = t & 3, first = level, E = 1u << (log_g - level);
  // entries of stream s; the tree last
  auto stream = [&](unsigned s) { return sh + (s <= first ? s * E : (first + 2) * E - (E >> (s - first - 1))); };
  xyzz *const sums = sh + (first + 2) * E; // the tree
  const xyzz *const s_in = streams + (size_t)w * stream_stride(log_g), *const t_in = tree + ((size_t)w << log_g);
  for (unsigned q = t; q < (first + 2) * E * 8; q += TAIL_THREADS) { // 16-byte words
    const unsigned entry = q / 8, s = entry / E, i = entry % E;
    const xyzz *from = s <= first ? s_in + stream_offset(log_g, s) + i : t_in + i;
    reinterpret_cast<uint4 *>(s <= first ? sh + entry : sums + i)[q % 8] = reinterpret_cast<const uint4 *>(from)[q % 8];
  }
  __syncthreads();
  for (; level < log_g; level++) {
    const unsigned half = 1u << (log_g - level - 1), jobs = (level + 2) * half;
    for (unsigned base = 0; base < jobs; base += TAIL_THREADS / 4) {
      const unsigned group = base + (t >> 2);
      const bool active = group < jobs;
      const unsigned job = active ? group / half : 0, i = active ? group % half : 0;
      const bool of_tree = job == level + 1;
      xyzz *const at = of_tree ? sums : stream(job);
      xyzz a, b;
      if (base + ((t & ~31u) >> 2) < jobs) { // the warp has a job
        a = at[2 * i];
        b = at[2 * i + 1];
        a = add_group4(a, b);
      }
      __syncthreads();
      if (active && role == 0) {
        if (of_tree)
          stream(level + 1)[i] = b;
        at[i] = a;
      }
      __syncthreads();
    }
  }
  out([&](unsigned s) { return *stream(s); });
}

} // namespace msm_b200
