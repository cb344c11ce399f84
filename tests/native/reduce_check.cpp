// CPU check of the reduction's end (era-bellman-cuda_b200/csrc/msm_reduce.cuh):
// reduce_tail itself, one block with its intrinsics emulated and its shared
// memory exactly as large as the launch makes it.  Also the accumulation's
// range rule.
//   reduce_check LOG_G...            exits 0 when every stream's sum is right
//   reduce_check ranges TOTAL RANGES THREADS   prints active_ranges
#include "warp_emulation.h"

#include "msm_reduce.cuh"

#include <string>

namespace msm_b200 {
uint4 tail_memory[(64 << 10) / 16];
}

using namespace msm_b200;

namespace {

bool equal(const xyzz &p, const xyzz &q) {
  if (curve::is_inf(p) || curve::is_inf(q))
    return curve::is_inf(p) == curve::is_inf(q);
  const bn254::affine a = curve::to_affine(p), b = curve::to_affine(q);
  return std::memcmp(&a, &b, sizeof(a)) == 0;
}

// Tree and streams as the levels before `tail_level` leave them, from points
// k G for small k (some infinite, some equal or opposite), and the sums that
// the remaining levels of reduce_level_kernel must give.
int check(unsigned log_g) {
  const unsigned level = tail_level(log_g), E = 1u << (log_g - level), windows = 2;
  bn254::affine g;
  fe one = fq::zero(), two = fq::zero();
  one.l[0] = 1, two.l[0] = 2;
  g.x = fq::to_mont(one), g.y = fq::to_mont(two);
  std::vector<xyzz> multiples(1, curve::infinity());
  for (int k = 1; k < 40; k++)
    multiples.push_back(curve::add_affine(multiples.back(), g));
  uint32_t seed = 12345 + log_g;
  auto some = [&] {
    seed = seed * 1664525u + 1013904223u;
    xyzz p = multiples[(seed >> 16) % multiples.size()];
    if (seed >> 31)
      p.y = fq::neg(p.y);
    return p;
  };
  std::vector<xyzz> tree((size_t)windows << log_g), streams(windows * stream_stride(log_g));
  for (auto &p : tree)
    p = some();
  for (auto &p : streams)
    p = some();
  for (unsigned w = 0; w < windows; w++) {
    std::vector<std::vector<xyzz>> want;
    for (unsigned s = 0; s <= level; s++) {
      const xyzz *from = &streams[w * stream_stride(log_g) + stream_offset(log_g, s)];
      want.emplace_back(from, from + E);
    }
    std::vector<xyzz> t(tree.begin() + ((size_t)w << log_g), tree.begin() + ((size_t)w << log_g) + E);
    for (unsigned l = level; l < log_g; l++) {
      std::vector<xyzz> odd;
      auto halve = [](std::vector<xyzz> &v) {
        for (size_t i = 0; i < v.size() / 2; i++)
          v[i] = curve::add(v[2 * i], v[2 * i + 1]);
        v.resize(v.size() / 2);
      };
      for (size_t i = 1; i < t.size(); i += 2)
        odd.push_back(t[i]);
      for (auto &s : want)
        halve(s);
      want.push_back(odd);
      halve(t);
    }
    const size_t bytes = tail_smem(log_g);
    std::memset(tail_memory, 0x5a, sizeof(tail_memory));
    std::vector<xyzz> got(log_g + 1);
    emulation::run(1, TAIL_THREADS, w == 1, [&](unsigned) {
      const unsigned thread = threadIdx.x;
      reduce_tail(tree.data(), streams.data(), w, log_g, level, [&](auto sum) {
        if (thread <= log_g)
          got[thread] = sum(thread);
      });
    });
    for (size_t i = bytes; i < sizeof(tail_memory); i++)
      if (reinterpret_cast<unsigned char *>(tail_memory)[i] != 0x5a) {
        std::fprintf(stderr, "log_g %u: byte %zu past the shared memory written\n", log_g, i - bytes);
        return 1;
      }
    for (unsigned s = 0; s <= log_g; s++)
      if (want[s].size() != 1 || !equal(got[s], want[s][0])) {
        std::fprintf(stderr, "log_g %u window %u: stream %u differs\n", log_g, w, s);
        return 1;
      }
  }
  return 0;
}

} // namespace

int main(int argc, char **argv) {
  if (argc == 5 && std::string(argv[1]) == "ranges") {
    std::printf("%llu\n", active_ranges(std::stoull(argv[2]), (unsigned)std::stoul(argv[3]), (unsigned)std::stoul(argv[4])));
    return 0;
  }
  int failed = 0;
  for (int k = 1; k < argc; k++)
    failed += check((unsigned)std::stoul(argv[k]));
  return failed ? 1 : 0;
}
