// CPU check of the final sum (era-bellman-cuda_b200/csrc/msm_final.cuh): the
// kernel's own device code, with the warp, block and cluster intrinsics
// emulated.  Built with array bounds checks; an index out of range ends it.
//   final_check sum IN OUT [descending]  254 Jacobian results (24 words each)
//                                        per sum -> 20 words each
//   final_check lanes IN OUT             pairs of Jacobian points -> per lane
//                                        the residues after each warp operation
//   final_check constants IN OUT         per split group a, b (4 words each) and
//                                        their signs, then beta (IN is not read)
//   final_check inverse IN OUT           values (8 words each, a multiple of
//                                        eight of them) -> their inverses, a
//                                        group of four lanes each
#include "warp_emulation.h"

#include "msm_final.cuh"

#include <fstream>
#include <iterator>
#include <string>

using namespace msm_b200;

namespace {

final_shared blocks[FINAL_BLOCKS];

// what final_sum_block uses of cooperative_groups::cluster_group
struct cluster_view {
  unsigned rank;
  unsigned block_rank() const { return rank; }
  void sync() const { emulation::meet(emulation::running->cluster_meeting, "cluster.sync"); }
  template <class T> T *map_shared_rank(T *at, unsigned of) const {
    return reinterpret_cast<T *>(reinterpret_cast<char *>(at) - reinterpret_cast<char *>(blocks + rank) + reinterpret_cast<char *>(blocks + of));
  }
};

std::vector<uint32_t> read_words(const char *path) {
  std::ifstream in(path, std::ios::binary);
  std::vector<char> bytes((std::istreambuf_iterator<char>(in)), {});
  std::vector<uint32_t> words(bytes.size() / 4);
  std::memcpy(words.data(), bytes.data(), words.size() * 4);
  return words;
}
void write_words(const char *path, const std::vector<uint32_t> &words) {
  std::ofstream(path, std::ios::binary).write(reinterpret_cast<const char *>(words.data()), words.size() * 4);
}

std::vector<uint32_t> sums(const std::vector<uint32_t> &in, bool descending) {
  constexpr size_t WORDS = RESULT_BITS * sizeof(jacobian) / 4;
  std::vector<uint32_t> out;
  std::vector<jacobian> results(RESULT_BITS);
  for (size_t k = 0; k + WORDS <= in.size(); k += WORDS) {
    std::memcpy(results.data(), in.data() + k, WORDS * 4);
    std::memset(blocks, 0xa5, sizeof(blocks)); // shared memory starts as anything
    msm_b200_affine_point point;
    emulation::run(FINAL_BLOCKS, FINAL_THREADS, descending,
                   [&](unsigned block) { final_sum_block(blocks[block], cluster_view{block}, results.data(), &point); });
    const size_t at = out.size();
    out.resize(at + sizeof(point) / 4);
    std::memcpy(out.data() + at, &point, sizeof(point));
  }
  return out;
}

// per pair, operation and lane: x.a x.b y.a y.b z.a z.b; operations: load p,
// load q, put and get p, 2 p, p + q, then whether the addition holds
std::vector<uint32_t> lanes(const std::vector<uint32_t> &in) {
  constexpr size_t WORDS = 2 * sizeof(jacobian) / 4, OPERATIONS = 5;
  std::vector<uint32_t> out;
  for (size_t k = 0; k + WORDS <= in.size(); k += WORDS) {
    jacobian pair[2];
    std::memcpy(pair, in.data() + k, sizeof(pair));
    const size_t at = out.size();
    out.resize(at + (OPERATIONS * 6 + 1) * 32);
    rns_stored stored;
    std::memset(&stored, 0xa5, sizeof(stored));
    emulation::run(1, 32, false, [&](unsigned) {
      const unsigned lane = threadIdx.x;
      const rns_warp w;
      auto record = [&](unsigned op, const rns_point &p) {
        const int32_t words[6] = {p.x.a, p.x.b, p.y.a, p.y.b, p.z.a, p.z.b};
        for (int i = 0; i < 6; i++)
          out[at + (op * 32 + lane) * 6 + i] = (uint32_t)words[i];
      };
      const rns_point p = w.load(curve::from_jacobian(pair[0])), q = w.load(curve::from_jacobian(pair[1]));
      record(0, p);
      record(1, q);
      w.put(stored, p);
      __syncwarp();
      record(2, w.get(stored));
      record(3, w.doubled(p));
      rns_point sum;
      const bool holds = w.added(p, q, sum);
      record(4, sum);
      out[at + OPERATIONS * 6 * 32 + lane] = holds;
    });
  }
  return out;
}

std::vector<uint32_t> constants() {
  std::vector<uint32_t> out;
  for (const split_power &p : split_powers) {
    out.insert(out.end(), p.a, p.a + 4);
    out.insert(out.end(), p.b, p.b + 4);
    out.push_back(p.a_negative);
    out.push_back(p.b_negative);
  }
  const fe beta = endomorphism_beta();
  out.insert(out.end(), beta.l, beta.l + 8);
  return out;
}

std::vector<uint32_t> inverses(const std::vector<uint32_t> &in) {
  std::vector<uint32_t> out(in.size());
  for (size_t k = 0; k + 64 <= in.size(); k += 64)
    emulation::run(1, 32, false, [&](unsigned) {
      const unsigned lane = threadIdx.x;
      fe a;
      std::memcpy(&a, in.data() + k + lane / 4 * 8, sizeof(a));
      const fe r = inverse_group4(a);
      fe first;
      for (int i = 0; i < 8; i++)
        first.l[i] = __shfl_sync(0xffffffffu, r.l[i], lane & 28);
      if (std::memcmp(&first, &r, sizeof(r)) != 0)
        emulation::fail("a group's lanes differ", "inverse_group4");
      std::memcpy(out.data() + k + lane / 4 * 8, &r, sizeof(r));
    });
  return out;
}

} // namespace

int main(int argc, char **argv) {
  if (argc < 4)
    return 2;
  const std::vector<uint32_t> in = read_words(argv[2]);
  const std::string mode = argv[1];
  write_words(argv[3], mode == "sum" ? sums(in, argc > 4) : mode == "lanes" ? lanes(in) : mode == "constants" ? constants() : inverses(in));
  return 0;
}
