// CPU check of the warp-wide residue-number-system products
// (era-bellman-cuda_b200/csrc/rns.cuh): the lanes of a group run one after
// another, with the device's per-lane arithmetic and tables.  Test
// infrastructure: loaded by tests/ via ctypes.
#include "rns.cuh"

#include <cstring>

using namespace msm_b200;

namespace {
constexpr int N = rns::RESIDUES;
struct value {
  rns::residues lane[N];
};

// runs F(lane, extend) for every lane; an extension's inputs come from a first
// run of every lane up to that point, so each of the two extensions repeats
// the group
template <class F> void run_group(F f) {
  int32_t first[N] = {}, second[N] = {};
  for (int pass = 0; pass < 3; pass++)
    for (int i = 0; i < N; i++) {
      int call = 0;
      f(i, [&](int32_t v, auto sum) {
        int32_t *inputs = call++ == 0 ? first : second;
        if (pass == (inputs == first ? 0 : 1))
          inputs[i] = v;
        for (int k = 0; k < N; k++)
          sum(k, inputs[k]);
      });
    }
}
} // namespace

extern "C" {

int rns_residues() { return N; }
void rns_moduli(int32_t *a, int32_t *b) {
  for (int i = 0; i < N; i++) {
    a[i] = rns::TABLES.lane[i].mod_a;
    b[i] = rns::TABLES.lane[i].mod_b;
  }
}

// stored residues (2 N words: base a, then base b) of an eight-word integer
void rns_from_words(const uint32_t *w, int32_t *out) {
  for (int i = 0; i < N; i++) {
    const rns::residues r = rns::from_words(rns::TABLES.lane[i], w);
    out[i] = r.a;
    out[N + i] = r.b;
  }
}

void rns_product(const int32_t *x, const int32_t *y, int32_t *out) {
  run_group([&](int i, auto extend) {
    const rns::residues r = rns::product(rns::TABLES.lane[i], {x[i], x[N + i]}, {y[i], y[N + i]}, extend);
    out[i] = r.a;
    out[N + i] = r.b;
  });
}

// eight words of p + (x y + q p) / A
void rns_product_words(const int32_t *x, const int32_t *y, uint32_t *out) {
  int64_t column[N];
  run_group([&](int i, auto extend) { column[i] = rns::product_column(rns::TABLES.lane[i], {x[i], x[N + i]}, {y[i], y[N + i]}, extend); });
  int64_t carry = 0;
  for (int k = 0; k < 8; k++) {
    carry += column[k];
    out[k] = (uint32_t)carry;
    carry >>= 32;
  }
}

// the warp's test for a multiple of p: the lanes' words and-ed
uint32_t rns_multiples(const int32_t *x) {
  uint32_t all = 0xffffffffu;
  for (int i = 0; i < N; i++)
    all &= rns::multiples_of_p(rns::TABLES.lane[i], {x[i], x[N + i]});
  return all;
}

void rns_constants(int32_t *enter, int32_t *leave) {
  for (int i = 0; i < N; i++) {
    enter[i] = rns::TABLES.lane[i].enter_a;
    enter[N + i] = rns::TABLES.lane[i].enter_b;
    leave[i] = rns::TABLES.lane[i].leave_a;
    leave[N + i] = rns::TABLES.lane[i].leave_b;
  }
}
}
