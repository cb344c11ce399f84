// Field products of Fq spread over the lanes of a warp, for one dependent
// chain of point doublings (the final sum of an MSM's 254 results).
//
// One thread's Montgomery product is a chain of some 136 wide multiplies (801
// cycles on a B200 with one warp per scheduler), and its carries leave nothing
// to split over lanes.  In a residue number system a value is held by its
// residues modulo small coprime moduli, and every step of a product works on
// all residues at once, one lane each, without carries: about 300 cycles.
// The method is Montgomery multiplication with two bases of moduli and base
// extensions (S. Kawamura, M. Koike, F. Sano, A. Shimbo, "Cox-Rower
// architecture for fast parallel Montgomery multiplication", EUROCRYPT 2000).
//
// Bases a_0..a_9 and b_0..b_9: the twenty largest primes below 2^27,
// alternately; A and B are their products (just under 2^270, p < 2^254).  Lane
// i < 10 of a group holds a value's residues modulo a_i and b_i; a warp holds
// three groups (lanes 30 and 31 repeat lanes 20 and 21), so three independent
// products run at once.  A product of x and y gives r = (x y + q p) / A with
// q = -x y / p (mod A):
//   q's mixed terms   xi_i = x y (-1/p) (A / a_i)^-1 mod a_i
//   to base b         zeta_j = r (B / b_j)^-1 mod b_j,
//                     r = x y / A + sum_i xi_i (A / a_i) p / A
//   back to base a    r = sum_j zeta_j (B / b_j) - alpha B       mod a_i,
//                     alpha = the nearest integer to sum_j zeta_j / b_j
// The first sum is left as it is, so r may be off by a few multiples of p
// (|r| < 6.5 p + |x y| / A); the second is exact, because |r| / B < 2^-10 and
// sum_j zeta_j 2^-27 is within 10 * 2^-17 of sum_j zeta_j / b_j.
//
// Residues are signed and not fully reduced: a stored residue is v 2^32 modulo
// the modulus (word-level Montgomery form), and a product's output words stay
// below 1.1 * 2^26 in magnitude (1.25 by the bounds: each word product adds at
// most half a modulus to what 2^-32 leaves of its argument), so sums of up to
// 20 outputs fit the 32-bit words that go into the next product.
#pragma once

#include "bn254_field.cuh"

namespace msm_b200 {
namespace rns {

constexpr unsigned RESIDUES = 10; // per base and group
constexpr unsigned GROUPS = 3;    // per warp

// What lane i of a group needs; all "mod" values are centred.
struct lane_table {
  int32_t mod_a, mod_b;           // a_i, b_i
  uint32_t ninv_a, ninv_b;        // -1 / modulus mod 2^32
  int32_t xi;                     // (-1/p) (A / a_i)^-1 mod a_i
  int32_t keep;                   // (B / b_i)^-1 / A mod b_i
  int32_t value;                  // (B / b_i) 2^64 mod b_i
  int32_t whole;                  // -B 2^64 mod a_i
  int32_t p_b;                    // (B / b_i)^-1 p 2^32 mod b_i
  uint32_t p_a;                   // p as a stored residue modulo a_i, in [0, a_i)
  int32_t to_b[RESIDUES];         // (B / b_i)^-1 (A / a_k) p / A 2^32 mod b_i
  int32_t to_a[RESIDUES];         // (B / b_k) 2^64 mod a_i
  uint32_t word_a[8], word_b[8];  // 2^(32 k + 64) mod a_i, b_i, in [0, modulus)
  int32_t enter_a, enter_b;       // the constant A^2 2^-256 mod p, as a stored residue
  int32_t leave_a, leave_b;       // the constant 2^256 mod p, as a stored residue
  uint32_t column[RESIDUES];      // 32-bit word i of B / b_k (i < 8)
  uint32_t column_whole, column_p; // word i of B mod 2^256 and of p
};

struct tables {
  lane_table lane[RESIDUES];
};

// ---------------------------------------------------------------------------
// the tables, from the moduli alone (compile time)
// ---------------------------------------------------------------------------
struct table_builder {
  uint32_t a[RESIDUES], b[RESIDUES];

  static constexpr uint32_t mulmod(uint32_t x, uint32_t y, uint32_t m) { return (uint32_t)((uint64_t)x * y % m); }
  static constexpr uint32_t power(uint32_t x, uint32_t e, uint32_t m) {
    uint32_t r = 1;
    for (; e; e >>= 1, x = mulmod(x, x, m))
      if (e & 1)
        r = mulmod(r, x, m);
    return r;
  }
  static constexpr uint32_t inverse(uint32_t x, uint32_t m) { return power(x % m, m - 2, m); } // m prime
  static constexpr int32_t centred(uint32_t x, uint32_t m) { return x > m / 2 ? (int32_t)x - (int32_t)m : (int32_t)x; }
  static constexpr uint32_t two_to(unsigned bits, uint32_t m) { return power(2, bits, m); }
  static constexpr uint32_t negative_inverse(uint32_t m) { // -1/m mod 2^32 by Newton's iteration
    uint32_t x = m;
    for (int k = 0; k < 5; k++)
      x *= 2 - m * x;
    return 0 - x;
  }
  // product of the moduli of `base` except index `skip`, modulo m
  static constexpr uint32_t product(const uint32_t *base, unsigned skip, uint32_t m) {
    uint32_t r = 1;
    for (unsigned k = 0; k < RESIDUES; k++)
      if (k != skip)
        r = mulmod(r, base[k] % m, m);
    return r;
  }
  static constexpr uint32_t words_mod(const uint32_t *w, uint32_t m) {
    uint64_t r = 0;
    for (int k = 8; k-- > 0;)
      r = ((r << 32) | w[k]) % m;
    return (uint32_t)r;
  }

  struct words {
    uint32_t l[8];
  };
  static constexpr uint32_t prime(int i) { return bn254::fq_params::mod(i); }
  // x y mod p for a small y < 2^27: 32-bit words, then subtractions of p 2^k
  static constexpr words mul_small_mod_p(const words &x, uint32_t y) {
    words r{};
    for (int bit = 26; bit >= 0; bit--) {
      r = add_mod_p(r, r);
      if ((y >> bit) & 1)
        r = add_mod_p(r, x);
    }
    return r;
  }
  static constexpr words add_mod_p(const words &x, const words &y) {
    words s{}, d{};
    uint64_t c = 0;
    for (int i = 0; i < 8; i++) {
      c += (uint64_t)x.l[i] + y.l[i];
      s.l[i] = (uint32_t)c;
      c >>= 32;
    }
    int64_t borrow = 0;
    for (int i = 0; i < 8; i++) {
      borrow += (int64_t)s.l[i] - prime(i);
      d.l[i] = (uint32_t)borrow;
      borrow >>= 32;
    }
    return borrow < 0 ? s : d;
  }
  static constexpr words half_mod_p(const words &x) {
    words s = x;
    uint64_t c = 0;
    if (x.l[0] & 1)
      for (int i = 0; i < 8; i++) {
        c += (uint64_t)x.l[i] + prime(i);
        s.l[i] = (uint32_t)c;
        c >>= 32;
      }
    words r{};
    for (int i = 0; i < 8; i++)
      r.l[i] = (s.l[i] >> 1) | ((i < 7 ? s.l[i < 7 ? i + 1 : 7] : 0u) << 31);
    return r; // x + p < 2^256
  }

  constexpr tables build() const {
    tables t{};
    uint32_t p[8] = {};
    words one{};
    one.l[0] = 1;
    for (int k = 0; k < 8; k++)
      p[k] = prime(k);
    words enter = one, leave = one;
    for (int twice = 0; twice < 2; twice++)
      for (unsigned k = 0; k < RESIDUES; k++)
        enter = mul_small_mod_p(enter, a[k]);
    for (int k = 0; k < 256; k++) {
      enter = half_mod_p(enter);
      leave = add_mod_p(leave, leave);
    }
    for (unsigned i = 0; i < RESIDUES; i++) {
      lane_table &l = t.lane[i];
      const uint32_t ma = a[i], mb = b[i];
      l.mod_a = (int32_t)ma;
      l.mod_b = (int32_t)mb;
      l.ninv_a = negative_inverse(ma);
      l.ninv_b = negative_inverse(mb);
      const uint32_t inv_p = inverse(words_mod(p, ma), ma);
      l.xi = centred(mulmod(ma - inv_p, inverse(product(a, i, ma), ma), ma), ma);
      const uint32_t inv_a = inverse(product(a, RESIDUES, mb), mb);
      const uint32_t others = product(b, i, mb), zeta = inverse(others, mb);
      l.keep = centred(mulmod(zeta, inv_a, mb), mb);
      l.value = centred(mulmod(others, two_to(64, mb), mb), mb);
      l.whole = centred(ma - mulmod(product(b, RESIDUES, ma), two_to(64, ma), ma), ma);
      const uint32_t zeta_p = mulmod(mulmod(words_mod(p, mb), zeta, mb), two_to(32, mb), mb);
      l.p_b = centred(zeta_p, mb);
      l.p_a = mulmod(words_mod(p, ma), two_to(32, ma), ma);
      for (unsigned k = 0; k < RESIDUES; k++) {
        l.to_b[k] = centred(mulmod(mulmod(product(a, k, mb), inv_a, mb), zeta_p, mb), mb);
        l.to_a[k] = centred(mulmod(product(b, k, ma), two_to(64, ma), ma), ma);
      }
      for (unsigned k = 0; k < 8; k++) {
        l.word_a[k] = two_to(32 * k + 64, ma);
        l.word_b[k] = two_to(32 * k + 64, mb);
      }
      l.enter_a = centred(mulmod(words_mod(enter.l, ma), two_to(32, ma), ma), ma);
      l.enter_b = centred(mulmod(words_mod(enter.l, mb), two_to(32, mb), mb), mb);
      l.leave_a = centred(mulmod(words_mod(leave.l, ma), two_to(32, ma), ma), ma);
      l.leave_b = centred(mulmod(words_mod(leave.l, mb), two_to(32, mb), mb), mb);
    }
    // words of B / b_k and of B, modulo 2^256
    for (unsigned k = 0; k <= RESIDUES; k++) {
      words v = one;
      for (unsigned j = 0; j < RESIDUES; j++)
        if (j != k) {
          uint64_t c = 0;
          for (int i = 0; i < 8; i++) {
            c += (uint64_t)v.l[i] * b[j];
            v.l[i] = (uint32_t)c;
            c >>= 32;
          }
        }
      for (unsigned i = 0; i < 8; i++) {
        if (k < RESIDUES)
          t.lane[i].column[k] = v.l[i];
        else
          t.lane[i].column_whole = v.l[i];
        t.lane[i].column_p = p[i];
      }
    }
    return t;
  }
};

// 2^27 minus the twenty largest primes below 2^27, alternately for a and b
constexpr uint32_t below(uint32_t k) { return (1u << 27) - k; }
constexpr table_builder BASES = {
    {below(39), below(111), below(135), below(199), below(231), below(241), below(289), below(319), below(327), below(367)},
    {below(79), below(115), below(187), below(219), below(235), below(261), below(291), below(325), below(361), below(375)},
};
constexpr tables TABLES = BASES.build();

// ---------------------------------------------------------------------------
// one lane's arithmetic (also run on the host by the CPU tests)
// ---------------------------------------------------------------------------
// t 2^-32 modulo m, for |t| < 2^62: |result| <= |t| 2^-32 + m / 2
BN_HD int32_t word_redc(int64_t t, int32_t m, uint32_t ninv) {
  const int32_t k = (int32_t)((uint32_t)t * ninv);
  return (int32_t)((t + (int64_t)k * m) >> 32);
}

// a lane's two residues of a value
struct residues {
  int32_t a, b;
};

BN_HD residues operator+(const residues &x, const residues &y) { return {x.a + y.a, x.b + y.b}; }
BN_HD residues operator-(const residues &x, const residues &y) { return {x.a - y.a, x.b - y.b}; }
BN_HD residues scaled(const residues &x, int32_t k) { return {x.a * k, x.b * k}; }

// stored residues of the integer in eight 32-bit words
BN_HD residues from_words(const lane_table &t, const uint32_t *w) {
  uint64_t sa = 0, sb = 0; // eight terms below 2^59
  for (int k = 0; k < 8; k++) {
    sa += (uint64_t)w[k] * t.word_a[k];
    sb += (uint64_t)w[k] * t.word_b[k];
  }
  return {word_redc((int64_t)sa, t.mod_a, t.ninv_a), word_redc((int64_t)sb, t.mod_b, t.ninv_b)};
}

// the product's steps: EXTEND(value, sum) calls sum(k, value of lane k) for
// every lane k of the group
template <class EXTEND> BN_HD residues product(const lane_table &t, const residues &x, const residues &y, EXTEND extend) {
  const int32_t ta = word_redc((int64_t)x.a * y.a, t.mod_a, t.ninv_a), tb = word_redc((int64_t)x.b * y.b, t.mod_b, t.ninv_b);
  const int32_t xi = word_redc((int64_t)ta * t.xi, t.mod_a, t.ninv_a);
  int64_t sum = (int64_t)tb * t.keep;
  extend(xi, [&](int k, int32_t v) { sum += (int64_t)v * t.to_b[k]; });
  const int32_t zeta = word_redc(sum, t.mod_b, t.ninv_b);
  int64_t back = 0;
  int32_t all = 0;
  extend(zeta, [&](int k, int32_t v) {
    back += (int64_t)v * t.to_a[k];
    all += v;
  });
  back += (int64_t)((all + (1 << 26)) >> 27) * t.whole;
  return {word_redc(back, t.mod_a, t.ninv_a), word_redc((int64_t)zeta * t.value, t.mod_b, t.ninv_b)};
}

// A product's output is a multiple k p, |k| <= 6 (zero in the field), iff
// every lane of the group finds its residue equal for the same k: bit k of the
// result says so for this lane's residue and k, bit 16 + k for -k.
BN_HD uint32_t multiples_of_p(const lane_table &t, const residues &r) {
  const uint32_t m = (uint32_t)t.mod_a, c = (uint32_t)(r.a < 0 ? r.a + t.mod_a : r.a);
  uint32_t found = 0, kp = 0;
  for (unsigned k = 0; k <= 6; k++) {
    found |= (uint32_t)(c == kp) << k | (uint32_t)(c == (kp ? m - kp : 0)) << (16 + k);
    kp += t.p_a;
    kp = kp >= m ? kp - m : kp;
  }
  return found;
}

// Word column `lane` (lane < 8) of p + (x y + q p) / A, q taken nearest to
// zero so that the value lies in (0, 2 p): the eight columns, carried, give
// its 32-bit words.
template <class EXTEND> BN_HD int64_t product_column(const lane_table &t, const residues &x, const residues &y, EXTEND extend) {
  const int32_t ta = word_redc((int64_t)x.a * y.a, t.mod_a, t.ninv_a), tb = word_redc((int64_t)x.b * y.b, t.mod_b, t.ninv_b);
  const int32_t xi = word_redc((int64_t)ta * t.xi, t.mod_a, t.ninv_a);
  int64_t sum = (int64_t)tb * t.keep;
  int32_t all = 0;
  extend(xi, [&](int k, int32_t v) {
    sum += (int64_t)v * t.to_b[k];
    all += v;
  });
  sum -= (int64_t)((all + (1 << 26)) >> 27) * t.p_b; // q mod A: every whole A taken out of q is one p of r
  const int32_t zeta = word_redc(sum, t.mod_b, t.ninv_b) + t.mod_b; // positive: one more whole B per term
  int64_t column = t.column_p;
  all = 0;
  extend(zeta, [&](int k, int32_t v) {
    column += (int64_t)((uint64_t)(uint32_t)v * t.column[k]);
    all += v;
  });
  return column - (int64_t)((all + (1 << 26)) >> 27) * t.column_whole;
}

} // namespace rns
} // namespace msm_b200
