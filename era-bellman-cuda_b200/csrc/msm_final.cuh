// The caller-side final reduction of an MSM on the GPU: sum over i < 254 of
// 2^i R_i of the 254 per-bit Jacobian results, written as one canonical
// affine point (standard form, fully reduced, infinity flagged).  The
// reference leaves this Horner pass to its callers, on the host
// (src/bellman-cuda.h:496-505; tests/msm_test.cu:116-126).
//
// Doublings are what the sum costs: 2^253 R_253 taken plainly needs 253
// dependent ones, whatever the order of the additions.  Here the chain is about
// half as long, because BN254 (j = 0) has the endomorphism phi(x, y) =
// (beta x, y) = lambda (x, y), and with it any multiple k P is a P + b phi(P)
// for some |a|, |b| < 2^126 (R. Gallant, R. Lambert, S. Vanstone, "Faster point
// multiplication on elliptic curves with efficient endomorphisms", CRYPTO
// 2001).  A cluster of eight blocks works in three steps:
//   groups   V_g = sum of 2^i R_(16 g + i) over 16 bits, two groups per block,
//            as a pairwise tree over the bits (15 doublings, 4 additions deep)
//   digits   2^(16 g) V_g = a_g V_g + b_g phi(V_g) for g >= 8, so the sum is
//            that of 2^j Q_j over j < 126, Q_j adding the V_g and phi(V_g)
//            whose a_g or b_g has bit j (and V_(j / 16) itself for j = 0, 16,
//            ..., 112); 16 bits j per block, at most 16 terms each
//   bits     the sum of 2^j Q_j, a pairwise tree over the bits: 16 in each
//            block, the last three levels in the first block
// so 15 + 127 doublings are dependent, and about 12 additions between them.
//
// Levels of one or two doublings share each one between four lanes
// (dbl_group4).  The others give a warp to each point and double and add in a
// residue number system (rns.cuh), where a product of the whole warp takes less
// than half of one thread's: about 1,030 cycles per doubling on a B200 against
// 3,236 for dbl_group4.  The affine conversion takes one inversion
// (inverse_group4).  One final sum takes 307 K cycles, 0.157 ms on a B200 (0.161
// per call, one behind the other), of a batched instance's results (20 bits)
// 0.068 ms.  Measured on the way there: 0.230 ms in
// one block without phi, the 253 doublings one after another; 0.189 ms with the
// steps' code repeated; 0.169 ms with four-lane additions (and a conversion out
// of the residues and back) at every level.
// The kernel's device code is in this header, without anything that only nvcc
// knows beyond the warp and block intrinsics, so that the CPU tests can run it
// with those emulated.
#pragma once

#include "bellman-cuda-b200.h"
#include "msm_group4.cuh"
#include "rns.cuh"

namespace msm_b200 {

constexpr unsigned FINAL_BLOCKS = 8; // one cluster
constexpr unsigned FINAL_PARTS = 16; // per block: pairs of results, then bits of the sum
constexpr unsigned FINAL_THREADS = 256, FINAL_WARPS = FINAL_THREADS / 32;
constexpr unsigned FINAL_RNS_DOUBLINGS = 4; // levels of at least this many doublings take a warp per point
constexpr unsigned GROUP_BITS = 16, GROUPS = FINAL_BLOCKS * 2, SPLIT_GROUPS = GROUPS / 2; // groups g >= SPLIT_GROUPS are split by phi
static_assert(FINAL_BLOCKS * FINAL_PARTS * 2 >= RESULT_BITS && GROUPS * GROUP_BITS >= RESULT_BITS, "all results");

// 2^(16 g) = (-1)^a_negative a + (-1)^b_negative b lambda modulo the group
// order for g = 8..15, lambda = 0xb3c4d79d41a917585bfc41088d8daaa78b17ea66b99c90dd
struct split_power {
  uint32_t a[4], b[4];
  bool a_negative, b_negative;
};
__device__ const split_power split_powers[SPLIT_GROUPS] = {
    {{0xdbbdb5ea, 0xe8363d57, 0x228f4c05, 0x2164fb6e}, {0x29a427c6, 0x13a64ad1, 0x00000001, 0x00000000}, false, true},
    {{0xc9e237e5, 0x539f4c9e, 0x75c1faee, 0x06ebdd48}, {0xdb8b788d, 0x6ba77562, 0x00013d00, 0x00000000}, true, true},
    {{0xa24c59e7, 0xf85004a5, 0x0a6de4a2, 0x267f96d2}, {0x8c8a719f, 0x915e63d2, 0x3d006315, 0x00000001}, true, true},
    {{0x0b0af5fc, 0xd6058217, 0xf8e2c5d6, 0x13a5b87b}, {0xd7e617dc, 0x6f7e2430, 0x631561b2, 0x00013d00}, true, true},
    {{0x9768ca72, 0x62da6d02, 0x5343de7f, 0x3540c909}, {0xc9c5e8eb, 0xe101e709, 0x6a76b6cb, 0x10e823c5}, false, false},
    {{0xa407db0b, 0xdb74ec20, 0x9daeb672, 0x109889d3}, {0x23f8f66c, 0x72aec238, 0x5407a725, 0x0f4befa4}, true, true},
    {{0x22dd5037, 0xecc76690, 0xae9818db, 0x18d59a49}, {0x9d7fbb5c, 0x93928275, 0x6100ad02, 0x18668fff}, false, false},
    {{0x4941ded8, 0x1f927622, 0xdb80324c, 0x221b5563}, {0x772a38ab, 0x2d4e87c5, 0x710052ca, 0x211ca5f3}, true, false},
};

// beta 2^256 mod p, beta = 0x59e26bcea0d48bacd4f263f1acdb5c4f5763473177fffffe
__device__ __forceinline__ fe endomorphism_beta() {
  return {{0xd782e155, 0x71930c11, 0xffbe3323, 0xa6bb947c, 0xd4741444, 0xaa303344, 0x26594943, 0x2c3b3f0d}};
}

__device__ const rns::tables rns_tables = rns::TABLES;

// Doublings and additions of points by a whole warp.  All lanes hold their
// residues of X and Y of a Jacobian point, the lanes of groups 1 and 2 those of
// Z (x = X / Z^2, y = Y / Z^3; infinity: Z = 0 mod p).
struct rns_point {
  rns::residues x, y, z;
};
// the same between steps, one entry per residue index
struct rns_stored {
  rns::residues x[rns::RESIDUES], y[rns::RESIDUES], z[rns::RESIDUES];
};

struct rns_warp {
  unsigned group, index; // of this lane: 0..2, and its residue 0..9
  rns::lane_table t;

  __device__ __forceinline__ rns_warp() {
    const unsigned lane = threadIdx.x & 31;
    group = min(lane / rns::RESIDUES, rns::GROUPS - 1);
    index = lane % rns::RESIDUES; // lanes 30 and 31 hold what lanes 20 and 21 hold: group 2, residues 0 and 1
    // every word through a volatile move: the table stays in registers instead
    // of being read again inside the doubling loop
    const uint32_t *from = reinterpret_cast<const uint32_t *>(rns_tables.lane + index);
    uint32_t *to = reinterpret_cast<uint32_t *>(&t);
#pragma unroll
    for (unsigned k = 0; k < sizeof(rns::lane_table) / 4; k++)
#if defined(__CUDA_ARCH__)
      asm volatile("mov.b32 %0, %1;" : "=r"(to[k]) : "r"(from[k]));
#else
      to[k] = from[k];
#endif
  }
  __device__ __forceinline__ auto extension() const {
    return [first = group * rns::RESIDUES](int32_t v, auto sum) {
#pragma unroll
      for (int k = 0; k < (int)rns::RESIDUES; k++)
        sum(k, __shfl_sync(0xffffffffu, v, first + k));
    };
  }
  __device__ __forceinline__ rns::residues product(const rns::residues &x, const rns::residues &y) const {
    return rns::product(t, x, y, extension());
  }
  // group g's residues, in every lane
  __device__ __forceinline__ rns::residues from_group(const rns::residues &v, unsigned g) const {
    const unsigned src = g * rns::RESIDUES + index;
    return {__shfl_sync(0xffffffffu, v.a, src), __shfl_sync(0xffffffffu, v.b, src)};
  }
  __device__ __forceinline__ rns::residues pick(const rns::residues &g0, const rns::residues &g1, const rns::residues &g2) const {
    return {group == 0 ? g0.a : group == 1 ? g1.a : g2.a, group == 0 ? g0.b : group == 1 ? g1.b : g2.b};
  }

  // The point of an XYZZ value: X ZZ^2, Y ZZZ^2, Z = ZZZ (as to_jacobian).  A
  // coordinate c comes as the integer c 2^256 mod p and a stored value stands
  // for its integer / A, so with k = 2^256 / A the loaded coordinates carry a
  // factor k; X is freed of it by one product, which leaves (X k^2, Y k^3,
  // Z k): the same point.
  __device__ __forceinline__ rns_point load(const xyzz &p) const {
    const fe &c0 = group == 0 ? p.zz : group == 1 ? p.zzz : p.x, &c1 = group == 0 ? p.zzz : p.y;
    const rns::residues u = rns::from_words(t, c0.l), v = rns::from_words(t, c1.l);
    const rns::residues enter = {t.enter_a, t.enter_b};
    const rns::residues s = product(u, pick(u, u, enter)); // ZZ^2 | ZZZ^2 | X
    const rns::residues x = from_group(s, 2);
    const rns::residues m = product(pick(x, v, v), s); // X ZZ^2 | Y ZZZ^2 |
    return {from_group(m, 0), from_group(m, 1), from_group(v, 0)};
  }

  // 2 p (dbl-2009-l with Z3 = 2 Y Z), three products deep:
  //   A = X^2 | B = Y^2 | B;  E^2 | S = X B | B^2, E = 3 A;
  //   E (4 S - X3) with X3 = E^2 - 8 S | Y Z |;  Y3 = that - 8 B^2.
  // B is computed twice so that nothing moves between the first two products.
  // In units of the largest product output the words of X3 and Y3 stay below
  // 9, of 4 S - X3 below 13, of E below 3; as multiples of p (outputs below
  // 6.5): 59, 85 and 20, so |x y| / A < 0.1 p in every product.
  __device__ __forceinline__ rns_point doubled(const rns_point &p) const {
    const rns::residues xy = pick(p.x, p.y, p.y);
    const rns::residues r1 = product(xy, xy);
    const rns::residues e = {group == 0 ? 3 * r1.a : r1.a, group == 0 ? 3 * r1.b : r1.b}; // E | B | B
    const rns::residues r2 = product(e, pick(e, p.x, e));
    const rns::residues S = from_group(r2, 1);
    const rns::residues D = rns::scaled(S, 4), x = r2 - rns::scaled(S, 8); // group 0
    const rns::residues r3 = product(pick(e, p.y, p.y), pick(D - x, p.z, p.z));
    const rns::residues y = r3 - rns::scaled(from_group(r2, 2), 8);
    return {from_group(x, 0), from_group(y, 0), rns::scaled(r3, 2)};
  }

  // p + q, six products deep (add-2007-bl without its doublings):
  //   Z1^2 | Z2^2 | Z1 Z2;  U1 = X1 Z2^2 | U2 = X2 Z1^2 | Z2^3;
  //   S1 = Y1 Z2^3 | Z1^3 | H^2, H = U2 - U1;  S2 = Y2 Z1^3 | H^3 | V = U1 H^2;
  //   R^2 | S1 H^3 | Z3 = Z1 Z2 H, R = S2 - S1;
  //   R (V - X3) with X3 = R^2 - H^3 - 2 V;  Y3 = that - S1 H^3.
  // false when Z3 is zero (an infinite operand, equal or opposite points): the
  // formula does not hold then.  Sums stay below those of doubled().
  __device__ __forceinline__ bool added(const rns_point &p, const rns_point &q, rns_point &sum) const {
    const rns::residues z1 = from_group(p.z, 1), z2 = from_group(q.z, 1);
    const rns::residues r1 = product(pick(z1, z2, z1), pick(z1, z2, z2));
    const rns::residues zz1 = from_group(r1, 0), zz2 = from_group(r1, 1);
    const rns::residues r2 = product(pick(p.x, q.x, z2), pick(zz2, zz1, zz2));
    const rns::residues U1 = from_group(r2, 0), H = from_group(r2, 1) - U1;
    const rns::residues r3 = product(pick(p.y, z1, H), pick(from_group(r2, 2), zz1, H));
    const rns::residues HH = from_group(r3, 2), S1 = from_group(r3, 0);
    const rns::residues r4 = product(pick(q.y, H, U1), pick(from_group(r3, 1), HH, HH));
    const rns::residues R = from_group(r4, 0) - S1, HHH = from_group(r4, 1), V = from_group(r4, 2);
    const rns::residues r5 = product(pick(R, S1, r1), pick(R, HHH, H));
    const uint32_t zero = __reduce_and_sync(0xffffffffu, group == 2 ? rns::multiples_of_p(t, r5) : 0xffffffffu);
    const rns::residues x = from_group(r5, 0) - HHH - rns::scaled(V, 2);
    const rns::residues y = product(R, V - x) - from_group(r5, 1);
    sum = {x, y, from_group(r5, 2)};
    return (zero & 0x007f007fu) == 0;
  }

  __device__ __forceinline__ void put(rns_stored &to, const rns_point &p) const {
    const rns::residues z = from_group(p.z, 1);
    if ((threadIdx.x & 31) < rns::RESIDUES) {
      to.x[index] = p.x;
      to.y[index] = p.y;
      to.z[index] = z;
    }
  }
  __device__ __forceinline__ rns_point get(const rns_stored &from) const {
    return {from.x[index], from.y[index], from.z[index]};
  }

  // X, Y, Z as Montgomery-form field elements in (0, 2p), the same in every
  // lane; columns: 24 words of shared memory of this warp
  __device__ __forceinline__ jacobian store(const rns_point &p, int64_t (*columns)[8]) const {
    const rns::residues leave = {t.leave_a, t.leave_b};
    const int64_t column = rns::product_column(t, pick(p.x, p.y, p.z), leave, extension());
    const unsigned lane = threadIdx.x & 31;
    if (lane < rns::GROUPS * rns::RESIDUES && index < 8)
      columns[group][index] = column;
    __syncwarp();
    fe c; // lane g < 3 carries coordinate g
    int64_t carry = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      carry += columns[min(lane, rns::GROUPS - 1)][k];
      c.l[k] = (uint32_t)carry;
      carry >>= 32;
    }
    __syncwarp();
    return {shfl_fe(c, 0), shfl_fe(c, 1), shfl_fe(c, 2)};
  }
};

struct final_shared {
  xyzz part[FINAL_PARTS];
  xyzz group[GROUPS];            // every block's two group sums
  xyzz choice[SPLIT_GROUPS][3];  // of a split group, signed: V, phi(V), their sum
  rns_stored stored[FINAL_PARTS]; // parts between two steps of a warp per point
  bool empty[FINAL_PARTS];        // infinite ones among them
  int64_t columns[FINAL_WARPS][rns::GROUPS][8];
};

// copies one XYZZ point from block `rank`'s shared memory (8 lanes)
template <class CLUSTER> __device__ __forceinline__ void copy_remote(CLUSTER &cluster, xyzz *to, xyzz *from, unsigned rank, unsigned lane8) {
  reinterpret_cast<uint4 *>(to)[lane8] = reinterpret_cast<const uint4 *>(cluster.map_shared_rank(from, rank))[lane8];
}

// The digits step: part[b] = Q_(16 rank + b) from sh.group.  Sixteen lanes per
// bit, four per share; share s takes the split groups 2 s and 2 s + 1.
__device__ __forceinline__ void sum_digits(final_shared &sh, unsigned rank) {
  const unsigned t = threadIdx.x, j = rank * FINAL_PARTS + (t >> 4), share = (t >> 2) & 3;
  auto chosen = [&](unsigned g) {
    const split_power &power = split_powers[g];
    const unsigned a = (power.a[j >> 5] >> (j & 31)) & 1, b = (power.b[j >> 5] >> (j & 31)) & 1;
    return a + b ? sh.choice[g][a + 2 * b - 1] : curve::infinity();
  };
  xyzz acc = curve::infinity(), p = curve::infinity();
  // every addition of the step through one place: the code is too large to
  // repeat (each copy is fetched once per call)
#pragma unroll 1
  for (unsigned pass = 0; pass < 5; pass++) {
    const bool first_warp = t < 32, run = first_warp || (pass != 0 && pass != 4);
    if (pass == 0) {
      if (first_warp) {
        const unsigned g = t >> 2;
        acc = sh.group[SPLIT_GROUPS + g];
        p = acc;
        p.x = fq::mul(p.x, endomorphism_beta());
        acc.y = select_fe(split_powers[g].a_negative, fq::neg(acc.y), acc.y);
        p.y = select_fe(split_powers[g].b_negative, fq::neg(p.y), p.y);
        if ((t & 3) == 0) {
          sh.choice[g][0] = acc;
          sh.choice[g][1] = p;
        }
      }
    } else if (pass == 1) {
      acc = chosen(2 * share);
      p = chosen(2 * share + 1);
    } else if (pass < 4) {
      p = shfl_xyzz(acc, (t & 31) ^ (1u << pass));
    } else { // bit 16 rank also takes the unsplit group of that weight
      p = select_xyzz(t < 4, sh.group[rank], curve::infinity());
    }
    if (run && __any_sync(0xffffffffu, !curve::is_inf(p)))
      acc = add_group4(acc, p);
    if (pass == 0) {
      if (first_warp && (t & 3) == 0)
        sh.choice[t >> 2][2] = acc;
      __syncthreads();
    }
  }
  if ((t & 15) == 0)
    sh.part[t >> 4] = acc;
  __syncthreads();
}

// The whole sum, by every thread of the cluster; `point` is written by the
// first block.
template <class CLUSTER>
__device__ __forceinline__ void final_sum_block(final_shared &sh, CLUSTER cluster, const jacobian *__restrict__ results,
                                                msm_b200_affine_point *point) {
  const unsigned t = threadIdx.x, role = t & 3, rank = cluster.block_rank();
  const rns_warp w;
  // One tree level per step: part[g 2^L] += 2^n part[g 2^L + 2^(L-1)].  Step 0
  // forms the pairs R_2p + 2 R_2p+1; steps 1..3 are the groups' levels, 4..7
  // the bits' levels, 8..10 the last three in block 0.  One loop, so that every
  // step runs the same code (copies per step cost an instruction fetch each).
#pragma unroll 1
  for (unsigned step = 0; step < 11; step++) {
    if (step == 4) {
      cluster.sync();
      if (t < 8 * GROUPS) // group g: part 0 or 8 of block g / 2
        copy_remote(cluster, &sh.group[t >> 3], &sh.part[((t >> 3) & 1) * (FINAL_PARTS / 2)], t >> 4, t & 7);
      cluster.sync(); // every block has read the parts before they change
      sum_digits(sh, rank);
    } else if (step == 8) {
      cluster.sync();
      if (rank == 0 && t >= 32) { // block k's sum, of bits from 16 k on, into part 2 k
        constexpr unsigned WORDS = sizeof(rns_stored) / 8;
        for (unsigned q = t - 32; q < (FINAL_BLOCKS - 1) * WORDS; q += FINAL_THREADS - 32) {
          const unsigned k = 1 + q / WORDS;
          reinterpret_cast<uint2 *>(&sh.stored[2 * k])[q % WORDS] =
              reinterpret_cast<const uint2 *>(cluster.map_shared_rank(&sh.stored[0], k))[q % WORDS];
        }
        if (t - 32 < FINAL_BLOCKS - 1)
          sh.empty[2 * (t - 31)] = *cluster.map_shared_rank(&sh.empty[0], t - 31);
      }
      cluster.sync(); // the other blocks stay until their sums are read
      if (rank != 0)
        return;
    }
    const unsigned level = step < 4 ? step : step < 8 ? step - 3 : step - 6;
    const unsigned n = step < 4 ? 1u << level : step < 8 ? 1u << (level - 1) : 4u << level;
    const unsigned pairs = FINAL_PARTS >> level, half = (1u << level) >> 1;
    const bool by_lanes = n < FINAL_RNS_DOUBLINGS; // four lanes per pair, or a warp
    if (by_lanes && (t & ~31u) >> 2 < pairs) { // the warp has a pair; groups of lanes without one redo the first
      const bool active = t >> 2 < pairs;
      const unsigned pair = active ? t >> 2 : 0, target = pair << level;
      xyzz q, o;
      if (step == 0) {
        const unsigned r = 2 * (rank * FINAL_PARTS + pair);
        jacobian lo, hi;
        lo.x = lo.y = lo.z = hi.x = hi.y = hi.z = fq::zero();
        if (r + 1 < RESULT_BITS) {
          lo = results[r];
          hi = results[r + 1];
        }
        const fe z = select_fe(role & 1, hi.z, lo.z); // Z^2 and Z^3 of both points, one per lane
        const fe zz = fq::sqr(z), zzz = fq::mul(zz, z);
        q = {lo.x, lo.y, shfl_fe(zz, t & 28), shfl_fe(zzz, t & 28)};
        o = {hi.x, hi.y, shfl_fe(zz, (t & 28) + 1), shfl_fe(zzz, (t & 28) + 1)};
      } else {
        q = sh.part[target];
        o = sh.part[target + half];
      }
      // an infinite partner adds nothing (the batched path's results are infinity above bit c - 1)
      if (!__all_sync(0xffffffffu, curve::is_inf(o))) {
#pragma unroll 1
        for (unsigned k = 0; k < n; k++)
          o = dbl_group4(o);
        q = add_group4(q, o);
      }
      __syncwarp();
      if (active && role == 0)
        sh.part[target] = q;
    }
    if (!by_lanes && t >> 5 < pairs) {
      // steps 2 and 6 start from part[], 3 and 10 end there; between, the
      // points stay residues
      const bool enters = step == 2 || step == 6, leaves = step == 3 || step == 10;
      const unsigned target = (t >> 5) << level, partner = target + half;
      bool empty = enters ? curve::is_inf(sh.part[target]) : sh.empty[target];
      const bool adds = !(enters ? curve::is_inf(sh.part[partner]) : sh.empty[partner]);
      rns_point q{}, o{};
#pragma unroll 1
      for (unsigned k = empty; k <= adds; k++) { // 0: the target, 1: its partner
        const rns_point p = enters ? w.load(sh.part[k ? partner : target]) : w.get(sh.stored[k ? partner : target]);
        if (k)
          o = p;
        else
          q = p;
      }
      if (adds) {
#pragma unroll 1
        for (unsigned k = 0; k < n; k++)
          o = w.doubled(o);
        rns_point sum;
        if (empty) {
          q = o;
          empty = false;
        } else if (w.added(q, o, sum)) {
          q = sum;
        } else { // equal or opposite points
          const jacobian a = w.store(q, sh.columns[t >> 5]), b = w.store(o, sh.columns[t >> 5]);
          const xyzz s = add_group4(curve::from_jacobian(a), curve::from_jacobian(b));
          __syncwarp();
          if ((t & 31) == 0)
            sh.part[target] = s;
          __syncwarp();
          q = w.load(sh.part[target]);
          empty = curve::is_inf(s);
        }
      }
      __syncwarp();
      if (leaves) {
        xyzz p = curve::infinity();
        if (!empty)
          p = curve::from_jacobian(w.store(q, sh.columns[t >> 5]));
        if ((t & 31) == 0)
          sh.part[target] = p;
      } else {
        w.put(sh.stored[target], q);
        if ((t & 31) == 0)
          sh.empty[target] = empty;
      }
    }
    __syncthreads();
  }
  // affine: one inversion of ZZ ZZZ gives 1 / ZZ = ZZZ / (ZZ ZZZ) and 1 / ZZZ;
  // lane 0 finishes x, lane 1 y
  if (t < 32) {
    const xyzz p = sh.part[0];
    const fe inverse = fq::to_mont(inverse_group4(fq::from_mont(fq::mul(p.zz, p.zzz))));
    const bool is_x = t == 0, infinity = curve::is_inf(p);
    const fe c = fq::from_mont(fq::mul(select_fe(is_x, p.x, p.y), fq::mul(select_fe(is_x, p.zzz, p.zz), inverse)));
    if (t < 2)
      for (int i = 0; i < 8; i++)
        (is_x ? point->x : point->y)[i] = infinity ? 0 : c.l[i];
    if (t == 0) {
      point->infinity = infinity ? 1u : 0u;
      for (int i = 0; i < 3; i++)
        point->reserved[i] = 0;
    }
  }
}

} // namespace msm_b200
