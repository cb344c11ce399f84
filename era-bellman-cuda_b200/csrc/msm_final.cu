// The caller-side final reduction of an MSM on the GPU: sum over i < 254 of
// 2^i R_i of the 254 per-bit Jacobian results, written as one canonical
// affine point (standard form, fully reduced, infinity flagged).  The
// reference leaves this Horner pass to its callers, on the host
// (src/bellman-cuda.h:496-505; tests/msm_test.cu:116-126).
//
// Whatever the order of the additions, the term 2^253 R_253 needs 253
// dependent doublings, so the sum is latency-bound: one block, and what counts
// is the time of one doubling.  A Horner pass also puts 253 additions on that
// chain; a pairwise tree over the bits puts 8: part t starts from R_2t + 2
// R_2t+1, and at level L = 1..7 the sum starting at bit 2t (t mod 2^L = 0)
// takes its partner's (t + 2^(L-1)), doubled 2^L times.
//
// Levels 0 to 2 (many points, few doublings) share each doubling between four
// lanes (dbl_group4).  From level 3 on a warp takes one point and doubles it in
// a residue number system (rns.cuh), where a product of the whole warp takes
// less than half of one thread's: about 1,030 cycles per doubling on a B200
// against 3,236 for dbl_group4; one final sum 0.544 -> 0.230 ms, of a batched
// instance's results (20 bits) 0.083 ms.
// The affine conversion takes one inversion (inverse_group4).
#include "bellman-cuda-b200.h"
#include "msm_device.cuh"
#include "msm_group4.cuh"
#include "pointer_access.h"
#include "rns.cuh"

#include <cuda_runtime.h>

namespace msm_b200 {

constexpr unsigned FINAL_PARTS = 128; // parts t < 127 start from results 2t, 2t + 1
constexpr unsigned FINAL_THREADS = 4 * FINAL_PARTS;
constexpr unsigned FINAL_WARPS = FINAL_THREADS / 32;
constexpr unsigned FINAL_RNS_LEVEL = 3; // the first level with a warp per point
static_assert(FINAL_PARTS >> FINAL_RNS_LEVEL <= FINAL_WARPS, "a warp per point");

__device__ const rns::tables rns_tables = rns::TABLES;

// Doublings of one point by a whole warp.  All lanes hold their residues of X
// and Y of a Jacobian point, the lanes of groups 1 and 2 those of Z
// (x = X / Z^2, y = Y / Z^3).
struct rns_point {
  rns::residues x, y, z;
};

struct rns_warp {
  unsigned group, base; // of this lane: 0..2, its group's first lane
  rns::lane_table t;

  __device__ __forceinline__ rns_warp() {
    const unsigned lane = threadIdx.x & 31;
    group = min(lane / rns::RESIDUES, rns::GROUPS - 1); // lanes 30, 31 repeat lanes 20, 21
    base = group * rns::RESIDUES;
    // every word through a volatile move: the table stays in registers instead
    // of being read again inside the doubling loop
    const uint32_t *from = reinterpret_cast<const uint32_t *>(rns_tables.lane + lane % rns::RESIDUES);
    uint32_t *to = reinterpret_cast<uint32_t *>(&t);
#pragma unroll
    for (unsigned k = 0; k < sizeof(rns::lane_table) / 4; k++)
      asm volatile("mov.b32 %0, %1;" : "=r"(to[k]) : "r"(from[k]));
  }
  __device__ __forceinline__ auto extension() const {
    return [first = base](int32_t v, auto sum) {
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
    const unsigned src = g * rns::RESIDUES + (threadIdx.x & 31) - base;
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

  // X, Y, Z as Montgomery-form field elements in (0, 2p), the same in every
  // lane; columns: 24 words of shared memory of this warp
  __device__ __forceinline__ jacobian store(const rns_point &p, int64_t (*columns)[8]) const {
    const rns::residues leave = {t.leave_a, t.leave_b};
    const int64_t column = rns::product_column(t, pick(p.x, p.y, p.z), leave, extension());
    const unsigned lane = threadIdx.x & 31;
    if (lane < rns::GROUPS * rns::RESIDUES && lane - base < 8)
      columns[group][lane - base] = column;
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

__global__ void __launch_bounds__(FINAL_THREADS) final_sum_kernel(const jacobian *__restrict__ results, msm_b200_affine_point *point) {
  __shared__ xyzz part[FINAL_PARTS]; // part[t]: the sum of the bits starting at 2t (weights relative to 2^2t)
  __shared__ int64_t columns[FINAL_WARPS][rns::GROUPS][8];
  const unsigned t = threadIdx.x, group = t >> 2, role = t & 3, warp = t >> 5;
  { // level 0, four lanes per pair of results
    const unsigned lane_base = t & 28;
    jacobian lo, hi;
    lo.x = lo.y = lo.z = hi.x = hi.y = hi.z = fq::zero();
    if (2 * group + 1 < RESULT_BITS) {
      lo = results[2 * group];
      hi = results[2 * group + 1];
    }
    const fe z = select_fe(role & 1, hi.z, lo.z); // Z^2 and Z^3 of both points, one per lane
    const fe zz = fq::sqr(z), zzz = fq::mul(zz, z);
    const xyzz a = {lo.x, lo.y, shfl_fe(zz, lane_base), shfl_fe(zzz, lane_base)};
    const xyzz b = {hi.x, hi.y, shfl_fe(zz, lane_base + 1), shfl_fe(zzz, lane_base + 1)};
    const xyzz q = add_group4(a, dbl_group4(b));
    if (role == 0)
      part[group] = q;
  }
  __syncthreads();
  // levels 1 and 2: group g of four lanes adds part[g 2^L + 2^(L-1)], doubled
  // 2^L times, into part[g 2^L] (whole warps: 64 and 32 groups)
  for (unsigned level = 1; level < FINAL_RNS_LEVEL; level++) {
    if (group < FINAL_PARTS >> level) {
      const unsigned target = group << level;
      xyzz o = part[target + (1u << (level - 1))];
      if (!__all_sync(0xffffffffu, curve::is_inf(o)))
        for (unsigned k = 0; k < (1u << level); k++)
          o = dbl_group4(o);
      const xyzz q = add_group4(part[target], o);
      __syncwarp();
      if (role == 0)
        part[target] = q;
    }
    __syncthreads();
  }
  // the other levels, a warp per point; an infinite partner adds nothing (the
  // batched path's results are infinity above bit c - 1)
  const rns_warp w;
  for (unsigned level = FINAL_RNS_LEVEL; (1u << level) <= FINAL_PARTS; level++) {
    if (warp < FINAL_PARTS >> level) {
      const unsigned target = warp << level, partner = target + (1u << (level - 1));
      if (!curve::is_inf(part[partner])) {
        rns_point o = w.load(part[partner]);
        for (unsigned k = 0; k < (1u << level); k++)
          o = w.doubled(o);
        const jacobian j = w.store(o, columns[warp]);
        const xyzz q = add_group4(part[target], curve::from_jacobian(j));
        __syncwarp();
        if ((t & 31) == 0)
          part[target] = q;
      }
    }
    __syncthreads();
  }
  // affine: one inversion of ZZ ZZZ gives 1 / ZZ = ZZZ / (ZZ ZZZ) and 1 / ZZZ;
  // lane 0 finishes x, lane 1 y
  if (t < 32) {
    const xyzz p = part[0];
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

// A pointer the kernel can dereference (pointer_access.h): device memory of
// the current device or of a peer it has access to, managed memory, or pinned
// host memory through its device alias; anything else is refused.
static cudaError_t device_view(const void *ptr, void **view) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess)
    return err;
  cudaPointerAttributes attr{};
  if ((err = cudaPointerGetAttributes(&attr, ptr)) != cudaSuccess)
    return err;
  const bool peer = attr.type == cudaMemoryTypeDevice && attr.device != device && peer_access_recorded(device, attr.device);
  return kernel_view(ptr, attr, device, peer, host_memory::device_alias, view);
}

cudaError_t final_sum(const void *results, msm_b200_affine_point *point, cudaStream_t stream) {
  if (!results || !point || reinterpret_cast<uintptr_t>(results) % 16 || reinterpret_cast<uintptr_t>(point) % 4)
    return cudaErrorInvalidValue;
  void *r = nullptr, *p = nullptr;
  cudaError_t err = device_view(results, &r);
  if (err == cudaSuccess)
    err = device_view(point, &p);
  if (err != cudaSuccess)
    return err;
  final_sum_kernel<<<1, FINAL_THREADS, 0, stream>>>(static_cast<const jacobian *>(r), static_cast<msm_b200_affine_point *>(p));
  return cudaGetLastError();
}

} // namespace msm_b200

extern "C" bc_error msm_b200_final_sum_async(const void *results, msm_b200_affine_point *point, bc_stream stream) {
  return static_cast<bc_error>(msm_b200::final_sum(results, point, static_cast<cudaStream_t>(stream.handle)));
}
