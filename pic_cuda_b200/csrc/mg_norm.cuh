// mg_norm.cuh — the level-0 residual norm, summed so that the result does not depend on the order.
//
// Level 0's up leg runs as tiles, strips or general tiles by what fits the jobs of a launch, and each adds
// up r^2 over other groups of nodes.  A job's norm decides where its solve stops, so it must not depend
// on the jobs beside it: every kernel forms the same values, one per pair of columns 2 k and 2 k + 1 of
// a row, and adds them exactly.
//
// A lane adds into two FP64 accumulators that start at 1.5 times a power of two, 2^e1 and 2^e2: adding a value to the
// first rounds it to a multiple of u1 = 2^(e1 - 52), what that leaves over goes to the second and is
// rounded to a multiple of u2 = 2^(e2 - 52), each value by itself (its last bit is set, so that no tie
// is decided by the sum).  Multiples of one power of two add without rounding while they stay below 2^53 of
// it (the first parts, as FP64) or 2^63 (the second parts, as integers from the end of a lane on), so any
// grouping gives the same total, which is rounded once at the end.  e1 comes from the job's norm before
// the cycle (64 times its square fits), e2 from the number of pairs; all kernels read the same state.
//
// Against an extended-precision sum of the same r (129^2, 1025^2, 4097^2; after 1, 2 and 4 cycles) relres is
// off by at most 1.2e-16 of itself, as it was with plain FP64 sums in a fixed order.  If the norm grows by
// more than a factor of 8 in one cycle the sum is as accurate, but its last bits may depend on the order.
#pragma once
#include "common.cuh"

namespace mgn {

__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }   // -1022 <= e <= 1023
constexpr int kLeastE2 = -1022;   // u2 is then the least FP64 number: nothing is rounded, no tie to break

// Exponents for a job of side n whose norm's square before the cycle was rnorm2.
struct Scale {
  int e1, e2;
  __device__ __forceinline__ Scale(double rnorm2, int n) {
    const int e = ((__double2hiint(rnorm2) >> 20) & 0x7ff) - 1023;
    e1 = min(max(e + 8, -1000), 1000);
    // at most 2^bits pairs, whose left-overs of u1 / 2 each make less than 2^62 u2; a lane's 128 fit 2^51 u2
    const int bits = 1 + 2 * (32 - __clz((n + 1) / 2 - 1));
    e2 = max(e1 + max(bits - 63, -45), kLeastE2);
  }
};

// What a lane, a CTA or a launch has added up: the first part, and the second in units of u2.
struct __align__(16) Part {
  double first;
  long long second;
  __device__ __forceinline__ void add(const Part& p) { first += p.first; second += p.second; }
};
static_assert(sizeof(Part) == 16, "two FP64 values of JobDev::partials");

struct Sum {
  double a, b;
  int odd;
  __device__ __forceinline__ explicit Sum(const Scale& s)
      : a(1.5 * pow2(s.e1)), b(1.5 * pow2(s.e2)), odd(s.e2 > kLeastE2 ? 1 : 0) {}
  __device__ __forceinline__ void add(double v) {
    const double s = __dadd_rn(a, v), left = __dadd_rn(v, -__dadd_rn(s, -a));
    a = s;
    b = __dadd_rn(b, __hiloint2double(__double2hiint(left), __double2loint(left) | odd));
  }
  // count: the most values that a lane adds.  Left-overs above count u1 / 2 mean that the first part outgrew
  // its exponent; they are kept with it then.
  __device__ __forceinline__ Part part(const Scale& s, int count) const {
    const Sum zero(s);
    const double first = __dadd_rn(a, -zero.a), second = __dadd_rn(b, -zero.b);
    if (!(fabs(second) <= count * (0x1p-53 * pow2(s.e1)))) return Part{isfinite(first) ? first + second : first, 0};
    return Part{first, __double2ll_rn(second * pow2(-s.e2) * 0x1p52)};
  }
};
// The square of the norm.  The second part gives all its whole u1 to the first, so that one rounding is left.
__device__ __forceinline__ double total(const Part& p, const Scale& s) {
  const int shift = s.e1 - s.e2;
  const long long whole = (p.second + (1ll << (shift - 1))) >> shift;
  const double rest = (double)(p.second - (whole << shift)) * 0x1p-52 * pow2(s.e2);
  return __dadd_rn(__dadd_rn(p.first, (double)whole * 0x1p-52 * pow2(s.e1)), rest);
}

// Squares of a pair's residuals, added.
__device__ __forceinline__ double pair_of(double r0, double r1) { return __dadd_rn(__dmul_rn(r0, r0), __dmul_rn(r1, r1)); }

// Sum over the warp (over its first LANES lanes, in those).
template <int LANES = 32>
__device__ __forceinline__ Part warp_part(Part p) {
#pragma unroll
  for (int o = LANES / 2; o; o >>= 1)
    p.add(Part{__shfl_xor_sync(0xffffffffu, p.first, o), __shfl_xor_sync(0xffffffffu, p.second, o)});
  return p;
}
// Sum over a CTA of WARPS warps, in its first thread.
template <int WARPS>
__device__ __forceinline__ Part cta_part(Part p, Part (&ws)[WARPS]) {
  p = warp_part(p);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) ws[warp] = p;
  __syncthreads();
  if (warp == 0) p = warp_part<WARPS>(ws[lane & (WARPS - 1)]);
  return p;
}
// Sum of n partials by a CTA of WARPS warps, in its first thread.  Eight loads of a thread are issued ahead of the
// additions (16.4k partials at 4097^2 as tiles).
template <int WARPS>
__device__ __forceinline__ Part sum_partials(const double* partials, int n, Part (&ws)[WARPS]) {
  Part p{0.0, 0};
#pragma unroll 8
  for (int k = threadIdx.x; k < n; k += 32 * WARPS) p.add(reinterpret_cast<const Part*>(partials)[k]);
  return cta_part(p, ws);
}

// The pairs of four rows of a tile: the lanes of a warp hold the residuals r of those rows in the column
// of their number (0 outside the grid), and a lane pair adds two rows' pairs each.
__device__ __forceinline__ void add_rows4(Sum& S, const double (&r)[4]) {
  const bool odd = threadIdx.x & 1;
  double h[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const double v = __dmul_rn(r[u], r[u]);
    h[u] = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
  }
  S.add(odd ? h[2] : h[0]);
  S.add(odd ? h[3] : h[1]);
}

}  // namespace mgn
