// mg_coarse.cuh — the lower V-cycle (levels of side 65 and below) of one job in one CTA, with every
// node of the level at hand in a register of the thread that owns it.
//
// The V-cycle's small levels are a chain of some sixty dependent half-sweeps, residuals and transfers,
// and only the length of one link counts.  With the level arrays in shared memory a half-sweep of 65^2
// took 860 cycles and one of 5^2 270 (B200, clock stamps): five shared accesses and their addresses per
// node and a 1024-thread barrier.  Here a half-sweep reads what it needs of the row above and below
// from shared memory (one value each), of the columns beside it by shuffle, and publishes what it
// changed:
//   65^2            16 warps, 4 rows x 2 columns per thread: one node per row and colour
//   33^2 and below  a thread per column and pair of rows: one node per colour; 512 threads, 128 at
//                   17^2, one warp from 9^2 down
// The levels below 65^2 share one piece of code with run-time sizes, and the sweeps before and after a
// level's correction share theirs: the CTA lands on an SM whose instruction cache does not hold the
// kernel, and code that is unrolled by level (tried: 42 k cycles instead of the shared-memory solver's
// 29 k with stamps) waits for its instructions.
// Same expressions in the same order at every node as the shared-memory solver (coarse_solve), so
// the results are the same bits.  Measured on B200, from f in memory to the stored correction of 65^2 .. 3^2 at
// 2 + 2 sweeps: 29.4 k cycles with the shared-memory solver, 19.0 k here (a half-sweep of 65^2 410, of 33^2 270,
// of the others 180-200: one shared access, one shuffle, seven dependent operations and a barrier);
// V-cycle at 129^2 28.6 -> 22.4 us, at 1025^2 63.4 -> 56.6 us.  Tables of the levels' places in shared memory in
// place of the selects below were slower (24.4 us).
#pragma once
#include "common.cuh"
#include "mg_strips.cuh"
#include "tma.cuh"

namespace mgc {

using mgs::relax;

constexpr int kThreads = 512;
constexpr int kTop = 65;              // largest side

// Levels below 65^2: index 0 is 33^2, 4 is 3^2.  Row pitches put the row pairs of a warp in distinct
// banks; the arrays hold the grid's zero boundary.
constexpr int kPairs = 5;
__host__ __device__ constexpr int pitch_of(int k) { return k == 0 ? 34 : k == 1 ? 24 : k == 2 ? 12 : k == 3 ? 6 : 4; }
__host__ __device__ constexpr int offset_of(int k) {
  int o = 0;
  for (int q = 0; q < k; ++q) o += ((32 >> q) + 1) * pitch_of(q);
  return o;
}

struct __align__(16) Shared {
  // 65^2: the first and last row of every warp's four, by column of the pair: [first, last][column][1 +
  // warp][lane], zero beyond the grid; and the first row's residuals
  float edge[2][2][18][32];
  // the other levels' corrections, right-hand sides and residuals of odd rows
  float e[(offset_of(kPairs) + 3) & ~3];
  float f[offset_of(kPairs)], r[offset_of(kPairs)];
  float res[2][18][33];
  float h2[6], ih2[6];   // 65^2 .. 3^2
};
constexpr int kZeroed = (sizeof(Shared::edge) + sizeof(Shared::e)) / 16;   // what starts as zero comes first

struct Params {
  float omega, om1;
  int nu_pre, nu_post, nu_coarse, bottom;   // index of the coarsest level (-1: 65^2)
};

// Barrier of the first n threads (a multiple of 32) on hardware barrier 1.  Where a level's other threads
// wait for the levels below it they use a barrier of the level's own (2 or 3): those below still
// meet on 1, and the waiting threads of 33^2 are at theirs while 17^2 waits for 9^2 at its own.
__device__ __forceinline__ void sync_first(int n) { asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory"); }
__device__ __forceinline__ void join_33() { asm volatile("bar.sync 2, 512;" ::: "memory"); }
__device__ __forceinline__ void join_17() { asm volatile("bar.sync 3, 128;" ::: "memory"); }

// The V-cycle of the levels from index top down, whose right-hand side is in S.f; its correction is in
// S.e on return (for the threads of the top level, after their last barrier).  A thread owns column i of
// rows j and j + 1 (j odd).
__device__ __forceinline__ void pair_levels(Shared& S, const Params& A, int top) {
  const int t = threadIdx.x;
  int k = top;
  bool down = true;
  for (;;) {
    const int sh = 5 - k, C = 1 << sh, n = C + 1;            // C = side - 1
    const int T = k == 0 ? 512 : k == 1 ? 128 : 32, P = k == 0 ? 34 : k == 1 ? 24 : k == 2 ? 12 : k == 3 ? 6 : 4;
    const int off = k == 0 ? offset_of(0) : k == 1 ? offset_of(1) : k == 2 ? offset_of(2) : k == 3 ? offset_of(3) : offset_of(4);
    const int below = k == 0 ? offset_of(1) : k == 1 ? offset_of(2) : k == 2 ? offset_of(3) : offset_of(4);
    const int PB = k == 0 ? 24 : k == 1 ? 12 : k == 2 ? 6 : 4;   // the next level's pitch
    const bool bottom = k == A.bottom;
    if (t < T) {
      const bool on = (t >> sh) < (C >> 1);
      const int c = t & (C - 1), i = c + 1, j = on ? 2 * (t >> sh) + 1 : 1;
      const bool ok0 = on && i < n - 1, ok1 = ok0 && j + 1 < n - 1;   // inside the boundary
      float* const E = S.e + off + j * P + i;                         // this thread's node of row j
      const float* const F = S.f + off + j * P + i;
      const float h2 = S.h2[k + 1];
      const float f0 = ok0 ? F[0] : 0.f, f1 = ok1 ? F[P] : 0.f;
      float e0 = 0.f, e1 = 0.f;
      auto west = [&](float v) {
        const float w = __shfl_up_sync(0xffffffffu, v, 1);
        return c == 0 ? 0.f : w;
      };
      auto east = [&](float v) { return __shfl_down_sync(0xffffffffu, v, 1); };
      if (!down) {
        // bilinear prolongation (Multigrid.cu:351-407) of the next level's correction
        if (k == 0) join_33();
        else if (k == 1) join_17();
        const float* q = S.e + below + (j >> 1) * PB + (i >> 1);
        const bool io = i & 1;
        const float a = q[0], b = q[PB], a1 = io ? q[1] : 0.f, b1 = io ? q[PB + 1] : 0.f;
        e0 = ok0 ? E[0] + (io ? 0.25f : 0.5f) * (a + a1 + b + b1) : 0.f;
        e1 = ok1 ? E[P] + (io ? 0.5f : 1.f) * (b + b1) : 0.f;
        if (ok0) E[0] = e0;
        if (ok1) E[P] = e1;
        sync_first(T);
      }
      // Half-sweeps, colour (i + j) odd first.  Row j's node has the colour of c; the node of the other
      // colour in the column beside it is the one that column does not update, so one value per
      // thread serves both neighbours.
      const int half_sweeps = 2 * (!down ? A.nu_post : bottom ? A.nu_coarse : A.nu_pre);
      bool up = (c & 1) == 0;                                // the node of the colour is row j + 1's
#pragma unroll 1
      for (int s = 0; s < half_sweeps; ++s) {
        const float mine = up ? e1 : e0, other = up ? e0 : e1;
        const float out = E[up ? 2 * P : -P];
        const float w = west(other), x = east(other);
        const float v = relax(up ? out : other, up ? other : out, x, w, up ? f1 : f0, mine, h2, A.omega, A.om1);
        if (up ? ok1 : ok0) {
          E[up ? P : 0] = v;
          if (up) e1 = v;
          else e0 = v;
        }
        up = !up;
        sync_first(T);
      }
      if (down && !bottom) {
        // residual and its full weighting (Multigrid.cu:299-349) to the next level; row j + 2's
        // residuals come from the thread of the next pair of rows
        const float ih2 = S.ih2[k + 1];
        const float n0 = E[-P], s1 = E[2 * P];
        const float w0 = west(e0), x0 = east(e0), w1 = west(e1), x1 = east(e1);
        const float l0 = n0 + e1 + w0 + x0 - 4.f * e0, l1 = e0 + s1 + w1 + x1 - 4.f * e1;
        const float r0 = ok0 ? fmaf(-l0, ih2, f0) : 0.f, r1 = ok1 ? fmaf(-l1, ih2, f1) : 0.f;
        float* const R = S.r + off + j * P + i;
        if (ok0) R[0] = r0;
        sync_first(T);
        const float nw = west(r0), ne = east(r0), w = west(r1), x = east(r1);
        if ((c & 1) && ok1) {
          const float* q = R + 2 * P;
          const float sum = 4.f * r1 + 2.f * w + 2.f * x + 2.f * r0 + 2.f * q[0] + nw + ne + q[-1] + q[1];
          S.f[below + ((j + 1) >> 1) * PB + (i >> 1)] = sum * 0.0625f;
        }
        sync_first(T);
      }
    }
    if (down && !bottom) {
      ++k;
    } else {
      if (k == top) break;
      --k;
      down = false;
    }
  }
}

// The 65^2 level: warp w's rows 4 w + 1 .. 4 w + 4, lane l's columns 2 l + 1 and 2 l + 2.
struct Block {
  float e[4][2], f[4][2];
  int w, l;
  __device__ __forceinline__ bool ok(int a, int b) const { return !(w == 15 && a == 3) && !(l == 31 && b == 1); }
  __device__ __forceinline__ float west(float v) const {
    const float x = __shfl_up_sync(0xffffffffu, v, 1);
    return l == 0 ? 0.f : x;
  }
  __device__ __forceinline__ float east(float v) const { return __shfl_down_sync(0xffffffffu, v, 1); }
  // One half-sweep of colour kOdd (row a's node of the colour sits in column (a + kOdd) & 1).
  template <int kOdd>
  __device__ __forceinline__ void half_sweep(Shared& S, const Params& A, float h2) {
    const float above = S.edge[1][kOdd][w][l], below = S.edge[0][1 - kOdd][w + 2][l];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int b = (a + kOdd) & 1;
      const float n = a == 0 ? above : e[a == 0 ? 0 : a - 1][b], s = a == 3 ? below : e[a == 3 ? 3 : a + 1][b];
      const float x = b ? east(e[a][0]) : e[a][1], y = b ? e[a][0] : west(e[a][1]);
      const float v = relax(s, n, x, y, f[a][b], e[a][b], h2, A.omega, A.om1);
      e[a][b] = ok(a, b) ? v : 0.f;
    }
    S.edge[0][kOdd][w + 1][l] = e[0][kOdd];
    S.edge[1][1 - kOdd][w + 1][l] = e[3][1 - kOdd];
    __syncthreads();
  }
  __device__ __forceinline__ void restrict_to(Shared& S, float ih2) {
    constexpr int PC = pitch_of(0);
    float r[4][2], right[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const float x = east(e[a][0]), y = west(e[a][1]);
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const float n = a == 0 ? S.edge[1][b][w][l] : e[a == 0 ? 0 : a - 1][b];
        const float s = a == 3 ? S.edge[0][b][w + 2][l] : e[a == 3 ? 3 : a + 1][b];
        const float lap = n + s + (b ? e[a][0] : y) + (b ? x : e[a][1]) - 4.f * e[a][b];
        r[a][b] = ok(a, b) ? fmaf(-lap, ih2, f[a][b]) : 0.f;
      }
      right[a] = east(r[a][0]);
    }
    S.res[0][w + 1][l] = r[0][0];
    S.res[1][w + 1][l] = r[0][1];
    __syncthreads();
    const float s0 = S.res[0][w + 2][l], s1 = S.res[1][w + 2][l], s2 = S.res[0][w + 2][l + 1];
    if (l < 31) {
      float* const F = S.f + (2 * w + 1) * PC + l + 1;
      const float up = 4.f * r[1][1] + 2.f * r[1][0] + 2.f * right[1] + 2.f * r[0][1] + 2.f * r[2][1] + r[0][0] + right[0] +
                       r[2][0] + right[2];
      F[0] = up * 0.0625f;
      if (w < 15) {
        const float lo = 4.f * r[3][1] + 2.f * r[3][0] + 2.f * right[3] + 2.f * r[2][1] + 2.f * s1 + r[2][0] + right[2] + s0 +
                         s2;
        F[PC] = lo * 0.0625f;
      }
    }
    __syncthreads();
  }
  __device__ __forceinline__ void prolong_from(Shared& S) {
    constexpr int PC = pitch_of(0);
    const float* q = S.e + 2 * w * PC + l;
    const float a = q[0], a1 = q[1], b = q[PC], b1 = q[PC + 1], c = q[2 * PC], c1 = q[2 * PC + 1];
    e[0][0] += 0.25f * (a + a1 + b + b1);
    e[0][1] += 0.5f * (a1 + b1);
    e[1][0] += 0.5f * (b + b1);
    e[1][1] += b1;
    e[2][0] += 0.25f * (b + b1 + c + c1);
    e[2][1] += 0.5f * (b1 + c1);
    e[3][0] += 0.5f * (c + c1);
    e[3][1] += c1;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      S.edge[0][u][w + 1][l] = e[0][u];
      S.edge[1][u][w + 1][l] = e[3][u];
    }
    __syncthreads();
  }
};

// Coarse solve of one job per CTA, for jobs whose first coarse level has at most 65 nodes a side.  The
// correction's boundary stays as job creation zeroed it.
__global__ void __launch_bounds__(kThreads) mg_coarse_reg_kernel(const int* __restrict__ job_list,
                                                                 const JobDev* __restrict__ jobs,
                                                                 const JobState* __restrict__ st) {
  __shared__ __align__(16) Shared S;
  tma::pdl_trigger();
  const int job = job_list[blockIdx.x];
  const JobDev& J = jobs[job];
  if (st[job].converged) { tma::pdl_wait(); return; }   // waits all the same: see pdl_wait
  const int t = threadIdx.x, lc = J.lc, n = J.nl[lc], pitch = J.pl[lc];
  Params A;
  A.omega = J.omega;
  A.om1 = 1.f - A.omega;
  A.nu_pre = J.nu_pre; A.nu_post = J.nu_post; A.nu_coarse = J.nu_coarse;
  const int top = n >= kTop ? -1 : 4 - (31 - __clz(n - 1)) + 1;   // index of the job's first level (-1: 65^2)
  A.bottom = top + J.levels - 1 - lc;
  float* const e = J.e[lc];
  const float* const f = (lc == 0 && st[job].fsel) ? J.f0b : J.f[lc];
  // zero: the grid boundaries, and corrections that no sweep touches
  for (int k = t; k < kZeroed; k += kThreads) reinterpret_cast<float4*>(&S)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (t < 6) {
    // constants of side 2^(6 - t) + 1, which is level lc + t - (top + 1)
    const double hl = J.h * (double)(1 << (lc + max(0, t - 1 - top)));
    S.h2[t] = (float)(hl * hl);
    S.ih2[t] = (float)(1.0 / (hl * hl));
  }
  __syncthreads();
  tma::pdl_wait();
  if (top >= 0) {
    // a first level of 33^2 or less goes through the shared arrays (pitch by index as above)
    const int P = pitch_of(top), off = offset_of(top);
    for (int k = t; k < (n - 2) * (n - 2); k += kThreads) {
      const int j = 1 + k / (n - 2), i = 1 + k % (n - 2);
      S.f[off + j * P + i] = __ldg(f + j * pitch + i);
    }
    __syncthreads();
    pair_levels(S, A, top);
    __syncthreads();
    for (int k = t; k < (n - 2) * (n - 2); k += kThreads) {
      const int j = 1 + k / (n - 2), i = 1 + k % (n - 2);
      e[j * pitch + i] = S.e[off + j * P + i];
    }
    return;
  }
  Block q;
  q.w = t >> 5;
  q.l = t & 31;
  const int at = (4 * q.w + 1) * pitch + 2 * q.l + 1;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      q.e[a][b] = 0.f;
      q.f[a][b] = q.ok(a, b) ? __ldg(f + at + a * pitch + b) : 0.f;
    }
  const float h2 = S.h2[0];
#pragma unroll 1
  for (int leg = 0;; ++leg) {
    const int nu = leg ? A.nu_post : A.bottom < 0 ? A.nu_coarse : A.nu_pre;
#pragma unroll 1
    for (int it = 0; it < nu; ++it) {
      q.half_sweep<1>(S, A, h2);
      q.half_sweep<0>(S, A, h2);
    }
    if (leg || A.bottom < 0) break;
    q.restrict_to(S, S.ih2[0]);
    pair_levels(S, A, 0);
    __syncthreads();
    q.prolong_from(S);
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
      if (q.ok(a, b)) e[at + a * pitch + b] = q.e[a][b];
}

}  // namespace mgc
