// mg_strips.cuh — the V-cycle's tile-free level kernels: red-black SOR sweeps as a pipeline of
// rows in registers.
//
// One warp owns a strip of 64 grid columns (lane: the even column c0 = x0 + 2 lane and c1 = c0 + 1)
// and walks it row by row.  T = 2 NU half-sweeps follow one another down the strip, one row
// apart: while the newest row enters, half-sweep k relaxes the row k behind it, which has
// everything it needs (the row below was relaxed by half-sweep k - 1 a moment ago).  The last
// T + 2 rows stay in registers; the neighbours in a row are a lane's other column or one
// shuffle away.  Each lane holds one node of each colour per row, and at one row step every
// half-sweep works on the same column of the pair (the colours and the row parities advance
// together), so no lane idles.  Half-sweeps invalidate one column per side and one row at the
// start, so a strip's owned columns are fewer than 64 and its rows start early (the lane ranges
// below); neighbouring strips recompute those columns.  Every node goes through the same
// expressions in the same order as in the tile kernels, so the results are the same bits.
//
// Why this shape: sweeps on 32 x 32 tiles in shared memory are bound by instruction issue (157
// thread instructions per node down, 289 up on level 0 at 4097^2: five shared accesses, address
// arithmetic and a block barrier per half-sweep, on 1.7 nodes per owned node).  Here a half-sweep
// of two nodes is one shuffle and six arithmetic instructions, nothing waits at a barrier, and the
// recomputed halo is 64 / 54 columns: 49 and 99 instructions per node.  Level 0 at 4097^2 (ncu,
// cold): down 100 -> 40 us (issue 71% active), up 199 -> 131 us (55% of DRAM, 586 MB against 554 MB
// of inputs and outputs; short and long scoreboard of the shared-memory ring).
#pragma once
#include "common.cuh"
#include "kernels.h"
#include "mg_norm.cuh"
#include "tma.cuh"

namespace mgs {

constexpr int kWarps = 4;                 // strips per CTA
constexpr int up_warps(int mode) { return mode ? 3 : kWarps; }   // the same of the up kernel

// Owned lanes [lo, lo + lanes) of a strip and its owned columns, for the down leg (residual and
// full weighting after the sweeps), the up leg and the up leg of level 0 (FP64 residual after
// the sweeps).
__host__ __device__ constexpr int down_lo(int nu) { return nu + 1; }
__host__ __device__ constexpr int down_lanes(int nu) { return 31 - 2 * nu; }
__host__ __device__ constexpr int up_lo(int nu, int x) { return nu + x; }
__host__ __device__ constexpr int up_lanes(int nu, int x) { return 32 - 2 * nu - 2 * x; }
__host__ __device__ constexpr int down_strips(int nu, int n) { return (n + 2 * down_lanes(nu) - 1) / (2 * down_lanes(nu)); }
__host__ __device__ constexpr int up_strips(int nu, int x, int n) {
  return (n + 2 * up_lanes(nu, x) - 1) / (2 * up_lanes(nu, x));
}
constexpr int kMinRows = 8;               // fewest rows of an item

// Row steps in flight in a strip's ring, and per unrolled step of its loop.
constexpr int kDownRing = 8;
__host__ __device__ constexpr int up_ring(int x) { return x ? 6 : 8; }
// Most rows per item, at most `at_most`, whose row steps fill whole unrolled steps (leg 0: down; 1:
// up, x = 1 on level 0); 0 if no size of at least kMinRows does.
inline int rows_fit(int leg, int nu, int x, int at_most) {
  const int lead = leg == 0 ? 4 * nu + 2 : x ? 4 * nu + 4 : 4 * nu, d = leg == 0 ? kDownRing : up_ring(x);
  const int rows = (at_most + lead) / d * d - lead;
  return rows >= kMinRows ? rows : 0;
}

// One relaxation, the expression of every smoother here (Multigrid.cu:246-265).
__device__ __forceinline__ float relax(float below, float above, float east, float west, float f, float e, float h2,
                                       float omega, float om1) {
  const float s = below + above + east + west;
  // fused explicitly: f stays in registers over several half-sweeps, and the compiler would share its
  // product with h2 between them instead
  const float nv = 0.25f * fmaf(-h2, f, s);
  return fmaf(omega, nv, om1 * e);
}
__device__ __forceinline__ float left_of(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ float right_of(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double left_of(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double right_of(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }

// Inputs arrive by per-lane asynchronous copies (cp.async) into a ring of row steps in shared
// memory: every lane reads back only what it copied itself, so nothing waits but the lane's own
// copy groups (one per pair of rows).  Loads held in registers wait on one of a warp's six
// scoreboards, and a row asked for early then waits for the rows asked for after it.
template <bool EDGE>
__device__ __forceinline__ void copy8(void* dst, const void* src, const void* safe, bool ok) {
  if (EDGE) tma::cp_async8(dst, ok ? src : safe, ok);
  else tma::cp_async8(dst, src, true);
}
template <bool EDGE>
__device__ __forceinline__ void copy4(void* dst, const void* src, const void* safe, bool ok) {
  if (EDGE) tma::cp_async4(dst, ok ? src : safe, ok);
  else tma::cp_async4(dst, src, true);
}

// Predicated stores: no branch, so a step of several rows stays one basic block whose independent
// chains the compiler can interleave.
__device__ __forceinline__ void store1(float* p, float a, bool ok) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.f32 [%0], %1;\n\t}" ::"l"(p), "f"(a),
               "r"((unsigned)ok)
               : "memory");
}
__device__ __forceinline__ void store2(float* p, float a, float b, bool ok) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q st.global.v2.f32 [%0], {%1, %2};\n\t}" ::"l"(p), "f"(a),
               "f"(b), "r"((unsigned)ok)
               : "memory");
}
__device__ __forceinline__ void store1(double* p, double a, bool ok) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.f64 [%0], %1;\n\t}" ::"l"(p), "d"(a),
               "r"((unsigned)ok)
               : "memory");
}

// The FP64 defect rhs_scale rho - lap / h^2 of a node in row j.  Which product is rounded on its own is
// spelled out, so that the tile and the strip kernels agree to the bit whichever a level is given
// to (a job's result must not depend on the jobs beside it); it alternates by the row as it always
// has in the tile kernel, whose four passes over a tile's rows the compiler fused differently.
__device__ __forceinline__ double defect(double lap, double inv_h2, double rhs_scale, double rho, int j) {
  return (j & 31) < 24 ? fma(rhs_scale, rho, -__dmul_rn(lap, inv_h2)) : fma(-lap, inv_h2, __dmul_rn(rhs_scale, rho));
}

// Down leg of level l: NU pre-sweeps from a zero correction, the smoothed correction to e_l, its
// residual full-weighted to f_{l+1}.
struct DownArgs {
  const float* f;      // right-hand side (whole array)
  float* e;
  float* fc;
  int n, nc, pf, pc, c0, r0, r1;
  float h2, inv_h2, omega;
};
// EDGE: the strip or its rows touch the grid's boundary, so loads and updates are masked.
template <int NU, bool EDGE>
__device__ __forceinline__ void down_strip(const DownArgs& A, float2* ring) {
  constexpr int T = 2 * NU, WIN = T + 1, LO = down_lo(NU), LANES = down_lanes(NU), D = kDownRing;
  const int lane = threadIdx.x & 31;
  const int n = A.n, c0 = A.c0, pf = A.pf;
  const float h2 = A.h2, inv_h2 = A.inv_h2, omega = A.omega, om1 = 1.f - omega;
  const bool colin = !EDGE || (unsigned)c0 < (unsigned)n;
  const bool mine = lane >= LO && lane < LO + LANES && colin;
  const bool upd0 = !EDGE || (c0 >= 1 && c0 <= n - 2), upd1 = !EDGE || (c0 >= 0 && c0 + 1 <= n - 2);
  const bool fine_ic = !EDGE || (c0 >= 2 && c0 <= n - 3);   // an interior coarse column
  const int js = A.r0 - T - 2, je = A.r1 - 1 + T;           // first and last row step
  const float* src = A.f + ((ptrdiff_t)js * pf + c0);       // the next row to request
  int next = js;
  float2* const slot = ring + lane;
  auto request = [&](int g) {
    copy8<EDGE>(slot + g * 32, src, A.f, colin && (unsigned)next < (unsigned)n);
    src += pf;
    ++next;
  };
  // the row the last half-sweep has just completed, and the coarse row, of a row step
  static_assert(NU > 0, "without sweeps the general kernels run");
  constexpr int kDone = T - 1;
  float* eout = A.e + ((ptrdiff_t)(js - kDone) * pf + c0);
  float* cout = A.fc + ((ptrdiff_t)((js - T) >> 1) * A.pc + (c0 >> 1));
  float E[WIN + D][2], F[WIN + D][2];
  float ra[3] = {0.f, 0.f, 0.f}, rb[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int a = 0; a < WIN; ++a) E[a][0] = E[a][1] = F[a][0] = F[a][1] = 0.f;
#pragma unroll
  for (int g = 0; g < D; ++g) {
    if (EDGE || js + g <= je) request(g);
    if (g & 1) tma::cp_async_commit();
  }
  for (int jg = js; jg <= je; jg += D) {
    const bool more = EDGE || jg + D <= je;
#pragma unroll
    for (int g = 0; g < D; ++g) {
      const int a = WIN + g, j = jg + g;
      if (!(g & 1)) tma::cp_async_wait<D / 2 - 1>();
      const float2 fv = slot[g * 32];
      F[a][0] = fv.x;
      F[a][1] = fv.y;
      if (more) request(g);
      if (g & 1) tma::cp_async_commit();
      E[a][0] = E[a][1] = 0.f;
      // half-sweep k on row j - k; the column of its colour is c1 on even row steps, c0 on odd
#pragma unroll
      for (int k = 0; k < T; ++k) {
        const int b = a - k, b1 = k == 0 ? b : b + 1;
        const bool row = !EDGE || (unsigned)(j - k - 1) < (unsigned)(n - 2);
        if (g & 1) {
          const float w = k == 0 ? 0.f : left_of(E[b][1]);
          const float v = k == 0 ? relax(0.f, 0.f, 0.f, 0.f, F[b][0], 0.f, h2, omega, om1)
                                 : relax(E[b1][0], E[b - 1][0], E[b][1], w, F[b][0], E[b][0], h2, omega, om1);
          E[b][0] = (row && upd0) ? v : E[b][0];
        } else {
          const float e = k == 0 ? 0.f : right_of(E[b][0]);
          const float v = k == 0 ? relax(0.f, 0.f, 0.f, 0.f, F[b][1], 0.f, h2, omega, om1)
                                 : relax(E[b1][1], E[b - 1][1], e, E[b][0], F[b][1], E[b][1], h2, omega, om1);
          E[b][1] = (row && upd1) ? v : E[b][1];
        }
      }
      {
        const int b = a - kDone, q = j - kDone;
        const bool own = mine && (unsigned)(q - A.r0) < (unsigned)(A.r1 - A.r0) && (!EDGE || q < n);
        const bool pair = !EDGE || c0 + 1 < n;
        store2(eout, E[b][0], E[b][1], own && pair);
        if (EDGE) store1(eout, E[b][0], own && !pair);
        eout += pf;
      }
      // residual of row j - T, one column further to the left by shuffle, and on odd rows the
      // full weighting of the three last rows to coarse row (j - T - 1) / 2
      float rc[3];
      {
        const int b = a - T;
        const float w = left_of(E[b][1]), e = right_of(E[b][0]);
        const float l0 = E[b - 1][0] + E[b + 1][0] + w + E[b][1] - 4.f * E[b][0];
        const float l1 = E[b - 1][1] + E[b + 1][1] + E[b][0] + e - 4.f * E[b][1];
        rc[1] = fmaf(-l0, inv_h2, F[b][0]);
        rc[2] = fmaf(-l1, inv_h2, F[b][1]);
        rc[0] = left_of(rc[2]);
      }
      if (g & 1) {
        const int q = j - T, jc = (q - 1) >> 1;
        const float sum = 4.f * rb[1] + 2.f * rb[0] + 2.f * rb[2] + 2.f * ra[1] + 2.f * rc[1] + ra[0] + ra[2] + rc[0] +
                          rc[2];
        store1(cout, (!EDGE || (fine_ic && jc > 0 && jc < A.nc - 1)) ? sum * 0.0625f : 0.f,
               mine && (unsigned)(q - A.r0) < (unsigned)(A.r1 - A.r0) && (!EDGE || jc < A.nc));
        cout += A.pc;
#pragma unroll
        for (int u = 0; u < 3; ++u) ra[u] = rc[u];
      } else {
#pragma unroll
        for (int u = 0; u < 3; ++u) rb[u] = rc[u];
      }
    }
#pragma unroll
    for (int a = 0; a < WIN; ++a) {
      E[a][0] = E[a + D][0]; E[a][1] = E[a + D][1];
      F[a][0] = F[a + D][0]; F[a][1] = F[a + D][1];
    }
  }
  tma::cp_async_wait<0>();
}

template <int NU>
__global__ void __launch_bounds__(32 * kWarps) mg_down_strip_kernel(const TileRef* __restrict__ items, int n_items,
                                                                    const JobDev* __restrict__ jobs,
                                                                    const JobState* __restrict__ st, int l) {
  __shared__ __align__(16) float2 ring[kWarps][kDownRing * 32];
  constexpr int T = 2 * NU;
  tma::pdl_trigger();
  const int warp = threadIdx.x >> 5, item = blockIdx.x * kWarps + warp, lane = threadIdx.x & 31;
  if (item >= n_items) return;
  // item, job and job-state fields: none of them is written by the previous level's launch
  const TileRef tr = items[item];
  const int rows = tr.nlocal;
  const JobDev& J = jobs[tr.job];
  const JobState& S = st[tr.job];
  if (S.converged) { tma::pdl_wait(); return; }   // waits all the same: see pdl_wait
  DownArgs A;
  A.n = J.nl[l]; A.nc = J.nl[l + 1]; A.pf = J.pl[l]; A.pc = J.pl[l + 1];
  const double hl = J.h * (double)(1 << l);
  A.h2 = (float)(hl * hl);
  A.inv_h2 = (float)(1.0 / (hl * hl));
  A.omega = J.omega;
  const int x0 = tr.ti * 2 * down_lanes(NU) - 2 * down_lo(NU);
  A.c0 = x0 + 2 * lane;
  A.r0 = tr.tj * rows;
  A.r1 = min(A.r0 + rows, A.n + 1);   // n is odd: whole pairs of rows
  A.f = (l == 0 && S.fsel) ? J.f0b : J.f[l];
  A.e = J.e[l];
  A.fc = J.f[l + 1];
  tma::pdl_wait();
  const bool edge = x0 < 1 || x0 + 63 > A.n - 2 || A.r0 - T - 2 < 1 || A.r1 + T + 9 > A.n - 1;
  if (edge) down_strip<NU, true>(A, ring[warp]);
  else down_strip<NU, false>(A, ring[warp]);
}

// Up leg: the bilinear prolongation of the coarser correction added to the pre-smoothed one and
// NU post-sweeps.  MODE 0 (level l >= 1): the result to eu_l.  MODE 1 (level 0): phi <- phi + e
// in FP64, the new FP64 defect and the strip's partial of its norm.
struct UpArgs {
  const float *e, *f, *c;    // pre-smoothed correction, right-hand side, coarser correction
  float* out;                // MODE 0: eu_l; MODE 1: the new defect
  const double* phi;
  double* phi_new;
  const void* rho;
  int rmode;
  double inv_h2, rhs_scale;
  int n, nc, pf, pc, c0, r0, r1;
  float h2, omega;
};
// One row step's inputs of a strip: e of row j, f of row j - 1, on odd j the coarse row
// (j + 1) / 2 (two columns per lane), on level 0 phi of row j - T and rho of row j - T - 1 (FP32
// charge in the first half).  phi and rho have the odd row length of the caller's arrays, so no
// copy of theirs can be wider than one value: lane k copies columns k and k + 32, which keeps each
// copy contiguous over the warp, and the lanes read their pairs after a warp barrier.
template <int MODE>
struct __align__(16) UpStep {
  float2 e[32], f[32], c[32];
  double phi[MODE ? 64 : 1], rho[MODE ? 64 : 1];
};

template <int NU, int MODE, bool EDGE>
__device__ __forceinline__ void up_strip(const UpArgs& A, UpStep<MODE>* ring, mgn::Sum& norm) {
  constexpr int T = 2 * NU, WIN = T + 1, WF = T, LO = up_lo(NU, MODE), LANES = up_lanes(NU, MODE), D = up_ring(MODE);
  const int lane = threadIdx.x & 31;
  const int n = A.n, c0 = A.c0, pf = A.pf;
  const float h2 = A.h2, omega = A.omega, om1 = 1.f - omega;
  const bool colin = !EDGE || (unsigned)c0 < (unsigned)n, colin1 = !EDGE || (c0 >= 0 && c0 + 1 < n);
  const bool mine = lane >= LO && lane < LO + LANES && colin;
  const bool upd0 = !EDGE || (c0 >= 1 && c0 <= n - 2), upd1 = !EDGE || (c0 >= 0 && c0 + 1 <= n - 2);
  const int js = A.r0 - T - 2 * MODE, je = A.r1 - 1 + T + MODE;
  // the next row step's sources (see UpStep)
  int next = js;
  const float* esrc = A.e + ((ptrdiff_t)js * pf + c0);
  const float* fsrc = A.f + ((ptrdiff_t)(js - 1) * pf + c0);
  const float* csrc = A.c + ((ptrdiff_t)(js >> 1) * A.pc + (c0 >> 1));
  const int k0 = c0 - lane;                // the column of the lane's first phi and rho copies
  const bool kin = !EDGE || (unsigned)k0 < (unsigned)n, kin1 = !EDGE || (unsigned)(k0 + 32) < (unsigned)n;
  const double* psrc = MODE ? A.phi + ((ptrdiff_t)(js - T) * n + k0) : nullptr;
  const int rsize = A.rmode == 0 ? 4 : 8;
  const char* rsrc = MODE ? static_cast<const char*>(A.rho) + ((ptrdiff_t)(js - T - 1) * n + k0) * rsize : nullptr;
  auto request_c = [&](UpStep<MODE>& s, int m) {
    const bool in = (unsigned)m < (unsigned)A.nc;
    copy4<EDGE>(&s.c[lane].x, csrc, A.c, in && colin);
    copy4<EDGE>(&s.c[lane].y, csrc + 1, A.c, in && colin1);
    csrc += A.pc;
  };
  auto request = [&](int g) {
    UpStep<MODE>& s = ring[g];
    const int j = next;
    copy8<EDGE>(&s.e[lane], esrc, A.e, colin && (unsigned)j < (unsigned)n);
    copy8<EDGE>(&s.f[lane], fsrc, A.f, colin && (unsigned)(j - 1) < (unsigned)n);
    if (g & 1) request_c(s, (j + 1) >> 1);
    if (MODE) {
      const bool qin = (unsigned)(j - T) < (unsigned)n, din = (unsigned)(j - T - 1) < (unsigned)n;
      copy8<EDGE>(&s.phi[lane], psrc, A.phi, qin && kin);
      copy8<EDGE>(&s.phi[lane + 32], psrc + 32, A.phi, qin && kin1);
      if (A.rmode == 0) {
        float* r = reinterpret_cast<float*>(s.rho);
        copy4<EDGE>(r + lane, rsrc, A.rho, din && kin);
        copy4<EDGE>(r + lane + 32, rsrc + 4 * 32, A.rho, din && kin1);
      } else {
        copy8<EDGE>(&s.rho[lane], rsrc, A.rho, din && kin);
        copy8<EDGE>(&s.rho[lane + 32], rsrc + 8 * 32, A.rho, din && kin1);
      }
      psrc += n;
      rsrc += (ptrdiff_t)n * rsize;
    }
    esrc += pf;
    fsrc += pf;
    ++next;
  };
  float* out = A.out + ((ptrdiff_t)(js - T - MODE) * pf + c0);
  double* pout = MODE ? A.phi_new + ((ptrdiff_t)(js - T - 1) * n + c0) : nullptr;
  float E[WIN + D][2], F[WF + D][2];
  double P[2 + D][2];                      // rows j - T - 2, j - T - 1 and the group's
#pragma unroll
  for (int a = 0; a < WIN; ++a) E[a][0] = E[a][1] = 0.f;
#pragma unroll
  for (int a = 0; a < WF; ++a) F[a][0] = F[a][1] = 0.f;
  P[0][0] = P[0][1] = P[1][0] = P[1][1] = 0.0;
  // the coarse row of the first step's row goes through the ring's last slot
  request_c(ring[D - 1], js >> 1);
  tma::cp_async_commit();
  tma::cp_async_wait<0>();
  float2 cc = ring[D - 1].c[lane];
#pragma unroll
  for (int g = 0; g < D; ++g) {
    if (EDGE || js + g <= je) request(g);
    if (g & 1) tma::cp_async_commit();
  }
  for (int jg = js; jg <= je; jg += D) {
    const bool more = EDGE || jg + D <= je;
#pragma unroll
    for (int g = 0; g < D; ++g) {
      const int a = WIN + g, j = jg + g;
      if (!(g & 1)) {
        // the two rows of this pair have arrived for every lane, and every lane has read the rows
        // of the previous pair, whose slots take the next request
        tma::cp_async_wait<D / 2 - 2>();
        __syncwarp();
        if (g > 0 ? more : jg > js) {
          request((g + D - 2) % D);
          request((g + D - 1) % D);
        }
        tma::cp_async_commit();
      }
      const UpStep<MODE>& s = ring[g];
      const float2 ev = s.e[lane], fv = s.f[lane];
      const float2 cn = (g & 1) ? s.c[lane] : cc;
      double2 pv = make_double2(0.0, 0.0), rv = pv;
      if (MODE) {
        pv = reinterpret_cast<const double2*>(s.phi)[lane];
        if (A.rmode == 0) {
          const float2 r = reinterpret_cast<const float2*>(s.rho)[lane];
          rv = make_double2((double)r.x, (double)r.y);
        } else {
          rv = reinterpret_cast<const double2*>(s.rho)[lane];
          if (A.rmode == 1) {
            rv.x = (double)__double_as_longlong(rv.x) * 0x1p-40;
            rv.y = (double)__double_as_longlong(rv.y) * 0x1p-40;
          }
        }
      }
      // row j enters: pre-smoothed correction + bilinear prolongation (Multigrid.cu:378-404);
      // the right-hand side one row behind it
      F[WF + g][0] = fv.x;
      F[WF + g][1] = fv.y;
      if (g & 1) {
        E[a][0] = ev.x + 0.5f * (cc.x + cn.x);
        E[a][1] = ev.y + 0.25f * (cc.x + cc.y + cn.x + cn.y);
        cc = cn;
      } else {
        E[a][0] = ev.x + cc.x;
        E[a][1] = ev.y + 0.5f * (cc.x + cc.y);
      }
      // half-sweep k on row j - 1 - k; its colour sits in c0 on even row steps, c1 on odd
#pragma unroll
      for (int k = 0; k < T; ++k) {
        const int b = a - 1 - k;
        const bool row = !EDGE || (unsigned)(j - k - 2) < (unsigned)(n - 2);
        if (g & 1) {
          const float e = right_of(E[b][0]);
          const float v = relax(E[b + 1][1], E[b - 1][1], e, E[b][0], F[WF + g - k][1], E[b][1], h2, omega, om1);
          E[b][1] = (row && upd1) ? v : E[b][1];
        } else {
          const float w = left_of(E[b][1]);
          const float v = relax(E[b + 1][0], E[b - 1][0], E[b][1], w, F[WF + g - k][0], E[b][0], h2, omega, om1);
          E[b][0] = (row && upd0) ? v : E[b][0];
        }
      }
      const int b = a - T;                   // row j - T, which the last half-sweep completed
      if (MODE == 0) {
        const bool own = mine && (unsigned)(j - T - A.r0) < (unsigned)(A.r1 - A.r0);
        store2(out, E[b][0], E[b][1], own && colin1);
        if (EDGE) store1(out, E[b][0], own && !colin1);
      } else {
        // FP64 update of row j - T, then the defect of row d = j - T - 1
        P[2 + g][0] = pv.x + (double)E[b][0];
        P[2 + g][1] = pv.y + (double)E[b][1];
        const double w = left_of(P[1 + g][1]), e = right_of(P[1 + g][0]);
        const int d = j - T - 1;
        const bool own = mine && (unsigned)(d - A.r0) < (unsigned)(A.r1 - A.r0);
        const bool rowin = !EDGE || (d > 0 && d < n - 1);
        const double lap0 = P[g][0] + P[2 + g][0] + w + P[1 + g][1] - 4.0 * P[1 + g][0];
        const double lap1 = P[g][1] + P[2 + g][1] + P[1 + g][0] + e - 4.0 * P[1 + g][1];
        const double d0 = (rowin && upd0) ? defect(lap0, A.inv_h2, A.rhs_scale, rv.x, d) : 0.0;
        const double d1 = (rowin && upd1) ? defect(lap1, A.inv_h2, A.rhs_scale, rv.y, d) : 0.0;
        store1(pout, P[1 + g][0], own);
        store1(pout + 1, P[1 + g][1], own && colin1);
        store2(out, (float)d0, (float)d1, own && colin1);
        if (EDGE) store1(out, (float)d0, own && !colin1);
        pout += n;
        norm.add(own ? mgn::pair_of(d0, d1) : 0.0);
      }
      out += pf;
    }
#pragma unroll
    for (int a = 0; a < WIN; ++a) { E[a][0] = E[a + D][0]; E[a][1] = E[a + D][1]; }
#pragma unroll
    for (int a = 0; a < WF; ++a) { F[a][0] = F[a + D][0]; F[a][1] = F[a + D][1]; }
    if (MODE) { P[0][0] = P[D][0]; P[0][1] = P[D][1]; P[1][0] = P[D + 1][0]; P[1][1] = P[D + 1][1]; }
  }
  tma::cp_async_wait<0>();
}

// Level 0: 15 warps per SM at 128 registers (five CTAs of three warps; with four of four the norm's sums
// spill more: V-cycle at 2049^2 116.1 us against 114.2, 4097^2 274.8 against 272).
template <int NU, int MODE>
__global__ void __launch_bounds__(32 * up_warps(MODE), 5) mg_up_strip_kernel(const TileRef* __restrict__ items, int n_items,
                                                                  const JobDev* __restrict__ jobs,
                                                                  JobState* __restrict__ st, int l) {
  __shared__ __align__(16) UpStep<MODE> ring[up_warps(MODE)][up_ring(MODE)];
  constexpr int T = 2 * NU;
  tma::pdl_trigger();
  const int warp = threadIdx.x >> 5, item = blockIdx.x * up_warps(MODE) + warp, lane = threadIdx.x & 31;
  if (item >= n_items) return;
  // the job state changes only in mg_finish_kernel, at the end of a V-cycle (the next V-cycle's
  // first launch waits for it), so it is read before waiting for the previous launch
  const TileRef tr = items[item];
  const int rows = tr.nlocal;
  const JobDev& J = jobs[tr.job];
  const JobState& S = st[tr.job];
  if (S.converged) { tma::pdl_wait(); return; }   // waits all the same: see pdl_wait
  UpArgs A;
  A.n = J.nl[l]; A.nc = J.nl[l + 1]; A.pf = J.pl[l]; A.pc = J.pl[l + 1];
  const double hl = J.h * (double)(1 << l);
  A.h2 = (float)(hl * hl);
  A.omega = J.omega;
  const int x0 = tr.ti * 2 * up_lanes(NU, MODE) - 2 * up_lo(NU, MODE);
  A.c0 = x0 + 2 * lane;
  A.r0 = tr.tj * rows;
  A.r1 = min(A.r0 + rows, A.n);
  const int fsel = S.fsel;
  A.e = J.e[l];
  A.f = (l == 0 && fsel) ? J.f0b : J.f[l];
  A.c = l + 1 == J.lc ? J.e[l + 1] : J.eu[l + 1];
  A.out = MODE == 0 ? J.eu[l] : fsel ? J.f[0] : J.f0b;   // the new defect goes to the other buffer
  if (MODE) {
    A.phi = J.phi64[S.phi_cur];
    A.phi_new = J.phi64[S.phi_nxt];
    A.rmode = J.deposit_mode;
    A.rho = A.rmode == 0 ? (const void*)J.rho_f : A.rmode == 1 ? (const void*)J.rho_i : (const void*)J.rho_d;
    A.inv_h2 = 1.0 / (J.h * J.h);
    A.rhs_scale = J.rhs_scale;
  }
  const double rnorm2 = MODE ? S.rnorm2 : 0.0;
  tma::pdl_wait();
  const bool edge = x0 < 1 || x0 + 63 > A.n - 2 || A.r0 - (MODE ? 2 * T + 3 : T + 1) < 0 || A.r1 + T + 9 > A.n - 1;
  const mgn::Scale scale(rnorm2, A.n);
  mgn::Sum norm(scale);
  if (edge) up_strip<NU, MODE, true>(A, ring[warp], norm);
  else up_strip<NU, MODE, false>(A, ring[warp], norm);
  if (MODE) {
    const mgn::Part p = mgn::warp_part(norm.part(scale, rows));
    if (lane == 0) reinterpret_cast<mgn::Part*>(J.partials)[tr.pbase + tr.local] = p;
  }
}

}  // namespace mgs
