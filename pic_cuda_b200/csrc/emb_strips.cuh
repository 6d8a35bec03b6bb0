// emb_strips.cuh — the embedded-boundary multigrid's smoothing kernels as pipelines of rows in
// registers, for levels with enough nodes (the FP64, masked counterpart of mg_strips.cuh).
//
// One warp owns a strip of 64 columns (lane: the even column c0 = x0 + 2 lane and c1 = c0 + 1) and walks
// it row by row; the T = 2 NU half-sweeps follow one another down the strip one row apart, each lane
// holding one node of either colour per row.  Inputs arrive through a per-warp ring of row steps in
// shared memory (cp.async): phi and the right-hand side have the caller's row length, so no copy can
// be wider than one value, and lane k copies columns k and k + 32; the node kinds come as the
// aligned words around the row's 64 bytes.  Every node goes through the expressions of the tile
// kernels in the same order, so results are the same bits.
//
// Why: the tile kernels (colour-split FP64 tiles in shared memory, a block barrier per half-sweep, 44 x
// 44 nodes for 32 x 32) are bound by instruction issue at a quarter of the memory rate.  At 4097^2 (ncu,
// cold) the down leg went from 265 to 168 us and the post-smoothing from 250 to 131 us; both are bound
// by the FP64 chains of a row step with 16 warps per SM (issue 50% active, DRAM 38%).
#pragma once
#include <type_traits>
#include "common.cuh"
#include "tma.cuh"

namespace embs {

constexpr int kWarps = 4;   // strips per CTA
constexpr int kRing = 6;    // row steps in flight, and rows per unrolled step
constexpr int kMaxNu = 3;   // largest sweep count with a strip kernel

// First owned lane and owned lanes of a strip: down leg (residual and full weighting follow the
// sweeps) and smoothing alone.
__host__ __device__ constexpr int lo(int nu, bool down) { return down ? nu + 1 : nu; }
__host__ __device__ constexpr int lanes(int nu, bool down) { return down ? 30 - 2 * nu : 32 - 2 * nu; }
__host__ __device__ constexpr int strips(int nu, bool down, int n) {
  return (n + 2 * lanes(nu, down) - 1) / (2 * lanes(nu, down));
}
// Most rows per item, at most `at_most`, that fill whole unrolled steps (0 if fewer than 8).
inline int rows_fit(int nu, bool down, int at_most) {
  const int lead = down ? 4 * nu + 4 : 4 * nu;
  const int rows = (at_most + lead) / kRing * kRing - lead;
  return rows >= 8 ? rows : 0;
}

struct Args {
  const double* phi;
  double* out;
  const double* rhs;
  const uint8_t* mask;
  const double* bc;       // DIRICHLET values, or null
  const double* coarse;   // coarser phi (PRO)
  double *rhs_c, *phi_c;  // down leg's outputs
  uint8_t* mask_c;
  int nx, ny, nxc, nyc;
  double h2;
  int bilinear, any;
  int rows, strips_x, items;
  const int* done;        // solver's flag (null: none): nothing to do where it is set
};

// Inputs of one row step (read back as 16-byte pairs, so its size is a multiple of 16).
template <bool PRO>
struct __align__(16) Step {
  double phi[64], rhs[64], c[PRO ? 34 : 2];
  uint32_t kind[20];
};
static_assert(sizeof(Step<false>) % 16 == 0 && sizeof(Step<true>) % 16 == 0, "aligned row steps");

__device__ __forceinline__ double left_of(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double right_of(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }

__device__ __forceinline__ void store_if(uint8_t* p, uint32_t v, bool ok) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.u8 [%0], %1;\n\t}" ::"l"(
                   __cvta_generic_to_global(p)), "r"(v), "r"((unsigned)ok) : "memory");
}
__device__ __forceinline__ void store_if(double* p, double v, bool ok) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.f64 [%0], %1;\n\t}" ::"l"(
                   __cvta_generic_to_global(p)), "d"(v), "r"((unsigned)ok) : "memory");
}

// Node kinds of a lane's pair in one word: bits 0-1 column c0, bits 2-3 column c1; 0 FLUID,
// 1 DIRICHLET, 2 SOLID or anything else, 3 grid boundary or outside.
__device__ __forceinline__ uint32_t kind_code(uint32_t m) {
  return m == PIC_NODE_FLUID ? 0u : m == PIC_NODE_DIRICHLET ? 1u : 2u;
}

// DOWN: NU pre-sweeps, the smoothed phi, and the full-weighted residual, kinds and zero phi of the
// coarser level.  Otherwise NU sweeps, after adding the coarse correction with PRO.  EDGE: the strip or
// its rows touch the grid's boundary, so loads and nodes are tested.
template <int NU, bool DOWN, bool PRO, bool EDGE>
__device__ __forceinline__ void strip(const Args& A, Step<PRO>* ring, int x0, int r0) {
  constexpr int T = 2 * NU, WIN = T + (DOWN ? 2 : 1), D = kRing, LO = lo(NU, DOWN), LANES = lanes(NU, DOWN);
  const int lane = threadIdx.x & 31;
  const int nx = A.nx, ny = A.ny, c0 = x0 + 2 * lane;
  const double h2 = A.h2, h2i = 1.0 / A.h2;
  const bool has_bc = A.bc != nullptr;
  const bool mine = lane >= LO && lane < LO + LANES && (!EDGE || c0 < nx);
  const bool mine1 = mine && (!EDGE || c0 + 1 < nx);
  const bool in0 = !EDGE || (c0 > 0 && c0 < nx - 1), in1 = !EDGE || (c0 >= 0 && c0 + 1 < nx - 1);   // interior columns
  const int rend = min(r0 + A.rows, ny);                    // owned rows [r0, rend)
  const int js = DOWN ? r0 - T - 2 : r0 - T, je = DOWN ? r0 + A.rows + T : r0 + A.rows - 1 + T;
  const int last = EDGE ? je : min(je, rend + T + 1);
  // the next row step's sources: 32-bit positions, so that the array bases stay in constant memory
  // (levels of less than 2^30 nodes only)
  const int k0 = x0 + lane;
  int next = js, pos = js * nx + k0, cpos = PRO ? (js >> 1) * A.nxc + (x0 >> 1) + lane : 0;
  const bool kin = !EDGE || (unsigned)k0 < (unsigned)nx, kin1 = !EDGE || (unsigned)(k0 + 32) < (unsigned)nx;
  auto request_c = [&](Step<PRO>& s, int m) {
    const bool row = !EDGE || (unsigned)m < (unsigned)A.nyc;
    const bool a = row && (!EDGE || (unsigned)((x0 >> 1) + lane) < (unsigned)A.nxc);
    const bool b = row && lane == 0 && (!EDGE || (unsigned)((x0 >> 1) + 32) < (unsigned)A.nxc);
    tma::cp_async8(&s.c[lane], A.coarse + (a ? cpos : 0), a);
    if (lane == 0) tma::cp_async8(&s.c[32], A.coarse + (b ? cpos + 32 : 0), b);
    cpos += A.nxc;
  };
  auto request = [&](int g) {
    Step<PRO>& s = ring[g];
    const bool row = !EDGE || (unsigned)next < (unsigned)ny;
    const bool a = row && kin, b = row && kin1;
    tma::cp_async8(&s.phi[lane], A.phi + (a ? pos : 0), a);
    tma::cp_async8(&s.phi[lane + 32], A.phi + (b ? pos + 32 : 0), b);
    tma::cp_async8(&s.rhs[lane], A.rhs + (a ? pos : 0), a);
    tma::cp_async8(&s.rhs[lane + 32], A.rhs + (b ? pos + 32 : 0), b);
    if (!EDGE && lane < 17) {
      const uintptr_t w = reinterpret_cast<uintptr_t>(A.mask + (pos - lane)) & ~(uintptr_t)3;
      tma::cp_async4(&s.kind[lane], reinterpret_cast<const uint32_t*>(w) + lane, true);
    }
    if (PRO && (g & 1)) request_c(s, (next + 1) >> 1);
    pos += nx;
    ++next;
  };
  const uint32_t mask_low = (uint32_t)(reinterpret_cast<uintptr_t>(A.mask) & 3);
  int at = js * nx + c0;                       // the entering row's node c0
  double E[WIN + D][2], F[WIN + D][2];
  uint32_t K[WIN + D];
#pragma unroll
  for (int a = 0; a < WIN; ++a) { E[a][0] = E[a][1] = F[a][0] = F[a][1] = 0.0; K[a] = 15u; }
  // what the full weighting needs of the two rows before: residuals of column c0 and partial sums
  double a1 = 0.0, corners = 0.0, b1 = 0.0, cross = 0.0;
  uint32_t fluid_rows = 0;                                  // bit k: row j - k is FLUID in all 64 columns
  uint32_t ka = 0, kb = 0;                                  // OR of the kinds of three columns, two rows back
  double cc0 = 0.0, cc1 = 0.0;
  if (PRO) {
    request_c(ring[D - 1], js >> 1);   // the coarse row at the first step's row, through the last slot
    tma::cp_async_commit();
    tma::cp_async_wait<0>();
    __syncwarp();
    cc0 = ring[D - 1].c[lane];
    cc1 = ring[D - 1].c[lane + 1];
    __syncwarp();
  }
#pragma unroll
  for (int g = 0; g < D; ++g) {
    if (EDGE || js + g <= last) request(g);
    if (g & 1) tma::cp_async_commit();
  }
  for (int jg = js; jg <= last; jg += D) {
    const bool more = EDGE || jg + D <= last;
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
      const Step<PRO>& s = ring[g];
      const double2 pv = reinterpret_cast<const double2*>(s.phi)[lane];
      double2 fv = reinterpret_cast<const double2*>(s.rhs)[lane];
      uint32_t m0, m1;
      if (EDGE) {
        const bool row = j > 0 && j < ny - 1;
        m0 = row && in0 ? kind_code(A.mask[at]) : 3u;
        m1 = row && in1 ? kind_code(A.mask[at + 1]) : 3u;
      } else {
        const uint8_t* w = reinterpret_cast<const uint8_t*>(s.kind) + ((mask_low + (uint32_t)(at - 2 * lane)) & 3u) + 2 * lane;
        m0 = kind_code(w[0]);
        m1 = kind_code(w[1]);
      }
      K[a] = m0 | m1 << 2;
      // right-hand side slot: rhs on FLUID, phi_bc on DIRICHLET nodes with phi_bc, 0 otherwise
      const bool plain = !EDGE && __all_sync(0xffffffffu, (m0 | m1) == 0u);
      fluid_rows = fluid_rows << 1 | (plain ? 1u : 0u);
      if (!plain) {
        if (m0) fv.x = 0.0;
        if (m1) fv.y = 0.0;
        if (has_bc) {
          const double* b = A.bc + at;
          if (m0 == 1u) fv.x = b[0];
          if (m1 == 1u) fv.y = b[1];
        }
      }
      E[a][0] = pv.x; E[a][1] = pv.y;
      F[a][0] = fv.x; F[a][1] = fv.y;
      if (PRO) {
        // bilinear, or the coarse node (i / 2, j / 2), on FLUID nodes
        double v0, v1;
        if (g & 1) {
          const double d0 = s.c[lane], d1 = s.c[lane + 1];
          v0 = A.bilinear ? 0.5 * (cc0 + d0) : cc0;
          v1 = A.bilinear ? 0.25 * (cc0 + cc1 + d0 + d1) : cc0;
          cc0 = d0;
          cc1 = d1;
        } else {
          v0 = cc0;
          v1 = A.bilinear ? 0.5 * (cc0 + cc1) : cc0;
        }
        if (!m0) E[a][0] += v0;
        if (!m1) E[a][1] += v1;
      }
      // half-sweep k on row j - 1 - k (even colour first); its colour sits in c1 on even row steps.
      // Where every row in the window is all FLUID (nearly everywhere) without looking at the kinds.
      auto sweeps = [&](auto masked) {
#pragma unroll
        for (int k = 0; k < T; ++k) {
          const int b = a - 1 - k, u = (g & 1) ? 0 : 1;
          const double w = u ? E[b][0] : left_of(E[b][1]), e = u ? right_of(E[b][0]) : E[b][1];
          const double sum = E[b - 1][u] + E[b + 1][u] + w + e;
          const double v = 0.25 * fma(-h2, F[b][u], sum);
          if constexpr (decltype(masked)::value) {
            const uint32_t m = (K[b] >> (2 * u)) & 3u;
            E[b][u] = m == 0u ? v : (m == 1u && has_bc) ? F[b][u] : E[b][u];
          } else {
            E[b][u] = v;
          }
        }
      };
      constexpr uint32_t kWindow = (1u << (T + (DOWN ? 4 : 2))) - 1u;   // rows back to the oldest one looked at
      const bool window = !EDGE && (fluid_rows & kWindow) == kWindow;
      if (window) sweeps(std::false_type{});
      else sweeps(std::true_type{});
      {
        const int b = a - T, q = j - T;      // the row the last half-sweep completed
        const bool row = q >= r0 && q < rend;
        double* out = A.out + (at - T * nx);
        store_if(out, E[b][0], row && mine);
        store_if(out + 1, E[b][1], row && mine1);
      }
      if (DOWN) {
        // residual of row q = j - T - 1, and on odd q the full weighting of the three last rows
        const int b = a - T - 1, q = j - T - 1;
        double rc[3];
        const double w = left_of(E[b][1]), e = right_of(E[b][0]);
        const double l0 = E[b - 1][0] + E[b + 1][0] + w + E[b][1] - 4.0 * E[b][0];
        const double l1 = E[b - 1][1] + E[b + 1][1] + E[b][0] + e - 4.0 * E[b][1];
        rc[1] = fma(-h2i, l0, F[b][0]);
        rc[2] = fma(-h2i, l1, F[b][1]);
        if (!window) {
          if (K[b] & 3u) rc[1] = 0.0;
          if (K[b] & 12u) rc[2] = 0.0;
        }
        rc[0] = left_of(rc[2]);
        // kinds of columns c0 - 1, c0, c0 + 1 as two flags: 1 some DIRICHLET, 2 some other non-FLUID
        const uint32_t kl = __shfl_up_sync(0xffffffffu, K[b], 1) >> 2, kc = K[b] & 3u, kr = K[b] >> 2;
        const uint32_t kk = (kl | kc | kr);
        if (!(g & 1)) {                      // odd q
          const int jc = (q - 1) >> 1, ic = c0 >> 1;
          const bool own = mine && q > r0 && jc < (r0 + A.rows) / 2 && (!EDGE || (jc < A.nyc && ic < A.nxc));
          const bool inner = !EDGE || (ic > 0 && jc > 0 && ic < A.nxc - 1 && jc < A.nyc - 1);
          uint32_t kind = PIC_NODE_FLUID;
          if (!window) {
            const uint32_t three = ka | kb | kk, centre = K[b - 1] & 3u;
            if (A.any) kind = (three & 1u) ? PIC_NODE_DIRICHLET : (three & 2u) ? PIC_NODE_SOLID : PIC_NODE_FLUID;
            else kind = centre == 0u ? (uint32_t)PIC_NODE_FLUID : centre == 1u ? (uint32_t)PIC_NODE_DIRICHLET
                        : own && inner ? A.mask[2 * jc * nx + c0] : (uint32_t)PIC_NODE_SOLID;
            if (!inner) kind = PIC_NODE_FLUID;
          }
          double sum = b1;                   // the tile kernel's order: centre, cross, corners
          sum += 0.5 * (cross + rc[1]);
          sum += 0.25 * (corners + rc[0] + rc[2]);
          const int id = jc * A.nxc + ic;
          store_if(A.phi_c + id, 0.0, own);
          store_if(A.rhs_c + id, inner && kind == PIC_NODE_FLUID ? sum / 4.0 : 0.0, own);
          store_if(A.mask_c + id, kind, own);
          a1 = rc[1];
          corners = rc[0] + rc[2];
          ka = kk;
        } else {
          b1 = rc[1];
          cross = rc[0] + rc[2] + a1;
          kb = kk;
        }
      }
      at += nx;
    }
#pragma unroll
    for (int a = 0; a < WIN; ++a) {
      E[a][0] = E[a + D][0]; E[a][1] = E[a + D][1];
      F[a][0] = F[a + D][0]; F[a][1] = F[a + D][1];
      K[a] = K[a + D];
    }
  }
  tma::cp_async_wait<0>();
}

template <int NU, bool DOWN, bool PRO>
__global__ void __launch_bounds__(32 * kWarps, NU < 3 ? 4 : 3) emb_strip_kernel(const __grid_constant__ Args A) {
  __shared__ __align__(16) Step<PRO> ring[kWarps][kRing];
  constexpr int T = 2 * NU;
  tma::pdl_trigger();
  const int warp = threadIdx.x >> 5, item = blockIdx.x * kWarps + warp;
  if (item >= A.items) return;
  tma::pdl_wait();
  if (A.done && *A.done) return;
  const int tj = item / A.strips_x, ti = item - tj * A.strips_x;
  const int x0 = ti * 2 * lanes(NU, DOWN) - 2 * lo(NU, DOWN), r0 = tj * A.rows;
  // rows read: down to r0 - T - 2 and up to r0 + rows + T + 7 (the last unrolled step runs over)
  const bool edge = x0 < 1 || x0 + 67 > A.nx - 1 || r0 - T - 3 < 1 || r0 + A.rows + T + 8 > A.ny - 1;
  if (edge) strip<NU, DOWN, PRO, true>(A, ring[warp], x0, r0);
  else strip<NU, DOWN, PRO, false>(A, ring[warp], x0, r0);
}

}  // namespace embs
