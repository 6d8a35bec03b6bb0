// mg_embedded.cu — embedded-boundary multigrid: lap(phi) = rhs on the FLUID nodes of a node
// mask, with interior electrodes (DIRICHLET nodes held at phi_bc) and excluded regions (SOLID
// nodes left as they are).  Algorithm of the reference's Multigrid_embedded.cu:1-190
// (Multigrid::vcycle, :159-188), FP64 like the reference:
//   pre-smoothing   nu_pre red-black Gauss-Seidel sweeps, colour (i+j) even first
//                   (smooth_redblack :15-33, with the intended colour test: the reference's
//                   `(i + j) & 1 != redblack` parses as (i + j) & (1 != redblack))
//   restriction     r = rhs - lap(phi)/h^2 on FLUID nodes (residual_kernel :35-55), full
//                   weighting onto FLUID coarse nodes (restrict_kernel :57-86); coarse mask =
//                   the fine node (2i, 2j)'s, or with PIC_EMB_COARSEN_ANY the rule the
//                   reference's comment at :73 states (any DIRICHLET fine node of the 3x3
//                   stencil makes the coarse node DIRICHLET; else any other non-FLUID one
//                   makes it SOLID)
//   coarse level    phi = 0 (:151), recursion; the coarsest level runs the pre-sweeps only
//   prolongation    FLUID fine nodes add coarse (i/2, j/2) (prolongate_add_kernel :88-104),
//                   or with PIC_EMB_PROLONG_BILINEAR the bilinear interpolant
//   post-smoothing  nu_post sweeps
// Level l has spacing h 2^l.  DIRICHLET nodes take phi_bc of their level; without a phi_bc
// array they keep the value phi holds (coarse levels start from phi = 0, so that is 0, what
// the reference's zeroed coarse phi_bc arrays give).
//
// Kernels of one V-cycle:
//   emb_down_kernel<NU>  pre-smoothing fused with the restriction: a 32 x 32 output tile with
//       a halo of 2 NU + 2 nodes (phi, node kinds and the right-hand side, DIRICHLET nodes'
//       phi_bc in the same slot, staged in shared memory with every load of a thread issued
//       at once); the NU sweeps run there (after k half-sweeps every node at least k nodes
//       inside the tile edge is exact); the smoothed output region is written back, and the
//       16 x 16 coarse nodes of the tile get the full-weighted residual of their nine fine
//       nodes (from shared memory), their kind, and phi = 0.  No residual array.
//   emb_smooth_kernel<NU, PRO>  the same tile scheme with a halo of 2 NU for the
//       post-smoothing: the coarse correction is prolongated while staging (PRO).  Tiles read
//       halos that neighbouring CTAs own, so results go to the level's other phi buffer.
//   Levels with enough nodes (strip_args) run the same smoothing as pipelines of rows in registers
//       (emb_strip_kernel, emb_strips.cuh), with the same bits.
//   emb_coarse_kernel  every level from the first one with at most 65 x 65 nodes down, in one
//       CTA's shared memory (one launch for the whole lower V-cycle).
//   emb_norm_kernel  ||r||^2 and ||rhs||^2 over the FLUID nodes in a fixed order (per-CTA
//       partials, then the last CTA), for the convergence test, which that CTA makes: it sets the solve's done flag, and the host sends cycles in groups instead of
//       waiting for each one's norm (385 x 257, 50 cycles: 4.78 -> 3.69 ms, the wait, the copy and
//       the restart having taken 20 us of a cycle's 97).
// At 385 x 257 a cycle is a chain of eight short launches, each bound by its own chain of loads,
// half-sweeps and barriers, not by bandwidth: programmatic launches overlap each one's start-up with its
// predecessor's end (V-cycle 77.8 -> 76.4 us; 1025^2 133.8 -> 123.4), and a CTA of 1024 threads, one node
// of each colour per thread, shortens the chain (76 -> 54 us; 1025^2 124 -> 103; with 256 threads on
// 16 x 16 tiles 61 and 127); with the one-CTA kernel's share 48 and 95 us.
// The shared tiles store each colour's nodes contiguously (struct Tile), so a red-black
// half-sweep reads its FP64 neighbours at unit stride.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <vector>
#include "common.cuh"
#include "emb_strips.cuh"
#include "kernels.h"

int pic_fail(int code, const char* msg);

namespace {

constexpr uint8_t kFluid = PIC_NODE_FLUID, kDir = PIC_NODE_DIRICHLET, kSolid = PIC_NODE_SOLID;
constexpr uint8_t kFixed = 255;            // grid boundary / outside the grid: never updated
constexpr int kTile = 32;
constexpr int kSmoothThreads = 1024;
constexpr int kCoarseThreads = 1024;
constexpr int kCoarseMaxNodes = 65 * 65;   // first level at or below this size: one-CTA solve
constexpr int kNormBlocks = 592;

// Coarse correction at fine node (gx, gy) (an interior node, so every coarse index used
// lies inside the coarse grid: gx <= nx - 2 gives (gx + 1) / 2 <= nxc - 1).
__device__ __forceinline__ double prolong_at(const double* __restrict__ c, int nxc, int gx, int gy, bool bilinear) {
  const int ic = gx >> 1, jc = gy >> 1;
  const size_t a = (size_t)jc * nxc + ic;
  if (!bilinear) return c[a];
  const bool io = gx & 1, jo = gy & 1;
  if (!io && !jo) return c[a];
  if (io && !jo) return 0.5 * (c[a] + c[a + 1]);
  if (!io && jo) return 0.5 * (c[a] + c[a + nxc]);
  return 0.25 * (c[a] + c[a + 1] + c[a + nxc] + c[a + nxc + 1]);
}

// Node kind as the smoother treats it: FLUID, DIRICHLET (value in the rhs slot) or SOLID.
__device__ __forceinline__ uint8_t smoother_kind(uint8_t m, bool has_bc) {
  if (m == kFluid) return kFluid;
  if (m == kDir && has_bc) return kDir;
  return kSolid;
}

// Shared-memory tile of W x W nodes (W even) whose node (0, 0) is grid node (x0, y0), with
// x0 + y0 even, so a node's colour is (tx + ty) & 1.  Each colour is stored on its own: node
// (tx, ty) sits at [colour][ty * W/2 + tx/2].  A red-black half-sweep then reads the other
// colour's neighbours at consecutive FP64 words across a warp (the interleaved layout reads
// them at a stride of two words, two-way bank conflicts), and the rows of one colour share
// the parity of tx, so W/E neighbours are at q - 1 + (tx & 1) and q + (tx & 1).
template <int W>
struct Tile {
  static constexpr int HW = W / 2;
  double p[2][HW * W];    // phi
  double rb[2][HW * W];   // rhs (FLUID), phi_bc (DIRICHLET with phi_bc), 0 otherwise
  uint8_t m[2][HW * W];   // the caller's node kinds; kFixed on the grid boundary and outside
  __device__ __forceinline__ static int at(int tx, int ty) { return ty * HW + (tx >> 1); }
  __device__ __forceinline__ static int colour(int tx, int ty) { return (tx + ty) & 1; }
  __device__ __forceinline__ double phi(int tx, int ty) const { return p[colour(tx, ty)][at(tx, ty)]; }
  __device__ __forceinline__ uint8_t kind(int tx, int ty) const { return m[colour(tx, ty)][at(tx, ty)]; }
  // residual_kernel's expression at an interior tile node: rhs - (S + N + W + E - 4 phi) / h^2
  __device__ __forceinline__ double residual(int tx, int ty, double h2i) const {
    const int c = colour(tx, ty), o = c ^ 1, i = at(tx, ty);
    if (m[c][i] != kFluid) return 0.0;
    const int w = i - 1 + (tx & 1);
    const double lap = p[o][i - HW] + p[o][i + HW] + p[o][w] + p[o][w + 1] - 4.0 * p[c][i];
    return rb[c][i] - h2i * lap;
  }
};

// NU sweeps of smooth_redblack on the interior tile nodes, colour (i + j) even first.  Thread k has one
// node of each colour, the (k % H)-th one of its colour in row 1 + k / H (H = (W - 2) / 2 per row), and a
// second pair 1024 nodes further on where the tile is that large (four sweeps): their kinds and
// right-hand sides stay in registers, and a half-sweep is four shared loads, the FP64 chain and a
// barrier.  FLUID nodes relax, DIRICHLET nodes take their phi_bc when the caller gave one, others stay.
template <int W, int NU>
__device__ __forceinline__ void tile_sweeps(Tile<W>& T, double h2, bool has_bc) {
  if (NU == 0) return;
  constexpr int HW = W / 2, HALF = (W - 2) / 2, CNT = (W - 2) * HALF;
  constexpr int IT = (CNT + kSmoothThreads - 1) / kSmoothThreads;
  int at[IT], par[IT];        // place of the pair in its row; tx parity of the colour-0 node
  double rb[IT][2];
  uint8_t m[IT][2];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int k = threadIdx.x + it * kSmoothThreads;
    const int r = k / HALF, ty = 1 + r;
    const int base = ty * HW + (k - r * HALF);
    at[it] = base;
    par[it] = ty & 1;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int i = base + ((par[it] ^ c) ? 0 : 1);
      m[it][c] = kFixed; rb[it][c] = 0.0;
      if (k < CNT) { m[it][c] = T.m[c][i]; rb[it][c] = T.rb[c][i]; }
    }
  }
#pragma unroll 1
  for (int s = 0; s < NU; ++s) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      double* __restrict__ own = T.p[c];
      const double* __restrict__ oth = T.p[c ^ 1];
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int odd = par[it] ^ c, i = at[it] + 1 - odd;
        if (m[it][c] == kFluid) {
          const double sum = oth[i - HW] + oth[i + HW] + oth[at[it]] + oth[at[it] + 1];
          own[i] = 0.25 * fma(-h2, rb[it][c], sum);   // written out: h2 * rb must not be kept as a product
        } else if (m[it][c] == kDir && has_bc) {
          own[i] = rb[it][c];
        }
      }
      __syncthreads();
    }
  }
}

// Stages the tile: phi, the node kind and the rhs slot of every node.  Every load of a thread
// is issued before any is used, so a tile waits for one memory latency; the DIRICHLET values
// (rare) and, with PRO, the coarse correction of the FLUID nodes follow in a second round.
template <int W, bool PRO>
__device__ __forceinline__ void stage_tile(Tile<W>& T, const double* __restrict__ phi, const double* __restrict__ rhs,
                                           const uint8_t* __restrict__ mask, const double* __restrict__ bc,
                                           const double* __restrict__ coarse, int nx, int ny, int nxc, int x0, int y0,
                                           bool bilinear) {
  constexpr int IT = (W * W + kSmoothThreads - 1) / kSmoothThreads;
  double p[IT], r[IT];
  uint8_t m[IT];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int k = threadIdx.x + it * kSmoothThreads;
    p[it] = 0.0; r[it] = 0.0; m[it] = kFixed;
    if (k < W * W) {
      const int ty = k / W, tx = k - ty * W;
      const int gx = x0 + tx, gy = y0 + ty;
      if (gx >= 0 && gy >= 0 && gx < nx && gy < ny) {
        const size_t id = (size_t)gy * nx + gx;
        p[it] = phi[id];
        if (gx > 0 && gy > 0 && gx < nx - 1 && gy < ny - 1) {
          m[it] = mask[id];
          r[it] = rhs[id];
        }
      }
    }
  }
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int k = threadIdx.x + it * kSmoothThreads;
    if (k < W * W) {
      const int ty = k / W, tx = k - ty * W;
      const int gx = x0 + tx, gy = y0 + ty;
      double pv = p[it], rv = r[it];
      if (m[it] == kFluid) {
        if (PRO) pv += prolong_at(coarse, nxc, gx, gy, bilinear);
      } else {
        rv = (m[it] == kDir && bc) ? bc[(size_t)gy * nx + gx] : 0.0;
      }
      const int c = Tile<W>::colour(tx, ty), i = Tile<W>::at(tx, ty);
      T.p[c][i] = pv; T.rb[c][i] = rv; T.m[c][i] = m[it];
    }
  }
}

// The 32 x 32 output region of a staged tile (halo H) back to global memory.
template <int W, int H>
__device__ __forceinline__ void store_tile(const Tile<W>& T, double* __restrict__ out, int nx, int ny, int x0,
                                           int y0) {
  for (int k = threadIdx.x; k < kTile * kTile; k += kSmoothThreads) {
    const int ty = k / kTile, tx = k - ty * kTile;
    const int gx = x0 + H + tx, gy = y0 + H + ty;
    if (gx < nx && gy < ny) out[(size_t)gy * nx + gx] = T.phi(tx + H, ty + H);
  }
}

// Start of every kernel of a solve: the next launch may begin its own start-up, this one waits for the
// previous one's results, and where the solver's flag is set there is nothing left to do.
__device__ __forceinline__ bool skip_launch(const int* done) {
  tma::pdl_trigger();
  tma::pdl_wait();
  return done && *done;
}

// NU sweeps (post-smoothing with PRO: after adding the coarse correction) of one tile.
template <int NU, bool PRO>
__global__ void __launch_bounds__(kSmoothThreads) emb_smooth_kernel(
    const double* __restrict__ phi_in, double* __restrict__ phi_out, const double* __restrict__ rhs,
    const uint8_t* __restrict__ mask, const double* __restrict__ bc, const double* __restrict__ coarse, int nx, int ny,
    int nxc, double h2, int bilinear, const int* done) {
  constexpr int H = 2 * NU, W = kTile + 2 * H;
  __shared__ Tile<W> T;
  if (skip_launch(done)) return;
  const int x0 = blockIdx.x * kTile - H, y0 = blockIdx.y * kTile - H;
  stage_tile<W, PRO>(T, phi_in, rhs, mask, bc, coarse, nx, ny, nxc, x0, y0, bilinear != 0);
  __syncthreads();
  tile_sweeps<W, NU>(T, h2, bc != nullptr);
  store_tile<W, H>(T, phi_out, nx, ny, x0, y0);
}

// Coarse node kind from the fine kinds around fine node (tx, ty): the kind of that node, or
// (any) DIRICHLET if any of the 3x3 is, else SOLID if any is not FLUID, else FLUID.
template <class M>
__device__ __forceinline__ uint8_t coarse_kind_of(M kind, bool any) {
  if (!any) return kind(0, 0);
  bool dir = false, other = false;
#pragma unroll
  for (int dj = -1; dj <= 1; ++dj)
#pragma unroll
    for (int di = -1; di <= 1; ++di) {
      const uint8_t m = kind(di, dj);
      dir |= m == kDir;
      other |= m != kFluid && m != kDir;
    }
  return dir ? kDir : other ? kSolid : kFluid;
}

// Full weighting of the fine residual (restrict_kernel's sum order) around a fine node;
// res(di, dj) is the residual at offset (di, dj).
template <class R>
__device__ __forceinline__ double full_weight(R res) {
  double sum = 0.0;
  sum += res(0, 0);
  sum += 0.5 * (res(-1, 0) + res(1, 0) + res(0, -1) + res(0, 1));
  sum += 0.25 * (res(-1, -1) + res(1, -1) + res(-1, 1) + res(1, 1));
  return sum / 4.0;
}

// Pre-smoothing of one tile fused with the restriction: NU sweeps on a tile with a halo of
// 2 NU + 2 (so the smoothed phi is exact two nodes beyond the output region), the 32 x 32
// output region written back, then for the 16 x 16 coarse nodes whose fine node (2i, 2j)
// lies in the output region: the residual of the nine fine nodes from shared memory
// (residual_kernel's expression), full weighting, the coarse kind, and coarse phi = 0.
template <int NU>
__global__ void __launch_bounds__(kSmoothThreads) emb_down_kernel(
    const double* __restrict__ phi_in, double* __restrict__ phi_out, const double* __restrict__ rhs,
    const uint8_t* __restrict__ mask, const double* __restrict__ bc, int nx, int ny, double h2,
    double* __restrict__ rhs_c, uint8_t* __restrict__ mask_c, double* __restrict__ phi_c, int nxc, int nyc, int any,
    const int* done) {
  constexpr int H = 2 * NU + 2, W = kTile + 2 * H;
  __shared__ Tile<W> T;
  if (skip_launch(done)) return;
  const int x0 = blockIdx.x * kTile - H, y0 = blockIdx.y * kTile - H;
  stage_tile<W, false>(T, phi_in, rhs, mask, bc, nullptr, nx, ny, 0, x0, y0, false);
  __syncthreads();
  tile_sweeps<W, NU>(T, h2, bc != nullptr);
  store_tile<W, H>(T, phi_out, nx, ny, x0, y0);
  const double h2i = 1.0 / h2;
  constexpr int CT = kTile / 2;
  const int k = threadIdx.x;            // one coarse node each
  const int ic = blockIdx.x * CT + k % CT, jc = blockIdx.y * CT + k / CT;
  if (k >= CT * CT || ic >= nxc || jc >= nyc) return;
  const size_t idc = (size_t)jc * nxc + ic;
  phi_c[idc] = 0.0;
  if (ic == 0 || jc == 0 || ic == nxc - 1 || jc == nyc - 1) {
    rhs_c[idc] = 0.0;
    mask_c[idc] = kFluid;
    return;
  }
  const int tx = 2 * ic - x0, ty = 2 * jc - y0;
  const uint8_t kc = coarse_kind_of([&](int di, int dj) { return T.kind(tx + di, ty + dj); }, any != 0);
  mask_c[idc] = kc;
  rhs_c[idc] = kc == kFluid ? full_weight([&](int di, int dj) { return T.residual(tx + di, ty + dj, h2i); }) : 0.0;
}

// Residual of fine node id (interior): restatement of residual_kernel's expression.
__device__ __forceinline__ double fine_residual(const double* phi, const double* rhs, const uint8_t* mask, size_t id,
                                                int nx, double h2i) {
  if (mask[id] != kFluid) return 0.0;
  const double lap = phi[id - nx] + phi[id + nx] + phi[id - 1] + phi[id + 1] - 4.0 * phi[id];
  return rhs[id] - h2i * lap;
}

// ---------------------------------------------------------------- one-CTA lower V-cycle
struct CoarseLevelArgs {
  int n;                     // levels lc .. lc + n - 1
  int nx[PIC_MAX_LEVELS], ny[PIC_MAX_LEVELS];
  double* phi[PIC_MAX_LEVELS];
  double* rhs[PIC_MAX_LEVELS];
  uint8_t* mask[PIC_MAX_LEVELS];
  const double* bc[PIC_MAX_LEVELS];
  double h2[PIC_MAX_LEVELS], h2i[PIC_MAX_LEVELS];
  int soff[PIC_MAX_LEVELS];  // byte offsets in shared memory: phi, rb (doubles), then both kinds
  int nu1, nu2, coarsen_any, bilinear;
  const int* done;
};

// One node of a half-sweep: phi in shared memory at p, the rows' stride nx.
__device__ __forceinline__ void relax_node(double* p, int nx, uint8_t kind, double f, double h2) {
  const double s = p[-nx], n = p[nx], w = p[-1], e = p[1];
  if (kind == kFluid) {
    const double sum = s + n + w + e;
    *p = 0.25 * fma(-h2, f, sum);      // written out: h2 * f must not be kept as a product
  } else if (kind == kDir) {
    *p = f;
  }
}

// nu sweeps of one level in shared memory by one CTA of 32 warps: a warp takes a row, its lanes the row's
// nodes of one colour.  A level of at most 66 x 66 nodes gives a thread two nodes of each colour at most;
// their places, kinds and right-hand sides are then read once, and a half-sweep is the neighbours' loads,
// the FP64 chain and a barrier.  (Narrower and longer levels take the loop over rows and lane groups.)
__device__ __forceinline__ void cta_sweeps(double* p, const double* rb, const uint8_t* m, int nx, int ny, int nu,
                                           double h2) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = kCoarseThreads / 32;
  if (nx <= 66 && ny <= 2 * NW + 2) {
    int t[2][2];
    double f[2][2];
    uint8_t kind[2][2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int j = 1 + warp + NW * r, i = 1 + ((1 + j + c) & 1) + 2 * lane;
        const bool in = j < ny - 1 && i < nx - 1;
        t[r][c] = in ? j * nx + i : nx + 1;      // an interior node: its loads stay inside the level
        f[r][c] = rb[t[r][c]];
        kind[r][c] = in ? m[t[r][c]] : kFixed;
      }
    const bool two = 1 + warp + NW < ny - 1;
#pragma unroll 1
    for (int s = 0; s < nu; ++s)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        relax_node(p + t[0][c], nx, kind[0][c], f[0][c], h2);
        if (two) relax_node(p + t[1][c], nx, kind[1][c], f[1][c], h2);
        __syncthreads();
      }
    return;
  }
  for (int s = 0; s < 2 * nu; ++s) {
    for (int j = 1 + warp; j < ny - 1; j += NW)
      for (int i = 1 + ((1 + j + s) & 1) + 2 * lane; i < nx - 1; i += 64)
        relax_node(p + j * nx + i, nx, m[j * nx + i], rb[j * nx + i], h2);
    __syncthreads();
  }
}

// The lower levels in one CTA.  Bound by the latency of the chain of half-sweeps and barriers on one SM
// (65 x 65 and below with 2 + 2 sweeps, of which 385 x 257 uses 49 x 33: 20.5 -> 16.7 us, each sweep reading
// its nodes' places, kinds and right-hand sides again before).
__global__ void __launch_bounds__(kCoarseThreads) emb_coarse_kernel(CoarseLevelArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (skip_launch(A.done)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  auto P = [&](int l) { return reinterpret_cast<double*>(smem + A.soff[l]); };
  auto RB = [&](int l) { return reinterpret_cast<double*>(smem + A.soff[l]) + A.nx[l] * A.ny[l]; };
  auto M = [&](int l) { return reinterpret_cast<uint8_t*>(smem + A.soff[l] + 16 * A.nx[l] * A.ny[l]); };
  auto K = [&](int l) { return M(l) + A.nx[l] * A.ny[l]; };   // the reference's kinds (M: the smoother's)
  // stage the first level: phi, kinds, rhs (DIRICHLET: phi_bc)
  {
    const int nx = A.nx[0], ny = A.ny[0];
    double* p = P(0); double* rb = RB(0); uint8_t* m = M(0); uint8_t* kinds = K(0);
#pragma unroll 4
    for (int j = warp; j < ny; j += nwarp)
      for (int i = lane; i < nx; i += 32) {
        const int k = j * nx + i;
        p[k] = A.phi[0][k];
        uint8_t kk = kFixed;
        const uint8_t raw = A.mask[0][k];
        double v = A.rhs[0][k];
        if (i > 0 && j > 0 && i < nx - 1 && j < ny - 1) kk = smoother_kind(raw, A.bc[0] != nullptr);
        if (kk != kFluid) v = kk == kDir ? A.bc[0][k] : 0.0;
        m[k] = kk; rb[k] = v; kinds[k] = raw;
      }
  }
  __syncthreads();
  // down leg
  int l = 0;
  for (;; ++l) {
    const int nx = A.nx[l], ny = A.ny[l];
    cta_sweeps(P(l), RB(l), M(l), nx, ny, A.nu1, A.h2[l]);
    if (l == A.n - 1) break;
    // restriction from the staged fine level
    const int nxc = A.nx[l + 1], nyc = A.ny[l + 1];
    const double* pf = P(l);
    const double* rbf = RB(l);
    const uint8_t* mk = K(l);
    const double h2i = A.h2i[l];
    double* pc = P(l + 1); double* rbc = RB(l + 1); uint8_t* mc = M(l + 1); uint8_t* kinds_c = K(l + 1);
    for (int jc = warp; jc < nyc; jc += nwarp)
      for (int ic = lane; ic < nxc; ic += 32) {
        const int k = jc * nxc + ic;
        pc[k] = 0.0;
        uint8_t kc = kFluid;
        double fc = 0.0;
        const bool interior = ic > 0 && jc > 0 && ic < nxc - 1 && jc < nyc - 1;
        if (interior) {
          const int idf = 2 * jc * nx + 2 * ic;
          uint8_t kind[9];
#pragma unroll
          for (int q = 0; q < 9; ++q) kind[q] = mk[idf + (q / 3 - 1) * nx + (q % 3 - 1)];
          kc = coarse_kind_of([&](int di, int dj) { return kind[(dj + 1) * 3 + di + 1]; }, A.coarsen_any != 0);
          if (kc == kFluid)
            fc = full_weight([&](int di, int dj) {
                   const int id = idf + dj * nx + di;
                   if (kind[(dj + 1) * 3 + di + 1] != kFluid) return 0.0;
                   const double lap = pf[id - nx] + pf[id + nx] + pf[id - 1] + pf[id + 1] - 4.0 * pf[id];
                   return rbf[id] - h2i * lap;
                 });
        }
        A.mask[l + 1][k] = kc;       // the reference writes the coarse kinds and rhs of every level
        A.rhs[l + 1][k] = fc;
        const uint8_t sk = interior ? smoother_kind(kc, A.bc[l + 1] != nullptr) : kFixed;
        mc[k] = sk;
        kinds_c[k] = kc;
        rbc[k] = sk == kFluid ? fc : sk == kDir ? A.bc[l + 1][k] : 0.0;
      }
    __syncthreads();
  }
  // up leg
  for (l = A.n - 2; l >= 0; --l) {
    const int nx = A.nx[l], ny = A.ny[l], nxc = A.nx[l + 1];
    double* p = P(l);
    const double* pc = P(l + 1);
    const uint8_t* m = M(l);
    for (int j = 1 + warp; j < ny - 1; j += nwarp)
      for (int i = 1 + lane; i < nx - 1; i += 32) {
        const int k = j * nx + i;
        if (m[k] == kFluid) p[k] += prolong_at(pc, nxc, i, j, A.bilinear != 0);
      }
    __syncthreads();
    cta_sweeps(p, RB(l), m, nx, ny, A.nu2, A.h2[l]);
  }
  // every level's phi back to global memory (the reference keeps them in its level arrays)
  for (l = 0; l < A.n; ++l) {
    const int N = A.nx[l] * A.ny[l];
    const double* p = P(l);
    for (int k = threadIdx.x; k < N; k += blockDim.x) A.phi[l][k] = p[k];
  }
}

// ---------------------------------------------------------------- norms
// Sums of a and b over a CTA of 8 warps, in a fixed order, in thread 0.
__device__ __forceinline__ void cta_sums(double& a, double& b, double (*red)[2]) {
  for (int o = 16; o; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) { red[w][0] = a; red[w][1] = b; }
  __syncthreads();
  a = b = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < 8; ++k) { a += red[k][0]; b += red[k][1]; }
}

// What a solve knows of itself, on the device and (copied) on the host.
struct SolveState {
  double r2, f2;       // ||r||^2 and ||rhs||^2 of the last norms
  double r0;           // ||r||^2 of the initial guess
  double rel, before;  // relative residual of the last check, and of the one before
  int cycles, done;
  int ticket;          // CTAs of emb_norm_kernel that have left their partials
};

__device__ __forceinline__ double emb_relative(double r2, double f2, double r0) {
  if (f2 > 0.0) return sqrt(r2 / f2);
  if (r0 > 0.0) return sqrt(r2 / r0);
  return sqrt(r2);
}

// CTA b sums the interior rows 1 + b, 1 + b + gridDim.x, ... (threads along the row), so every
// partial is formed in a fixed order; the CTA that finishes last adds the partials, in a fixed order too
// (a launch of its own for that: 3 us).  cycle >= 0: the norms belong to a V-cycle of the solve, which is
// counted and ends the solve below tol; -1: to the initial guess.
__global__ void __launch_bounds__(256) emb_norm_kernel(const double* __restrict__ phi, const double* __restrict__ rhs,
                                                       const uint8_t* __restrict__ mask, int nx, int ny, double h2i,
                                                       double* partials, SolveState* S, int cycle, double tol,
                                                       const int* done) {
  __shared__ double red[8][2];
  __shared__ bool last;
  if (skip_launch(done)) return;
  double a = 0.0, b = 0.0;
  for (int j = 1 + blockIdx.x; j < ny - 1; j += gridDim.x) {
    const size_t row = (size_t)j * nx;
    for (int i = 1 + threadIdx.x; i < nx - 1; i += 256) {
      const size_t k = row + i;
      if (mask[k] != kFluid) continue;
      const double r = fine_residual(phi, rhs, mask, k, nx, h2i);
      a += r * r;
      b += rhs[k] * rhs[k];
    }
  }
  cta_sums(a, b, red);
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = a;
    partials[2 * blockIdx.x + 1] = b;
    __threadfence();
    last = atomicAdd(&S->ticket, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  a = b = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += 256) {
    a += __ldcg(partials + 2 * k);
    b += __ldcg(partials + 2 * k + 1);
  }
  cta_sums(a, b, red);
  if (threadIdx.x == 0) {
    S->ticket = 0;
    S->r2 = a; S->f2 = b;
    if (cycle < 0) S->r0 = a;
    S->before = S->rel;
    S->rel = emb_relative(a, b, S->r0);
    if (cycle >= 0) {
      S->cycles = cycle + 1;
      if (S->rel < tol) S->done = 1;
    }
  }
}

}  // namespace

// ---------------------------------------------------------------- host side
// Level sizes (nx_{l+1} = (nx_l - 1) / 2 + 1, Multigrid_embedded.cu:140-141) and the first
// level solved by the one-CTA kernel.
void emb_layout(EmbLevels& P, int nx, int ny, int levels) {
  P.L = levels;
  int a = nx, b = ny;
  P.lc = -1;
  for (int l = 0; l < levels; ++l) {
    P.nx[l] = a; P.ny[l] = b;
    if (P.lc < 0 && (int64_t)a * b <= kCoarseMaxNodes) P.lc = l;
    a = (a - 1) / 2 + 1; b = (b - 1) / 2 + 1;
  }
  if (P.lc < 0) P.lc = levels;   // never: the sizes halve down to 2
}

namespace {

int coarse_smem_bytes(const EmbLevels& P, int l0, int offs[PIC_MAX_LEVELS]) {
  int off = 0;
  for (int l = l0; l < P.L; ++l) {
    offs[l - l0] = off;
    const int N = P.nx[l] * P.ny[l];
    off += 16 * N + ((2 * N + 15) / 16) * 16;
  }
  return off;
}

// Launch with programmatic stream serialisation (every kernel here waits in skip_launch or pdl_wait before
// it reads its predecessor's results).
template <typename... KArgs, typename... Args>
void launch_emb(void (*k)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, args...);
}

// Arguments of the strip kernels (emb_strips.cuh) for nu sweeps of a level (down: with the
// restriction); rows = 0 where the tile kernels take it.  An item is one warp with FP64 chains to hide, so
// a level needs about 14 of them per SM; the largest row count that still gives as many wastes
// least on the rows a strip recomputes, up to 36 (more leave the last wave empty).  Measured on
// B200, V-cycle with the line at 10 / 14 / 20 / 28 items per SM, and with tiles alone: 4097^2 494 / 488 /
// 496 / 496, 755 us; 2049^2 202 / 200 / 203 / 206, 231; 1409^2 133 / 123 / 135 / 132, 132; 1025^2 (strips
// only at 10) 100 / 95.  At most 36 rows: with 48 or 60 the 4097^2 V-cycle was 1 % slower.
embs::Args strip_args(const EmbLevels& P, int l, int nu, bool down, const double* in, double* out) {
  constexpr int kItemsPerSm = 14, kMaxRows = 36;
  embs::Args A{};
  const int nx = P.nx[l], ny = P.ny[l];
  if (nu > embs::kMaxNu || (int64_t)nx * ny >= 1 << 30) return A;   // 32-bit node positions
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return A;
  }
  A.done = P.done;
  A.phi = in; A.out = out; A.rhs = P.rhs[l]; A.mask = P.mask[l]; A.bc = P.bc[l];
  A.nx = nx; A.ny = ny;
  A.h2 = P.h * P.h * std::ldexp(1.0, 2 * l);
  A.strips_x = embs::strips(nu, down, nx);
  for (int rows = embs::rows_fit(nu, down, kMaxRows); rows > 0; rows = embs::rows_fit(nu, down, rows - 1)) {
    const int64_t items = (int64_t)A.strips_x * ((ny + rows - 1) / rows);
    if (items >= (int64_t)kItemsPerSm * sms) { A.rows = rows; A.items = (int)items; break; }
  }
  return A;
}

template <int NU, bool PRO>
void launch_smooth(const EmbLevels& P, int l, const double* in, double* out, const double* coarse, bool bilinear,
                   cudaStream_t s) {
  if constexpr (NU <= embs::kMaxNu) {
    embs::Args A = strip_args(P, l, NU, false, in, out);
    if (A.rows) {
      A.coarse = coarse;
      A.bilinear = bilinear ? 1 : 0;
      if (PRO) { A.nxc = P.nx[l + 1]; A.nyc = P.ny[l + 1]; }
      launch_emb(embs::emb_strip_kernel<NU, false, PRO>, dim3((A.items + embs::kWarps - 1) / embs::kWarps), 32 * embs::kWarps, 0, s,
                 A);
      return;
    }
  }
  const dim3 grid((P.nx[l] + kTile - 1) / kTile, (P.ny[l] + kTile - 1) / kTile);
  const double h2 = P.h * P.h * std::ldexp(1.0, 2 * l);
  launch_emb(emb_smooth_kernel<NU, PRO>, grid, kSmoothThreads, 0, s, in, out, (const double*)P.rhs[l],
             (const uint8_t*)P.mask[l], P.bc[l], coarse, P.nx[l], P.ny[l], PRO ? P.nx[l + 1] : 0, h2, bilinear ? 1 : 0, P.done);
}

void smooth_chunk(const EmbLevels& P, int l, int nu, bool pro, const double* in, double* out, bool bilinear,
                  cudaStream_t s) {
  const double* c = pro ? P.phi[l + 1] : nullptr;
  switch (nu * 2 + (pro ? 1 : 0)) {
    case 1: launch_smooth<0, true>(P, l, in, out, c, bilinear, s); break;
    case 2: launch_smooth<1, false>(P, l, in, out, c, bilinear, s); break;
    case 3: launch_smooth<1, true>(P, l, in, out, c, bilinear, s); break;
    case 4: launch_smooth<2, false>(P, l, in, out, c, bilinear, s); break;
    case 5: launch_smooth<2, true>(P, l, in, out, c, bilinear, s); break;
    case 6: launch_smooth<3, false>(P, l, in, out, c, bilinear, s); break;
    case 7: launch_smooth<3, true>(P, l, in, out, c, bilinear, s); break;
    case 8: launch_smooth<4, false>(P, l, in, out, c, bilinear, s); break;
    case 9: launch_smooth<4, true>(P, l, in, out, c, bilinear, s); break;
    default: break;
  }
}

template <int NU>
void launch_down(const EmbLevels& P, int l, const double* in, double* out, int any, cudaStream_t s) {
  if constexpr (NU <= embs::kMaxNu) {
    embs::Args A = strip_args(P, l, NU, true, in, out);
    if (A.rows) {
      A.nxc = P.nx[l + 1]; A.nyc = P.ny[l + 1];
      A.rhs_c = P.rhs[l + 1]; A.mask_c = P.mask[l + 1]; A.phi_c = P.phi[l + 1];
      A.any = any;
      launch_emb(embs::emb_strip_kernel<NU, true, false>, dim3((A.items + embs::kWarps - 1) / embs::kWarps), 32 * embs::kWarps, 0, s,
                 A);
      return;
    }
  }
  const dim3 grid((P.nx[l] + kTile - 1) / kTile, (P.ny[l] + kTile - 1) / kTile);
  const double h2 = P.h * P.h * std::ldexp(1.0, 2 * l);
  launch_emb(emb_down_kernel<NU>, grid, kSmoothThreads, 0, s, in, out, (const double*)P.rhs[l], (const uint8_t*)P.mask[l],
             P.bc[l], P.nx[l], P.ny[l], h2, P.rhs[l + 1], P.mask[l + 1], P.phi[l + 1], P.nx[l + 1], P.ny[l + 1], any, P.done);
}

// nu sweeps of level l (chunks of at most 4 per launch; the first applies the prolongation
// when pro is set); `cur` tracks which of phi[l] / alt[l] holds the level's current values.
void smooth_level(const EmbLevels& P, int l, int nu, bool pro, double*& cur, bool bilinear, cudaStream_t s) {
  while (nu > 0 || pro) {
    const int c = std::min(nu, 4);
    double* out = cur == P.phi[l] ? P.alt[l] : P.phi[l];
    smooth_chunk(P, l, c, pro, cur, out, bilinear, s);
    cur = out;
    nu -= c;
    pro = false;
  }
}

}  // namespace

// One V-cycle of Multigrid::vcycle(l0) on the level arrays of P (results in P.phi[l]).
int emb_vcycle(const EmbLevels& P, int l0, int nu1, int nu2, int options, cudaStream_t s) {
  // the one-CTA kernel's shared memory above the 48 KB default, once per device
  static std::atomic<int> smem_set[64];
  int dev = 0;
  cudaError_t e0 = cudaGetDevice(&dev);
  if (e0 != cudaSuccess) return pic_fail(PIC_ERR_CUDA, cudaGetErrorString(e0));
  if (dev >= 64) return pic_fail(PIC_ERR_ARG, "device index beyond the solver's table");
  if (!smem_set[dev].load()) {
    e0 = cudaFuncSetAttribute(emb_coarse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e0 != cudaSuccess) return pic_fail(PIC_ERR_CUDA, cudaGetErrorString(e0));
    smem_set[dev].store(1);
  }
  const bool bilinear = options & PIC_EMB_PROLONG_BILINEAR;
  const int any = (options & PIC_EMB_COARSEN_ANY) ? 1 : 0;
  const int lc = std::max(P.lc, l0);
  double* cur[PIC_MAX_LEVELS];
  for (int l = l0; l < lc; ++l) {
    cur[l] = P.phi[l];
    if (l < P.L - 1) {
      // all but the last (up to 4) pre-sweeps, then those fused with the restriction
      const int last = nu1 == 0 ? 0 : (nu1 - 1) % 4 + 1;
      smooth_level(P, l, nu1 - last, false, cur[l], bilinear, s);
      double* out = cur[l] == P.phi[l] ? P.alt[l] : P.phi[l];
      switch (last) {
        case 0: launch_down<0>(P, l, cur[l], out, any, s); break;
        case 1: launch_down<1>(P, l, cur[l], out, any, s); break;
        case 2: launch_down<2>(P, l, cur[l], out, any, s); break;
        case 3: launch_down<3>(P, l, cur[l], out, any, s); break;
        default: launch_down<4>(P, l, cur[l], out, any, s); break;
      }
      cur[l] = out;
      continue;
    }
    smooth_level(P, l, nu1, false, cur[l], bilinear, s);
    {   // coarsest level on the tile path: pre-sweeps only
      if (cur[l] != P.phi[l]) {
        const cudaError_t e = cudaMemcpyAsync(P.phi[l], cur[l], sizeof(double) * P.nx[l] * P.ny[l],
                                              cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return pic_fail(PIC_ERR_CUDA, cudaGetErrorString(e));
      }
    }
  }
  if (lc < P.L) {
    CoarseLevelArgs A{};
    A.n = P.L - lc;
    for (int k = 0; k < A.n; ++k) {
      const int l = lc + k;
      A.nx[k] = P.nx[l]; A.ny[k] = P.ny[l];
      A.phi[k] = P.phi[l]; A.rhs[k] = P.rhs[l]; A.mask[k] = P.mask[l]; A.bc[k] = P.bc[l];
      A.h2[k] = P.h * P.h * std::ldexp(1.0, 2 * l);
      A.h2i[k] = 1.0 / A.h2[k];
    }
    const int bytes = coarse_smem_bytes(P, lc, A.soff);
    A.nu1 = nu1; A.nu2 = nu2; A.coarsen_any = any; A.bilinear = bilinear ? 1 : 0;
    A.done = P.done;
    launch_emb(emb_coarse_kernel, dim3(1), kCoarseThreads, bytes, s, A);
  }
  for (int l = std::min(lc, P.L - 1) - 1; l >= l0; --l) {
    smooth_level(P, l, nu2, true, cur[l], bilinear, s);
    if (cur[l] != P.phi[l]) {
      cudaError_t e = cudaMemcpyAsync(P.phi[l], cur[l], sizeof(double) * P.nx[l] * P.ny[l], cudaMemcpyDeviceToDevice, s);
      if (e != cudaSuccess) return pic_fail(PIC_ERR_CUDA, cudaGetErrorString(e));
    }
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return pic_fail(PIC_ERR_CUDA, cudaGetErrorString(e));
  return PIC_OK;
}

namespace {

// ||r||^2 and ||rhs||^2 over level 0's FLUID nodes into S; see emb_norm_kernel.
int emb_norms(const EmbLevels& P, double* partials, SolveState* S, int cycle, double tol, cudaStream_t s) {
  const double h2i = 1.0 / (P.h * P.h);
  const int nb = std::max(1, std::min(kNormBlocks, P.ny[0] - 2));
  launch_emb(emb_norm_kernel, dim3(nb), 256, 0, s, (const double*)P.phi[0], (const double*)P.rhs[0],
             (const uint8_t*)P.mask[0], P.nx[0], P.ny[0], h2i, partials, S, cycle, tol, P.done);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return pic_fail(PIC_ERR_CUDA, cudaGetErrorString(e));
  return PIC_OK;
}

}  // namespace

namespace {

// Working arrays of pic_solve_embedded_f64, one set per (device, nx, ny, levels), kept until
// the process exits.
struct EmbScratch {
  int device, nx, ny, levels;
  EmbLevels P;           // coarse-level pointers (level 0 is filled per call)
  double* alt0;
  double* partials;
  SolveState* state;       // device
  SolveState* host_state;  // pinned
};
std::mutex g_emb_mu;
std::vector<EmbScratch> g_emb;

int emb_scratch(int device, int nx, int ny, int levels, EmbScratch** out) {
  for (auto& c : g_emb)
    if (c.device == device && c.nx == nx && c.ny == ny && c.levels == levels) { *out = &c; return PIC_OK; }
  EmbScratch c{};
  c.device = device; c.nx = nx; c.ny = ny; c.levels = levels;
  emb_layout(c.P, nx, ny, levels);
  std::vector<void*> got;
  auto A = [&](void** p, size_t b) {
    const cudaError_t e = cudaMalloc(p, b);
    if (e == cudaSuccess) got.push_back(*p);
    return e;
  };
  cudaError_t e = A((void**)&c.alt0, sizeof(double) * nx * ny);
  for (int l = 1; l < levels && e == cudaSuccess; ++l) {
    const size_t N = (size_t)c.P.nx[l] * c.P.ny[l];
    e = A((void**)&c.P.phi[l], 8 * N);
    if (e == cudaSuccess && l < c.P.lc) e = A((void**)&c.P.alt[l], 8 * N);
    if (e == cudaSuccess) e = A((void**)&c.P.rhs[l], 8 * N);
    if (e == cudaSuccess) e = A((void**)&c.P.mask[l], N);
  }
  if (e == cudaSuccess) e = A((void**)&c.partials, sizeof(double) * 2 * kNormBlocks);
  if (e == cudaSuccess) e = A((void**)&c.state, sizeof(SolveState));
  if (e == cudaSuccess) {
    e = cudaMallocHost((void**)&c.host_state, sizeof(SolveState));
  }
  if (e != cudaSuccess) {
    for (void* p : got) cudaFree(p);
    cudaGetLastError();
    return pic_fail(e == cudaErrorMemoryAllocation ? PIC_ERR_OOM : PIC_ERR_CUDA, cudaGetErrorString(e));
  }
  g_emb.push_back(c);
  *out = &g_emb.back();
  return PIC_OK;
}

// V-cycles to send before the next look at the norms: one fewer than the last two residuals' ratio says
// are needed (the kernels of cycles behind the converged one return at once, but each still costs its
// launches).
int cycles_ahead(const SolveState& S, double tol, int left) {
  int n = 1;
  if (S.cycles >= 2 && S.rel > tol && S.rel < S.before && S.rel > 0.0)
    n = (int)std::min(16.0, std::ceil(std::log(tol / S.rel) / std::log(S.rel / S.before))) - 1;
  return std::max(1, std::min(n, left));
}

}  // namespace

extern "C" int pic_solve_embedded_f64(double* phi, const double* rhs, const uint8_t* mask, const double* phi_bc, int nx,
                                      int ny, int levels, double h, int nu_pre, int nu_post, int options, double tol,
                                      int max_cycles, void* stream, int* cycles_out, double* relres_out) {
  if (!phi || !rhs || !mask) return pic_fail(PIC_ERR_ARG, "null grid pointers");
  if (nx < 3 || ny < 3) return pic_fail(PIC_ERR_ARG, "grid needs at least 3 x 3 nodes");
  if ((int64_t)nx * ny > (int64_t)1 << 31) return pic_fail(PIC_ERR_ARG, "grid too large");
  if (levels < 1 || levels > PIC_MAX_LEVELS) return pic_fail(PIC_ERR_ARG, "levels must be in 1..14");
  if (!(h > 0)) return pic_fail(PIC_ERR_ARG, "h must be positive");
  if (nu_pre < 0 || nu_post < 0 || nu_pre > 64 || nu_post > 64) return pic_fail(PIC_ERR_ARG, "sweep counts out of range");
  if (options & ~(PIC_EMB_COARSEN_ANY | PIC_EMB_PROLONG_BILINEAR)) return pic_fail(PIC_ERR_ARG, "unknown option bits");
  if (max_cycles < 1 || !(tol >= 0)) return pic_fail(PIC_ERR_ARG, "max_cycles >= 1 and tol >= 0 required");
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) { cudaGetLastError(); return pic_fail(PIC_ERR_NO_DEVICE, cudaGetErrorString(e)); }
  std::lock_guard<std::mutex> lk(g_emb_mu);
  EmbScratch* S = nullptr;
  int rc = emb_scratch(device, nx, ny, levels, &S);
  if (rc) return rc;
  EmbLevels P = S->P;
  P.phi[0] = phi; P.alt[0] = S->alt0; P.rhs[0] = const_cast<double*>(rhs);
  P.mask[0] = const_cast<uint8_t*>(mask); P.bc[0] = phi_bc; P.h = h;
  cudaStream_t s = (cudaStream_t)stream;
  // With a tolerance the norms follow every cycle on the device, where the first cycle below tol sets the
  // done flag, and the host sends several cycles at a time.  The kernels of a cycle behind the converged
  // one return at once; its cudaMemcpyAsync copies (an odd number of smoothing launches per level) repeat
  // the converged cycle's copies from arrays that nothing has written since.
  const bool check = tol > 0;
  auto read_state = [&]() -> int {
    cudaError_t e2 = cudaMemcpyAsync(S->host_state, S->state, sizeof(SolveState), cudaMemcpyDeviceToHost, s);
    if (e2 == cudaSuccess) e2 = cudaStreamSynchronize(s);
    return e2 == cudaSuccess ? PIC_OK : pic_fail(PIC_ERR_CUDA, cudaGetErrorString(e2));
  };
  int cyc = 0;
  double rel = 0.0;
  if (check || relres_out) {
    e = cudaMemsetAsync(S->state, 0, sizeof(SolveState), s);
    if (e != cudaSuccess) return pic_fail(PIC_ERR_CUDA, cudaGetErrorString(e));
    if ((rc = emb_norms(P, S->partials, S->state, -1, tol, s))) return rc;
  }
  if (check) {
    P.done = &S->state->done;
    for (int ahead = std::min(2, max_cycles);;) {
      for (int k = 0; k < ahead; ++k) {
        if ((rc = emb_vcycle(P, 0, nu_pre, nu_post, options, s))) return rc;
        if ((rc = emb_norms(P, S->partials, S->state, cyc + k, tol, s))) return rc;
      }
      if ((rc = read_state())) return rc;
      cyc = S->host_state->cycles;
      rel = S->host_state->rel;
      if (S->host_state->done || cyc >= max_cycles) break;
      ahead = cycles_ahead(*S->host_state, tol, max_cycles - cyc);
    }
  } else {
    for (; cyc < max_cycles; ++cyc)
      if ((rc = emb_vcycle(P, 0, nu_pre, nu_post, options, s))) return rc;
    if (relres_out) {
      if ((rc = emb_norms(P, S->partials, S->state, max_cycles - 1, 0.0, s))) return rc;
      if ((rc = read_state())) return rc;
      rel = S->host_state->rel;
    }
  }
  if (cycles_out) *cycles_out = cyc;
  if (relres_out) *relres_out = rel;
  // tol == 0 never converges (as in pic_solve_multigrid_f64): exactly max_cycles V-cycles
  if (!(rel < tol)) return pic_fail(PIC_ERR_NOT_CONVERGED, "embedded multigrid stopped at max_cycles above tol");
  return PIC_OK;
}
