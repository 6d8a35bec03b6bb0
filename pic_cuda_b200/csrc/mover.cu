// mover.cu — the fused particle pass of one PIC step.
//
// One pass over each particle slot does, in the reference's order (main.cu:64-134):
//   kick     updateParticleVelocities (kernels.cu:71-131): E bilinearly gathered from the
//            node field that efield32_kernel computes once per step from the FP64 potential
//            with the computeElectricField stencils (kernels.cu:134-191)
//   MCC      null-collision Monte Carlo (or the reference's elastic form, mcc.cu:56-85)
//   drift    update_coordinates (kernels.cu:8-23) on cell-relative FP32 positions
//   walls    detect_intersections (collisions.cu:7-54) / box absorption; hits are appended
//            with one atomic per warp item (compaction happens in compact.cu)
//   deposit  updateDensity (kernels.cu:26-69) at the new position: runs of equal cells are
//            summed in registers (particles are counting-sorted by cell), then a warp-segmented
//            reduction and one atomic per node per segment; FP32 or int64 fixed point.
// The kick + MCC of step k are fused into the pass of step k+1 (the job's kick_pending
// flag); an explicit flush applies them before any read-back.
#include <algorithm>
#include "common.cuh"
#include "kernels.h"
#include "particle_ops.cuh"

namespace {

__device__ __forceinline__ float xs_lookup(const ProcDev& p, float E) {
  const float* e = p.e;
  const int n = p.n;
  if (E <= e[0]) return p.s[0];
  if (E >= e[n - 1]) return p.s[n - 1];
  int k;
  if (p.inv_dlog > 0.f) {
    k = (int)((__logf(E) - p.log_e0) * p.inv_dlog);
    k = max(0, min(k, n - 2));
    while (k > 0 && E < e[k]) --k;
    while (k < n - 2 && E >= e[k + 1]) ++k;
  } else {
    int lo = 0, hi = n - 2;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (e[mid] <= E) lo = mid; else hi = mid - 1;
    }
    k = lo;
  }
  const float t = (E - e[k]) / (e[k + 1] - e[k]);
  return p.s[k] + t * (p.s[k + 1] - p.s[k]);
}

__device__ __forceinline__ void iso_dir(float ua, float ub, float d[3]) {
  const float c = 1.f - 2.f * ua;
  const float sn = sqrtf(fmaxf(0.f, 1.f - c * c));
  float s, co;
  sincospif(2.f * ub, &s, &co);
  d[0] = sn * co; d[1] = sn * s; d[2] = c;
}

__device__ __forceinline__ void neutral_velocity(uint64_t seed, uint32_t pid, uint32_t step, float sig, float v[3]) {
  float u[4];
  draw4(seed, pid, step, 2u, u);
  const float r0 = sqrtf(-2.f * logf(u[0])), r1 = sqrtf(-2.f * logf(u[2]));
  float s, c, s2, c2;
  sincospif(2.f * u[1], &s, &c);
  sincospif(2.f * u[3], &s2, &c2);
  v[0] = sig * r0 * c; v[1] = sig * r0 * s; v[2] = sig * r1 * c2;
}

}  // namespace

// A warp's work item is 64 consecutive particles: lane l holds particles 2 l and 2 l + 1 in registers, loaded
// with one 8-byte load per array.  Capacities are multiples of PIC_CHUNK, so every item lies inside
// the arrays.  Small CTAs let the register file hold 28 warps of 72 registers.  Measured on B200, ms per
// pass at 1025^2 (2e7 particles, FP32 deposit) / 4097^2 (2e8) / 4097^2 with the int64 deposit: 128
// threads x 7 CTAs per SM 0.341 / 3.22 / 3.50; x 6 0.352 / 3.40 / 3.67; x 8 0.361 / 3.43 / 3.71; x 9 0.380 /
// 3.61 / 3.91; 256 x 4 0.356 / 3.36 / 3.67; items of twice as many particles, 128 x 5 0.345 / 3.30 /
// 3.71; x 6 0.362 / 3.37 / 3.82.
constexpr int kPPL = 2;   // particles per lane
constexpr int kItem = 32 * kPPL;

// The two 4-byte values of one lane, as one evict-first load / store (p: the lane's first).
__device__ __forceinline__ void ld_lane(const float* p, float (&a)[kPPL]) {
  const float2 v = __ldcs(reinterpret_cast<const float2*>(p));
  a[0] = v.x; a[1] = v.y;
}
__device__ __forceinline__ void ld_lane(const uint32_t* p, uint32_t (&a)[kPPL]) {
  const uint2 v = __ldcs(reinterpret_cast<const uint2*>(p));
  a[0] = v.x; a[1] = v.y;
}
__device__ __forceinline__ void st_lane(float* p, const float (&a)[kPPL]) {
  __stcs(reinterpret_cast<float2*>(p), make_float2(a[0], a[1]));
}
__device__ __forceinline__ void st_lane(uint32_t* p, const uint32_t (&a)[kPPL]) {
  __stcs(reinterpret_cast<uint2*>(p), make_uint2(a[0], a[1]));
}
constexpr int kWarps = PIC_MOVER_THREADS / 32;
#ifndef PIC_MOVER_MIN_BLOCKS
#define PIC_MOVER_MIN_BLOCKS 7
#endif

// One real-or-null collision of a null-collision candidate (Vahedi & Surendra 1995): the
// candidate's process is chosen with u1 * nu_max against the cumulative n sigma_j(E) v.
__device__ void collide(const JobDev& J, const SlotDev& S, const SlotDev* slots, JobState& T, uint32_t pid,
                        uint32_t cell, float fx, float fy, float& vx, float& vy, float& vz, const float u[4],
                        uint32_t step, unsigned* proc_count) {
  const float v2 = vx * vx + vy * vy + vz * vz;
  const float sp = sqrtf(v2);
  const float E = S.half_m_over_e * v2;
  const float target = u[1] * S.numax;
  float acc = 0.f;
  int chosen = -1;
  for (int q = 0; q < S.n_proc; ++q) {
    acc += J.gas_density * xs_lookup(J.procs[S.first_proc + q], E) * sp;
    if (target < acc) { chosen = q; break; }
  }
  if (chosen < 0) return;
  const ProcDev& P = J.procs[S.first_proc + chosen];
  float d[3];
  if (P.type == PIC_PROC_ELASTIC) {
    iso_dir(u[2], u[3], d);
    const float cosx = sp > 0.f ? (vx * d[0] + vy * d[1] + vz * d[2]) / sp : 1.f;
    const float Ep = E * (1.f - 2.f * S.mass / J.gas_mass * (1.f - cosx));
    const float vn = sqrtf(fmaxf(0.f, Ep) / S.half_m_over_e);
    vx = vn * d[0]; vy = vn * d[1]; vz = vn * d[2];
  } else if (P.type == PIC_PROC_EXCITATION) {
    if (E < P.threshold) return;
    iso_dir(u[2], u[3], d);
    const float vn = sqrtf((E - P.threshold) / S.half_m_over_e);
    vx = vn * d[0]; vy = vn * d[1]; vz = vn * d[2];
  } else if (P.type == PIC_PROC_IONIZATION) {
    if (E < P.threshold) return;
    float u2[4];
    draw4(J.seed, pid, step, 1u, u2);
    const float Er = E - P.threshold, B = 10.f;
    const float Eej = B * tanf(u2[0] * atanf(Er / (2.f * B)));
    const float Esc = fmaxf(0.f, Er - Eej);
    iso_dir(u[2], u[3], d);
    const float vs = sqrtf(Esc / S.half_m_over_e);
    Event ev;
    ev.parent_pid = pid; ev.cell = cell; ev.fx = fx; ev.fy = fy;
    float d2[3];
    iso_dir(u2[1], u2[2], d2);
    const SlotDev& SE = slots[J.slot0 + J.ion_e_species];
    const float ve = sqrtf(Eej / SE.half_m_over_e);
    ev.ve[0] = ve * d2[0]; ev.ve[1] = ve * d2[1]; ev.ve[2] = ve * d2[2];
    neutral_velocity(J.seed, pid, step, J.vth_neutral, ev.vi);
    const int k = atomicAdd(&T.event_count, 1);
    if (k < J.event_capacity) J.events[k] = ev;
    else atomicOr(&T.status, PIC_ST_EVENTS);
    vx = vs * d[0]; vy = vs * d[1]; vz = vs * d[2];
  } else if (P.type == PIC_PROC_CHARGE_EXCHANGE) {
    float vn[3];
    neutral_velocity(J.seed, pid, step, J.vth_neutral, vn);
    vx = vn[0]; vy = vn[1]; vz = vn[2];
  }
  atomicAdd(&proc_count[chosen & 7], 1u);
}

// E per unit cell (-dphi across one cell) at node k of a job, from its current FP64 potential with the
// computeElectricField stencils (kernels.cu:134-191): (phi[i-1] - phi[i+1]) / 2 inside, phi[i] -
// phi[i+1] on the first and phi[i-1] - phi[i] on the last node of a row, the same along columns;
// rounded to FP32 once.
__device__ __forceinline__ float2 efield_at(const double* __restrict__ phi, int nx, int ny, int k) {
  const int j = k / nx, i = k - j * nx;
  const int il = i > 0 ? i - 1 : 0, ir = i < nx - 1 ? i + 1 : nx - 1;
  const int jl = j > 0 ? j - 1 : 0, jr = j < ny - 1 ? j + 1 : ny - 1;
  const double sx = (i > 0 && i < nx - 1) ? 0.5 : 1.0, sy = (j > 0 && j < ny - 1) ? 0.5 : 1.0;
  const double ex = (phi[j * nx + il] - phi[j * nx + ir]) * sx;
  const double ey = (phi[jl * nx + i] - phi[jr * nx + i]) * sy;
  return make_float2((float)ex, (float)ey);
}

// The node field of every job.  Job j uses blockIdx.y == j and a grid-stride loop over its nodes.
__global__ void __launch_bounds__(256) efield32_kernel(const JobDev* __restrict__ jobs, const JobState* __restrict__ st) {
  const JobDev& J = jobs[blockIdx.y];
  float2* const out = J.efield;
  if (!out) return;
  const double* __restrict__ phi = J.phi64[st[blockIdx.y].phi_cur];
  const int nx = J.nx, ny = J.ny, N = nx * ny;
  for (int k = blockIdx.x * 256 + threadIdx.x; k < N; k += gridDim.x * 256) out[k] = efield_at(phi, nx, ny, k);
}

// Exclusive prefix of mover work items (kItem particles) per active slot, by one thread.
__device__ void item_prefix_of(const int* __restrict__ counts, const uint8_t* __restrict__ active, int* prefix,
                               int nslots) {
  int a = 0;
  for (int s = 0; s < nslots; ++s) {
    prefix[s] = a;
    if (!active || active[s]) a += (counts[s] + kItem - 1) / kItem;
  }
  prefix[nslots] = a;
}
__global__ void chunk_table_kernel(const int* __restrict__ counts, const uint8_t* __restrict__ active,
                                   int* __restrict__ chunk_prefix, int nslots) {
  if (threadIdx.x == 0) item_prefix_of(counts, active, chunk_prefix, nslots);
}

// What a full step does before its particle pass, in one launch: the node field of every job, its charge
// grid zeroed, the step's diagnostics reset and the work items counted.  (Four launches of 2-4 us each
// before, most of it launch latency on small jobs: 129^2 step 123 -> 113 us together with the merged
// V-cycle end and the memsets that moved into the solver's kernels.)
__global__ void __launch_bounds__(256) step_head_kernel(const JobDev* __restrict__ jobs, JobState* __restrict__ st,
                                                        const int* __restrict__ counts,
                                                        const uint8_t* __restrict__ active, int* __restrict__ prefix,
                                                        int nslots) {
  const JobDev& J = jobs[blockIdx.y];
  if (blockIdx.x == gridDim.x - 1) {   // the block with the fewest nodes
    if (blockIdx.y == 0 && threadIdx.x == 0) item_prefix_of(counts, active, prefix, nslots);
    JobState& T = st[blockIdx.y];
    const int t = (int)threadIdx.x - 32;
    if (t >= 0 && t < PIC_MAX_SPECIES) T.ke[t] = 0.0;
    if (t >= 32 && t < 32 + 8 * PIC_MAX_SPECIES) T.collisions[(t - 32) >> 3][(t - 32) & 7] = 0ull;
  }
  float2* const out = J.efield;
  if (!out) return;                    // no such job
  const double* __restrict__ phi = J.phi64[st[blockIdx.y].phi_cur];
  const int nx = J.nx, ny = J.ny, N = nx * ny;
  float* const rf = J.deposit_mode == 0 ? J.rho_f : nullptr;
  long long* const ri = J.deposit_mode == 1 ? J.rho_i : nullptr;
  for (int k = blockIdx.x * 256 + threadIdx.x; k < N; k += gridDim.x * 256) {
    out[k] = efield_at(phi, nx, ny, k);
    if (rf) rf[k] = 0.f;
    else if (ri) ri[k] = 0;
  }
}

// The slot and job tables of the slot a warp works on, copied to shared memory when the
// warp moves to another slot (every parameter read in the per-particle code is then a
// shared-memory load, and the functions shared with the ionisation kernel take them as is).
struct WarpTables {
  SlotDev S;
  JobDev J;
};

__device__ __forceinline__ void copy_words(void* dst, const void* src, int bytes, int lane) {
  int* d = reinterpret_cast<int*>(dst);
  const int* s = reinterpret_cast<const int*>(src);
  for (int q = lane; q < bytes / 4; q += 32) d[q] = s[q];
}

// CIC weights of one particle (updateDensity, kernels.cu:56-68) in deposit units: FP32, or
// int64 fixed point whose four parts sum to the particle's quantised charge exactly.
__device__ __forceinline__ void cic_f32(float q, float fx, float fy, float& a, float& b, float& c, float& d) {
  a = q * ((1.f - fx) * (1.f - fy)); b = q * (fx * (1.f - fy)); c = q * ((1.f - fx) * fy); d = q * (fx * fy);
}
__device__ __forceinline__ void cic_i64(long long qf, float fx, float fy, long long& a, long long& b, long long& c,
                                        long long& d) {
  const double Q = (double)qf;
  a = __double2ll_rn((double)((1.f - fx) * (1.f - fy)) * Q);
  b = __double2ll_rn((double)(fx * (1.f - fy)) * Q);
  c = __double2ll_rn((double)((1.f - fx) * fy) * Q);
  d = qf - a - b - c;
}

// Deposit of an item's 64 particles, two per lane (keys in lane order): equal keys of a lane's pair are summed
// in registers (of two different ones the first goes to rho at once), then the lanes' runs of equal
// keys are summed over the warp (lane order) and the first lane of each adds the totals to rho.
// Called by all lanes.
template <typename V, typename W>
__device__ __forceinline__ void lane_deposit(V* rho, int nx, const uint32_t (&key)[kPPL], const float (&fx)[kPPL],
                                             const float (&fy)[kPPL], W weights) {
  const int lane = lane_id();
  V v[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0};
  uint32_t rk = key[0];
  if (rk != PIC_CELL_OUT) weights(fx[0], fy[0], v[0], v[1], v[2], v[3]);
  if (key[1] != PIC_CELL_OUT) weights(fx[1], fy[1], b[0], b[1], b[2], b[3]);
  if (key[1] == rk) {
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] += b[u];
  } else {
    if (rk != PIC_CELL_OUT) {
      V* r = rho + (size_t)cell_j(rk) * nx + cell_i(rk);
      red_add(r, v[0]); red_add(r + 1, v[1]); red_add(r + nx, v[2]); red_add(r + nx + 1, v[3]);
    }
    rk = key[1];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = b[u];
  }
  const uint32_t prev = __shfl_up_sync(0xffffffffu, rk, 1);
  const bool head = (lane == 0) || (rk != prev);
  const unsigned heads = __ballot_sync(0xffffffffu, head);
  // the lane after this lane's segment, and the longest segment of the warp
  const unsigned after = lane == 31 ? 0u : heads & (0xfffffffeu << lane);
  const int first = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
  const int end = after ? __ffs(after) - 1 : 32;
  const int longest = (int)__reduce_max_sync(0xffffffffu, (unsigned)(end - first));
  // only as many shuffle levels as the longest segment needs
  for (int o = 1; o < longest; o <<= 1) {
    V t[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) t[u] = __shfl_down_sync(0xffffffffu, v[u], o);
    if (lane + o < end) {
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] += t[u];
    }
  }
  if (head && rk != PIC_CELL_OUT) {
    V* r = rho + (size_t)cell_j(rk) * nx + cell_i(rk);
    red_add(r, v[0]);
    red_add(r + 1, v[1]);
    red_add(r + nx, v[2]);
    red_add(r + nx + 1, v[3]);
  }
}

// Deferred collision candidates of a warp: cell fx fy vx vy vz pid index, up to one round of
// 32 left over plus one item's worth.
constexpr int kQueue = 32 + kItem;
constexpr int kQFields = 8;
constexpr size_t kMoverSmem = (size_t)kWarps * kQFields * kQueue * sizeof(uint32_t);

// The fused particle pass.  Warp w of the grid takes items w, w + W, w + 2W, ... (W warps in
// the grid) over the concatenated items of all active slots; the slot of an item comes from
// the item prefix, and a warp's items only move forward through the slots.  Per item:
//   loads    cell, fx, fy, vx, vy (+ vz, pid with collisions): one evict-first vector load
//            per array and lane
//   pass A   kick (E gathered from the per-step node field; particles are cell-sorted, so a
//            warp's gathers hit a few cache lines) and the null-collision test: candidates
//            (~nu_max dt of the particles) whose collision is real (u1 nu_max below the
//            species' total n sigma_T v, one table lookup) leave the item for the warp's queue
//            in shared memory.  Whenever 32 are queued (and when the warp leaves a slot), one
//            round chooses the process and collides, drifts, deposits and stores them, one
//            per lane, after their owners have stored the rest of their items.
//   pass B   drift, absorption (hits appended with one atomic per item), CIC deposit
//   stores   evict-first vector stores of what changed (vz only in the queue rounds; the
//            cell word only when some particle of the warp crossed a cell edge)
// The particle stream bypasses L2 retention (evict-first loads and stores) so the grids the
// gathers and deposits touch stay resident.  No block-level synchronisation.
__global__ void __launch_bounds__(PIC_MOVER_THREADS, PIC_MOVER_MIN_BLOCKS)
mover_kernel(const JobDev* __restrict__ jobs, JobState* __restrict__ st, const SlotDev* __restrict__ slots,
             const int* __restrict__ counts, int* __restrict__ hit_counts, const int* __restrict__ item_prefix,
             int nslots, int flags, uint32_t explicit_step) {
  extern __shared__ __align__(16) uint32_t qbuf[];
  __shared__ WarpTables tab[kWarps];
  __shared__ unsigned pcount[kWarps][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int total = item_prefix[nslots];
  const SlotDev& S = tab[warp].S;
  const JobDev& J = tab[warp].J;
  unsigned* const pc = pcount[warp];
  uint32_t* const cq = qbuf + (size_t)warp * kQFields * kQueue;   // field f of entry e: cq[f * kQueue + e]
  int qn = 0;                                                      // queued candidates (warp-uniform)
  if (lane < 8) pc[lane] = 0u;
  __syncwarp();
  int cur = -1, cur_first = 0, cur_end = 0;   // the warp's slot, its first item and the one after its last
  double ke = 0.0;
  bool do_kick = false, do_mcc = false, do_drift = false, do_walls = false, do_dep = false, want_ke = false;
  uint32_t mcc_step = 0;
  uint32_t cand_below = 0;   // draws m with u01 = (2 m + 1) 2^-24 < pnull: exactly those m < cand_below
  int n = 0;
  // One round over the first cnt queued candidates (one per lane): collide (Philox stream
  // (seed, pid, step) as for the candidate test), drift, absorb, deposit, store at the
  // particle's index; then the queue moves down by cnt.  The owners' stores of these
  // particles were issued before (the barrier orders them first).
  auto round = [&](int cnt) {
    __syncwarp();
    const int s = cur;
    bool absorbed = false;
    int idx = 0;
    if (lane < cnt) {
      uint32_t qc = cq[0 * kQueue + lane];
      float qfx = __uint_as_float(cq[1 * kQueue + lane]), qfy = __uint_as_float(cq[2 * kQueue + lane]);
      float qvx = __uint_as_float(cq[3 * kQueue + lane]), qvy = __uint_as_float(cq[4 * kQueue + lane]);
      float qvz = __uint_as_float(cq[5 * kQueue + lane]);
      const uint32_t qpid = cq[6 * kQueue + lane];
      idx = (int)cq[7 * kQueue + lane];
      float u[4];
      draw4(J.seed, qpid, mcc_step, 0u, u);
      collide(J, S, slots, st[S.job], qpid, qc, qfx, qfy, qvx, qvy, qvz, u, mcc_step, pc);
      if (want_ke) ke += (double)(qvx * qvx + qvy * qvy + qvz * qvz);
      if (do_drift) {
        const Drifted d = drift_particle(J, S, qc, qfx, qfy, qvx, qvy, do_walls);
        absorbed = d.absorbed; qc = d.cell; qfx = d.fx; qfy = d.fy;
        S.cell[idx] = qc; S.fx[idx] = qfx; S.fy[idx] = qfy;
      }
      if (do_dep && !absorbed) deposit_one(J, S, qc, qfx, qfy);
      S.vx[idx] = qvx; S.vy[idx] = qvy; S.vz[idx] = qvz;
    }
    if (do_walls) {
      const int h = warp_append(lane < cnt && absorbed, hit_counts + s);
      if (h >= 0) S.hits[h] = idx;
    }
    __syncwarp();
    for (int q = lane; q < qn - cnt; q += 32)
#pragma unroll
      for (int f = 0; f < kQFields; ++f) cq[f * kQueue + q] = cq[f * kQueue + q + cnt];
    __syncwarp();
    qn -= cnt;
  };
  // kinetic energy and collision counts of the slot a warp leaves go to its job's state
  auto flush = [&]() {
    if (cur < 0) return;
    if (qn > 0) round(qn);
    if (want_ke) {
      double v = ke;
#pragma unroll
      for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0 && v != 0.0) atomicAdd(&st[S.job].ke[S.species], v * S.ke_factor);
    }
    ke = 0.0;
    if (lane < 8) {
      const unsigned c = pc[lane];
      if (c) { atomicAdd(&st[S.job].collisions[S.species][lane], (unsigned long long)c); pc[lane] = 0u; }
    }
    __syncwarp();
  };
  const int nwarps = gridDim.x * kWarps;
  for (int item = blockIdx.x * kWarps + warp; item < total; item += nwarps) {
    if (item >= cur_end) {
      int s = cur < 0 ? 0 : cur;
      while (s < nslots - 1 && item_prefix[s + 1] <= item) ++s;
      flush();
      cur_first = item_prefix[s];
      cur_end = item_prefix[s + 1];
      copy_words(&tab[warp].S, slots + s, sizeof(SlotDev), lane);
      __syncwarp();
      copy_words(&tab[warp].J, jobs + S.job, sizeof(JobDev), lane);
      __syncwarp();
      cur = s;
      const JobState& T0 = st[S.job];
      const bool gated = flags & PIC_PHASE_GATED_I;
      const bool pending = T0.kick_pending != 0;
      do_kick = (flags & PIC_PHASE_KICK_I) && (!gated || pending);
      do_mcc = (flags & PIC_PHASE_MCC_I) && (!gated || pending) && J.mcc_mode != 0 && S.n_proc > 0;
      do_drift = flags & PIC_PHASE_DRIFT_I;
      do_walls = (flags & PIC_PHASE_WALLS_I) && J.wall_mode != 0;
      do_dep = flags & PIC_PHASE_DEPOSIT_I;
      want_ke = do_kick || do_mcc;
      mcc_step = gated ? (uint32_t)(T0.step - 1) : explicit_step;
      n = counts[s];
      cand_below = (uint32_t)ceil((fmin((double)S.pnull, 1.0) * 16777216.0 - 1.0) * 0.5);
    }
    const int s = cur;
    const int i0 = (item - cur_first) * kItem + 2 * lane;
    // ---- loads
    uint32_t c[kPPL], pid[kPPL];
    float fx[kPPL], fy[kPPL], vx[kPPL], vy[kPPL], vz[kPPL];
    {
      ld_lane(S.cell + i0, c);
      ld_lane(S.fx + i0, fx);
      ld_lane(S.fy + i0, fy);
      ld_lane(S.vx + i0, vx);
      ld_lane(S.vy + i0, vy);
      if (do_mcc) {
        ld_lane(S.vz + i0, vz);
        ld_lane(S.pid + i0, pid);
      } else {
#pragma unroll
        for (int k = 0; k < kPPL; ++k) { vz[k] = 0.f; pid[k] = 0u; }
      }
    }
    bool valid[kPPL];
#pragma unroll
    for (int k = 0; k < kPPL; ++k) valid[k] = i0 + k < n;
    // ---- pass A: kick and collisions
    if (do_kick) {
      const float2* __restrict__ ef = J.efield;
      const int enx = J.nx;
      const float kx = S.kx, ky = S.ky;
#pragma unroll
      for (int k = 0; k < kPPL; ++k)
        if (valid[k] && c[k] != PIC_CELL_OUT) {
          const float2* e0 = ef + cell_j(c[k]) * enx + cell_i(c[k]);
          const float2 e00 = __ldg(e0), e10 = __ldg(e0 + 1), e01 = __ldg(e0 + enx), e11 = __ldg(e0 + enx + 1);
          const float x = fx[k], y = fy[k];
          const float w00 = (1.f - x) * (1.f - y), w10 = x * (1.f - y), w01 = (1.f - x) * y, w11 = x * y;
          const float gx = w00 * e00.x + w10 * e10.x + w01 * e01.x + w11 * e11.x;
          const float gy = w00 * e00.y + w10 * e10.y + w01 * e01.y + w11 * e11.y;
          vx[k] += kx * gx;
          vy[k] += ky * gy;
        }
    }
    if (do_mcc) {
      if (J.mcc_mode == 2) {
        const ProcDev& P = J.procs[S.first_proc];
#pragma unroll
        for (int k = 0; k < kPPL; ++k)
          if (valid[k]) {
            float u[4];
            draw4(J.seed, pid[k], mcc_step, 0u, u);
            const float v2 = vx[k] * vx[k] + vy[k] * vy[k];
            const float sp = sqrtf(v2);
            const float Pc = 1.f - expf(-J.gas_density * xs_lookup(P, S.half_m_over_e * v2) * sp * J.dt);
            if (u[0] < Pc) {
              float sn, cs;
              sincospif(2.f * u[1], &sn, &cs);
              vx[k] = sp * cs; vy[k] = sp * sn;
              atomicAdd(&pc[0], 1u);
            }
          }
      } else {
        // candidate with probability nu_max dt; a candidate's collision is real when
        // u1 nu_max < n sigma_T(E) v (the process is chosen in the queue round, with the
        // same draw).  Null candidates stay in the item like every other particle.
        bool cand[kPPL];
        uint32_t x1[kPPL];
        unsigned m[kPPL];
        int before[kPPL];
        int ncand = 0;
#pragma unroll
        for (int k = 0; k < kPPL; ++k) {
          uint32_t x[4] = {pid[k], mcc_step, 0u, 0u};
          philox4x32_10(x, (uint32_t)J.seed, (uint32_t)(J.seed >> 32));
          x1[k] = x[1];
          cand[k] = valid[k] && (x[0] >> 9) < cand_below;
        }
        // The cross-section lookup is a chain of dependent loads that the whole warp waits for
        // whenever one lane needs it, so each pass of this loop takes one candidate of every lane
        // that has any left: one pass where each lane has at most one.
        unsigned left = 0;
#pragma unroll
        for (int k = 0; k < kPPL; ++k) left |= cand[k] ? 1u << k : 0u;
        while (left) {
          const int k = __ffs(left) - 1;
          left &= left - 1u;
          float v2 = 0.f, u1 = 0.f;
#pragma unroll
          for (int q = 0; q < kPPL; ++q)
            if (q == k) { v2 = vx[q] * vx[q] + vy[q] * vy[q] + vz[q] * vz[q]; u1 = u01(x1[q]); }
          const bool real = u1 * S.numax < J.gas_density * xs_lookup(S.total, S.half_m_over_e * v2) * sqrtf(v2);
#pragma unroll
          for (int q = 0; q < kPPL; ++q)
            if (q == k) cand[q] = real;
        }
#pragma unroll
        for (int k = 0; k < kPPL; ++k) {
          m[k] = __ballot_sync(0xffffffffu, cand[k]);
          before[k] = ncand;
          ncand += __popc(m[k]);
        }
        // rank of candidate (lane, k): item order k-major, then lane
        int rank[kPPL];
#pragma unroll
        for (int k = 0; k < kPPL; ++k) rank[k] = before[k] + __popc(m[k] & ((1u << lane) - 1u));
        // candidates leave the item for the warp's queue
#pragma unroll
        for (int k = 0; k < kPPL; ++k)
          if (cand[k]) {
            const int q = qn + rank[k];
            cq[0 * kQueue + q] = c[k];
            cq[1 * kQueue + q] = __float_as_uint(fx[k]); cq[2 * kQueue + q] = __float_as_uint(fy[k]);
            cq[3 * kQueue + q] = __float_as_uint(vx[k]); cq[4 * kQueue + q] = __float_as_uint(vy[k]);
            cq[5 * kQueue + q] = __float_as_uint(vz[k]); cq[6 * kQueue + q] = pid[k];
            cq[7 * kQueue + q] = (uint32_t)(i0 + k);
            valid[k] = false;   // the queue round finishes this particle
          }
        qn += ncand;
      }
    }
    if (want_ke) {
#pragma unroll
      for (int k = 0; k < kPPL; ++k)
        if (valid[k]) ke += (double)(vx[k] * vx[k] + vy[k] * vy[k] + vz[k] * vz[k]);
    }
    // ---- pass B: drift, walls, deposit
    uint32_t c_in[kPPL];
#pragma unroll
    for (int k = 0; k < kPPL; ++k) c_in[k] = c[k];
    uint32_t key[kPPL];
    bool absorbed[kPPL];
#pragma unroll
    for (int k = 0; k < kPPL; ++k) {
      absorbed[k] = false;
      key[k] = valid[k] ? c[k] : PIC_CELL_OUT;
    }
    if (do_drift) {
      // no particle of the warp leaves its cell (ions, nearly always): the drifted offsets are the
      // new ones and nothing is absorbed, without the cell arithmetic
      bool stay = !(do_walls && (J.wall_mode & 2));
      float ax[kPPL], ay[kPPL];
#pragma unroll
      for (int k = 0; k < kPPL; ++k) {
        ax[k] = fx[k] + vx[k] * S.dtdx;
        ay[k] = fy[k] + vy[k] * S.dtdy;
        stay = stay && (!valid[k] || (c[k] != PIC_CELL_OUT && ax[k] >= 0.f && ax[k] < 1.f && ay[k] >= 0.f && ay[k] < 1.f));
      }
      if (__all_sync(0xffffffffu, stay)) {
#pragma unroll
        for (int k = 0; k < kPPL; ++k)
          if (valid[k]) { fx[k] = ax[k]; fy[k] = ay[k]; }
      } else {
#pragma unroll
        for (int k = 0; k < kPPL; ++k)
          if (valid[k]) {
            const Drifted d = drift_particle(J, S, c[k], fx[k], fy[k], vx[k], vy[k], do_walls);
            absorbed[k] = d.absorbed; c[k] = d.cell; fx[k] = d.fx; fy[k] = d.fy;
            key[k] = d.absorbed ? PIC_CELL_OUT : d.cell;
          }
      }
    }
    if (do_walls) {
      unsigned hm[kPPL];
      int nh = 0, hb[kPPL];
#pragma unroll
      for (int k = 0; k < kPPL; ++k) {
        hm[k] = __ballot_sync(0xffffffffu, valid[k] && absorbed[k]);
        hb[k] = nh;
        nh += __popc(hm[k]);
      }
      if (nh) {
        int base = 0;
        if (lane == 0) base = atomicAdd(hit_counts + s, nh);
        base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
        for (int k = 0; k < kPPL; ++k)
          if (valid[k] && absorbed[k]) S.hits[base + hb[k] + __popc(hm[k] & ((1u << lane) - 1u))] = i0 + k;
      }
    }
    if (do_dep) {
      if (J.deposit_mode == 0) {
        const float q = S.qdep;
        lane_deposit<float>(J.rho_f, J.nx, key, fx, fy,
                            [q](float x, float y, float& a, float& b, float& cc, float& d) { cic_f32(q, x, y, a, b, cc, d); });
      } else {
        const long long qf = S.qfix;
        lane_deposit<unsigned long long>(
            reinterpret_cast<unsigned long long*>(J.rho_i), J.nx, key, fx, fy,
            [qf](float x, float y, unsigned long long& a, unsigned long long& b, unsigned long long& cc,
                 unsigned long long& d) {
              long long a_, b_, c_, d_;
              cic_i64(qf, x, y, a_, b_, c_, d_);
              a = (unsigned long long)a_; b = (unsigned long long)b_; cc = (unsigned long long)c_;
              d = (unsigned long long)d_;
            });
      }
    }
    // ---- stores
    if (do_drift) {
      // the cell word changes only when a particle crosses a cell edge (rare for ions): a warp
      // whose cells all stayed leaves them in place
      bool moved = false;
#pragma unroll
      for (int k = 0; k < kPPL; ++k) moved |= c[k] != c_in[k];
      if (__any_sync(0xffffffffu, moved)) st_lane(S.cell + i0, c);
      st_lane(S.fx + i0, fx);
      st_lane(S.fy + i0, fy);
    }
    if (do_kick || do_mcc) {
      st_lane(S.vx + i0, vx);
      st_lane(S.vy + i0, vy);
    }
    // vz changes only in a collision, and the queue round stores the collided particles
    // full rounds of queued candidates, after this item's stores
    while (qn >= 32) round(32);
  }
  flush();
}

int mover_blocks_per_sm() {
  cudaFuncSetAttribute(mover_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMoverSmem);
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, mover_kernel, PIC_MOVER_THREADS, kMoverSmem) != cudaSuccess ||
      b < 1) {
    cudaGetLastError();
    b = 1;
  }
  return b;
}

int launch_step_head(const EngineLaunch& L, cudaStream_t stream) {
  if (!L.njobs) return 0;
  const int gx = std::max(1, std::min(4096, 8 * L.num_sms / L.njobs));
  step_head_kernel<<<dim3(gx, L.njobs), 256, 0, stream>>>(L.jobs, L.st, L.counts, L.active, L.chunk_prefix, L.nslots);
  return 1;
}

int launch_mover(const EngineLaunch& L, int flags, uint32_t explicit_step, bool after_head, cudaStream_t stream) {
  int k = 1;
  if (!after_head) {
    if ((flags & PIC_PHASE_KICK_I) && L.njobs > 0) {
      // the node field of every job's current potential, for the kick
      const int gx = std::max(1, std::min(4096, 8 * L.num_sms / L.njobs));
      efield32_kernel<<<dim3(gx, L.njobs), 256, 0, stream>>>(L.jobs, L.st);
      ++k;
    }
    chunk_table_kernel<<<1, 32, 0, stream>>>(L.counts, L.active, L.chunk_prefix, L.nslots);
    ++k;
  }
  if (L.ev_mover_begin) cudaEventRecord(L.ev_mover_begin, stream);
  mover_kernel<<<L.mover_grid, PIC_MOVER_THREADS, kMoverSmem, stream>>>(L.jobs, L.st, L.slots, L.counts,
                                                                          L.hit_counts, L.chunk_prefix, L.nslots, flags,
                                                                          explicit_step);
  if (L.ev_mover_end) cudaEventRecord(L.ev_mover_end, stream);
  return k;
}
