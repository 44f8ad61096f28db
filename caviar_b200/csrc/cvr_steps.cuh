// cvr_steps.cuh -- many velocity-Verlet steps of a small short-range system
// in one launch.
//
// A step of a system of a few thousand atoms is a few microseconds of work
// per kernel, and with one kernel per stage (position update, rebuild
// condition, list build, pair force, kick, thermostat) the launches and the
// gaps between dependent kernels cost more than the work.  Here one
// cooperative launch runs all steps of a run.  The blocks stay resident and
// meet at grid barriers (1.5 us each at 148 blocks): one per step, two with a
// thermostat or a thermo record, four more on a step that rebuilds the list.
// Per step (runs without records, one kernel per stage -> k_steps): 500 LJ
// atoms mixed 20.5 -> 7.0 us, 4000 mixed 22.8 -> 9.1 and FP64 26.1 -> 11.8,
// 16,001 mixed 33.1 -> 14.3, 32,001 37.6 -> 23.5, 65,001 50.1 -> 40.7 and FP64
// 62.1 -> 50.6, 32,001 of two types under Berendsen 51.4 -> 32.9.  Of the 9.1
// us at 4000 atoms, 1.9 are the barrier (waiting included), 4.7 the pair force
// and update, and 33 per rebuild (one step in 10) the build.
//
// The stage that ends one step starts the next: the warp that summed atom
// i's force applies both half kicks and the drift to it at once, writing the
// new pair coordinates into the other of two buffers, so that neighbours
// still read the old ones and no barrier is needed in between.  On a rebuild
// the warp that searches atom i's neighbours sums its force right after (the
// search reads a copy of the positions: other atoms may have drifted on).
// The per-atom functions are those of the one-kernel-per-stage path, so the
// trajectories agree bit for bit (with a thermostat the kinetic energy is
// summed in another order).
//
// The barriers' waits are bounded; one that runs out sets ERR_BARRIER and the
// block leaves.  A block passes a barrier only when all have arrived at it, so
// the blocks still running never see a stage half done; the state and the
// build's counters are left as they are, and the host drops both.
#pragma once
#include "cvr_build.cuh"
#include "cvr_device.cuh"
#include "cvr_force.cuh"

namespace cvr {

// Most threads per block, one block per SM: 28 warps at 72 registers, so that
// 4000 atoms are one per warp (24 warps: 12.7 us per step, mixed, 16 FP64
// warps 13.1, against 9.1 and 11.8; 32 warps spill: 10.1).  A block takes
// only the warps its atoms need.
constexpr int STEP_THREADS = 896;

// Control words (64 bits): a pair of barrier words for this launch and one
// for the next, which this launch clears.
constexpr int SC_WORDS = 4;

template <typename real> struct StepArgs {
  const PairCoef<real> *coef;
  real fscale;
  int ignore_intra, use_mol, log2_tpa;
  double dt;
  int nsteps;
  typename V4<real>::t *x4b;  // second pair-coordinate buffer
  double *bx, *by, *bz;       // positions at the build
  unsigned long long *ctrl;
  int *share_atoms;           // [gridDim.x], zero between builds (scan_cells)
  int launch;                 // parity: which pair of control words is this launch's
  unsigned polls;             // most polls of a barrier's wait
  long long *counters;
  ThermostatArgs ts;
  double *part;               // [gridDim.x][4]: the thermostat's block sums
  // warps' sums of a thermo record, one half per parity of the record: pair
  // energies and virial [warps of k_pair][3], kinetic energy and momentum [n / 32][4]
  double *ev_warp[2], *ke_warp[2];
  int every, done;            // thermo record after steps k with (done + k + 1) % every == 0 (0: none)
  ThermoArgs th;
};

constexpr unsigned BARRIER_POLLS = 1u << 22;  // a barrier's wait: some seconds
// Steps per launch (the need field holds 2^24 / 148 of them).  The blocks hold
// their SMs for the whole launch, and other streams wait that long: at most
// about 15 ms (1024 steps of 500 atoms 6.2 ms, of 16,000 13-16; 256 of 65,000
// 10-12), which the 10 us of a launch do not lengthen (0.2 %).
constexpr int STEPS_MAX = 1024;
constexpr int64_t STEPS_ATOMS_MAX = 1 << 24;  // steps x atoms

// Grid barrier on a counter per parity of the barrier: every block adds 1,
// plus 2^32 if it asks for a list rebuild and 2^56 if it met an error, and
// polls until all blocks of this barrier have added theirs.  A block adds to
// a counter again only two barriers later, when all have left this one, so
// everybody reads the same word: the arrivals and both answers come with one
// load, and all blocks leave a failed run at the same barrier.
// The bookkeeping lives in shared memory: only thread 0 needs it.
struct GridBarrier {
  unsigned long long *word;  // [2]
  unsigned count[2];         // arrivals awaited, per parity
  unsigned needs[2];         // rebuild requests before this barrier, per parity
  unsigned limit;            // most polls of a wait
  int parity;
  int need, bad;             // set by any thread that asks for a rebuild or met an error
  int answer;

  __device__ __forceinline__ void init(unsigned long long *w, unsigned polls) {
    if (threadIdx.x == 0) {
      word = w;
      limit = polls;
      count[0] = count[1] = needs[0] = needs[1] = 0;
      parity = need = bad = 0;
    }
    __syncthreads();
  }

  // 1: a block asked for a rebuild; 2: a block met an error (for every thread alike)
  __device__ __forceinline__ int meet(int *err) {
    __syncthreads();
    if (threadIdx.x == 0) {
      const int p = parity;
      const unsigned long long add = 1ull + (need ? 1ull << 32 : 0ull) + (bad ? 1ull << 56 : 0ull);
      unsigned long long *w = word + p, v;
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"(add) : "memory");
      need = 0;
      parity = p ^ 1;
      const unsigned want = count[p] + gridDim.x;
      count[p] = want;
      unsigned polls = 0;
      do {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(w) : "memory");
      } while ((unsigned)v < want && ++polls < limit);
      int a = (v >> 56) ? 2 : 0;
      if ((unsigned)v < want) {
        atomicOr(err, ERR_BARRIER);
        a = 2;
      }
      const unsigned total = (unsigned)(v >> 32) & 0xffffffu;
      if (total != needs[p]) a |= 1;
      needs[p] = total;
      answer = a;
    }
    __syncthreads();
    return answer;
  }
};

// The scan of the cell counts, every block its own share of the cells, needs
// the atoms of the shares before it.  The binning counts them, once per warp
// and share (the atoms are in the last build's cell order, and single adds
// would queue at a few addresses: 32,001 atoms 37.3 us per step).  Summing the
// cells before the share instead costs blocks x cells: a build of 500 atoms at
// density 1e-3 (175,000 cells) took 338 us that way, 53 with the shares'
// atoms, 74 with one kernel per stage; dense systems, summed / counted: 500
// atoms 8.6 / 8.7 us per step, 4000 FP64 24.5 / 24.5, 32,001 36.5 / 35.7.
__device__ __forceinline__ int cell_share(int ncells) { return (ncells + gridDim.x - 1) / gridDim.x; }
__device__ __forceinline__ bool few_cells(int ncells) { return ncells <= 8 * (int)blockDim.x; }

// Bins the atoms, counting them per cell and per share.
template <typename real>
__device__ __forceinline__ void bin_atoms(const DevState<real> &s, int *share_atoms, int tid, int nthreads) {
  const int share = cell_share(s.cells.ncells), lane = threadIdx.x & 31;
  for (int i = tid; i < s.n; i += nthreads) {
    const int b = bin_atom(s, i) / share;
    const unsigned same = __match_any_sync(__activemask(), b);
    if (lane == __ffs(same) - 1) atomicAdd(&share_atoms[b], __popc(same));
  }
}

// Exclusive scan of cell_count into cell_start: what lies before the block's
// share, then a block scan over it, four cells per thread.  Not inlined: inside
// k_steps it costs the pair stage registers.
__device__ __noinline__ void scan_cells(const int *count, int *start, const int *share_atoms, int ncells, int *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int share = cell_share(ncells);
  const int c0 = min(ncells, (int)blockIdx.x * share), c1 = min(ncells, c0 + share);
  int before = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += blockDim.x) before += share_atoms[b];
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 0) red[warp] = before;
  __syncthreads();
  before = 0;
  for (int w = 0; w < nw; ++w) before += red[w];
  for (int base = c0; base < c1; base += 4 * blockDim.x) {
    const int c = base + 4 * threadIdx.x;
    int v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = c + u < c1 ? count[c + u] : 0;
    const int mine = (v[0] + v[1]) + (v[2] + v[3]);
    int x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) red[warp] = x;
    __syncthreads();
    int ahead = 0, total = 0;
    for (int w = 0; w < nw; ++w) {
      const int t = red[w];
      if (w < warp) ahead += t;
      total += t;
    }
    int at = before + ahead + x - mine;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c + u < c1) start[c + u] = at;
      at += v[u];
    }
    before += total;
  }
  if (c1 == ncells && c0 < c1 && threadIdx.x == 0) start[ncells] = before;
}

// One warp's list-search pieces inside the block's dynamic shared memory.
__device__ __forceinline__ WarpPieces warp_pieces(unsigned char *sm, int warp, int warps) {
  float4 *geo = reinterpret_cast<float4 *>(sm);
  int *off = reinterpret_cast<int *>(geo + warps * PIECES_MAX);
  uint32_t *pc = reinterpret_cast<uint32_t *>(off + warps * (PIECES_MAX + 1));
  return WarpPieces{off + warp * (PIECES_MAX + 1), geo + warp * PIECES_MAX, pc + warp * PIECES_MAX};
}

// Block-wide sum of NV doubles into out[0..NV) (fixed order).
template <int NV>
__device__ __forceinline__ void block_sum_to(double (&v)[NV], double *out) {
  __shared__ double red[NV][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();  // the array is free again
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    double x = v[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[q][warp] = x;
  }
  __syncthreads();
  if ((int)threadIdx.x < NV) {
    double x = 0.0;
    for (int w = 0; w < nw; ++w) x += red[threadIdx.x][w];
    out[threadIdx.x] = x;
  }
}

template <typename real, int TPA, bool ONE_TYPE, bool FIXED>
__global__ void __launch_bounds__(STEP_THREADS, 1) k_steps(DevState<real> s, StepArgs<real> a) {
  using real4 = typename V4<real>::t;
  constexpr int GPW = 32 / TPA;
  const int THREADS = blockDim.x, WARPS = THREADS >> 5;
  extern __shared__ __align__(16) unsigned char smraw[];  // the warps' list-search pieces
  __shared__ PairCoef<real> coef[ONE_TYPE ? 1 : MAX_TYPES * MAX_TYPES];
  __shared__ GridBarrier grid;
  __shared__ int red[STEP_THREADS / 32];
  __shared__ double ke_sum[4], rec_red[7][32];
  const int n = s.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tid = blockIdx.x * THREADS + threadIdx.x, nthreads = gridDim.x * THREADS;
  const int gwarp = blockIdx.x * WARPS + warp, nwarps = gridDim.x * WARPS;
  for (int t = threadIdx.x; t < (ONE_TYPE ? 1 : s.n_types * s.n_types); t += THREADS) coef[t] = a.coef[t];
  if (tid < 2) a.ctrl[2 * (a.launch ^ 1) + tid] = 0;
  grid.init(a.ctrl + 2 * a.launch, a.polls);
  const Stencil<real> st = stencil_of(s);
  const EwrArgs<real> no_ewald{};
  const WarpPieces wp = warp_pieces(smraw, warp, WARPS);
  real4 *buf[2] = {s.x4, a.x4b};
  DevState<real> built = s;  // as the list search sees it
  built.x = a.bx;
  built.y = a.by;
  built.z = a.bz;
  const double h = 0.5 * a.dt;
  const int ts = a.ts.kind;
  double zeta = ts == 2 ? a.ts.scal[1] : 0.0, lambda = 1.0;
  const long long step0 = a.counters[0];  // block 0 writes the counters after the last barrier
  // an atom's stored drift: rebuild request and NaN error
  const auto drifted = [&](int i, const double (&acc)[3], const double (&v)[3], const double (&p)[3], const real4 *in,
                           real4 *out) {
    if (store_drift(s, i, acc, v, p, in, out)) grid.need = 1;
    if (isnan(acc[0]) || isnan(acc[1]) || isnan(acc[2])) grid.bad = 1;
  };

  // the first step's kick and drift, one thread per atom
  for (int i = tid; i < n; i += nthreads) {
    const double acc[3] = {(double)s.ax[i], (double)s.ay[i], (double)s.az[i]};
    double v[3], p[3];
    kick_drift_atom(s, i, a.dt, 0.0, acc[0], acc[1], acc[2], v, p);
    drifted(i, acc, v, p, buf[0], buf[1]);
  }
  // Step k's thermo record, by one block beside the next step's work (which
  // writes the other half of the sums).  The sums are those of k_pair's and
  // k_kick's blocks and k_thermo's threads, in their order: the record is
  // theirs bit for bit.
  long long records = a.counters[1];
  const auto record = [&](int k, int which) {
    const long long at = records++;
    if (blockIdx.x != 0) return;
    const double *ew = a.ev_warp[which], *kw = a.ke_warp[which];
    const int n_ew = (n + GPW - 1) / GPW, n_kw = (n + 31) >> 5;
    const auto warp_value = [](const double *p, int w, int nw, int stride, int q) {
      return w < nw ? p[(size_t)w * stride + q] : 0.0;
    };
    const auto tree = [&](double x) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      return x;
    };
    for (int vw = warp; vw < THERMO_THREADS / 32; vw += WARPS) {
      double v[7] = {0, 0, 0, 0, 0, 0, 0};
      for (int b = vw * 32 + lane; b < (n + 255) / 256; b += THERMO_THREADS)
        for (int q = 0; q < 4; ++q) {
          double w[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) w[u] = warp_value(kw, 8 * b + u, n_kw, 4, q);
          v[q] += ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
        }
      for (int b = vw * 32 + lane; b < (n_ew + 3) / 4; b += THERMO_THREADS)
        for (int q = 0; q < 3; ++q) {
          double w[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) w[u] = warp_value(ew, 4 * b + u, n_ew, 3, q);
          v[4 + q] += (w[0] + w[2]) + (w[1] + w[3]);
        }
#pragma unroll
      for (int q = 0; q < 7; ++q) {
        const double x = tree(v[q]);
        if (lane == 0) rec_red[q][vw] = x;
      }
    }
    __syncthreads();
    if (warp == 0) {
      double acc[8];
      acc[7] = 0.0;
#pragma unroll
      for (int q = 0; q < 7; ++q) acc[q] = tree(rec_red[q][lane]);
      if (lane == 0) thermo_record(a.th, acc, step0 + k + 1, a.th.out + at * 10);
    }
    __syncthreads();
  };

  int cur = 0, half = 0;
  bool record_due = false;
  for (int k = 0; k < a.nsteps; ++k) {
    const int answer = grid.meet(s.err);
    if (answer & 2) return;
    cur ^= 1;
    if (record_due) {
      record(k - 1, half);
      half ^= 1;
    }
    const bool build = answer & 1;
    if (build) {
      bin_atoms(s, a.share_atoms, tid, nthreads);
      if (grid.meet(s.err) & 2) return;
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        *s.build_epoch += 1;
        atomicAdd(s.n_builds, 1);
      }
      scan_cells(s.cell_count, s.cell_start, a.share_atoms, s.cells.ncells, red);
      if (grid.meet(s.err) & 2) return;
      for (int i = tid; i < n; i += nthreads) scatter_atom(s, i);
      if (grid.meet(s.err) & 2) return;
      for (int c = tid; c < s.cells.ncells; c += nthreads) s.cell_count[c] = s.cell_fill[c] = 0;
      if (tid < (int)gridDim.x) a.share_atoms[tid] = 0;
      for (int t = tid; t < n; t += nthreads) {
        const int i = s.slot_atom[t];
        const int to = place_of(s, i);
        place_atom(s, to, i, buf[cur]);
        a.bx[to] = s.tx[i];
        a.by[to] = s.ty[i];
        a.bz[to] = s.tz[i];
      }
      if (grid.meet(s.err) & 2) return;
    }
    const bool last = k + 1 == a.nsteps;
    record_due = a.every > 0 && (a.done + k + 1) % a.every == 0;
    const bool two_pass = ts || record_due;  // forces and kick, then (all sums known) thermostat and drift
    const auto pair_stage = [&](auto with_record) {
      constexpr bool EV = decltype(with_record)::value;
      double ke[4] = {0, 0, 0, 0};
      for (int base = gwarp * GPW; base < n; base += nwarps * GPW) {
        if (build) {
#pragma unroll 1
          for (int g = 0; g < GPW; ++g)
            if (base + g < n && list_search_warp(built, base + g, lane, wp, 0, a.log2_tpa) > s.cap) grid.bad = 1;
          __syncwarp();
        }
        const int i = base + lane / TPA, sub = lane % TPA;
        const bool valid = i < n;
        if (valid && sub < 7) {  // what the update below reads, into L1 meanwhile
          const void *w = sub == 0   ? (const void *)(s.vx + i)
                          : sub == 1 ? (const void *)(s.vy + i)
                          : sub == 2 ? (const void *)(s.vz + i)
                          : sub == 3 ? (const void *)(s.x + i)
                          : sub == 4 ? (const void *)(s.y + i)
                          : sub == 5 ? (const void *)(s.z + i)
                                     : (const void *)(s.xb + i);
          asm volatile("prefetch.global.L1 [%0];" ::"l"(w));
        }
        PairAcc<real> A{0, 0, 0, 0.0, 0.0, 0.0, 0, 0, 0};
        int ti = 0;
        if (valid)
          pair_row<real, TPA, true, false, EV, ONE_TYPE, FIXED>(A, ti, s, buf[cur], i, sub, coef, st, no_ewald,
                                                                a.ignore_intra, a.use_mol);
#pragma unroll
        for (int o = TPA / 2; o > 0; o >>= 1) {
          A.fx += __shfl_xor_sync(0xffffffffu, A.fx, o);
          A.fy += __shfl_xor_sync(0xffffffffu, A.fy, o);
          A.fz += __shfl_xor_sync(0xffffffffu, A.fz, o);
        }
        if (EV) {  // full list: each pair twice
          double e[3] = {0.5 * A.e_lj, 0.0, 0.5 * A.vir};
#pragma unroll
          for (int q = 0; q < 3; ++q) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) e[q] += __shfl_down_sync(0xffffffffu, e[q], o);
            if (lane == 0) a.ev_warp[half][(size_t)(base / GPW) * 3 + q] = e[q];
          }
        }
        if (!valid || sub != 0) continue;
        const real mi = (real)s.mass_inv[ti] * a.fscale;
        const real ax = A.fx * mi, ay = A.fy * mi, az = A.fz * mi;
        const double acc[3] = {(double)ax, (double)ay, (double)az};
        if (last || two_pass) {  // the step's second half kick by itself
          s.ax[i] = ax;
          s.ay[i] = ay;
          s.az[i] = az;
          const double v0 = s.vx[i] + h * acc[0], v1 = s.vy[i] + h * acc[1], v2 = s.vz[i] + h * acc[2];
          s.vx[i] = v0;
          s.vy[i] = v1;
          s.vz[i] = v2;
          if (ts) {
            const double m = s.mass[s.type[i]];
            ke[0] += m * (v0 * v0 + v1 * v1 + v2 * v2);
            ke[1] += m * v0;
            ke[2] += m * v1;
            ke[3] += m * v2;
          }
        } else {
          double v[3], p[3];
          kick_drift_atom(s, i, a.dt, h, acc[0], acc[1], acc[2], v, p);
          drifted(i, acc, v, p, buf[cur], buf[cur ^ 1]);
        }
      }
      if (ts) block_sum_to<4>(ke, a.part + 4 * blockIdx.x);
    };
    if (record_due)
      pair_stage(std::true_type{});
    else
      pair_stage(std::false_type{});
    if (two_pass) {
      if (grid.meet(s.err) & 2) return;
      if (ts) {
        for (int q = warp; q < 4; q += WARPS) {  // every block sums the partials in the same order
          double x = 0.0;
          for (int b = lane; b < (int)gridDim.x; b += 32) x += a.part[4 * b + q];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
          if (lane == 0) ke_sum[q] = x;
        }
        __syncthreads();
        const double sums[4] = {ke_sum[0], ke_sum[1], ke_sum[2], ke_sum[3]};
        thermostat_update(a.ts, sums, step0 + k, lambda, zeta);
      }
      for (int b = gwarp * 32; b < n; b += nthreads) {
        const int i = b + lane;
        double ke[4] = {0, 0, 0, 0};
        if (i < n) {
          double v0 = s.vx[i], v1 = s.vy[i], v2 = s.vz[i];
          if (ts == 1) {
            v0 *= lambda;
            v1 *= lambda;
            v2 *= lambda;
            s.vx[i] = v0;
            s.vy[i] = v1;
            s.vz[i] = v2;
          }
          if (record_due) {
            const double m = s.mass[s.type[i]];
            ke[0] = m * (v0 * v0 + v1 * v1 + v2 * v2);
            ke[1] = m * v0;
            ke[2] = m * v1;
            ke[3] = m * v2;
          }
          if (ts == 2) {
            s.ax[i] = (real)((double)s.ax[i] - zeta * v0);
            s.ay[i] = (real)((double)s.ay[i] - zeta * v1);
            s.az[i] = (real)((double)s.az[i] - zeta * v2);
          }
          if (!last) {
            const double acc[3] = {(double)s.ax[i], (double)s.ay[i], (double)s.az[i]};
            double v[3], p[3];
            kick_drift_atom(s, i, a.dt, 0.0, acc[0], acc[1], acc[2], v, p);
            drifted(i, acc, v, p, buf[cur], buf[cur ^ 1]);
          }
        }
        if (record_due) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ke[q] += __shfl_down_sync(0xffffffffu, ke[q], o);
            if (lane == 0) a.ke_warp[half][(size_t)(b >> 5) * 4 + q] = ke[q];
          }
        }
      }
    }
  }
  if (record_due) {  // the last step's record
    if (grid.meet(s.err) & 2) return;
    record(a.nsteps - 1, half);
  }
  // the coordinates of the last step into the context's own buffer (only
  // the other one is still being read)
  if (cur == 1)
    for (int i = tid; i < n; i += nthreads) s.x4[i] = a.x4b[i];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.counters[0] = step0 + a.nsteps;
    a.counters[1] = records;
    if (ts) {
      a.ts.scal[0] = lambda;
      a.ts.scal[1] = zeta;
    }
  }
}

// A forced list build (count_only: the neighbour counts alone) in one launch
// for the systems k_steps takes: the stages of launch_build between grid
// barriers.  Eight launches of 2-4 us each and their gaps otherwise.  Returns
// at once if the rebuild flag is not set.
template <typename real>
__global__ void __launch_bounds__(STEP_THREADS, 1)
    k_build_once(DevState<real> s, unsigned long long *ctrl, int *share_atoms, int launch, unsigned polls, int count_only,
                 int log2_tpa) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ GridBarrier grid;
  __shared__ int red[STEP_THREADS / 32];
  const int n = s.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
  if (tid < 2) ctrl[2 * (launch ^ 1) + tid] = 0;
  if (*s.flag == 0) return;
  grid.init(ctrl + 2 * launch, polls);
  bin_atoms(s, share_atoms, tid, nthreads);
  if (grid.meet(s.err) & 2) return;
  if (tid == 0) {
    *s.build_epoch += 1;
    if (!count_only) atomicAdd(s.n_builds, 1);
  }
  scan_cells(s.cell_count, s.cell_start, share_atoms, s.cells.ncells, red);
  if (grid.meet(s.err) & 2) return;
  for (int i = tid; i < n; i += nthreads) scatter_atom(s, i);
  if (grid.meet(s.err) & 2) return;
  for (int c = tid; c < s.cells.ncells; c += nthreads) s.cell_count[c] = s.cell_fill[c] = 0;
  if (tid < (int)gridDim.x) share_atoms[tid] = 0;
  for (int t = tid; t < n; t += nthreads) {
    const int i = s.slot_atom[t];
    place_atom(s, place_of(s, i), i, s.x4);
  }
  if (grid.meet(s.err) & 2) return;
  const WarpPieces wp = warp_pieces(smraw, warp, warps);
  for (int i = blockIdx.x * warps + warp; i < n; i += gridDim.x * warps)
    list_search_warp(s, i, lane, wp, count_only, log2_tpa);
}

// one record's sums for n atoms (at most one k_pair warp per atom)
inline size_t steps_record_doubles(size_t n) { return 3 * n + 4 * ((n + 31) / 32); }

inline size_t steps_smem(int warps) {
  constexpr size_t pieces = PIECES_MAX;
  return warps * (pieces * (sizeof(float4) + sizeof(uint32_t)) + (pieces + 1) * sizeof(int));
}

}  // namespace cvr
