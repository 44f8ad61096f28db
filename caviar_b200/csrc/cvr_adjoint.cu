// cvr_adjoint.cu -- gradient of a trajectory loss through velocity Verlet on
// the GPU: forces, their vector-Jacobian product (VJP) w.r.t. positions and
// force-field parameters, and a checkpointed reverse sweep.
//
// No reference counterpart: the reference has no gradients.  The forward
// follows the reference's force definitions (LJ with the linear force shift,
// lj.cpp:439-448; Ewald real space, electrostatic_ewald_r.cpp:196-198, here
// with an explicit cutoff; Ewald k space over the reference's k-set,
// initialize.cpp:184-222 and electrostatic_ewald_k.cpp:197-234; velocity
// Verlet, md_simulator.cpp:555-668) on one periodic cube under the minimum
// image (every cutoff <= L/2).
//
// Every force evaluation of a trajectory uses the same kernels (the energy
// terms sit behind a uniform branch), so the segments the reverse sweep
// re-runs are bit-identical to the forward pass.
//
// Loss J = (1/M) sum_{t=1..M} U(r_t).  Reverse sweep over the state (r, v, a)
// with cotangents (Gr, Gv, Ga); for step t (r' = r_{t+1}):
//   Gr -= F(r')/M;  Ga += dt/2 Gv;  Gr += (dF/dr)^T (Ga/m);  theta_bar += (dF/dtheta)^T (Ga/m)
//   (Gr, Gv, Ga) <- (Gr, Gv + dt Gr, dt/2 Gv + dt^2/2 Gr)
// and finally the VJP at r_0 for a_0 = F(r_0)/m.  Positions, velocities and
// (memory allowing) forces are checkpointed every K steps; the reverse sweep
// re-runs each segment forward, keeping its K positions and forces (the last segment's
// are kept by the forward pass itself).
//
// Atoms are stored sorted by type (type 0 first), so that the partners of
// one species are one index range and an atom chunk holds one species.
//
// Kernels (real = float for the mixed form, double for FP64), five launches
// per evaluation:
//   k_adj_prep     the state update before the evaluation (position drift,
//                  or the reverse step's first half), phase tables
//                  e^{i 2 pi m x / L}, and the mixed form's packed coordinates
//   k_adj_pair     one to eight warps per atom over all partners: distance
//                  tests, the pairs inside each cutoff queued in shared memory
//                  and evaluated 32 at a time
//   k_adj_sk       species-resolved S_a(k) = sum_{i in a} e^{ik.r_i} and, for
//                  the VJP, T_a(k) = sum_{i in a} (k.u_i) e^{ik.r_i}, per atom
//                  chunk (FP32 sub-sums of 16 atoms, FP64 chunk sums)
//   k_adj_kreduce  chunks -> per-(column, m) force coefficients; energy and
//                  charge-gradient terms
//   k_adj_kforce   k-space force or VJP per atom, added to the pair part, and
//                  the state update after the evaluation (kick, or the
//                  reverse step's second half)
//   k_adj_accum    once per call: sums of the per-block parameter partials,
//                  which every evaluation adds to in place
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/caviar_b200.h"
#include "cvr_device.cuh"

namespace {

constexpr int NT = 2;         // types
constexpr int NTT = NT * NT;  // ordered type pairs
constexpr int KMAX_ADJ = 10;
constexpr int PAIR_WARPS = 8;   // warps per block of k_adj_pair
// partners per lane and round of k_adj_pair, and its queued pairs per warp and
// kind (at most 31 left over + a round)
template <typename real> constexpr int PAIR_ROUND = sizeof(real) == 4 ? 2 : 1;
template <typename real> constexpr int QCAP = 32 * (PAIR_ROUND<real> + 1);
constexpr int SK_STAGE = 64;    // atoms per shared-memory stage of k_adj_sk
constexpr int SK_THREADS = 128;
constexpr int SK_MG = 2;        // m-values per thread of k_adj_sk
constexpr int SK_MAXCHUNKS = 1024;
constexpr int KRED_E = 16, KRED_G = 16;  // k_adj_kreduce: entries and chunk groups per block
constexpr int KF_WARPS = 16;    // k_adj_kforce: warps per block of 32 atoms
constexpr int NPV = 3 * NTT;    // pair partials per block: three sums per ordered type pair

// FP64 sums over a call (device), each the sum of a per-block partial array
enum : int {
  A_PE = 0,             // pairs, energy form: sum Ue, Us, Uq per ordered type pair
  A_PV = A_PE + NPV,    // pairs, VJP form: sum dce ud, dcs ud, cq ud
  A_KE = A_PV + NPV,    // k space, energy form: E_k, dE_k/dq
  A_KV = A_KE + 1 + NT, // k space, VJP form: u . dF_k/dq
  A_N = A_KV + NT
};

template <typename real> struct R2;
template <> struct R2<float> { using t = float2; };
template <> struct R2<double> { using t = double2; };

struct Params {
  int n, n0, kmax, kp;      // n0 atoms of type 0, stored first
  int ncol, M;              // k-space columns summed, k_max + 1
  double L, invL, alpha, k_e, dt, kf;  // kf = 2 pi / L
  double mass_inv[NT], charge[NT];
};

// Pair constants of the ordered type pair; the cutoffs^2 are in the units of
// the tested displacements (fixed-point coordinates: L / 2^32).
template <typename real> struct LjC {
  real sg2, e, shift, shiftS, U0, U1, S0, S1;
  int on;
};
template <typename real> struct PairC {
  real rl2, rr2;            // rr2 < 0: no Ewald
  real rc2;                 // LJ cutoff^2 as a length
  double unit;              // fixed-point unit
  real alpha, alpha2, beta, ke;
  LjC<real> lj[NTT];
};

__device__ __forceinline__ void sincospi_a(float a, float *s, float *c) { sincospif(a, s, c); }
__device__ __forceinline__ void sincospi_a(double a, double *s, double *c) { sincospi(a, s, c); }

template <typename T2> __device__ __forceinline__ T2 cmul(T2 a, T2 b) {
  T2 r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
template <typename T2> __device__ __forceinline__ T2 conj_if(T2 a, bool c) {
  if (c) a.y = -a.y;
  return a;
}

// What k_adj_prep does before an evaluation at positions x:
//   PREP_EVAL   nothing (x = X)
//   PREP_DRIFT  x = Xin + dt V + dt^2/2 F/m, stored (md_simulator.cpp:591-593)
//   PREP_REV    the reverse step's first half: Gr -= F/M; Ga += dt/2 Gv; u = Ga/m
//   PREP_REV0   u = Ga/m (the VJP at r_0)
enum : int { PREP_EVAL = 0, PREP_DRIFT = 1, PREP_REV = 2, PREP_REV0 = 3 };
struct PrepArgs {
  int op;
  const double *X;      // positions in
  double *Xout;         // PREP_DRIFT
  const double *V, *F;  // PREP_DRIFT: velocities, forces; PREP_REV: F = forces at X
  double *Gr, *Ga, *u;
  const double *Gv;
  double invM;
};

// One thread per (atom, axis, four m-values); the m = 0 thread does the state
// update and packs the mixed form's coordinate.  tab[(axis*kp + m)*n + slot].
template <typename real, bool VJP>
__global__ void __launch_bounds__(256) k_adj_prep(Params p, PrepArgs a, typename R2<real>::t *__restrict__ tab,
                                                  uint32_t *__restrict__ xs, float *__restrict__ us) {
  const int n3 = 3 * p.n, t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n3) return;
  const int slot = t % p.n, ax = t / p.n, m4 = 4 * blockIdx.y;
  const double mi = slot >= p.n0 ? p.mass_inv[1] : p.mass_inv[0];
  const auto position = [&](int s) {
    return a.op == PREP_DRIFT ? a.X[s] + a.V[s] * p.dt + a.F[s] * mi * 0.5 * p.dt * p.dt : a.X[s];
  };
  const double x = position(t);
  if (m4 == 0) {
    if (a.op == PREP_DRIFT) a.Xout[t] = x;
    if (a.op == PREP_REV) {
      a.Gr[t] -= a.invM * a.F[t];
      const double ga = a.Ga[t] + 0.5 * p.dt * a.Gv[t];
      a.Ga[t] = ga;
      a.u[t] = ga * mi;
    } else if (a.op == PREP_REV0) {
      a.u[t] = a.Ga[t] * mi;
    }
    if (sizeof(real) == 4) {
      xs[4 * slot + ax] = (uint32_t)(unsigned long long)__double2ll_rn(x * (4294967296.0 * p.invL));
      if (ax == 0) {
        const bool fine = isfinite(x) && isfinite(position(slot + p.n)) && isfinite(position(slot + 2 * p.n));
        xs[4 * slot + 3] = fine ? 0u : 0x7fffffffu;
      }
      if (VJP) us[4 * slot + ax] = (float)a.u[t];
    }
  }
  const double w = x * p.invL;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int m = m4 + q;
    if (m >= p.kp) break;
    const double u = (double)m * w;
    real sn, cs;
    sincospi_a((real)(2.0 * (u - rint(u))), &sn, &cs);
    typename R2<real>::t v;
    v.x = cs;
    v.y = sn;
    tab[(size_t)(ax * p.kp + m) * p.n + slot] = v;
  }
}

// Species-resolved structure factors of one atom chunk (blockIdx.y; chunks
// of type 0 first) over columns (nx, ny), nx < 0 or nx = 0, ny <= 0 (for real
// charges the others are mirrors: S(-k) = conj(S(k)), T(-k) = -conj(T(k))).
// One thread holds a column's m = m0 .. m0 + SK_MG - 1: per atom the phase
// W = X Y and, with s = kf (nx ux + ny uy), t = kf uz, the products of W, sW,
// tW with Z[m]; S(+-m) and T(+-m) are sums and differences of the four (twelve)
// sums.  part[((chunk*NV + v)*M + m)*ncol + col], v = S+, S-, (T+, T-).
// Latency-bound at 4000 atoms (two blocks per SM): SK_MG and the stage are
// small to spread the sums.  One thread per k-vector over 256 atoms took 73 us
// (VJP 145; FP64 VJP at 1372 atoms 196); now 10, 14 and 14.
template <typename real, bool VJP>
__global__ void __launch_bounds__(SK_THREADS) k_adj_sk(Params p, const typename R2<real>::t *__restrict__ tab,
                                                       const double *__restrict__ U, int chunk, int nch0,
                                                       double2 *__restrict__ part) {
  using T2 = typename R2<real>::t;
  constexpr int NV = VJP ? 4 : 2, NA = VJP ? 12 : 4;
  extern __shared__ __align__(16) unsigned char smraw[];
  T2 *st = reinterpret_cast<T2 *>(smraw);                      // [SK_STAGE][3 kp]
  real *su = reinterpret_cast<real *>(st + SK_STAGE * 3 * p.kp);  // [SK_STAGE][3], times kf
  const int row = 3 * p.kp;
  const int ngr = (p.M + SK_MG - 1) / SK_MG;
  const int item = blockIdx.x * SK_THREADS + threadIdx.x;
  const bool live = item < p.ncol * ngr;
  const int col = live ? item % p.ncol : 0, m0 = live ? item / p.ncol * SK_MG : 0;
  const int nx = col / (2 * p.kmax + 1) - p.kmax, ny = col % (2 * p.kmax + 1) - p.kmax;
  const int mx = abs(nx), my = p.kp + abs(ny);
  const bool second = (int)blockIdx.y >= nch0;
  const int a0 = second ? p.n0 + ((int)blockIdx.y - nch0) * chunk : (int)blockIdx.y * chunk;
  const int a1 = min(second ? p.n : p.n0, a0 + chunk);
  real sub[SK_MG][NA];
  double acc[SK_MG][2 * NV];
#pragma unroll
  for (int u = 0; u < SK_MG; ++u) {
#pragma unroll
    for (int q = 0; q < NA; ++q) sub[u][q] = (real)0;
#pragma unroll
    for (int q = 0; q < 2 * NV; ++q) acc[u][q] = 0.0;
  }
  for (int s0 = a0; s0 < a1; s0 += SK_STAGE) {
    const int na = min(SK_STAGE, a1 - s0);
    __syncthreads();
    for (int t = threadIdx.x; t < row * SK_STAGE; t += SK_THREADS) {
      const int at = t % SK_STAGE, r = t / SK_STAGE;
      if (at < na) st[at * row + r] = tab[(size_t)r * p.n + s0 + at];
    }
    if (VJP)
      for (int t = threadIdx.x; t < 3 * SK_STAGE; t += SK_THREADS) {
        const int at = t % SK_STAGE, r = t / SK_STAGE;
        if (at < na) su[at * 3 + r] = (real)p.kf * (real)U[(size_t)r * p.n + s0 + at];
      }
    __syncthreads();
    if (!live) continue;
    for (int at = 0; at < na; ++at) {
      const T2 *tb = st + at * row;
      const T2 w = cmul(conj_if(tb[mx], nx < 0), conj_if(tb[my], ny < 0));
      T2 ws{}, wt{};
      if (VJP) {
        const real s = (real)nx * su[3 * at] + (real)ny * su[3 * at + 1], tt = su[3 * at + 2];
        ws.x = s * w.x;
        ws.y = s * w.y;
        wt.x = tt * w.x;
        wt.y = tt * w.y;
      }
#pragma unroll
      for (int u = 0; u < SK_MG; ++u) {
        const T2 z = tb[2 * p.kp + min(m0 + u, p.kmax)];
        sub[u][0] += w.x * z.x;
        sub[u][1] += w.y * z.y;
        sub[u][2] += w.x * z.y;
        sub[u][3] += w.y * z.x;
        if (VJP) {
          sub[u][4] += ws.x * z.x;
          sub[u][5] += ws.y * z.y;
          sub[u][6] += ws.x * z.y;
          sub[u][7] += ws.y * z.x;
          sub[u][8] += wt.x * z.x;
          sub[u][9] += wt.y * z.y;
          sub[u][10] += wt.x * z.y;
          sub[u][11] += wt.y * z.x;
        }
      }
      if ((at & 15) == 15 || at == na - 1) {
#pragma unroll
        for (int u = 0; u < SK_MG; ++u) {
          const double m = (double)(m0 + u);
          double q[NA];
#pragma unroll
          for (int k = 0; k < NA; ++k) {
            q[k] = (double)sub[u][k];
            sub[u][k] = (real)0;
          }
          acc[u][0] += q[0] - q[1];
          acc[u][1] += q[2] + q[3];
          acc[u][2] += q[0] + q[1];
          acc[u][3] += q[3] - q[2];
          if (VJP) {
            acc[u][4] += (q[4] - q[5]) + m * (q[8] - q[9]);
            acc[u][5] += (q[6] + q[7]) + m * (q[10] + q[11]);
            acc[u][6] += (q[4] + q[5]) - m * (q[8] + q[9]);
            acc[u][7] += (q[7] - q[6]) - m * (q[11] - q[10]);
          }
        }
      }
    }
  }
  if (!live) return;
#pragma unroll
  for (int u = 0; u < SK_MG; ++u) {
    if (m0 + u >= p.M) break;
#pragma unroll
    for (int v = 0; v < NV; ++v)
      part[(((size_t)blockIdx.y * NV + v) * p.M + m0 + u) * p.ncol + col] = make_double2(acc[u][2 * v], acc[u][2 * v + 1]);
  }
}

// Chunk sums -> force coefficients of every (column, m), weights kw =
// C f_k (C = 4 pi k_e / V) times the number of k and -k in the set, for +m
// and -m: with A+- = kw conj(S+-) = (a, b), (c, d) the four values a + c, d - b,
// b + d, a - c and, for the VJP, the same of B+- = kw T+-: a + c, b - d, b + d,
// c - a (see k_adj_kforce).  Energy form: {E_k, dE_k/dq}, VJP: {u . dF_k/dq},
// times scale, added to this block's partial.
template <typename real, bool VJP>
__global__ void __launch_bounds__(KRED_E *KRED_G) k_adj_kreduce(Params p, const double2 *__restrict__ part, int nch0,
                                                                int nch, const double2 *__restrict__ kw,
                                                                real *__restrict__ kc, double scale,
                                                                double *__restrict__ kpart) {
  constexpr int NV = VJP ? 4 : 2, NQ = VJP ? NT : 1 + NT;
  __shared__ double2 sums[KRED_G][NT * NV][KRED_E];
  __shared__ double red[NQ][KRED_E];
  const int E = p.M * p.ncol, e = blockIdx.x * KRED_E + threadIdx.x, g = threadIdx.y;
  double2 s[NT][NV];
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int v = 0; v < NV; ++v) s[t][v] = make_double2(0.0, 0.0);
  if (e < E) {
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int c1 = t ? nch : nch0;
#pragma unroll 2
      for (int c = (t ? nch0 : 0) + g; c < c1; c += KRED_G)
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const double2 x = part[((size_t)c * NV + v) * E + e];
          s[t][v].x += x.x;
          s[t][v].y += x.y;
        }
    }
  }
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int v = 0; v < NV; ++v) sums[g][t * NV + v][threadIdx.x] = s[t][v];
  __syncthreads();
  // one thread per (entry, quantity) adds the groups in order
  const int tid = g * KRED_E + threadIdx.x;
  if (tid < NT * NV * KRED_E) {
    const int v = tid / KRED_E, x = tid % KRED_E;
    double2 r = sums[0][v][x];
#pragma unroll
    for (int q = 1; q < KRED_G; ++q) {
      r.x += sums[q][v][x].x;
      r.y += sums[q][v][x].y;
    }
    sums[0][v][x] = r;
  }
  __syncthreads();
  if (g != 0) return;
  double v[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) v[q] = 0.0;
  if (e < E) {
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int q = 0; q < NV; ++q) s[t][q] = sums[0][t * NV + q][threadIdx.x];
    const double2 w2 = kw[e];
    const double w[2] = {w2.x, w2.y};
    double ab[2][2], tb[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // +m, -m
      const double Sx = p.charge[0] * s[0][h].x + p.charge[1] * s[1][h].x;
      const double Sy = p.charge[0] * s[0][h].y + p.charge[1] * s[1][h].y;
      ab[h][0] = w[h] * Sx;
      ab[h][1] = -w[h] * Sy;
      if (!VJP) {
        v[0] += 0.5 * w[h] * (Sx * Sx + Sy * Sy);
#pragma unroll
        for (int t = 0; t < NT; ++t) v[1 + t] += w[h] * (s[t][h].x * Sx + s[t][h].y * Sy);  // Re(S_t conj S)
      } else {
        const double Tx = p.charge[0] * s[0][2 + h].x + p.charge[1] * s[1][2 + h].x;
        const double Ty = p.charge[0] * s[0][2 + h].y + p.charge[1] * s[1][2 + h].y;
        tb[h][0] = w[h] * Tx;
        tb[h][1] = w[h] * Ty;
#pragma unroll
        for (int t = 0; t < NT; ++t)  // Im(T_t conj S + T conj S_t)
          v[t] += w[h] * ((s[t][2 + h].y * Sx - s[t][2 + h].x * Sy) + (Ty * s[t][h].x - Tx * s[t][h].y));
      }
    }
    const int col = e % p.ncol, m = e / p.ncol;
    real *out = kc + ((size_t)col * p.M + m) * (VJP ? 8 : 4);
    out[0] = (real)(ab[0][0] + ab[1][0]);
    out[1] = (real)(ab[1][1] - ab[0][1]);
    out[2] = (real)(ab[0][1] + ab[1][1]);
    out[3] = (real)(ab[0][0] - ab[1][0]);
    if (VJP) {
      out[4] = (real)(tb[0][0] + tb[1][0]);
      out[5] = (real)(tb[0][1] - tb[1][1]);
      out[6] = (real)(tb[0][1] + tb[1][1]);
      out[7] = (real)(tb[1][0] - tb[0][0]);
    }
  }
  if (scale == 0.0) return;
#pragma unroll
  for (int q = 0; q < NQ; ++q) red[q][threadIdx.x] = v[q];
  __syncwarp((1u << KRED_E) - 1u);
  if (threadIdx.x < NQ) {
    double x = 0.0;
    for (int k = 0; k < KRED_E; ++k) x += red[threadIdx.x][k];
    kpart[(size_t)blockIdx.x * NQ + threadIdx.x] += scale * x;
  }
}

// FP32 (mixed) pair terms use the hardware reciprocal / reciprocal square
// root / exponential and erfc from Abramowitz & Stegun 7.1.26 sharing the
// Gaussian (erfc_as); FP64 takes the library's functions and erfc_ex.
__device__ __forceinline__ float adj_rcp(float x) { return __fdividef(1.f, x); }
__device__ __forceinline__ double adj_rcp(double x) { return 1.0 / x; }

// Coordinates in the pair kernel: the displacement r_j - r_i (minimum image)
// that the distance test takes (test) and the queues hold (Diff), and its
// three lengths at the evaluation (length).
//  FixedCoord  mixed form: the wrapping difference of 32-bit fixed-point
//              coordinates in units L / 2^32, exact, turned into a length
//              through FP64 with one rounding to FP32.
//  WideCoord   mixed form in boxes where L / 2^32 is too coarse
//              (FIXED_MAX_SIGMA): FP64 differences rounded once.
//  FullCoord   FP64: the differences themselves.
struct FixedCoord {
  static constexpr int MIN_BLOCKS = 4;
  struct Diff {
    int x, y, z, j;
  };
  uint32_t x, y, z;
  float bad;  // 0, or NaN where the position is not finite (a fixed-point coordinate cannot say so)
  __device__ __forceinline__ static FixedCoord load(const uint4 *xs, const double *, int, int j) {
    const uint4 v = xs[j];
    return {v.x, v.y, v.z, __uint_as_float(v.w)};
  }
  __device__ __forceinline__ Diff to(const FixedCoord &o, const Params &, int j) const {
    return {(int)(o.x - x), (int)(o.y - y), (int)(o.z - z), j};
  }
  __device__ __forceinline__ static float test(const Diff &d, const FixedCoord &o) {
    const float a = (float)d.x + o.bad, b = (float)d.y, c = (float)d.z;
    return a * a + b * b + c * c;
  }
  // j's sign bit: the pair's r^2 was NaN
  __device__ __forceinline__ static Diff marked(Diff d, float r2) {
    if (r2 != r2) d.j |= 1 << 31;
    return d;
  }
  template <typename PC> __device__ __forceinline__ static int length(const Diff &e, const PC &pc, float (&d)[3]) {
    d[0] = (float)((double)e.x * pc.unit);
    d[1] = (float)((double)e.y * pc.unit);
    d[2] = (float)((double)e.z * pc.unit);
    if (e.j < 0) d[0] = __int_as_float(0x7fffffff);
    return e.j & 0x7fffffff;
  }
};
template <typename real> struct RealDiff {
  real x, y, z;
  int j;
};
template <typename real> struct RealCoord {
  static constexpr int MIN_BLOCKS = sizeof(real) == 4 ? 3 : 2;  // 4 in the mixed form spill
  using Diff = RealDiff<real>;
  double x, y, z;
  static constexpr double bad = 0.0;  // the differences carry a NaN themselves
  __device__ __forceinline__ static RealCoord load(const uint4 *, const double *X, int n, int j) {
    return {X[j], X[n + j], X[2 * n + j]};
  }
  __device__ __forceinline__ Diff to(const RealCoord &o, const Params &p, int j) const {
    double d[3] = {o.x - x, o.y - y, o.z - z};
#pragma unroll
    for (int a = 0; a < 3; ++a) d[a] -= p.L * rint(d[a] * p.invL);
    return {(real)d[0], (real)d[1], (real)d[2], j};
  }
  __device__ __forceinline__ static real test(const Diff &d, const RealCoord &) {
    return d.x * d.x + d.y * d.y + d.z * d.z;
  }
  __device__ __forceinline__ static Diff marked(const Diff &d, real) { return d; }
  template <typename PC> __device__ __forceinline__ static int length(const Diff &e, const PC &, real (&d)[3]) {
    d[0] = e.x;
    d[1] = e.y;
    d[2] = e.z;
    return e.j;
  }
};
using WideCoord = RealCoord<float>;
using FullCoord = RealCoord<double>;
// Fixed-point coordinates in boxes of at most this many of the smallest LJ
// diameter: FP32 rounds a contact distance to 1.7e-8 of it (r.m.s.), the two
// coordinates' quanta add 9.5e-11 L / sigma, 1.6 % of that error at 32.
constexpr double FIXED_MAX_SIGMA = 32.0;

__device__ __forceinline__ void load_u(const float4 *us, const double *, int, int j, float (&u)[3]) {
  const float4 v = us[j];
  u[0] = v.x;
  u[1] = v.y;
  u[2] = v.z;
}
__device__ __forceinline__ void load_u(const float4 *, const double *U, int n, int j, double (&u)[3]) {
  u[0] = U[j];
  u[1] = U[n + j];
  u[2] = U[2 * n + j];
}

// One pair's contribution: c (F_i += c d); VJP: c (u_j - u_i) + c1 (d . (u_j - u_i)) d,
// c1 = (1/r) dc/dr.  Returns the parameter derivative's factor u_i . d (VJP).
template <typename real, bool VJP>
__device__ __forceinline__ real apply(real c, real c1, const real (&d)[3], const real (&ui)[3], const float4 *us,
                                      const double *U, int n, int j, real (&acc)[3]) {
  if (!VJP) {
#pragma unroll
    for (int a = 0; a < 3; ++a) acc[a] += c * d[a];
    return (real)0;
  }
  real uj[3];
  load_u(us, U, n, j, uj);
  const real du[3] = {uj[0] - ui[0], uj[1] - ui[1], uj[2] - ui[2]};
  const real w = c1 * (d[0] * du[0] + d[1] * du[1] + d[2] * du[2]);
#pragma unroll
  for (int a = 0; a < 3; ++a) acc[a] += c * du[a] + w * d[a];
  return ui[0] * d[0] + ui[1] * d[1] + ui[2] * d[2];
}

// Pair part of the forces (energy form: with sum Ue, Us, Uq per ordered type
// pair) or of the VJP (with sum dce ud, dcs ud, cq ud, ud = u_i . d): one atom
// per JS warps, lanes over partners.  All partners take the distance test
// (about 15 instructions); the pairs inside a cutoff (45 % of them at a
// real-space cutoff of L/2.1, 1.4 % for LJ) are queued per warp by ballot and
// evaluated 32 at a time, so the long terms run with full warps.  Partners of
// one species at a time: the type pair is uniform and its constants and sums
// are fixed registers.  Two partners per lane and round keep two loads in
// flight and halve the loop's own cost (68 -> 52 us for the energy form at
// 4000 atoms, rc 8, before the exact displacements, which took it to 58).
// Issue bound, mixed (77 % of the slots, 41 % of the warps); FP64 54 % at 22 %
// of the warps, its pipe 37 %.  4000 atoms, rc 8, mixed, with every lane
// evaluating its own partner under divergence and FP64 differences: 216 us
// energy form with k space, 270 VJP; now 58 and 69 (+ 11 and 15 for the
// k-space kernel).
template <typename real, typename Coord, bool VJP>
__global__ void __launch_bounds__(PAIR_WARPS * 32, Coord::MIN_BLOCKS)
    k_adj_pair(Params p, PairC<real> pc, const double *__restrict__ X, const double *__restrict__ U,
               const uint4 *__restrict__ xs, const float4 *__restrict__ us, int JS, double scale, double *__restrict__ out,
               double *__restrict__ part) {
  constexpr int PR = PAIR_ROUND<real>;
  using Diff = typename Coord::Diff;
  __shared__ Diff queue[PAIR_WARPS][2][QCAP<real>];
  __shared__ double red[PAIR_WARPS][2][3];  // per warp, partner type
  __shared__ real facc[PAIR_WARPS][3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per_block = PAIR_WARPS / JS;
  const int i = blockIdx.x * per_block + warp / JS, js = warp % JS;
  const bool live = i < p.n;
  const int ti = i >= p.n0;
  const bool param = scale != 0.0;
  const unsigned lt = (1u << lane) - 1u;
  Diff *qe = queue[warp][0], *ql = queue[warp][1];
  real acc[3] = {0, 0, 0}, ui[3] = {0, 0, 0};
  double sum[2][3] = {{0, 0, 0}, {0, 0, 0}};
  if (live) {
    const Coord ci = Coord::load(xs, X, p.n, i);
    if (VJP) load_u(us, U, p.n, i, ui);
    acc[0] = ci.bad;
#pragma unroll
    for (int tj = 0; tj < NT; ++tj) {
      const LjC<real> lj = pc.lj[ti * NT + tj];
      const real qq = (real)((ti ? p.charge[1] : p.charge[0]) * p.charge[tj]);
      const int j0 = tj ? p.n0 : 0, j1 = tj ? p.n : p.n0;
      const auto ewald = [&](int k) {
        real d[3];
        const int j = Coord::length(qe[k], pc, d);
        const real r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        real r, ri, G, ec;
        if constexpr (sizeof(real) == 4) {
          ri = rsqrtf(r2);
          r = r2 * ri;
          G = __expf(-pc.alpha2 * r2);
          ec = cvr::erfc_as(pc.alpha * r, G);
        } else {
          r = sqrt(r2);
          ri = (real)1 / r;
          G = exp(-pc.alpha2 * r2);
          ec = cvr::erfc_ex(pc.alpha * r, G);
        }
        const real E1 = -pc.beta * G * ri - ec * ri * ri, cq = pc.ke * E1 * ri;
        real c1 = (real)0;
        if (VJP) {
          const real E2 = pc.beta * G * ((real)2 * pc.alpha2 + (real)2 * ri * ri) + (real)2 * ec * ri * ri * ri;
          c1 = qq * pc.ke * (E2 - E1 * ri) * ri * ri;
        }
        const real ud = apply<real, VJP>(qq * cq, c1, d, ui, us, U, p.n, j, acc);
        if (param) sum[tj][2] += (double)(VJP ? cq * ud : pc.ke * ec * ri);
      };
      const auto lennard_jones = [&](int k) {
        real d[3];
        const int j = Coord::length(ql[k], pc, d);
        const real r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        const real r2i = adj_rcp(r2), s2 = lj.sg2 * r2i, s6 = s2 * s2 * s2, s12 = s6 * s6;
        const real ce = (real)4 * (((real)6 * s6 - (real)12 * s12) * r2i + lj.shift);
        const real c1 = VJP ? lj.e * (real)4 * ((real)168 * s12 - (real)48 * s6) * r2i * r2i : (real)0;
        const real ud = apply<real, VJP>(lj.e * ce, c1, d, ui, us, U, p.n, j, acc);
        if (param) {
          if (VJP) {
            const real cs = (real)4 * (((real)36 * s6 - (real)144 * s12) * r2i + lj.shiftS);
            sum[tj][0] += (double)(ce * ud);
            sum[tj][1] += (double)(cs * ud);
          } else {
            sum[tj][0] += (double)((real)4 * (s12 - s6) + (lj.U0 + lj.U1 * (r2 - pc.rc2)));
            sum[tj][1] += (double)((real)4 * ((real)12 * s12 - (real)6 * s6) + (lj.S0 + lj.S1 * (r2 - pc.rc2)));
          }
        }
      };
      int ne = 0, nl = 0;
      for (int b = j0 + 32 * PR * js; b < j1; b += 32 * PR * JS) {
        Coord cj[PR];
#pragma unroll
        for (int q = 0; q < PR; ++q) cj[q] = Coord::load(xs, X, p.n, min(b + 32 * q + lane, p.n - 1));
#pragma unroll
        for (int q = 0; q < PR; ++q) {
          const int j = b + 32 * q + lane;
          const bool ok = j < j1 && j != i;
          const Diff d = ci.to(cj[q], p, j);
          const real r2 = Coord::test(d, cj[q]);
          // a NaN (a position that is not finite) counts as inside, and so reaches the force
          const bool ie = ok && !(r2 > pc.rr2), il = ok && lj.on && r2 <= pc.rl2;
          const unsigned me = __ballot_sync(0xffffffffu, ie);
          if (ie) qe[ne + __popc(me & lt)] = Coord::marked(d, r2);
          ne += __popc(me);
          const unsigned ml = __ballot_sync(0xffffffffu, il);
          if (ml) {
            if (il) ql[nl + __popc(ml & lt)] = d;
            nl += __popc(ml);
          }
        }
        __syncwarp();
        while (ne >= 32) {
          ne -= 32;
          ewald(ne + lane);
        }
        while (nl >= 32) {
          nl -= 32;
          lennard_jones(nl + lane);
        }
        __syncwarp();
      }
      if (lane < ne) ewald(lane);
      if (lane < nl) lennard_jones(lane);
      __syncwarp();
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[a] += __shfl_xor_sync(0xffffffffu, acc[a], o);
    }
    if (param) {
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) sum[t][q] += __shfl_xor_sync(0xffffffffu, sum[t][q], o);
        }
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) facc[warp][a] = acc[a];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int q = 0; q < 3; ++q) red[warp][t][q] = sum[t][q];
  }
  __syncthreads();
  if (threadIdx.x < 3 * per_block) {
    const int at = threadIdx.x / 3, ax = threadIdx.x % 3, ia = blockIdx.x * per_block + at;
    if (ia < p.n) {
      real f = facc[at * JS][ax];
      for (int w = 1; w < JS; ++w) f += facc[at * JS + w][ax];
      out[(size_t)ax * p.n + ia] = (double)f;
    }
  }
  if (param && threadIdx.x >= 32 && threadIdx.x < 32 + NPV) {
    const int v = threadIdx.x - 32, tp = v / 3, q = v % 3;
    double x = 0.0;
    for (int w = 0; w < PAIR_WARPS; ++w) {
      const int iw = blockIdx.x * per_block + w / JS;
      if ((iw >= p.n0) == (tp / NT != 0)) x += red[w][tp % NT][q];  // warps past the last atom hold zeros
    }
    part[(size_t)blockIdx.x * NPV + v] += scale * x;
  }
}

// What k_adj_kforce does with the finished force or VJP f of an atom:
//   POST_STORE  out = f
//   POST_KICK   out = f; V += dt/2 (Fold + f)/m (md_simulator.cpp:616)
//   POST_REV    Gr += f; (Gv, Ga) <- (Gv + dt Gr, dt/2 Gv + dt^2/2 Gr)
//   POST_REV0   Gr += f
enum : int { POST_STORE = 0, POST_KICK = 1, POST_REV = 2, POST_REV0 = 3 };
struct PostArgs {
  int op;
  double *out;
  const double *Fold;
  double *V, *Gr, *Gv, *Ga;
};

// k-space part per atom (one lane per atom, the columns over KF_WARPS warps)
// plus the pair part fp, then the state update.  Per column, W = X Y:
//   C = sum_m A+ z + A- z*, D = sum_m m (A+ z - A- z*):
//   F_xy = q kf n_xy Im(W C), F_z = q kf Im(W D)
// and for the VJP, with s = kf (nx ux + ny uy), t = kf uz, G = sum_m m^2 (A+ z + A- z*),
// Cb = sum_m B+ z* + B- z, Db = sum_m m (B+ z* - B- z):
//   w_xy = q kf n_xy (s Re(W C) + t Re(W D) - Re(W* Cb)), w_z = q kf (s Re(W D) + t Re(W G) - Re(W* Db)).
// The warps' sums are added in warp order.  Latency bound: the atoms' phases and
// a column's coefficients come from shared memory, the latter fetched one
// column ahead (VJP at 4000 atoms, k_max 7: 20 us from global memory, 13.8).
template <typename real, bool VJP>
__global__ void __launch_bounds__(KF_WARPS * 32)
    k_adj_kforce(Params p, const typename R2<real>::t *__restrict__ tab, const real *__restrict__ kc,
                 const double *__restrict__ U, const double *__restrict__ fp, PostArgs post) {
  using T2 = typename R2<real>::t;
  constexpr int NC = VJP ? 8 : 4;
  __shared__ T2 ts[3 * (KMAX_ADJ + 1)][32];  // the atoms' phases, rows axis * kp + m
  constexpr int CMAX = (KMAX_ADJ + 1) * NC, CPL = (CMAX + 31) / 32;  // a column's coefficients, per lane
  __shared__ __align__(16) real cs[KF_WARPS][CMAX];
  __shared__ real fs[KF_WARPS][3][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane, ia = min(i, p.n - 1);
  real f[3] = {0, 0, 0};
  if (p.ncol > 0) {
    for (int r = warp; r < 3 * p.kp; r += KF_WARPS) ts[r][lane] = tab[(size_t)r * p.n + ia];
    real ux = 0, uy = 0, t = 0;
    if (VJP) {
      ux = (real)(p.kf * U[ia]);
      uy = (real)(p.kf * U[p.n + ia]);
      t = (real)(p.kf * U[2 * (size_t)p.n + ia]);
    }
    __syncthreads();
    // a column's coefficients are fetched by the whole warp one column ahead
    const int nc = p.M * NC;
    real next[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c)
      next[c] = (warp < p.ncol && 32 * c + lane < nc) ? kc[(size_t)warp * nc + 32 * c + lane] : (real)0;
    for (int col = warp; col < p.ncol; col += KF_WARPS) {
      __syncwarp();
#pragma unroll
      for (int c = 0; c < CPL; ++c)
        if (32 * c + lane < nc) cs[warp][32 * c + lane] = next[c];
      __syncwarp();
      const int ahead = col + KF_WARPS;
#pragma unroll
      for (int c = 0; c < CPL; ++c)
        next[c] = (ahead < p.ncol && 32 * c + lane < nc) ? kc[(size_t)ahead * nc + 32 * c + lane] : (real)0;
      const int nx = col / (2 * p.kmax + 1) - p.kmax, ny = col % (2 * p.kmax + 1) - p.kmax;
      const T2 w = cmul(conj_if(ts[abs(nx)][lane], nx < 0), conj_if(ts[p.kp + abs(ny)][lane], ny < 0));
      const real *q = cs[warp];
      real Cr = 0, Ci = 0, Dr = 0, Di = 0, Gr = 0, Gi = 0, Br = 0, Bi = 0, Er = 0, Ei = 0;
#pragma unroll 4
      for (int m = 0; m < p.M; ++m, q += NC) {
        const T2 z = ts[2 * p.kp + m][lane];
        const real fm = (real)m;
        const real cr = q[0] * z.x + q[1] * z.y, ci = q[2] * z.x + q[3] * z.y;
        const real dr = fm * (q[3] * z.x - q[2] * z.y), di = fm * (q[0] * z.y - q[1] * z.x);
        Cr += cr;
        Ci += ci;
        Dr += dr;
        Di += di;
        if (VJP) {
          Gr += fm * fm * cr;
          Gi += fm * fm * ci;
          Br += q[4] * z.x + q[5] * z.y;
          Bi += q[6] * z.x + q[7] * z.y;
          Er += fm * (q[6] * z.y - q[7] * z.x);
          Ei += fm * (q[5] * z.x - q[4] * z.y);
        }
      }
      real xy, zz;
      if (VJP) {
        const real s = (real)nx * ux + (real)ny * uy;
        const real rd = w.x * Dr - w.y * Di;
        xy = s * (w.x * Cr - w.y * Ci) + t * rd - (w.x * Br + w.y * Bi);
        zz = s * rd + t * (w.x * Gr - w.y * Gi) - (w.x * Er + w.y * Ei);
      } else {
        xy = w.x * Ci + w.y * Cr;
        zz = w.x * Di + w.y * Dr;
      }
      f[0] += (real)nx * xy;
      f[1] += (real)ny * xy;
      f[2] += zz;
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) fs[warp][a][lane] = f[a];
  __syncthreads();
  if (warp >= 3 || i >= p.n) return;
  real k = fs[0][warp][lane];
#pragma unroll
  for (int w = 1; w < KF_WARPS; ++w) k += fs[w][warp][lane];
  const size_t t = (size_t)warp * p.n + i;
  const double total = fp[t] + (i >= p.n0 ? p.charge[1] : p.charge[0]) * p.kf * (double)k;
  const double mi = i >= p.n0 ? p.mass_inv[1] : p.mass_inv[0];
  if (post.op <= POST_KICK) {
    post.out[t] = total;
    if (post.op == POST_KICK) post.V[t] += 0.5 * p.dt * (post.Fold[t] + total) * mi;
  } else {
    const double gr = post.Gr[t] + total;
    post.Gr[t] = gr;
    if (post.op == POST_REV) {
      const double gv = post.Gv[t];
      post.Gv[t] = gv + p.dt * gr;
      post.Ga[t] = 0.5 * p.dt * gv + 0.5 * p.dt * p.dt * gr;
    }
  }
}

// The four partial arrays (nparts x nv values each), one block per value.
constexpr int ACC_THREADS = 128;
struct AccumArgs {
  const double *part[4];
  int nparts[4], nv[4];
  double *dst;
};
__global__ void __launch_bounds__(ACC_THREADS) k_adj_accum(AccumArgs a) {
  __shared__ double red[ACC_THREADS / 32];
  int v = blockIdx.x, g = 0;
  while (v >= a.nv[g]) v -= a.nv[g++];
  double s = 0;
#pragma unroll 4
  for (int q = threadIdx.x; q < a.nparts[g]; q += ACC_THREADS) s += a.part[g][(size_t)q * a.nv[g] + v];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < ACC_THREADS / 32; ++w) s += red[w];
  a.dst[blockIdx.x] = s;
}

}  // namespace

struct cvr_adj {
  int device = 0, precision = CVR_PREC_MIXED;
  cudaStream_t stream = nullptr, kstream = nullptr;  // kstream: the S(k) chain beside the pair kernel
  cudaEvent_t fork = nullptr, join = nullptr;
  Params p{};
  bool params_set = false, state_set = false;
  std::vector<int> type_h;
  std::vector<double> mass_h, charge_h, eps_h, sig_h;
  int n_types = 0;
  std::vector<int> id_of;               // stored slot -> caller's atom index
  // device; every per-atom array SoA [3][n] in stored order, all inside mem; the k-space arrays inside kmem
  double *mem = nullptr, *kmem = nullptr;
  double *x0 = nullptr, *v0 = nullptr;  // the state the loss starts from
  double *X = nullptr, *Xb = nullptr, *V = nullptr, *F = nullptr, *Fb = nullptr;
  double *Gr = nullptr, *Gv = nullptr, *Ga = nullptr, *W = nullptr, *u = nullptr, *fp = nullptr;
  uint4 *xs = nullptr;                  // mixed form: fixed-point coordinates
  float4 *us = nullptr;                 // mixed form: cotangent
  void *tab = nullptr, *kc = nullptr;
  double2 *kw = nullptr;                // per (m, column): weights C f_k of +m and -m
  double2 *skpart = nullptr;
  double *parts = nullptr, *accum = nullptr;
  double *ck = nullptr, *seg = nullptr;  // checkpoints, segment positions + forces
  size_t ck_cap = 0, seg_cap = 0;
  int nch0 = 0, nch = 0, chunk = SK_STAGE;  // S(k) chunks: of type 0, of both; atoms per chunk
  int jsplit = 1;                           // warps per atom of k_adj_pair
  bool fixed = false;                       // mixed form: fixed-point pair displacements
  PairC<float> pcf{};
  PairC<double> pcd{};
  std::string err;
};

namespace {

int afail(cvr_adj *a, int code, const std::string &m) {
  if (a) a->err = m;
  return code;
}

int cuda_ok(cvr_adj *a, const char *what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return afail(a, CVR_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return CVR_OK;
}

template <typename T>
int dalloc(cvr_adj *a, T **ptr, size_t count) {
  if (*ptr) cudaFree(*ptr);
  *ptr = nullptr;
  if (cudaMalloc((void **)ptr, std::max<size_t>(count, 1) * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();  // not the next launch's
    *ptr = nullptr;
    return afail(a, CVR_ERR_NOMEM, "cudaMalloc");
  }
  return CVR_OK;
}

// At least count doubles in *ptr (an allocation that fails leaves none).
int reserve(cvr_adj *a, double **ptr, size_t *cap, size_t count) {
  if (count <= *cap) return CVR_OK;
  *cap = 0;
  if (int rc = dalloc(a, ptr, count)) return rc;
  *cap = count;
  return CVR_OK;
}

inline int blocks(int n, int t) { return (n + t - 1) / t; }

inline size_t real_bytes(const cvr_adj *a) { return a->precision == CVR_PREC_FP64 ? 8 : 4; }
inline int pair_blocks(const cvr_adj *a) { return blocks(a->p.n, PAIR_WARPS / a->jsplit); }
inline int kred_blocks(const cvr_adj *a) { return blocks(a->p.ncol * a->p.M, KRED_E); }

// the per-block partial arrays inside parts, in accumulator order
struct PartPtr {
  double *pe, *pv, *ke, *kv;
  size_t total;
};
PartPtr part_ptr(const cvr_adj *a) {
  const size_t pb = (size_t)pair_blocks(a) * NPV, kb = kred_blocks(a);
  PartPtr q;
  q.pe = a->parts;
  q.pv = q.pe + pb;
  q.ke = q.pv + pb;
  q.kv = q.ke + kb * (1 + NT);
  q.total = 2 * pb + kb * (1 + 2 * NT);
  return q;
}

// One force evaluation (energy form) or VJP: state update, evaluation, state
// update.  scale weights the parameter sums added to the call's partials.
template <typename real, bool VJP>
int eval(cvr_adj *a, const PairC<real> &pc, const PrepArgs &prep, const double *X, const PostArgs &post, double scale) {
  using T2 = typename R2<real>::t;
  const Params &p = a->p;
  cudaStream_t st = a->stream;
  T2 *tab = static_cast<T2 *>(a->tab);
  real *kc = static_cast<real *>(a->kc);
  const PartPtr parts = part_ptr(a);
  k_adj_prep<real, VJP><<<dim3(blocks(3 * p.n, 256), blocks(p.kp, 4)), 256, 0, st>>>(
      p, prep, tab, reinterpret_cast<uint32_t *>(a->xs), reinterpret_cast<float *>(a->us));
  // the S(k) chain on the side stream (highest priority: it is short and the
  // k-space force waits for it) beside the pair kernel
  if (p.ncol > 0) {
    cudaEventRecord(a->fork, st);
    cudaStreamWaitEvent(a->kstream, a->fork, 0);
    const size_t smem = (size_t)SK_STAGE * (3 * p.kp * sizeof(T2) + 3 * sizeof(real));
    dim3 g(blocks(p.ncol * blocks(p.M, SK_MG), SK_THREADS), a->nch);
    k_adj_sk<real, VJP><<<g, SK_THREADS, smem, a->kstream>>>(p, tab, a->u, a->chunk, a->nch0, a->skpart);
    k_adj_kreduce<real, VJP><<<kred_blocks(a), dim3(KRED_E, KRED_G), 0, a->kstream>>>(
        p, a->skpart, a->nch0, a->nch, a->kw, kc, scale, VJP ? parts.kv : parts.ke);
    cudaEventRecord(a->join, a->kstream);
  }
  const auto pair = [&](auto kernel) {
    kernel<<<pair_blocks(a), PAIR_WARPS * 32, 0, st>>>(p, pc, X, a->u, a->xs, a->us, a->jsplit, scale, a->fp,
                                                       VJP ? parts.pv : parts.pe);
  };
  if constexpr (sizeof(real) == 8)
    pair(k_adj_pair<real, FullCoord, VJP>);
  else if (a->fixed)
    pair(k_adj_pair<real, FixedCoord, VJP>);
  else
    pair(k_adj_pair<real, WideCoord, VJP>);
  if (p.ncol > 0) cudaStreamWaitEvent(st, a->join, 0);
  k_adj_kforce<real, VJP><<<blocks(p.n, 32), KF_WARPS * 32, 0, st>>>(p, tab, kc, a->u, a->fp, post);
  return cuda_ok(a, "adjoint evaluation launch");
}

template <bool VJP>
int evalp(cvr_adj *a, const PrepArgs &prep, const double *X, const PostArgs &post, double scale) {
  return a->precision == CVR_PREC_FP64 ? eval<double, VJP>(a, a->pcd, prep, X, post, scale)
                                       : eval<float, VJP>(a, a->pcf, prep, X, post, scale);
}

// forces at X into F
int eval_forces(cvr_adj *a, const double *X, double *F, double scale) {
  PrepArgs pre{};
  pre.X = X;
  PostArgs post{};
  post.out = F;
  return evalp<false>(a, pre, X, post, scale);
}

// the call's partials: cleared at its start, summed into host acc[A_N] at its end
int clear_parts(cvr_adj *a) {
  if (cudaMemsetAsync(a->parts, 0, part_ptr(a).total * sizeof(double), a->stream) != cudaSuccess)
    return afail(a, CVR_ERR_CUDA, "memset");
  return CVR_OK;
}
void sum_parts(cvr_adj *a, double *acc) {
  const PartPtr q = part_ptr(a);
  const int pb = pair_blocks(a), kb = kred_blocks(a);
  AccumArgs g{{q.pe, q.pv, q.ke, q.kv}, {pb, pb, kb, kb}, {NPV, NPV, 1 + NT, NT}, a->accum};
  k_adj_accum<<<A_N, ACC_THREADS, 0, a->stream>>>(g);
  cudaMemcpyAsync(acc, a->accum, A_N * sizeof(double), cudaMemcpyDeviceToHost, a->stream);
}

template <typename real>
void set_pair_consts(const cvr_adj *a, double rc_lj, double rc_r, PairC<real> &c) {
  const Params &p = a->p;
  const double unit = sizeof(real) == 4 && a->fixed ? p.L / 4294967296.0 : 1.0;
  c.unit = unit;
  c.rl2 = (real)(rc_lj * rc_lj / (unit * unit));
  c.rr2 = (real)(p.k_e != 0.0 ? rc_r * rc_r / (unit * unit) : -1.0);
  c.alpha = (real)p.alpha;
  c.alpha2 = (real)(p.alpha * p.alpha);
  c.beta = (real)(2.0 * p.alpha * 0.56418958354775628695);
  c.ke = (real)p.k_e;
  const double rc2 = rc_lj * rc_lj;
  c.rc2 = (real)rc2;
  for (int x = 0; x < NT; ++x)
    for (int y = 0; y < NT; ++y) {
      LjC<real> &l = c.lj[x * NT + y];
      const bool in = x < a->n_types && y < a->n_types;
      const double e = in ? a->eps_h[x * a->n_types + y] : 0.0, sg = in ? a->sig_h[x * a->n_types + y] : 1.0;
      const double s2 = sg * sg, c2 = s2 / rc2, c6 = c2 * c2 * c2, c12 = c6 * c6;
      l.sg2 = (real)s2;
      l.e = (real)e;
      l.on = e != 0.0;
      l.shift = (real)((12 * c12 - 6 * c6) / rc2);
      l.shiftS = (real)((144 * c12 - 36 * c6) / rc2);
      const double u1 = 4 * (12 * c12 - 6 * c6) / (2 * rc2), s1 = 4 * (144 * c12 - 36 * c6) / (2 * rc2);
      l.U1 = (real)u1;
      l.U0 = (real)(-4 * (c12 - c6));
      l.S1 = (real)s1;
      l.S0 = (real)(-4 * (12 * c12 - 6 * c6));
    }
}

int ready(cvr_adj *a) {
  if (!a) return CVR_ERR_INVALID;
  if (!a->params_set) return afail(a, CVR_ERR_STATE, "cvr_adj_set_params has not been called");
  if (!a->state_set) return afail(a, CVR_ERR_STATE, "cvr_adj_set_state has not been called");
  cudaSetDevice(a->device);
  return CVR_OK;
}

// host-side terms: self energy -(alpha/sqrt(pi)) k_e sum q^2 and its q-gradient
double self_energy(const cvr_adj *a, double *dq) {
  double e = 0;
  for (int t = 0; t < NT; ++t) dq[t] = 0;
  if (a->p.ncol == 0) return 0;
  for (int i = 0; i < a->p.n; ++i) {
    const double q = a->charge_h[a->type_h[i]];
    e += q * q;
    dq[a->type_h[i]] += 2 * q;
  }
  const double c = -0.56418958354775628695 * a->p.alpha * a->p.k_e;
  for (int t = 0; t < NT; ++t) dq[t] *= c;
  return c * e;
}

// The call's sums -> energies {lj, ewald_r, ewald_k} and gradients of the
// shared symmetric parameters: energy form (forward) plus VJP (reverse).
void energies(const cvr_adj *a, const double *acc, double *e) {
  const Params &p = a->p;
  e[0] = e[1] = 0.0;
  for (int x = 0; x < NT; ++x)
    for (int y = 0; y < NT; ++y) {
      const double *s = acc + A_PE + 3 * (x * NT + y);
      const bool in = x < a->n_types && y < a->n_types;
      e[0] += 0.5 * (in ? a->eps_h[x * a->n_types + y] : 0.0) * s[0];
      e[1] += 0.5 * p.charge[x] * p.charge[y] * s[2];
    }
  e[2] = acc[A_KE];
}

void fold(const cvr_adj *a, const double *acc, bool energy, bool vjp, const double *extra_q, double *g) {
  const Params &p = a->p;
  const int nt = a->n_types;
  double re[NTT] = {}, rs[NTT] = {}, rq[NT] = {};
  for (int x = 0; x < nt; ++x)
    for (int y = 0; y < nt; ++y) {
      const int t = x * NT + y;
      const double es = a->eps_h[x * nt + y] / a->sig_h[x * nt + y];
      const double *e = acc + A_PE + 3 * t, *v = acc + A_PV + 3 * t;
      if (energy) {
        re[t] += 0.5 * e[0];
        rs[t] += 0.5 * es * e[1];
        rq[x] += 0.5 * p.charge[y] * e[2];
        rq[y] += 0.5 * p.charge[x] * e[2];
      }
      if (vjp) {
        re[t] += v[0];
        rs[t] += es * v[1];
        rq[x] += p.charge[y] * v[2];
        rq[y] += p.charge[x] * v[2];
      }
    }
  for (int t = 0; t < nt; ++t) {
    if (energy) rq[t] += acc[A_KE + 1 + t];
    if (vjp) rq[t] += acc[A_KV + t];
  }
  for (int x = 0; x < nt; ++x)
    for (int y = 0; y < nt; ++y) {
      const int xy = x * NT + y, yx = y * NT + x;
      g[x * nt + y] = x == y ? re[xy] : re[xy] + re[yx];
      g[nt * nt + x * nt + y] = x == y ? rs[xy] : rs[xy] + rs[yx];
    }
  for (int t = 0; t < nt; ++t) g[2 * nt * nt + t] = rq[t] + (extra_q ? extra_q[t] : 0.0);
}

int download_soa(cvr_adj *a, const double *src, double *dst_aos) {
  const int n = a->p.n;
  std::vector<double> h(3 * (size_t)n);
  cudaMemcpyAsync(h.data(), src, 3 * (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, a->stream);
  if (cudaStreamSynchronize(a->stream) != cudaSuccess) return afail(a, CVR_ERR_CUDA, "download");
  for (int d = 0; d < 3; ++d)
    for (int s = 0; s < n; ++s) dst_aos[3 * (size_t)a->id_of[s] + d] = h[(size_t)d * n + s];
  return CVR_OK;
}

}  // namespace

extern "C" {

int cvr_adj_create(cvr_adj **out, int64_t n, double box_len, int n_types, const double *mass, int precision,
                   int device) {
  if (!out) return CVR_ERR_INVALID;
  *out = nullptr;
  if (n < 2 || n > (1 << 24) || !(box_len > 0) || n_types < 1 || n_types > NT || !mass) return CVR_ERR_INVALID;
  if (precision != CVR_PREC_MIXED && precision != CVR_PREC_FP64) return CVR_ERR_INVALID;
  for (int t = 0; t < n_types; ++t)
    if (!(mass[t] > 0)) return CVR_ERR_INVALID;
  if (cudaSetDevice(device) != cudaSuccess) return CVR_ERR_CUDA;
  cvr_adj *a = new cvr_adj();
  a->device = device;
  a->precision = precision;
  a->n_types = n_types;
  a->mass_h.assign(mass, mass + n_types);
  Params &p = a->p;
  p.n = (int)n;
  p.L = box_len;
  p.invL = 1.0 / box_len;
  p.kf = 6.28318530717958647692 / box_len;
  for (int t = 0; t < NT; ++t) p.mass_inv[t] = t < n_types ? 1.0 / mass[t] : 0.0;
  int prio_least = 0, prio_greatest = 0;
  cudaDeviceGetStreamPriorityRange(&prio_least, &prio_greatest);
  if (cudaStreamCreateWithFlags(&a->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaStreamCreateWithPriority(&a->kstream, cudaStreamNonBlocking, prio_greatest) != cudaSuccess ||
      cudaEventCreateWithFlags(&a->fork, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&a->join, cudaEventDisableTiming) != cudaSuccess) {
    cvr_adj_destroy(a);
    return CVR_ERR_CUDA;
  }
  // warps per atom: enough for 40 warps per SM on small systems; the FP64 form
  // takes 16, which fill its pipe, because a warp's last batch of each species
  // is partly empty
  const int want = (precision == CVR_PREC_FP64 ? 16 : 40) * 148;
  while (a->jsplit < PAIR_WARPS && n * a->jsplit < want) a->jsplit *= 2;
  // S(k) chunks of whole stages, at most SK_MAXCHUNKS of them (plus one: each type's last is its own)
  a->chunk = SK_STAGE * (int)((n + (int64_t)SK_STAGE * SK_MAXCHUNKS - 1) / ((int64_t)SK_STAGE * SK_MAXCHUNKS));
  const size_t N3 = 3 * (size_t)n;
  int rc = 0;
  // one allocation for every per-atom array and the accumulators
  double **arrays[] = {&a->x0, &a->v0, &a->X,  &a->Xb, &a->V, &a->F, &a->Fb,
                       &a->Gr, &a->Gv, &a->Ga, &a->W,  &a->u, &a->fp};
  const size_t pad3 = (N3 + 1) & ~(size_t)1;  // 16-byte alignment of every array
  const size_t n_arrays = sizeof(arrays) / sizeof(arrays[0]);
  if ((rc = dalloc(a, &a->mem, n_arrays * pad3 + 4 * (size_t)n + A_N))) {
    cvr_adj_destroy(a);
    return rc;
  }
  double *q = a->mem;
  for (double **w : arrays) {
    *w = q;
    q += pad3;
  }
  a->xs = reinterpret_cast<uint4 *>(q);
  a->us = reinterpret_cast<float4 *>(q + 2 * (size_t)n);
  a->accum = q + 4 * (size_t)n;
  *out = a;
  return CVR_OK;
}

void cvr_adj_destroy(cvr_adj *a) {
  if (!a) return;
  cudaSetDevice(a->device);
  if (a->stream) cudaStreamSynchronize(a->stream);
  if (a->kstream) cudaStreamSynchronize(a->kstream);
  void *ptrs[] = {a->mem, a->kmem, a->ck, a->seg};
  for (void *q : ptrs)
    if (q) cudaFree(q);
  if (a->fork) cudaEventDestroy(a->fork);
  if (a->join) cudaEventDestroy(a->join);
  if (a->kstream) cudaStreamDestroy(a->kstream);
  if (a->stream) cudaStreamDestroy(a->stream);
  delete a;
}

int cvr_adj_set_params(cvr_adj *a, const double *charge, const double *eps, const double *sigma, double rc_lj,
                       double alpha, double rc_r, int kmax, double k_e, double dt) {
  if (!a || !charge || !eps || !sigma) return CVR_ERR_INVALID;
  if (kmax < 0 || kmax > KMAX_ADJ) return afail(a, CVR_ERR_INVALID, "k_max must be in [0, 10]");
  if (!(alpha > 0) || !(dt >= 0) || !(rc_lj > 0) || !(rc_r >= 0))
    return afail(a, CVR_ERR_INVALID, "alpha > 0, rc_lj > 0, rc_r >= 0, dt >= 0");
  Params &p = a->p;
  if (rc_lj > 0.5 * p.L * (1 + 1e-12) || rc_r > 0.5 * p.L * (1 + 1e-12))
    return afail(a, CVR_ERR_GEOMETRY, "cutoffs must be at most half the box (minimum image)");
  const int nt = a->n_types;
  for (int x = 0; x < nt; ++x)
    for (int y = 0; y < nt; ++y)
      if (eps[x * nt + y] != eps[y * nt + x] || sigma[x * nt + y] != sigma[y * nt + x] || !(sigma[x * nt + y] > 0))
        return afail(a, CVR_ERR_INVALID, "eps and sigma must be symmetric, sigma > 0");
  cudaSetDevice(a->device);
  a->charge_h.assign(charge, charge + nt);
  a->eps_h.assign(eps, eps + nt * nt);
  a->sig_h.assign(sigma, sigma + nt * nt);
  for (int t = 0; t < NT; ++t) p.charge[t] = t < nt ? charge[t] : 0.0;
  p.alpha = alpha;
  p.k_e = k_e;
  p.dt = dt;
  a->fixed = a->precision == CVR_PREC_MIXED && p.L <= FIXED_MAX_SIGMA * *std::min_element(sigma, sigma + nt * nt);
  set_pair_consts(a, rc_lj, rc_r, a->pcf);
  set_pair_consts(a, rc_lj, rc_r, a->pcd);
  const bool kchanged = !a->params_set || kmax != p.kmax;
  a->params_set = false;  // until everything below is done
  p.kmax = kmax;
  p.kp = kmax + 1;
  p.M = kmax + 1;
  // the reference's k-set (initialize.cpp:184-222): the first (2k)^3 of the
  // nesting, 0 skipped.  Columns up to (0, 0) in that order are summed; a
  // vector's weight counts itself and its mirror -k (at the mirrored place of
  // the nesting), each if in the set.
  const int span = 2 * kmax + 1;
  const long long used = (long long)(2 * kmax) * (2 * kmax) * (2 * kmax), all = (long long)span * span * span,
                  zero = all / 2;
  p.ncol = used > 0 ? (span * span + 1) / 2 : 0;
  const auto in_set = [&](long long full) { return full != zero && (full < zero ? full : full - 1) < used; };
  std::vector<double2> kw((size_t)p.M * p.ncol);
  for (int m = 0; m < p.M; ++m)
    for (int col = 0; col < p.ncol; ++col) {
      const int nx = col / span - kmax, ny = col % span - kmax;
      const double two_pi_L = 6.28318530717958647692 * p.invL;
      const double ksq = two_pi_L * two_pi_L * (nx * nx + ny * ny + m * m);
      const double cf = ksq > 0 ? 12.56637061435917295384 * k_e / (p.L * p.L * p.L) * (std::exp(-ksq / (4 * alpha * alpha)) / ksq) : 0.0;
      const long long plus = (long long)col * span + kmax + m, minus = (long long)col * span + kmax - m;
      const bool mid = col == p.ncol - 1;  // (0, 0): +m and -m are each other's mirror
      const int wp = (int)in_set(plus) + (mid ? 0 : (int)in_set(all - 1 - plus));
      const int wm = m == 0 ? 0 : (int)in_set(minus) + (mid ? 0 : (int)in_set(all - 1 - minus));
      kw[(size_t)m * p.ncol + col] = make_double2(wp * cf, wm * cf);
    }
  if (kchanged) {
    const size_t rb = real_bytes(a), E = (size_t)p.M * p.ncol;
    // each type's last chunk may be partly filled: at most two more than n / chunk
    const size_t max_chunks = (size_t)(p.n / a->chunk) + 2;
    // doubles: weights, chunk partials, tables, coefficients, parameter partials (each of even length)
    const size_t tab_d = ((size_t)p.n * 3 * p.kp * 2 * rb + 15) / 16 * 2, kc_d = (E * 8 * rb + 15) / 16 * 2;
    if (int rc = dalloc(a, &a->kmem, 2 * E + max_chunks * 8 * E + tab_d + kc_d + part_ptr(a).total)) return rc;
    a->kw = reinterpret_cast<double2 *>(a->kmem);
    a->skpart = a->kw + E;
    double *q = a->kmem + 2 * E + max_chunks * 8 * E;
    a->tab = q;
    a->kc = q + tab_d;
    a->parts = q + tab_d + kc_d;
  }
  if (!kw.empty() &&
      cudaMemcpy(a->kw, kw.data(), kw.size() * sizeof(double2), cudaMemcpyHostToDevice) != cudaSuccess)
    return afail(a, CVR_ERR_CUDA, "k-space weights");
  a->params_set = true;
  return CVR_OK;
}

int cvr_adj_set_state(cvr_adj *a, const double *pos, const double *vel, const int32_t *type) {
  if (!a || !pos || !type) return CVR_ERR_INVALID;
  cudaSetDevice(a->device);
  const int n = a->p.n;
  for (int i = 0; i < n; ++i)
    if (type[i] < 0 || type[i] >= a->n_types) return afail(a, CVR_ERR_INVALID, "atom type out of range");
  a->type_h.assign(type, type + n);
  a->id_of.resize(n);
  int k = 0;
  for (int t = 0; t < NT; ++t) {
    for (int i = 0; i < n; ++i)
      if (type[i] == t) a->id_of[k++] = i;
    if (t == 0) a->p.n0 = k;
  }
  a->nch0 = blocks(a->p.n0, a->chunk);
  a->nch = a->nch0 + blocks(n - a->p.n0, a->chunk);
  std::vector<double> soa(6 * (size_t)n, 0.0);
  for (int d = 0; d < 3; ++d)
    for (int s = 0; s < n; ++s) {
      const size_t i = a->id_of[s];
      soa[(size_t)d * n + s] = pos[3 * i + d];
      soa[(size_t)(3 + d) * n + s] = vel ? vel[3 * i + d] : 0.0;
    }
  cudaMemcpyAsync(a->x0, soa.data(), 3 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice, a->stream);
  cudaMemcpyAsync(a->v0, soa.data() + 3 * (size_t)n, 3 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice,
                  a->stream);
  if (cudaStreamSynchronize(a->stream) != cudaSuccess) return afail(a, CVR_ERR_CUDA, "upload");
  a->state_set = true;
  return CVR_OK;
}

int cvr_adj_forces(cvr_adj *a, double *force, double *energy, double *dU) {
  if (int rc = ready(a)) return rc;
  if (int rc = clear_parts(a)) return rc;
  if (int rc = eval_forces(a, a->x0, a->F, 1.0)) return rc;
  double acc[A_N];
  sum_parts(a, acc);
  if (force) {
    if (int rc = download_soa(a, a->F, force)) return rc;
  }
  if (cudaStreamSynchronize(a->stream) != cudaSuccess) return afail(a, CVR_ERR_CUDA, "force evaluation failed");
  double dq_self[NT];
  const double es = self_energy(a, dq_self);
  if (energy) {
    energies(a, acc, energy);
    energy[3] = es;
  }
  if (dU) fold(a, acc, true, false, dq_self, dU);
  return CVR_OK;
}

int cvr_adj_force_vjp(cvr_adj *a, const double *u, double *w, double *g) {
  if (int rc = ready(a)) return rc;
  if (!u) return afail(a, CVR_ERR_INVALID, "u is required");
  const int n = a->p.n;
  std::vector<double> us(3 * (size_t)n);
  for (int d = 0; d < 3; ++d)
    for (int s = 0; s < n; ++s) us[(size_t)d * n + s] = u[3 * (size_t)a->id_of[s] + d];
  cudaMemcpyAsync(a->u, us.data(), 3 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice, a->stream);
  if (int rc = clear_parts(a)) return rc;
  PrepArgs pre{};
  pre.X = a->x0;
  pre.u = a->u;
  PostArgs post{};
  post.out = a->W;
  if (int rc = evalp<true>(a, pre, a->x0, post, 1.0)) return rc;
  double acc[A_N];
  sum_parts(a, acc);
  if (w) {
    if (int rc = download_soa(a, a->W, w)) return rc;
  }
  if (cudaStreamSynchronize(a->stream) != cudaSuccess) return afail(a, CVR_ERR_CUDA, "VJP failed");
  if (g) fold(a, acc, false, true, nullptr, g);
  return CVR_OK;
}

// Xout, Fout = one velocity-Verlet step from Xin, Fin; V is advanced in place.
static int forward_step(cvr_adj *a, const double *Xin, double *Xout, const double *Fin, double *Fout, double scale) {
  PrepArgs pre{};
  pre.op = PREP_DRIFT;
  pre.X = Xin;
  pre.Xout = Xout;
  pre.V = a->V;
  pre.F = Fin;
  PostArgs post{};
  post.op = POST_KICK;
  post.out = Fout;
  post.Fold = Fin;
  post.V = a->V;
  return evalp<false>(a, pre, Xout, post, scale);
}

int cvr_adj_loss(cvr_adj *a, int64_t nsteps, double *loss, double *pos_out, double *vel_out) {
  if (int rc = ready(a)) return rc;
  if (nsteps < 0) return afail(a, CVR_ERR_INVALID, "nsteps < 0");
  const size_t N3 = 3 * (size_t)a->p.n;
  if (int rc = clear_parts(a)) return rc;
  cudaMemcpyAsync(a->X, a->x0, N3 * sizeof(double), cudaMemcpyDeviceToDevice, a->stream);
  cudaMemcpyAsync(a->V, a->v0, N3 * sizeof(double), cudaMemcpyDeviceToDevice, a->stream);
  if (int rc = eval_forces(a, a->X, a->F, 0.0)) return rc;
  double *x = a->X, *xb = a->Xb, *f = a->F, *fb = a->Fb;
  const double scale = nsteps ? 1.0 / (double)nsteps : 0.0;
  for (int64_t t = 0; t < nsteps; ++t) {
    if (int rc = forward_step(a, x, xb, f, fb, scale)) return rc;
    std::swap(x, xb);
    std::swap(f, fb);
  }
  double acc[A_N];
  sum_parts(a, acc);
  if (pos_out) {
    if (int rc = download_soa(a, x, pos_out)) return rc;
  }
  if (vel_out) {
    if (int rc = download_soa(a, a->V, vel_out)) return rc;
  }
  if (cudaStreamSynchronize(a->stream) != cudaSuccess) return afail(a, CVR_ERR_CUDA, "loss run failed");
  double dq[NT], e[3];
  const double es = self_energy(a, dq);
  energies(a, acc, e);
  if (loss) *loss = nsteps ? e[0] + e[1] + e[2] + es : 0.0;
  return CVR_OK;
}

int cvr_adj_loss_grad(cvr_adj *a, int64_t nsteps, int64_t checkpoint_every, double *loss, double *g_pos,
                      double *g_vel, double *g_theta) {
  if (int rc = ready(a)) return rc;
  if (nsteps < 1 || checkpoint_every < 1) return afail(a, CVR_ERR_INVALID, "nsteps >= 1, checkpoint_every >= 1");
  const size_t N3 = 3 * (size_t)a->p.n, B3 = N3 * sizeof(double);
  const int64_t M = nsteps, K = std::min<int64_t>(checkpoint_every, nsteps);
  const int64_t nseg = (M + K - 1) / K, last0 = (nseg - 1) * K;
  // a checkpoint holds positions and velocities, and the forces (which save an
  // evaluation per segment) where memory allows
  size_t ckn = 3;
  if (reserve(a, &a->ck, &a->ck_cap, (size_t)nseg * 3 * N3) != CVR_OK) {
    ckn = 2;
    if (int rc = reserve(a, &a->ck, &a->ck_cap, (size_t)nseg * 2 * N3)) return rc;
  }
  if (int rc = reserve(a, &a->seg, &a->seg_cap, (size_t)(K + 1) * 2 * N3)) return rc;
  double *segX = a->seg, *segF = a->seg + (size_t)(K + 1) * N3;
  cudaStream_t st = a->stream;
  const double invM = 1.0 / (double)M;
  if (int rc = clear_parts(a)) return rc;
  // forward: loss, dU/dtheta, checkpoints; the last segment straight into the segment buffers
  double *x = last0 == 0 ? segX : a->X, *f = last0 == 0 ? segF : a->F;
  double *xb = a->Xb, *fb = a->Fb;
  cudaMemcpyAsync(x, a->x0, B3, cudaMemcpyDeviceToDevice, st);
  cudaMemcpyAsync(a->V, a->v0, B3, cudaMemcpyDeviceToDevice, st);
  if (int rc = eval_forces(a, x, f, 0.0)) return rc;
  for (int64_t t = 0; t < M; ++t) {
    if (t % K == 0 && t < last0) {
      double *c = a->ck + (size_t)(t / K) * ckn * N3;
      cudaMemcpyAsync(c, x, B3, cudaMemcpyDeviceToDevice, st);
      cudaMemcpyAsync(c + N3, a->V, B3, cudaMemcpyDeviceToDevice, st);
      if (ckn == 3) cudaMemcpyAsync(c + 2 * N3, f, B3, cudaMemcpyDeviceToDevice, st);
    }
    // step t's end is kept from the last segment's start on
    const bool keep = t + 1 >= last0;
    double *xn = keep ? segX + (size_t)(t + 1 - last0) * N3 : xb;
    double *fn = keep ? segF + (size_t)(t + 1 - last0) * N3 : fb;
    if (int rc = forward_step(a, x, xn, f, fn, invM)) return rc;
    if (!keep) {
      xb = x;
      fb = f;
    }
    x = xn;
    f = fn;
  }
  // reverse
  cudaMemsetAsync(a->Gr, 0, B3, st);
  cudaMemsetAsync(a->Gv, 0, B3, st);
  cudaMemsetAsync(a->Ga, 0, B3, st);
  PrepArgs pre{};
  pre.Gr = a->Gr;
  pre.Gv = a->Gv;
  pre.Ga = a->Ga;
  pre.u = a->u;
  pre.invM = invM;
  PostArgs post{};
  post.Gr = a->Gr;
  post.Gv = a->Gv;
  post.Ga = a->Ga;
  for (int64_t s = nseg - 1; s >= 0; --s) {
    const int64_t t0 = s * K, t1 = std::min(M, t0 + K);
    if (s < nseg - 1) {
      const double *c = a->ck + (size_t)s * ckn * N3;
      cudaMemcpyAsync(segX, c, B3, cudaMemcpyDeviceToDevice, st);
      cudaMemcpyAsync(a->V, c + N3, B3, cudaMemcpyDeviceToDevice, st);
      if (ckn == 3)
        cudaMemcpyAsync(segF, c + 2 * N3, B3, cudaMemcpyDeviceToDevice, st);
      else if (int rc = eval_forces(a, segX, segF, 0.0))
        return rc;
      for (int64_t t = t0; t < t1; ++t) {
        const int64_t q = t - t0;
        if (int rc = forward_step(a, segX + q * N3, segX + (q + 1) * N3, segF + q * N3, segF + (q + 1) * N3, 0.0))
          return rc;
      }
    }
    for (int64_t t = t1 - 1; t >= t0; --t) {
      const int64_t q = t - t0 + 1;
      pre.op = PREP_REV;
      pre.X = segX + q * N3;
      pre.F = segF + q * N3;
      post.op = POST_REV;
      if (int rc = evalp<true>(a, pre, pre.X, post, 1.0)) return rc;
    }
  }
  // a_0 = F(r_0)/m
  pre.op = PREP_REV0;
  pre.X = a->x0;
  post.op = POST_REV0;
  if (int rc = evalp<true>(a, pre, a->x0, post, 1.0)) return rc;
  double acc[A_N];
  sum_parts(a, acc);
  if (g_pos)
    if (int rc = download_soa(a, a->Gr, g_pos)) return rc;
  if (g_vel)
    if (int rc = download_soa(a, a->Gv, g_vel)) return rc;
  if (cudaStreamSynchronize(st) != cudaSuccess) return afail(a, CVR_ERR_CUDA, "adjoint run failed");
  double dq_self[NT], e[3];
  const double es = self_energy(a, dq_self);
  energies(a, acc, e);
  if (loss) *loss = e[0] + e[1] + e[2] + es;
  if (g_theta) fold(a, acc, true, true, dq_self, g_theta);
  return CVR_OK;
}

int cvr_adj_last_error(const cvr_adj *a, char *buf, size_t len) {
  if (!a || !buf || !len) return CVR_ERR_INVALID;
  std::snprintf(buf, len, "%s", a->err.c_str());
  return CVR_OK;
}

void *cvr_adj_stream(const cvr_adj *a) { return a ? (void *)a->stream : nullptr; }

}  // extern "C"
