// cvr_noalloc.cu -- Ewald structure factor S(k) for callers that cannot
// allocate device memory.
//
// Who needs this: code that runs inside a host program whose allocator owns
// the GPU's memory (a framework with a caching allocator or an MD engine
// that reserves its pool up front) and may not ask the CUDA runtime for more,
// plug-ins that are forbidden to allocate after start-up, and callers that
// cannot afford the device-wide synchronisation cudaMalloc/cudaFree imply in
// the middle of their own work.  They own their input and output buffers;
// this entry point brings no buffer of its own.
//
// The per-chunk partial sums the two kernels exchange live in the file-scope
// array g_sk_scratch below instead of a cudaMalloc'd buffer.  It holds
// CVR_NOALLOC_SK_SCRATCH complex doubles (4 MiB) on every GPU that loads the
// library, for the life of the process.  Host code may not use the symbol
// g_sk_scratch as a device address (in host code it names a host-side stand-in):
// the first call on each device looks up the real address with
// cudaGetSymbolAddress, with that device current, and passes it to the
// kernels.  Make that first call before any stream capture.  The address is
// kept per device ordinal for the rest of the process, so the entry point must
// not be used again on a device after cudaDeviceReset (the module is loaded
// anew there and the kept address no longer names the array).
//
// Every call on a device shares the one array, and the array keeps the last
// call's contents.  Each call writes every partial it later reads, so nothing
// needs clearing, but two calls whose kernels overlap on the GPU (different
// streams, no ordering between them) race on the array and give wrong sums.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>

#include <cuda_runtime.h>

#include "../../include/caviar_b200.h"

namespace {

constexpr int kMaxDevices = 64;
constexpr int kThreads = 512;     // most threads per block of k_sk_noalloc_partial
constexpr int kItems = 192;       // most (column, m-group) items per block
constexpr int kMaxMG = 6;         // most m-values per thread
constexpr int kMaxK = 30;         // largest k_max per axis
constexpr int kRedEntries = 32, kRedGroups = 8;  // k_sk_noalloc_reduce block
constexpr int kSMs = 148;
constexpr size_t kTableSmem = 160 * 1024;        // phase tables of one stage of atoms

// k_max <= 30 on every axis gives at most (61*61 + 1) / 2 summed (nx, ny)
// columns of 61 k-vectors; the array holds at least one chunk of them.
static_assert(((2 * kMaxK + 1) * (2 * kMaxK + 1) + 1) / 2 * (2 * kMaxK + 1) <= CVR_NOALLOC_SK_SCRATCH,
              "scratch must hold one chunk at k_max 30");
// the atom subgroups' partial sums reuse the tables' shared memory
static_assert((size_t)kThreads * 4 * kMaxMG * sizeof(double) <= kTableSmem, "subgroup sums must fit the table area");

__device__ __align__(256) double2 g_sk_scratch[CVR_NOALLOC_SK_SCRATCH];

std::mutex g_lock;
double2 *g_scratch_ptr[kMaxDevices] = {nullptr};

// The reference enumerates kx, ky, kz over [-kmax, kmax] (kz fastest), skips
// k = 0, and keeps the first (2kx)(2ky)(2kz) vectors
// (electrostatic_ewald_k/initialize.cpp:184-222).  In that order column
// (nx, ny) is c = (nx + kx)(2ky + 1) + ny + ky and its mirror (-nx, -ny) is
// C - 1 - c, C = (2kx + 1)(2ky + 1): for real charges
// S(-nx, -ny, -nz) = conj(S(nx, ny, nz)), so only columns 0 .. (C - 1) / 2
// (the last one (0, 0)) are summed.
struct KSpan {
  int kx, ky, kz, kp;   // kp = largest k_max + 1: phase-table row
  int ncol;             // summed columns, (C + 1) / 2
  int nmg;              // m-groups per column (of MG values each)
  int nk;               // k-vectors of the set
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// e^{i 2 pi m u}
__device__ __forceinline__ double2 phase(double u, int m) {
  const double v = (double)m * u;
  double sn, cs;
  sincospi(2.0 * (v - rint(v)), &sn, &cs);
  return make_double2(cs, sn);
}

// Chunk sums of S(k) over the summed columns, FP64 throughout.  One thread
// holds one column's m = m0 .. m0 + MG - 1 for one of SUB interleaved atom
// subgroups of the chunk: per atom one complex product W = q X Y, then four
// FMAs per +-m pair (sums of Wr Zr, Wi Zi, Wr Zi, Wi Zr; S(+m) and S(-m) are
// their sums and differences).  The phase tables of a stage of atoms sit in
// shared memory; every fourth m is evaluated directly and the others are
// products with the m = 1 phase (whose argument error, m times that of x / L,
// the direct form has too).  Per atom at k_max 8: 290 items x 24 FP64
// operations, against 4096 x 12 with one thread per k-vector.  20001 atoms,
// k_max 8, whole call: 172 -> 32.8 us (100,000 atoms: 37 us at k_max 4, 209
// at 10).  Two columns per thread (half the reads of Z): 31.9, 41 and 215 us,
// so the reads are not what bounds it; the FP64 pipe is 39 % busy, the rest
// is the table phase, which one block per SM cannot overlap with the sums.
template <int MG>
__global__ void __launch_bounds__(kThreads) k_sk_noalloc_partial(const double *__restrict__ pos,
                                                                 const double *__restrict__ q, int n, int chunk_atoms,
                                                                 int stage_atoms, double3 inv_L, KSpan s,
                                                                 double2 *__restrict__ partial) {
  extern __shared__ double2 tab[];  // [stage_atoms][3][kp], X rows times the charge
  const int items = blockDim.x, it = threadIdx.x, sub = threadIdx.y, nsub = blockDim.y;
  const int tid = sub * items + it, nthreads = items * nsub;
  const int item = blockIdx.x * items + it;
  const bool live = item < s.ncol * s.nmg;
  const int col = live ? item % s.ncol : 0, m0 = live ? item / s.ncol * MG : 0;
  const int nx = col / (2 * s.ky + 1) - s.kx, ny = col % (2 * s.ky + 1) - s.ky;
  const int kp = s.kp, row = 3 * kp, mx = abs(nx), my = kp + abs(ny);
  // a group's m-values past k_max_z read the last row entry; their sums are not stored
  int mz[MG];
#pragma unroll
  for (int u = 0; u < MG; ++u) mz[u] = 2 * kp + min(m0 + u, s.kz);
  double a[MG], b[MG], c[MG], d[MG];
#pragma unroll
  for (int u = 0; u < MG; ++u) a[u] = b[u] = c[u] = d[u] = 0.0;
  const int a_begin = blockIdx.y * chunk_atoms, a_end = min(n, a_begin + chunk_atoms);
  const int quads = (kp + 3) >> 2;  // table tasks per (atom, axis): m = 4g .. 4g + 3
  for (int s0 = a_begin; s0 < a_end; s0 += stage_atoms) {
    const int na = min(stage_atoms, a_end - s0);
    __syncthreads();
    for (int t = tid; t < na * 3 * quads; t += nthreads) {
      const int at = t / (3 * quads), rem = t % (3 * quads), ax = rem / quads, m4 = 4 * (rem % quads);
      const double il = (ax == 0) ? inv_L.x : ((ax == 1) ? inv_L.y : inv_L.z);
      const double u = pos[3 * (size_t)(s0 + at) + ax] * il;
      const double scale = ax == 0 ? q[s0 + at] : 1.0;
      const double2 e1 = phase(u, 1);
      // m = 0: 1, and NaN where u is not finite (every S(k) is NaN then)
      double2 v = m4 ? phase(u, m4) : make_double2(isfinite(u) ? 1.0 : u - u, 0.0);
      double2 *out = tab + at * row + ax * kp + m4;
      const int len = min(4, kp - m4);
      for (int m = 0; m < len; ++m) {
        out[m] = make_double2(scale * v.x, scale * v.y);
        v = cmul(v, e1);
      }
    }
    __syncthreads();
    if (live) {
#pragma unroll 2
      for (int at = sub; at < na; at += nsub) {
        const double2 *tb = tab + at * row;
        double2 px = tb[mx], py = tb[my];
        if (nx < 0) px.y = -px.y;
        if (ny < 0) py.y = -py.y;
        const double2 w = cmul(px, py);
#pragma unroll
        for (int u = 0; u < MG; ++u) {
          const double2 z = tb[mz[u]];
          a[u] = fma(w.x, z.x, a[u]);
          b[u] = fma(w.y, z.y, b[u]);
          c[u] = fma(w.x, z.y, c[u]);
          d[u] = fma(w.y, z.x, d[u]);
        }
      }
    }
  }
  // atom subgroups in order into subgroup 0
  double *red = reinterpret_cast<double *>(tab);
  __syncthreads();
  if (sub > 0) {
#pragma unroll
    for (int u = 0; u < MG; ++u) {
      double *r = red + (size_t)((sub - 1) * 4 * MG + 4 * u) * items + it;
      r[0] = a[u];
      r[items] = b[u];
      r[2 * items] = c[u];
      r[3 * items] = d[u];
    }
  }
  __syncthreads();
  if (sub > 0 || !live) return;
  for (int g = 1; g < nsub; ++g) {
#pragma unroll
    for (int u = 0; u < MG; ++u) {
      const double *r = red + (size_t)((g - 1) * 4 * MG + 4 * u) * items + it;
      a[u] += r[0];
      b[u] += r[items];
      c[u] += r[2 * items];
      d[u] += r[3 * items];
    }
  }
  double2 *out = partial + (size_t)blockIdx.y * s.ncol * (2 * s.kz + 1) + col;
#pragma unroll
  for (int u = 0; u < MG; ++u) {
    const int m = m0 + u;
    if (m > s.kz) break;
    out[(size_t)(s.kz + m) * s.ncol] = make_double2(a[u] - b[u], c[u] + d[u]);
    if (m > 0) out[(size_t)(s.kz - m) * s.ncol] = make_double2(a[u] + b[u], d[u] - c[u]);
  }
}

// S(k) = sum of the chunk partials (fixed order: kRedGroups interleaved chunk
// groups, then the groups), stored at k and, conjugated, at the mirror -k,
// where they are in the set.
__global__ void __launch_bounds__(kRedEntries *kRedGroups) k_sk_noalloc_reduce(const double2 *__restrict__ partial,
                                                                               int nchunks, KSpan s,
                                                                               double *__restrict__ sk) {
  __shared__ double2 sums[kRedGroups][kRedEntries];
  const int nz = 2 * s.kz + 1, total = s.ncol * nz;
  const int e = blockIdx.x * kRedEntries + threadIdx.x, g = threadIdx.y;
  double2 v = make_double2(0.0, 0.0);
  if (e < total) {
#pragma unroll 4
    for (int c = g; c < nchunks; c += kRedGroups) {
      const double2 p = partial[(size_t)c * total + e];
      v.x += p.x;
      v.y += p.y;
    }
  }
  sums[g][threadIdx.x] = v;
  __syncthreads();
  if (g > 0 || e >= total) return;
#pragma unroll
  for (int r = 1; r < kRedGroups; ++r) {
    v.x += sums[r][threadIdx.x].x;
    v.y += sums[r][threadIdx.x].y;
  }
  const int col = e % s.ncol, full = col * nz + e / s.ncol;  // place in the enumeration with k = 0
  const int zero = (s.ncol - 1) * nz + s.kz, mirror = 2 * zero - full;
  if (full == zero) return;
  const int k = full < zero ? full : full - 1;
  if (k < s.nk) {
    sk[2 * (size_t)k] = v.x;
    sk[2 * (size_t)k + 1] = v.y;
  }
  const int km = mirror - 1;  // a mirror column comes after k = 0
  if (col < s.ncol - 1 && km < s.nk) {
    sk[2 * (size_t)km] = v.x;
    sk[2 * (size_t)km + 1] = -v.y;
  }
}

using PartialFn = void (*)(const double *, const double *, int, int, int, double3, KSpan, double2 *);
constexpr PartialFn kPartial[kMaxMG] = {k_sk_noalloc_partial<1>, k_sk_noalloc_partial<2>, k_sk_noalloc_partial<3>,
                                        k_sk_noalloc_partial<4>, k_sk_noalloc_partial<5>, k_sk_noalloc_partial<6>};

int say(char *err, size_t len, int code, const char *msg) {
  if (err && len) std::snprintf(err, len, "%s", msg);
  return code;
}

}  // namespace

extern "C" int cvr_structure_factor_noalloc(const double *pos, const double *q, int64_t n, const double box_len[3],
                                            int kx_max, int ky_max, int kz_max, double *sk, void *stream, char *err,
                                            size_t err_len) {
  if (err && err_len) err[0] = '\0';
  if (!pos || !q || !sk || !box_len || n <= 0 || n > (int64_t)1 << 30)
    return say(err, err_len, CVR_ERR_INVALID, "pos, q, sk, box_len must be non-null and 0 < n <= 2^30");
  if (kx_max < 0 || ky_max < 0 || kz_max < 0 || kx_max > kMaxK || ky_max > kMaxK || kz_max > kMaxK)
    return say(err, err_len, CVR_ERR_INVALID, "k_max per axis must be in [0, 30]");
  for (int d = 0; d < 3; ++d)
    if (!(box_len[d] > 0)) return say(err, err_len, CVR_ERR_INVALID, "box lengths must be positive");
  const int nk = (2 * kx_max) * (2 * ky_max) * (2 * kz_max);  // <= 216000, see kMaxK
  if (nk == 0) return CVR_OK;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return say(err, err_len, CVR_ERR_CUDA, "no usable current CUDA device");
  double2 *scratch = nullptr;
  {
    std::lock_guard<std::mutex> g(g_lock);
    if (!g_scratch_ptr[dev]) {
      // Set-up, once per device with that device current: the array's device
      // address, and the kernel's shared-memory limit for the largest k_max
      // (set once here, so that concurrent calls never lower it for each other).
      void *p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_sk_scratch);
      if (e != cudaSuccess) return say(err, err_len, CVR_ERR_CUDA, cudaGetErrorString(e));
      for (PartialFn f : kPartial) {
        e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTableSmem);
        if (e != cudaSuccess) return say(err, err_len, CVR_ERR_CUDA, cudaGetErrorString(e));
      }
      g_scratch_ptr[dev] = static_cast<double2 *>(p);
    }
    scratch = g_scratch_ptr[dev];
  }
  KSpan s{kx_max, ky_max, kz_max, 0, 0, 0, nk};
  s.kp = std::max(kx_max, std::max(ky_max, kz_max)) + 1;
  s.ncol = ((2 * kx_max + 1) * (2 * ky_max + 1) + 1) / 2;
  // m-groups of equal size, at most kMaxMG m-values per thread (24 FP64 sums)
  const int M = kz_max + 1;
  s.nmg = (M + kMaxMG - 1) / kMaxMG;
  const int mg = (M + s.nmg - 1) / s.nmg;
  // items in whole warps over as few blocks as kItems allows (each block
  // builds its own phase tables); atom subgroups fill the block's threads
  const int items = s.ncol * s.nmg, gx = (items + kItems - 1) / kItems;
  const int per_block = ((items + gx - 1) / gx + 31) / 32 * 32;
  const int nsub = kThreads / per_block;
  // one block per SM: the chunks that make it so, as far as the scratch
  // holds them, and no chunk below 16 atoms
  int64_t nchunks = std::min<int64_t>(CVR_NOALLOC_SK_SCRATCH / ((int64_t)s.ncol * (2 * kz_max + 1)),
                                      std::max(1, kSMs / gx));
  nchunks = std::max<int64_t>(1, std::min<int64_t>(nchunks, n / 16));
  const int chunk_atoms = (int)((n + nchunks - 1) / nchunks);
  nchunks = (n + chunk_atoms - 1) / chunk_atoms;
  const size_t atom_bytes = (size_t)3 * s.kp * sizeof(double2);
  const int stage_atoms = (int)std::min<int64_t>(chunk_atoms, kTableSmem / atom_bytes);
  const size_t smem =
      std::max(stage_atoms * atom_bytes, (size_t)(nsub - 1) * per_block * 4 * mg * sizeof(double));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const double3 inv_L = make_double3(1.0 / box_len[0], 1.0 / box_len[1], 1.0 / box_len[2]);
  kPartial[mg - 1]<<<dim3(gx, (unsigned)nchunks), dim3(per_block, nsub), smem, st>>>(
      pos, q, (int)n, chunk_atoms, stage_atoms, inv_L, s, scratch);
  const int entries = s.ncol * (2 * kz_max + 1);
  k_sk_noalloc_reduce<<<(entries + kRedEntries - 1) / kRedEntries, dim3(kRedEntries, kRedGroups), 0, st>>>(
      scratch, (int)nchunks, s, sk);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return say(err, err_len, CVR_ERR_CUDA, cudaGetErrorString(e));
  return CVR_OK;
}
