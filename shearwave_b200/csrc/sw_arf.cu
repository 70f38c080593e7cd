// Acoustic radiation force from recorded pressure (and particle velocity):
// the producers that feed shear_fdtd's body force.
//
// Reference: compute_radiation_force and compute_radiation_force_velocity
// (src/shearwave/radiation_force.py:27-85, 88-157).  Inputs are the
// reference's (nx, ny, nz, nt) arrays, time fastest, so a cell's series is
// one contiguous row of nt values:
//
//  * arf_env_partial / arf_env_final: the auto-gate envelope
//    env[t] = mean over cells of p[cell, t]^2 (radiation_force.py:63-68),
//    a column reduction of the (cells x nt) matrix into FP64 partials that a
//    second kernel sums in a fixed order: deterministic.
//  * arf_force: per cell, a group of lanes reads the gated entries of its
//    row, reduces sum p*q in FP64 (q = p, or a velocity component), and the
//    group leader applies the reference's formula:
//      alpha_Np = alpha_coeff * f0_MHz / 8.685889638 * 100
//      scalar:  b = 2 alpha_Np (mean p^2 / (rho c)) / c
//      vector:  b_i = (2 alpha_Np / c) mean(p v_i)
// Both passes are HBM-bound reads of the pressure (and velocity) records.
#include <algorithm>
#include <type_traits>

#include "sw_common.cuh"

namespace sw {
namespace {

// The envelope reads the record once.  A block owns a band of rows and a
// chunk of `cn` columns (all of them up to 1024); its threads are k rows of cn
// columns, so a warp's loads are consecutive whatever nt is, and each thread
// keeps eight loads of its column in flight.  (With 256 threads striding
// over the columns, a row of 300 kept 300 of 1024 lanes busy: 473 us on a
// 128 x 96 x 112 x 300 float record; now 250, 6.6 TB/s.)
constexpr int kEnvMaxThreads = 1024;

template <typename T>
__global__ void __launch_bounds__(kEnvMaxThreads, 2)
    arf_env_partial(const T* __restrict__ p, long long ncell, int nt, int chunk0, int cn, int k,
                    long long rows_per_block, double* __restrict__ partials) {
  extern __shared__ double env_red[];  // [k][cn]
  const int cb = (chunk0 + blockIdx.y) * cn, w = min(cn, nt - cb);
  const int r = threadIdx.x / cn, c = threadIdx.x % cn;
  const long long r0 = (long long)blockIdx.x * rows_per_block;
  const long long r1 = r0 + rows_per_block < ncell ? r0 + rows_per_block : ncell;
  double acc = 0.0;
  if (r < k && c < w) {
    const T* q = p + (r0 + r) * nt + cb + c;
    const long long step = (long long)k * nt;
    long long left = r0 + r < r1 ? (r1 - r0 - r + k - 1) / k : 0;
    for (; left >= 8; left -= 8, q += 8 * step) {
      T v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldcs(q + u * step);
#pragma unroll
      for (int u = 0; u < 8; ++u) acc = fma((double)v[u], (double)v[u], acc);
    }
    for (; left > 0; --left, q += step) {
      const double v = (double)__ldcs(q);
      acc = fma(v, v, acc);
    }
  }
  if (r < k) env_red[r * cn + c] = acc;
  __syncthreads();
  if (threadIdx.x < w) {
    double t = 0.0;
    for (int u = 0; u < k; ++u) t += env_red[u * cn + threadIdx.x];
    partials[(long long)blockIdx.x * nt + cb + threadIdx.x] = t;
  }
}

// Sums the bands' partials: 32 columns per block, 32 threads per column (one
// thread walking all bands took 66 us).
constexpr int kEnvFinal = 32;
__global__ void __launch_bounds__(kEnvFinal * kEnvFinal)
    arf_env_final(const double* __restrict__ partials, int nblk, int nt, long long ncell,
                  double* __restrict__ env) {
  __shared__ double red[kEnvFinal][kEnvFinal + 1];
  const int t = blockIdx.x * kEnvFinal + threadIdx.x;
  double s = 0.0;
  if (t < nt) {
#pragma unroll 8
    for (int b = threadIdx.y; b < nblk; b += kEnvFinal) s += partials[(long long)b * nt + t];
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && t < nt) {
    double v = 0.0;
#pragma unroll
    for (int b = 0; b < kEnvFinal; ++b) v += red[b][threadIdx.x];
    env[t] = v / (double)ncell;
  }
}

// Sum over the G lanes of a group (G a power of two <= 32, groups aligned).
template <int G>
__device__ inline double group_sum(double v) {
#pragma unroll
  for (int off = G / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

struct ArfMaps {
  const double *c, *rho, *alpha;  // per cell, or one value when stride is 0
  long long stride;
};

// One 16-byte window of a row.
template <typename T>
struct ArfWin {
  static constexpr int V = 16 / (int)sizeof(T);
  T v[V];
};
template <typename T>
__device__ __forceinline__ ArfWin<T> arf_window(const T* __restrict__ row, long long j0) {
  ArfWin<T> w;
  if constexpr (ArfWin<T>::V == 4) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(row + j0));
    w.v[0] = f.x, w.v[1] = f.y, w.v[2] = f.z, w.v[3] = f.w;
  } else {
    const double2 f = __ldg(reinterpret_cast<const double2*>(row + j0));
    w.v[0] = f.x, w.v[1] = f.y;
  }
  return w;
}

// The gate as bits, from its first sample on (bit 4 + t - first; room for the
// elements a window holds before the first and after the last).
constexpr int kGateSpan = 4096, kGateWords = (kGateSpan + 64) / 32 + 1;
struct ArfGate {
  unsigned bits[kGateWords];
  int lo, hi, dup;
};

// One lane's sums over its windows of a row: every G-th 16-byte window from
// `sub` on, `nw` in all, the row's first window at element e0 of the records,
// the gate's first sample n0 elements after it; the gate's bits tell which of a
// window's elements count.  Four windows of one record, or one of four, are in
// flight per lane: with two of one record the reads did not fill DRAM (405 of
// 1349 samples on 90 x 96 x 100 cells 298 us, with four 248, with eight 250 and
// small grids slower), and with four records more windows take registers from
// the warps that hide the latency (four: 120 registers, 16 warps per SM, 15 %
// slower; two at 80 registers: no faster on large grids).
template <typename T, int NF, int G>
__device__ __forceinline__ void row_sums(const T* __restrict__ p, const T* __restrict__ q0,
                                         const T* __restrict__ q1, const T* __restrict__ q2,
                                         long long e0, int sub, int nw, int n0,
                                         const unsigned* bits, double (&s)[3]) {
  constexpr int V = ArfWin<T>::V;
  constexpr int B = NF == 1 ? 4 : 1;
  // four chains for the one sum, so that few lanes a cell round no more than
  // many would; one for each of three (two spill, and are 2 % slower)
  constexpr int C = NF == 1 ? 4 : 1, S = NF == 1 ? 1 : 3;
  double acc[S][C] = {};
  e0 += sub * V;
  for (int w0 = sub; w0 < nw; w0 += B * G, e0 += B * G * V) {
    ArfWin<T> a[B], b[B], c[B], d[B];
#pragma unroll
    for (int k = 0; k < B; ++k)
      if (k == 0 || w0 + k * G < nw) {
        a[k] = arf_window(p, e0 + k * G * V);
        if (NF == 3) {
          b[k] = arf_window(q0, e0 + k * G * V);
          c[k] = arf_window(q1, e0 + k * G * V);
          d[k] = arf_window(q2, e0 + k * G * V);
        }
      }
#pragma unroll
    for (int k = 0; k < B; ++k) {
      const int w = w0 + k * G, bit = w * V - n0 + 4;
      if (k > 0 && w >= nw) break;
      const unsigned in = __funnelshift_r(bits[bit >> 5], bits[(bit >> 5) + 1], bit & 31);
#pragma unroll
      for (int u = 0; u < V; ++u) {
        if (((in >> u) & 1u) == 0u) continue;
        const double pv = (double)a[k].v[u];
        const int n = (k * V + u) & (C - 1);
        if (NF == 1) {
          acc[0][n] = fma(pv, pv, acc[0][n]);
        } else {
          acc[0][n] = fma(pv, (double)b[k].v[u], acc[0][n]);
          acc[1 % S][n] = fma(pv, (double)c[k].v[u], acc[1 % S][n]);
          acc[2 % S][n] = fma(pv, (double)d[k].v[u], acc[2 % S][n]);
        }
      }
    }
  }
#pragma unroll
  for (int f = 0; f < S; ++f) {
#pragma unroll
    for (int n = C / 2; n > 0; n /= 2)
#pragma unroll
      for (int u = 0; u < n; ++u) acc[f][u] += acc[f][u + n];
    s[f] = acc[f][0];
  }
}

// The record is read once; what bounds the pass is the number of loads in
// flight and the instructions per element.  A gate without repeats whose
// samples lie close together (`dense`: the auto gate of a burst, a slice, a
// mask) is read as 16-byte windows of the row (row_sums); any other gate entry
// by entry through the index list, as are the rows whose windows would leave
// the record (its first and last).  Rows start on any element, so the windows'
// alignment is each row's own; records whose bases differ modulo 16 bytes
// take the entry path.  A window covers four (or two) samples, and a 32-byte
// sector is read whole anyway, so windows pay up to six samples of span per
// sample.  A warp takes `iters` times 32 / G cells, each a group of G lanes'
// sum, then evaluates the formula for all of them at once: its float64
// divisions in one lane per group took as long as the reads.  Measured against
// one gate entry at a time and one cell per warp: 109 of 300 samples of a float
// record on 128 x 96 x 112 cells 363 -> 134 us, 129 of 257 of four records on
// 80 x 72 x 101 cells 382 -> 242 us (6 TB/s of DRAM reads, whose granules are
// wider than the gate).
template <typename T, typename To, int NF, int G>
__global__ void __launch_bounds__(256, 4)
    arf_force(const T* __restrict__ p, const T* __restrict__ q0, const T* __restrict__ q1,
              const T* __restrict__ q2, long long ncell, int nt, const int* __restrict__ gate,
              int ngate, ArfMaps m, double f0_mhz, To* __restrict__ o0, To* __restrict__ o1,
              To* __restrict__ o2, int windows, int iters) {
  constexpr int V = ArfWin<T>::V, PER = 32 / G;
  const int lane = threadIdx.x & 31, sub = lane & (G - 1);
  __shared__ ArfGate sg;
  if (threadIdx.x == 0) sg.lo = 0x7fffffff, sg.hi = -1, sg.dup = 0;
  for (int k = threadIdx.x; k < kGateWords; k += blockDim.x) sg.bits[k] = 0u;
  __syncthreads();
  {
    int lo = 0x7fffffff, hi = -0x7fffffff;
    for (int j = threadIdx.x; j < ngate; j += blockDim.x) {
      const int g = __ldg(gate + j);
      lo = min(lo, g);
      hi = max(hi, g);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) {
      atomicMin(&sg.lo, lo);
      atomicMax(&sg.hi, hi);
    }
  }
  __syncthreads();
  const int g0 = sg.lo;
  const long long wide = (long long)sg.hi - g0 + 1;
  bool dense = windows != 0 && g0 >= 0 && sg.hi < nt && wide <= kGateSpan && wide <= 6LL * ngate;
  const int span = dense ? (int)wide : 0;
  if (dense)
    for (int j = threadIdx.x; j < ngate; j += blockDim.x) {
      const int b = __ldg(gate + j) - g0 + 4;
      if (atomicOr(&sg.bits[b >> 5], 1u << (b & 31)) & (1u << (b & 31))) sg.dup = 1;
    }
  __syncthreads();
  dense = dense && sg.dup == 0;
  // elements of the base before its 16-byte boundary
  const int skew = (int)((reinterpret_cast<uintptr_t>(p) & 15u) / sizeof(T));
  const long long total = ncell * nt;
  // round `it` of a block's warps is a run of neighbouring cells
  const int wpb = blockDim.x >> 5, wib = threadIdx.x >> 5;
  const long long per_block = (long long)wpb * iters * PER;
  const double inv_n = 1.0 / (double)ngate;
  for (long long base = blockIdx.x * per_block + wib * PER; base < ncell;
       base += gridDim.x * per_block) {
    double keep[3] = {0.0, 0.0, 0.0};  // lane l: the sums of round l / PER, group l % PER
    for (int it = 0; it < iters; ++it) {
      const long long cell = base + it * wpb * PER + lane / G;
      double s[3] = {0.0, 0.0, 0.0};
      const long long lo = cell * nt + g0;
      // first window: the boundary at or before lo
      const long long e0 = (lo + skew) / V * V - skew;
      const int n0 = (int)(lo - e0), nw = (n0 + span + V - 1) / V;
      if (cell < ncell && dense && e0 >= 0 && e0 + (long long)nw * V <= total) {
        row_sums<T, NF, G>(p, q0, q1, q2, e0, sub, nw, n0, sg.bits, s);
      } else if (cell < ncell) {
        const long long row = cell * nt;
#pragma unroll 4
        for (int j = sub; j < ngate; j += G) {
          const int g = __ldg(gate + j);
          if ((unsigned)g >= (unsigned)nt) continue;  // the host validates; never read outside
          const long long k = row + g;
          const double pv = (double)p[k];
          if (NF == 1) {
            s[0] += pv * pv;
          } else {
            s[0] += pv * (double)q0[k];
            s[1] += pv * (double)q1[k];
            s[2] += pv * (double)q2[k];
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const double t = __shfl_sync(0xffffffffu, group_sum<G>(s[f]), (lane % PER) * G);
        if (lane / PER == it) keep[f] = t;
      }
    }
    const long long cell = base + lane / PER * wpb * PER + lane % PER;
    if (lane < iters * PER && cell < ncell) {
      const long long mi = cell * m.stride;
      const double c = m.c[mi], rho = m.rho[mi], alpha = m.alpha[mi];
      const double alpha_np = alpha * f0_mhz / 8.685889638 * 100.0;
      if (NF == 1) {
        const double isppa = (keep[0] * inv_n) / (rho * c);
        o0[cell] = (To)(2.0 * alpha_np * isppa / c);
      } else {
        const double coeff = 2.0 * alpha_np / c;
        o0[cell] = (To)(coeff * (keep[0] * inv_n));
        o1[cell] = (To)(coeff * (keep[1] * inv_n));
        o2[cell] = (To)(coeff * (keep[2] * inv_n));
      }
    }
  }
}

long long env_blocks(long long ncell) {
  const long long want = 8LL * kNumSMs;
  return ncell < want ? (ncell > 0 ? ncell : 1) : want;
}

template <typename T, typename To, int NF>
int launch_force(const void* p, const void* const* q, long long ncell, int nt, const int* gate,
                 int ngate, ArfMaps m, double f0_mhz, void* const* out, cudaStream_t s) {
  const T* pp = (const T*)p;
  const T* qa = NF == 3 ? (const T*)q[0] : nullptr;
  const T* qb = NF == 3 ? (const T*)q[1] : nullptr;
  const T* qc = NF == 3 ? (const T*)q[2] : nullptr;
  To* oa = (To*)out[0];
  To* ob = NF == 3 ? (To*)out[1] : nullptr;
  To* oc = NF == 3 ? (To*)out[2] : nullptr;
  // windows need element-aligned bases that agree modulo 16 bytes
  const uintptr_t al = (uintptr_t)p & 15u;
  const int windows =
      al % sizeof(T) == 0 &&
      (NF == 1 || (((uintptr_t)q[0] & 15u) == al && ((uintptr_t)q[1] & 15u) == al &&
                   ((uintptr_t)q[2] & 15u) == al));
  // lanes per cell: as few as keep a gate to several loads per lane (the
  // group's reduction costs log2 G shuffles a cell).  With four records a lane
  // has a quarter of the windows of one record in flight, and longer runs of
  // one row make up for it.  On 29 x 116 x 74 cells, us at 8, 16 and 32 lanes:
  // one record, 109 / 405 / 1200 samples: 31 40 61 / 83 84 90 / 208 206 217;
  // four records, 72 / 109 / 200 / 600 samples: 77 79 89 / 101 97 100 /
  // 165 157 160 / 443 410 392.
  // Rounds of 32 / g cells per warp: up to the 32 cells whose formula one warp
  // evaluates at once, fewer where the grid would not fill the 32 warps an SM
  // holds (four records, 405 samples on 34 x 33 x 23 cells: 41 us with half of
  // them, 35 us so).
  int iters = 1;
  auto blocks = [&](int g) {
    const long long warps = 32LL * kNumSMs, rounds = (ncell * g + 31) / 32;
    iters = (int)std::max<long long>(1, std::min<long long>(g, (rounds + warps - 1) / warps));
    const long long want = (rounds + iters * 8 - 1) / (iters * 8);
    return (int)std::max<long long>(1, std::min<long long>(want, 16LL * kNumSMs));
  };
  auto launch = [&](auto lanes) {
    constexpr int G = decltype(lanes)::value;
    const int nb = blocks(G);
    arf_force<T, To, NF, G><<<nb, 256, 0, s>>>(pp, qa, qb, qc, ncell, nt, gate, ngate, m, f0_mhz,
                                               oa, ob, oc, windows, iters);
  };
  using std::integral_constant;
  if (ngate <= 32)
    launch(integral_constant<int, 4>());
  else if (ngate <= (NF == 1 ? 1024 : 96))
    launch(integral_constant<int, 8>());
  else if (NF == 1 || ngate <= 256)
    launch(integral_constant<int, 16>());
  else if constexpr (NF == 3)
    launch(integral_constant<int, 32>());
  count_launches(1);
  SW_CHECK_LAUNCH("radiation force");
  return SW_OK;
}

}  // namespace
}  // namespace sw

using namespace sw;

extern "C" size_t sw_arf_workspace_bytes(int64_t ncell, int32_t nt) {
  if (ncell <= 0 || nt <= 0) return 0;
  return (size_t)env_blocks(ncell) * (size_t)nt * sizeof(double);
}

extern "C" int sw_arf_envelope(int dtype, const void* p, int64_t ncell, int32_t nt, double* env,
                               void* workspace, size_t workspace_bytes, void* stream) {
  if (p == nullptr || env == nullptr || ncell <= 0 || nt <= 0 ||
      (dtype != SW_F32 && dtype != SW_F64)) {
    set_error("sw_arf_envelope: bad arguments");
    return SW_EINVAL;
  }
  if (workspace == nullptr || workspace_bytes < sw_arf_workspace_bytes(ncell, nt)) {
    set_error("sw_arf_envelope: workspace must be >= %zu bytes", sw_arf_workspace_bytes(ncell, nt));
    return SW_EWORKSPACE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  // columns per block, and rows of them: the count that leaves the fewest
  // lanes of the last warp idle
  const int chunks = (nt - 1) / kEnvMaxThreads + 1;
  const int cn = (nt - 1) / chunks + 1;
  int k = 1;
  double best = 0.0;
  for (int c = 1; c * cn <= kEnvMaxThreads && c <= 64; ++c) {
    const double used = (double)(c * cn) / (((c * cn + 31) / 32) * 32);
    if (used >= best - 0.02 || c * cn <= kEnvMaxThreads / 2) {
      best = std::max(best, used);
      k = c;
    }
  }
  const int threads = (k * cn + 31) / 32 * 32;
  // four bands per resident block, within the workspace's room
  const int per_sm = std::max(1, 2048 / threads);
  const long long nblk = std::min(env_blocks(ncell), std::max(2LL, 4LL / chunks) * per_sm * kNumSMs);
  const long long rows = (ncell + nblk - 1) / nblk;
  const size_t smem = sizeof(double) * (size_t)k * cn;
  double* part = (double*)workspace;
  // one launch, unless a record has more than 65535 chunks
  for (int c0 = 0; c0 < chunks; c0 += 65535) {
    const dim3 grid((unsigned)nblk, (unsigned)std::min(chunks - c0, 65535));
    if (dtype == SW_F32)
      arf_env_partial<float><<<grid, threads, smem, s>>>((const float*)p, ncell, nt, c0, cn, k,
                                                         rows, part);
    else
      arf_env_partial<double><<<grid, threads, smem, s>>>((const double*)p, ncell, nt, c0, cn, k,
                                                          rows, part);
    count_launches(1);
  }
  arf_env_final<<<(nt + kEnvFinal - 1) / kEnvFinal, dim3(kEnvFinal, kEnvFinal), 0, s>>>(
      part, (int)nblk, nt, ncell, env);
  count_launches(1);
  SW_CHECK_LAUNCH("radiation-force envelope");
  return SW_OK;
}

extern "C" int sw_arf_force(int dtype, int n_fields, const void* p, const void* vx,
                            const void* vy, const void* vz, int64_t ncell, int32_t nt,
                            const int32_t* gate, int32_t n_gate, const double* c_map,
                            const double* rho_map, const double* alpha_map, int64_t map_stride,
                            double f0, int out_dtype, void* out0, void* out1, void* out2,
                            void* stream) {
  const bool ok_types = (dtype == SW_F32 || dtype == SW_F64) &&
                        (out_dtype == SW_F32 || out_dtype == SW_F64);
  if (!ok_types || p == nullptr || ncell <= 0 || nt <= 0 || gate == nullptr || n_gate <= 0 ||
      c_map == nullptr || rho_map == nullptr || alpha_map == nullptr ||
      (map_stride != 0 && map_stride != 1) || out0 == nullptr ||
      (n_fields != 1 && n_fields != 3) ||
      (n_fields == 3 && (vx == nullptr || vy == nullptr || vz == nullptr || out1 == nullptr ||
                         out2 == nullptr))) {
    set_error("sw_arf_force: bad arguments");
    return SW_EINVAL;
  }
  ArfMaps m{c_map, rho_map, alpha_map, map_stride};
  const void* q[3] = {vx, vy, vz};
  void* out[3] = {out0, out1, out2};
  const double f0_mhz = f0 / 1e6;
  cudaStream_t s = (cudaStream_t)stream;
  const bool f32 = dtype == SW_F32, o32 = out_dtype == SW_F32;
  if (n_fields == 1) {
    if (f32 && o32) return launch_force<float, float, 1>(p, q, ncell, nt, gate, n_gate, m, f0_mhz, out, s);
    if (f32) return launch_force<float, double, 1>(p, q, ncell, nt, gate, n_gate, m, f0_mhz, out, s);
    if (o32) return launch_force<double, float, 1>(p, q, ncell, nt, gate, n_gate, m, f0_mhz, out, s);
    return launch_force<double, double, 1>(p, q, ncell, nt, gate, n_gate, m, f0_mhz, out, s);
  }
  if (f32 && o32) return launch_force<float, float, 3>(p, q, ncell, nt, gate, n_gate, m, f0_mhz, out, s);
  if (f32) return launch_force<float, double, 3>(p, q, ncell, nt, gate, n_gate, m, f0_mhz, out, s);
  if (o32) return launch_force<double, float, 3>(p, q, ncell, nt, gate, n_gate, m, f0_mhz, out, s);
  return launch_force<double, double, 3>(p, q, ncell, nt, gate, n_gate, m, f0_mhz, out, s);
}
