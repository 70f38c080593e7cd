// Direct (spectral) solve of the projection's Poisson problem.
//
// The CG of src/shearwave/solver.py:1010-1050 inverts A = -div_c(grad_c .)
// with both central differences zeroed on the one-voxel shell.  Restricted to
// interior cells, A is a sum over axes of one-dimensional operators
//     A = A_x (x) I (x) I + I (x) A_y (x) I + I (x) I (x) A_z,
// because the gradient's shell mask along an axis only depends on the
// coordinate along that axis for the rows that matter.  Each 1-D operator is
// 1/(4h^2) times a matrix that couples index i to i+-2 only, i.e. two
// independent tridiagonal chains (even and odd grid indices) with -1
// off-diagonals, 2 on the diagonal, and 1 at a chain end that sits on grid
// index 1 or n-2 (the gradient term through the shell is dropped: a
// Neumann-like end) or 2 at an end next to the zero shell (Dirichlet).  The
// eigenvectors of such chains are the discrete sine / cosine bases, so
//     phi = Q_x Q_y Q_z  diag(1 / (lx_i + ly_j + lz_k))  Q_z^T Q_y^T Q_x^T rhs
// solves the problem exactly (pseudo-inverse on the constant modes of the
// all-Neumann sub-lattices, which is the solution CG converges to).
//
// The mixed form uses this exact solve in FP64: ~6 dense per-axis transforms
// instead of hundreds of CG iterations.  The plain FP64 form keeps the CG,
// whose truncated iterate is what the reference returns.
#include <math.h>

#include <algorithm>
#include <vector>

#include "sw_common.cuh"
#include "sw_project.cuh"

namespace sw {

// ---------------------------------------------------------------------------
// basis of one axis (host, closed form)
// ---------------------------------------------------------------------------
// Q (m x m, row-major Q[i*m + k]: interior index i = grid index i+1, mode k)
// and lam[k] (physical eigenvalues, 1/(4 h^2) included).  The interior
// indices form two chains, the even grid indices (columns 0..K0-1) and the
// odd ones (columns K0..); an entry is non-zero only where its row and
// column lie on the same chain.  One entry at a time, so that the host entry
// point and the device kernel share the formulas; `lam` (when not null)
// receives the column's eigenvalue.
__host__ __device__ inline double basis_entry(int n, double h, int row, int col, double* lam) {
  const int first0 = 2, first1 = 1;
  const int K0 = first0 > n - 2 ? 0 : (n - 2 - first0) / 2 + 1;
  const int par = col < K0 ? 0 : 1;
  const int first = par == 0 ? first0 : first1;
  const int k = par == 0 ? col : col - K0;
  const int last = first + 2 * ((n - 2 - first) / 2);
  const int K = (last - first) / 2 + 1;
  const bool nf = (first == 1), nl = (last == n - 2);  // Neumann-like ends
  if (lam != nullptr) {
    double lk;
    if (nf && nl) lk = 2.0 - 2.0 * cos(k * M_PI / K);
    else if (!nf && !nl) lk = 2.0 - 2.0 * cos((k + 1.0) * M_PI / (K + 1));
    else lk = 2.0 - 2.0 * cos((k + 0.5) * M_PI / (K + 0.5));
    *lam = lk * (1.0 / (4.0 * h * h));
  }
  const int gi = row + 1;  // grid index of the row
  if ((gi & 1) != (first & 1)) return 0.0;
  const int j = (gi - first) / 2;  // chain position
  if (nf && nl) {                  // N-N: cosines, k = 0..K-1
    const double c = (k == 0) ? sqrt(1.0 / K) : sqrt(2.0 / K);
    return c * cos((j + 0.5) * k * M_PI / K);
  }
  if (!nf && !nl)  // D-D: sines, k = 1..K
    return sqrt(2.0 / (K + 1)) * sin((j + 1.0) * (k + 1.0) * M_PI / (K + 1));
  const int jj = nf ? j : (K - 1 - j);  // one Neumann end: distance from it
  return sqrt(2.0 / (K + 0.5)) * cos((jj + 0.5) * (k + 0.5) * M_PI / (K + 0.5));
}

// One axis of the solve: its two chains (0: even grid indices, 1: odd ones),
// chain position j at grid index first + 2 j.  Mode k of a chain is stored at
// the grid index of position k, so every transform has one form,
//     out[first + 2 a] = sum_b W[b][a] in[first + 2 b],
// with W = Q forward and Q^T back (both K x K, row-major).
struct AxisBasis {
  double* W[2][2];  // [forward 0 / inverse 1][chain]
  double* lam;      // eigenvalue of the mode at grid index i, at i - 1
  int K[2];
};
__host__ __device__ inline int chain_first(int par) { return par == 0 ? 2 : 1; }
__host__ __device__ inline int chain_len(int n, int par) {
  const int first = chain_first(par);
  return first > n - 2 ? 0 : (n - 2 - first) / 2 + 1;
}

// The solve builds its bases on the device, one thread per entry of the two
// chains' matrices (the host would spend ~1 ms per solve on the cosines, with
// the GPU waiting).
__global__ void axis_basis_kernel(int n, double h, AxisBasis ax) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long n0 = (long long)ax.K[0] * ax.K[0];
  const int par = e < n0 ? 0 : 1;
  const long long q = par ? e - n0 : e;
  const int K = ax.K[par];
  if (q >= (long long)K * K) return;
  const int j = (int)(q / K), k = (int)(q % K);
  const int row = chain_first(par) + 2 * j - 1;  // interior index of the position
  const int col = par ? ax.K[0] + k : k;
  double lam;
  const double v = basis_entry(n, h, row, col, j == 0 ? &lam : nullptr);
  ax.W[0][par][(long long)j * K + k] = v;
  ax.W[1][par][(long long)k * K + j] = v;
  if (j == 0) ax.lam[chain_first(par) + 2 * k - 1] = lam;
}

// ---------------------------------------------------------------------------
// one-axis transforms in FP64
// ---------------------------------------------------------------------------
// A basis couples cells of one parity only, so an axis of n cells is two
// products with matrices of n/2 rows: half the multiply-adds of one n x n
// product.  What bounds them is the FP64 rate (64 multiply-adds per cycle and
// SM).  A warp owns 32 modes x 32 data columns as 16 m8n8k4 products on the
// FP64 matrix unit (eight 8-byte shared loads per 16 products; with fused
// multiply-adds, 8 x 4 accumulators a thread, half the instructions were not
// multiply-adds), operands come through a three-stage cp.async ring 16 deep.
// A block takes WM units of 32 modes: a chain of up to 128 modes reads its
// data once and pads its modes to a multiple of 32 only.  Measured: 64 x 64
// tiles of the full n x n matrices with 8-byte loads and no pipeline, then
// multiply-adds on the chains, then this: the six transforms of a 160 x 131 x
// 173 grid 1154, 339, 246 us (whole projection 1406, 523, 390 us), the 48 of
// eight 256 x 256 x 384 forces 75.4, 21.0, 15.0 ms (axes x and y at 28
// TFLOP/s of the multiply-adds a chain needs, axis z at 20).
constexpr int SG_K = 16, SG_STAGES = 3;
constexpr int SG_PAD = 8;  // rows 64 bytes apart modulo 128: the four depths of a fragment
// Resident blocks per SM that the registers are held to: 16 to 18 warps (a
// multiply-add's latency is covered by a thread's 32 accumulators; more warps
// cover the copies and barriers).  Shared memory leaves spec_rows 5, 4, 3, 2
// blocks (10 to 18 warps) for WM 1 to 4, and spec_lines, whose rings hold both
// chains, 4, 2, 2, 1 (8 to 12 warps).
#define SG_BLOCKS(WM) ((WM) == 1 ? 8 : (WM) == 2 ? 4 : (WM) == 3 ? 3 : 2)

__device__ __forceinline__ void cp_async8(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(ok ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A warp's 32 (modes) x 32 (data) tile of products for one 16-deep chunk on
// the FP64 matrix unit: w[b * LDW + mode], data column n of depth b at
// d[n * dn + b * db].  acc[i][j]: modes 8 i + lane / 4, data 8 j + 2 (lane % 4)
// and the next.
template <int LDW>
__device__ __forceinline__ void mma_chunk(const double* __restrict__ w,
                                          const double* __restrict__ d, int dn, int db,
                                          double (&acc)[4][4][2], int lane) {
  const double* wp = w + (lane & 3) * LDW + (lane >> 2);
  const double* dp = d + (lane & 3) * db + (lane >> 2) * dn;
#pragma unroll
  for (int kk = 0; kk < SG_K; kk += 4) {
    double a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = wp[kk * LDW + 8 * i];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = dp[kk * db + 8 * j * dn];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
            : "+d"(acc[i][j][0]), "+d"(acc[i][j][1])
            : "d"(a[i]), "d"(b[j]));
  }
}

// Rows b0 .. b0+15 of a chain's matrix, columns a0 .. a0+32 WM-1 (zero
// outside the matrix), by the 64 WM threads of a block: a thread keeps its
// column and copies every other row.
template <int WM>
__device__ __forceinline__ void load_w(double* __restrict__ ws, const double* __restrict__ W,
                                       int K, int b0, int a0, int tid) {
  constexpr int N = 32 * WM, LD = N + SG_PAD;
  const int half = tid >= N ? 1 : 0, a = tid - half * N;
  const bool col = a0 + a < K;
  const double* src = W + (long long)(b0 + half) * K + a0 + a;
  double* dst = ws + half * LD + a;
#pragma unroll
  for (int kk = 0; kk < SG_K; kk += 2) {
    const bool ok = col && (unsigned)(b0 + half + kk) < (unsigned)K;
    cp_async8(dst + kk * LD, ok ? src : W, ok);
    src += 2 * K;
  }
}

// Axes x and y: rows of the padded field are `rs` apart; the data columns are
// numbered n, `nper` of them contiguous and then `nstride` on (axis x: one
// run of a whole plane; axis y: the z rows of all interior planes).  nper is
// even, so the 16-byte pieces never straddle two runs.
template <int WM>
__global__ void __launch_bounds__(64 * WM, SG_BLOCKS(WM))
    spec_rows(AxisBasis ax, int inverse, const double* __restrict__ src, double* __restrict__ dst,
              long long rs, int nper, long long nstride, long long ntot) {
  constexpr int LDW = 32 * WM + SG_PAD, LDD = 64 + SG_PAD;
  extern __shared__ __align__(16) double smem[];
  double* wsm = smem;                               // [stage][16][32 WM + 8]
  double* dsm = smem + SG_STAGES * SG_K * LDW;      // [stage][16][64 + 8]
  const int par = blockIdx.z, K = ax.K[par];
  const int a0 = blockIdx.y * 32 * WM;
  if (a0 >= K) return;
  const double* W = ax.W[inverse][par];
  const long long n0 = blockIdx.x * 64ll;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = warp % WM, wn = warp / WM;
  const double* base = src + chain_first(par) * rs;
  // pieces of two columns: this thread copies piece tid % 32 of some rows
  const long long pn = n0 + 2 * (tid & 31);
  const bool pok = pn < ntot;
  const long long poff = pok ? (pn / nper) * nstride + pn % nper : 0;
  auto load = [&](int st, int b0) {
    load_w<WM>(wsm + st * SG_K * LDW, W, K, b0, a0, tid);
    const int k0 = tid >> 5;
    const double* p = base + 2 * (b0 + k0) * rs + poff;
    double* d = dsm + (st * SG_K + k0) * LDD + 2 * (tid & 31);
#pragma unroll
    for (int kk = 0; kk < SG_K; kk += 2 * WM) {
      if (k0 + kk >= SG_K) break;
      const bool ok = pok && b0 + k0 + kk < K;
      cp_async16(d + kk * LDD, ok ? p : src, ok);
      p += 4ll * WM * rs;
    }
  };
  double acc[4][4][2] = {};
  const int nk = (K + SG_K - 1) / SG_K;
#pragma unroll
  for (int st = 0; st < SG_STAGES - 1; ++st) {
    if (st < nk) load(st, st * SG_K);
    cp_async_commit();
  }
  for (int c = 0; c < nk; ++c) {
    cp_async_wait<SG_STAGES - 2>();
    __syncthreads();
    const int nx = c + SG_STAGES - 1;
    if (nx < nk) load(nx % SG_STAGES, nx * SG_K);
    cp_async_commit();
    mma_chunk<LDW>(wsm + (c % SG_STAGES) * SG_K * LDW + wm * 32,
                   dsm + (c % SG_STAGES) * SG_K * LDD + wn * 32, 1, LDD, acc, lane);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const long long n = n0 + wn * 32 + 8 * j + 2 * (lane & 3);
    if (n >= ntot) continue;
    double* out = dst + (n / nper) * nstride + n % nper;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int a = a0 + wm * 32 + 8 * i + (lane >> 2);
      if (a < K)
        *reinterpret_cast<double2*>(out + (chain_first(par) + 2ll * a) * rs) =
            make_double2(acc[i][j][0], acc[i][j][1]);
    }
  }
}

// Axis z: 32 lines (x, y) per block, both chains (the two halves of its
// warps), so each line is read and written in whole rows; the results pass
// through shared memory to leave in row order.  Lines are the interior
// (x, y).  With `scale` the results are divided by the eigenvalue sums (zero
// on the null modes), which ends the forward transforms.
template <int WM>
__global__ void __launch_bounds__(64 * WM, SG_BLOCKS(WM))
    spec_lines(AxisBasis ax, int inverse, const double* __restrict__ src,
               double* __restrict__ dst, Geom g, int scale, const double* __restrict__ lx,
               const double* __restrict__ ly, double lam_floor) {
  constexpr int THREADS = 64 * WM, LDW = 32 * WM + SG_PAD, LDD = 2 * SG_K + 2;
  constexpr int LDE = 64 * WM + 1;
  extern __shared__ __align__(16) double smem[];
  double* wsm = smem;                                // [stage][chain][16][32 WM + 8]
  double* dsm = smem + SG_STAGES * 2 * SG_K * LDW;   // [stage][32 lines][34]
  __shared__ long long loff[32];
  __shared__ double lsum[32];
  const int a0 = blockIdx.y * 32 * WM;
  const long long l0 = blockIdx.x * 32ll, nl = (long long)(g.nx - 2) * (g.ny - 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int par = warp / WM, wm = warp % WM;
  if (tid < 32) {
    const long long l = l0 + tid;
    const int x = (int)(l / (g.ny - 2)) + 1, y = (int)(l % (g.ny - 2)) + 1;
    loff[tid] = l < nl ? x * g.sxy + (long long)y * g.pz : -1;
    lsum[tid] = scale && l < nl ? lx[x - 1] + ly[y - 1] : 0.0;
  }
  __syncthreads();
  // 16-byte pieces: 16 per line, THREADS / 16 lines at a time
  auto load = [&](int st, int c) {
#pragma unroll
    for (int p = 0; p < 2; ++p)  // z = 32 c + 2 t: even chain position 16 c + t - 1
      load_w<WM>(wsm + (st * 2 + p) * SG_K * LDW, ax.W[inverse][p], ax.K[p],
                          c * SG_K - (p == 0 ? 1 : 0), a0, tid);
    const int z = 2 * SG_K * c + 2 * (tid & 15);
    for (int l = tid >> 4; l < 32; l += THREADS / 16) {
      const bool ok = loff[l] >= 0 && z < g.pz;
      cp_async16(dsm + (st * 32 + l) * LDD + 2 * (tid & 15), ok ? src + loff[l] + z : src, ok);
    }
  };
  double acc[4][4][2] = {};
  const int nk = (g.nz - 1 + 2 * SG_K - 1) / (2 * SG_K);  // z = 0 .. nz-2
#pragma unroll
  for (int st = 0; st < SG_STAGES - 1; ++st) {
    if (st < nk) load(st, st);
    cp_async_commit();
  }
  for (int c = 0; c < nk; ++c) {
    cp_async_wait<SG_STAGES - 2>();
    __syncthreads();
    const int nx = c + SG_STAGES - 1;
    if (nx < nk) load(nx % SG_STAGES, nx);
    cp_async_commit();
    mma_chunk<LDW>(wsm + ((c % SG_STAGES) * 2 + par) * SG_K * LDW + wm * 32,
                   dsm + (c % SG_STAGES) * 32 * LDD + (par == 0 ? 0 : 1), LDD, 2, acc, lane);
  }
  cp_async_wait<0>();
  __syncthreads();  // the ring is free: rows of results take its place
  // odd chain's mode a at z = 1 + 2 a, even chain's at 2 + 2 a
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int u = 0; u < 2; ++u)
        smem[(8 * j + 2 * (lane & 3) + u) * LDE + 2 * (wm * 32 + 8 * i + (lane >> 2)) +
             (par == 0 ? 1 : 0)] = acc[i][j][u];
  __syncthreads();
  const int z0 = 1 + 2 * a0, zn = min(64 * WM, g.nz - 2 + 1 - z0);
  for (int l = warp; l < 32; l += THREADS / 32) {
    if (loff[l] < 0) continue;
    for (int r = lane; r < zn; r += 32) {
      double v = smem[l * LDE + r];
      if (scale) {
        const double L = lsum[l] + ax.lam[z0 + r - 1];
        v = L > lam_floor ? v / L : 0.0;
      }
      dst[loff[l] + z0 + r] = v;
    }
  }
}

// Units of 32 modes per block for a chain of K modes: all of them up to four,
// else the count whose blocks pad the modes least.
static int mode_units(int K) {
  const int u = std::max(1, (K + 31) / 32);
  if (u <= 4) return u;
  int best = 4;
  for (int w = 3; w >= 2; --w)
    if ((u + w - 1) / w * w < (u + best - 1) / best * best) best = w;
  return best;
}

constexpr size_t spec_rows_smem(int wm) {
  return sizeof(double) * SG_STAGES * SG_K * (32 * wm + SG_PAD + 64 + SG_PAD);
}
constexpr size_t spec_lines_smem(int wm) {
  const size_t ring = sizeof(double) * SG_STAGES * (2 * SG_K * (32 * wm + SG_PAD) + 32 * (2 * SG_K + 2));
  const size_t rows = sizeof(double) * 32 * (64 * wm + 1);
  return ring > rows ? ring : rows;
}

template <int WM>
static int launch_axis(const Geom& g, int axis, const AxisBasis& ax, bool inverse,
                       const double* src, double* dst, bool scale, const double* lx,
                       const double* ly, double lam_floor, cudaStream_t s) {
  const int Kmax = std::max(ax.K[0], ax.K[1]);
  const unsigned mt = (unsigned)((Kmax + 32 * WM - 1) / (32 * WM));
  cudaError_t e;
  if (axis == 2) {
    const size_t sm = spec_lines_smem(WM);
    e = cudaFuncSetAttribute(spec_lines<WM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(spectral lines)");
    const long long nl = (long long)(g.nx - 2) * (g.ny - 2);
    spec_lines<WM><<<dim3((unsigned)((nl + 31) / 32), mt), 64 * WM, sm, s>>>(
        ax, inverse ? 1 : 0, src, dst, g, scale ? 1 : 0, lx, ly, lam_floor);
  } else {
    const size_t sm = spec_rows_smem(WM);
    e = cudaFuncSetAttribute(spec_rows<WM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(spectral rows)");
    const long long ntot = axis == 0 ? g.sxy : (long long)(g.nx - 2) * g.pz;
    const dim3 grid((unsigned)((ntot + 63) / 64), mt, 2);
    if (axis == 0)  // all (y, z) columns of the plane
      spec_rows<WM><<<grid, 64 * WM, sm, s>>>(ax, inverse ? 1 : 0, src, dst, g.sxy, (int)g.sxy, 0,
                                              ntot);
    else  // the z columns of every interior plane
      spec_rows<WM><<<grid, 64 * WM, sm, s>>>(ax, inverse ? 1 : 0, src + g.sxy, dst + g.sxy, g.pz,
                                              g.pz, g.sxy, ntot);
  }
  count_launches(1);
  SW_CHECK_LAUNCH("spectral transform");
  return SW_OK;
}

// Transform along `axis` (0 x, 1 y, 2 z) of the interior of the padded field
// src into dst.
static int axis_transform(const Geom& g, int axis, const AxisBasis& ax, bool inverse,
                          const double* src, double* dst, bool scale, const double* lx,
                          const double* ly, double lam_floor, cudaStream_t s) {
  switch (mode_units(std::max(ax.K[0], ax.K[1]))) {
    case 1: return launch_axis<1>(g, axis, ax, inverse, src, dst, scale, lx, ly, lam_floor, s);
    case 2: return launch_axis<2>(g, axis, ax, inverse, src, dst, scale, lx, ly, lam_floor, s);
    case 3: return launch_axis<3>(g, axis, ax, inverse, src, dst, scale, lx, ly, lam_floor, s);
    default: return launch_axis<4>(g, axis, ax, inverse, src, dst, scale, lx, ly, lam_floor, s);
  }
}

size_t spectral_extra_bytes(const Geom& g) {
  size_t b = 0;
  const int ns[3] = {g.nx, g.ny, g.nz};
  for (int a = 0; a < 3; ++a) {
    const size_t m = ns[a] > 2 ? ns[a] - 2 : 1;
    b += align_up(m * m * sizeof(double), 256) + align_up(m * sizeof(double), 256);
  }
  return b;
}

}  // namespace sw

using namespace sw;

namespace {

// Blocks of 32 (z) x 8 (y) threads over the padded cells, a few x planes per
// block: no division per cell, and the shell and padding are written here
// too, so neither the rhs nor the output is cleared beforehand.
constexpr int kSpecPlanes = 8;
dim3 spec_grid(const Geom& g) {
  return dim3((unsigned)((g.pz + TILE_Z - 1) / TILE_Z), (unsigned)((g.ny + TILE_Y - 1) / TILE_Y),
              (unsigned)((g.nx + kSpecPlanes - 1) / kSpecPlanes));
}

// rhs = -div_c(mask f) on interior cells (the CG's r0), 0 elsewhere; also max |div|
template <typename T>
__global__ void __launch_bounds__(TILE_THREADS)
    prep_rhs(const T* __restrict__ fx, const T* __restrict__ fy, const T* __restrict__ fz,
             InStride s, Geom g, double c2x, double c2y, double c2z, double* __restrict__ rhs,
             double* __restrict__ maxdiv) {
  __shared__ double red[32];
  double mx = 0.0;
  const int z = blockIdx.x * TILE_Z + threadIdx.x, y = blockIdx.y * TILE_Y + threadIdx.y;
  const int x0 = blockIdx.z * kSpecPlanes, x1 = min(x0 + kSpecPlanes, g.nx);
  if (z < g.pz && y < g.ny) {
    double* out = rhs + (long long)x0 * g.sxy + (long long)y * g.pz + z;
    if (y >= 1 && y <= g.ny - 2 && z >= 1 && z <= g.nz - 2) {
      // masked neighbours: those on the shell count as 0
      const bool yp = y + 1 <= g.ny - 2, ym = y - 1 >= 1, zp = z + 1 <= g.nz - 2, zm = z - 1 >= 1;
      const long long f0 = (long long)y * s.sy + (long long)z * s.sz;
      auto at = [&](const T* f, int x, long long off, bool in) -> double {
        return f != nullptr && in ? (double)f[(long long)x * s.sx + f0 + off] : 0.0;
      };
      auto fx_at = [&](int x) -> double { return at(fx, x, 0, x >= 1 && x <= g.nx - 2); };
      double xm = fx_at(x0 - 1), xc = fx_at(x0);
      for (int x = x0; x < x1; ++x, out += g.sxy) {
        const double xp = fx_at(x + 1);
        double div = 0.0;
        if (x >= 1 && x <= g.nx - 2) {
          const double tx = (xp - xm) * c2x;
          const double ty = (at(fy, x, s.sy, yp) - at(fy, x, -s.sy, ym)) * c2y;
          const double tz = (at(fz, x, s.sz, zp) - at(fz, x, -s.sz, zm)) * c2z;
          div = (tx + ty) + tz;
          mx = fmax(mx, fabs(div));
        }
        *out = -div;
        xm = xc;
        xc = xp;
      }
    } else {
      for (int x = x0; x < x1; ++x, out += g.sxy) *out = 0.0;
    }
  }
  // block max, then one atomic per block that raises it, on the bit pattern
  // (non-negative doubles)
  mx = block_max(mx, red);
  if (flat_tid() == 0 && mx > *(volatile double*)maxdiv)
    atomicMax((unsigned long long*)maxdiv, (unsigned long long)__double_as_longlong(mx));
}

// out = mask f - grad_c phi on interior cells (phi null: mask f), 0 elsewhere
template <typename T>
__global__ void __launch_bounds__(TILE_THREADS)
    finish_spectral(const T* __restrict__ fx, const T* __restrict__ fy, const T* __restrict__ fz,
                    InStride s, Geom g, double c2x, double c2y, double c2z,
                    const double* __restrict__ phi, double* __restrict__ out) {
  const int z = blockIdx.x * TILE_Z + threadIdx.x, y = blockIdx.y * TILE_Y + threadIdx.y;
  const int x0 = blockIdx.z * kSpecPlanes, x1 = min(x0 + kSpecPlanes, g.nx);
  if (z >= g.pz || y >= g.ny) return;
  for (int x = x0; x < x1; ++x) {
    const long long i = (long long)x * g.sxy + (long long)y * g.pz + z;
    double ox = 0.0, oy = 0.0, oz = 0.0;
    if (interior(g, x, y, z)) {
      const long long f = (long long)x * s.sx + (long long)y * s.sy + (long long)z * s.sz;
      double gx = 0.0, gy = 0.0, gz = 0.0;
      if (phi) {
        gx = (phi[i + g.sxy] - phi[i - g.sxy]) * c2x;
        gy = (phi[i + g.pz] - phi[i - g.pz]) * c2y;
        gz = (phi[i + 1] - phi[i - 1]) * c2z;
      }
      ox = (fx ? (double)fx[f] : 0.0) - gx;
      oy = (fy ? (double)fy[f] : 0.0) - gy;
      oz = (fz ? (double)fz[f] : 0.0) - gz;
    }
    out[i] = ox;
    out[i + g.ncell] = oy;
    out[i + 2 * g.ncell] = oz;
  }
}

template <typename T>
int spectral_one(const void* fx, const void* fy, const void* fz, InStride fs, const Geom& g,
                 double dX, double dY, double dZ, double* out, char* ws, size_t ws_bytes,
                 sw_cg_stats* stats, cudaStream_t s) {
  const size_t vec = align_up((size_t)g.ncell * sizeof(double), 256);
  // (the last 256 bytes: the maximum, and the room of align_workspace)
  const size_t need = 3 * vec + spectral_extra_bytes(g) + 256;
  static_assert(sizeof(double) + kWorkspaceAlign - 1 <= 256, "no room for align_workspace");
  if (ws == nullptr || ws_bytes < need) {
    set_error("spectral workspace of %zu bytes is smaller than the %zu bytes required", ws_bytes,
              need);
    return SW_EWORKSPACE;
  }
  ws = align_workspace(ws);
  double* v0 = (double*)ws;
  double* v1 = (double*)(ws + vec);
  double* v2 = (double*)(ws + 2 * vec);
  char* p = ws + 3 * vec;
  const int ns[3] = {g.nx, g.ny, g.nz};
  const double hs[3] = {dX, dY, dZ};
  const bool has_interior = g.nx > 2 && g.ny > 2 && g.nz > 2;
  if (!has_interior) {
    if (cudaError_t e = cudaMemsetAsync(out, 0, (size_t)g.ncell * 3 * sizeof(double), s))
      return cuda_status(e, "spectral setup");
    if (stats) *stats = sw_cg_stats{0, SW_CG_EARLY_EXIT, 0.0, 0.0};
    return SW_OK;
  }
  AxisBasis ax[3];
  for (int a = 0; a < 3; ++a) {
    const int m = ns[a] - 2;
    // the four chain matrices take at most m^2 + 1 values; m^2 + 1 > m^2 only
    // for odd m, whose m^2 values leave room below the 256-byte boundary
    double* q = (double*)p;
    for (int par = 0; par < 2; ++par) ax[a].K[par] = chain_len(ns[a], par);
    for (int dir = 0; dir < 2; ++dir)
      for (int par = 0; par < 2; ++par) {
        ax[a].W[dir][par] = q;
        q += (size_t)ax[a].K[par] * ax[a].K[par];
      }
    p += align_up((size_t)m * m * sizeof(double), 256);
    ax[a].lam = (double*)p;
    p += align_up((size_t)m * sizeof(double), 256);
    const long long cnt =
        (long long)ax[a].K[0] * ax[a].K[0] + (long long)ax[a].K[1] * ax[a].K[1];
    axis_basis_kernel<<<(unsigned)((cnt + 255) / 256), 256, 0, s>>>(ns[a], hs[a], ax[a]);
    count_launches(1);
    SW_CHECK_LAUNCH("spectral basis");
  }
  double* d_max = (double*)p;
  cudaError_t e = cudaMemsetAsync(d_max, 0, sizeof(double), s);
  if (e != cudaSuccess) return cuda_status(e, "spectral setup");
  double maxdiv = 0.0;
  const double c2x = 1.0 / (2.0 * dX), c2y = 1.0 / (2.0 * dY), c2z = 1.0 / (2.0 * dZ);
  const dim3 blk(TILE_Z, TILE_Y);
  prep_rhs<T><<<spec_grid(g), blk, 0, s>>>((const T*)fx, (const T*)fy, (const T*)fz, fs, g, c2x,
                                           c2y, c2z, v0, d_max);
  count_launches(1);
  SW_CHECK_LAUNCH("spectral prep");
  e = cudaMemcpyAsync(&maxdiv, d_max, sizeof(double), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_status(e, "spectral readback");
  const bool solve = !(maxdiv < 1e-12);
  if (solve) {
    // v0 -x-> v1 -y-> v2 -z-> v1 (scaled) -z-> v2 -y-> v1 -x-> v0.  Shell cells
    // stay zero throughout without being cleared: axis x writes whole planes
    // (from v0's zero shell), axis y whole rows, axis z the interior of lines
    // whose ends axis x or y wrote; v0 keeps the shell planes of the rhs.
    double lmax = 0.0;
    for (int a = 0; a < 3; ++a) lmax += 4.0 / (hs[a] * hs[a]);
    const double fl = 1e-13 * lmax;
    struct {
      int axis;
      bool inverse, scale;
      const double* src;
      double* dst;
    } const steps[6] = {{0, false, false, v0, v1}, {1, false, false, v1, v2},
                        {2, false, true, v2, v1},  {2, true, false, v1, v2},
                        {1, true, false, v2, v1},  {0, true, false, v1, v0}};
    for (const auto& t : steps) {
      const int rc = axis_transform(g, t.axis, ax[t.axis], t.inverse, t.src, t.dst, t.scale,
                                    ax[0].lam, ax[1].lam, fl, s);
      if (rc != SW_OK) return rc;
    }
  }
  finish_spectral<T><<<spec_grid(g), blk, 0, s>>>((const T*)fx, (const T*)fy, (const T*)fz, fs, g,
                                                  c2x, c2y, c2z, solve ? v0 : nullptr, out);
  count_launches(1);
  SW_CHECK_LAUNCH("spectral finish");
  if (stats) {
    stats->iters = 0;
    stats->reason = solve ? SW_CG_CONVERGED : SW_CG_EARLY_EXIT;
    stats->rel = 0.0;
    stats->max_div = maxdiv;
  }
  return SW_OK;
}

}  // namespace

extern "C" size_t sw_project_spectral_workspace_bytes(int nx, int ny, int nz) {
  if (nx <= 0 || ny <= 0 || nz <= 0) return 0;
  Geom g = make_geom(nx, ny, nz, pad_pitch(nz));
  return 3 * align_up((size_t)g.ncell * sizeof(double), 256) + spectral_extra_bytes(g) + 256;
}

extern "C" int sw_project_spectral(int in_dtype, const void* fx, const void* fy, const void* fz,
                                   int64_t in_sx, int64_t in_sy, int64_t in_sz, int nx, int ny,
                                   int nz, double dX, double dY, double dZ, double* out,
                                   void* workspace, size_t workspace_bytes, sw_cg_stats* stats,
                                   void* stream) {
  if (nx <= 0 || ny <= 0 || nz <= 0 || out == nullptr || !(dX > 0 && dY > 0 && dZ > 0)) {
    set_error("sw_project_spectral: bad grid, spacing or null output");
    return SW_EINVAL;
  }
  Geom g = make_geom(nx, ny, nz, pad_pitch(nz));
  InStride fs{in_sx, in_sy, in_sz};
  cudaStream_t s = (cudaStream_t)stream;
  if (in_dtype == SW_F32)
    return spectral_one<float>(fx, fy, fz, fs, g, dX, dY, dZ, out, (char*)workspace,
                               workspace_bytes, stats, s);
  if (in_dtype == SW_F64)
    return spectral_one<double>(fx, fy, fz, fs, g, dX, dY, dZ, out, (char*)workspace,
                                workspace_bytes, stats, s);
  set_error("sw_project_spectral: unknown dtype %d", in_dtype);
  return SW_EINVAL;
}

extern "C" int sw_spectral_basis(int n, double h, double* Q, double* lam) {
  if (n < 3 || !(h > 0) || Q == nullptr || lam == nullptr) {
    set_error("sw_spectral_basis: need n >= 3, h > 0 and host buffers");
    return SW_EINVAL;
  }
  const int m = n - 2;
  for (int row = 0; row < m; ++row)
    for (int col = 0; col < m; ++col)
      Q[(size_t)row * m + col] = basis_entry(n, h, row, col, row == 0 ? lam + col : nullptr);
  return SW_OK;
}
