// Collocated FD operators and the strain post-pass.
//
// Reference: laplacian_center / divergence_center / gradient_center
// (src/shearwave/solver.py:686-729), compute_strain_tensor and
// compute_strain_invariants (src/shearwave/strain.py:16-135).
//
// These kernels reproduce numpy's elementwise rounding: every operation is a
// separately rounded IEEE operation in the array dtype (no FMA contraction,
// true division by the same divisor numpy uses), so their outputs equal the
// reference's bit for bit in float32 and float64.  One exception: where the
// second invariant is NaN (a strain that overflowed), max_shear is 0; numpy's
// maximum keeps the NaN, as the other invariants do here too.
#include <math.h>

#include <algorithm>
#include <cmath>

#include "sw_common.cuh"

namespace sw {

template <typename T>
struct Ar;
template <>
struct Ar<float> {
  static __device__ inline float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ inline float sub(float a, float b) { return __fsub_rn(a, b); }
  static __device__ inline float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ inline float div(float a, float b) { return __fdiv_rn(a, b); }
  static __device__ inline float sqrt_(float a) { return __fsqrt_rn(a); }
};
template <>
struct Ar<double> {
  static __device__ inline double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ inline double sub(double a, double b) { return __dsub_rn(a, b); }
  static __device__ inline double mul(double a, double b) { return __dmul_rn(a, b); }
  static __device__ inline double div(double a, double b) { return __ddiv_rn(a, b); }
  static __device__ inline double sqrt_(double a) { return __dsqrt_rn(a); }
};

// Division by a constant, correctly rounded.  With r = RN(1/b), a
// faithful quotient q and the exact remainder a - b q, RN(q + (a - b q) r) is
// RN(a / b) (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", 1990); the first correction makes a r faithful.
// Five multiply-adds instead of a division subroutine, for quotients and
// remainders well inside the exponent range (`fast`, |a| in [lo, hi]);
// anything else but a zero is divided.
template <typename T>
struct ConstDiv {
  T b, r;
  int fast;
};
template <typename T>
struct DivRange;
template <>
struct DivRange<float> {
  static constexpr float lo = 0x1p-80f, hi = 0x1p80f, b_lo = 0x1p-40f, b_hi = 0x1p40f;
};
template <>
struct DivRange<double> {
  static constexpr double lo = 0x1p-800, hi = 0x1p800, b_lo = 0x1p-100, b_hi = 0x1p100;
};
template <typename T>
__host__ __device__ inline ConstDiv<T> const_div(T b) {
  return ConstDiv<T>{b, T(1) / b, b >= DivRange<T>::b_lo && b <= DivRange<T>::b_hi};
}
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) {
  return __fma_rn(a, b, c);
}
// The multiply-add sequence (the sign is a's, which it would lose of a -0).
template <typename T>
__device__ __forceinline__ T div_fast(T a, const ConstDiv<T>& d) {
  T q = Ar<T>::mul(a, d.r);
  q = fma_rn(fma_rn(-d.b, q, a), d.r, q);
  return copysign(fma_rn(fma_rn(-d.b, q, a), d.r, q), a);
}
template <typename T>
__device__ __forceinline__ T div_const(T a, const ConstDiv<T>& d) {
  const T m = fabs(a);
  if (d.fast && (a == T(0) || (m >= DivRange<T>::lo && m <= DivRange<T>::hi)))
    return div_fast(a, d);
  return Ar<T>::div(a, d.b);
}

// Whether every value of a set is a zero or in the sequence's range: the
// largest magnitude, and the smallest one that is not zero (a magnitude's bits
// less one, which puts zero last).
struct RangeF {
  float hi = 0.f;
  unsigned lo = 0xffffffffu;
  __device__ __forceinline__ void add(float a) {
    hi = fmaxf(hi, fabsf(a));
    lo = min(lo, (__float_as_uint(a) & 0x7fffffffu) - 1u);
  }
  __device__ __forceinline__ bool ok() const {
    return hi <= DivRange<float>::hi && lo >= __float_as_uint(DivRange<float>::lo) - 1u;
  }
};
struct RangeD {  // by the high words: exponent and the top of the mantissa
  unsigned hi = 0u, lo = 0xffffffffu;
  __device__ __forceinline__ void add(double a) {
    const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
    hi = max(hi, h);
    // a zero goes last; a subnormal with a zero high word counts as small
    lo = min(lo, a == 0.0 ? 0xffffffffu : h);
  }
  __device__ __forceinline__ bool ok() const {
    return hi < (unsigned)__double2hiint(DivRange<double>::hi) &&
           lo >= (unsigned)__double2hiint(DivRange<double>::lo);
  }
};
__device__ __forceinline__ RangeF range_of(float) { return RangeF(); }
__device__ __forceinline__ RangeD range_of(double) { return RangeD(); }

// A dense (nx, ny, nz) grid, z fastest.  The stencil kernels give each
// thread one (z, y) column of a 32 x 8 block and walk x across the grid's z
// dimension of blocks, so a cell's coordinates cost no division.
constexpr int kCellBlockZ = 32, kCellBlockY = 8;
struct Dense {
  int nx, ny, nz;
  __device__ inline bool inner(int x, int y, int z) const {
    return x >= 1 && y >= 1 && z >= 1 && x <= nx - 2 && y <= ny - 2 && z <= nz - 2;
  }
};

template <typename T>
__global__ void laplacian_kernel(const T* __restrict__ f, T* __restrict__ out, Dense d,
                                 ConstDiv<T> hx2, ConstDiv<T> hy2, ConstDiv<T> hz2) {
  using A = Ar<T>;
  const long long sx = (long long)d.ny * d.nz, sy = d.nz;
  const int z = blockIdx.x * kCellBlockZ + threadIdx.x, y = blockIdx.y * kCellBlockY + threadIdx.y;
  if (z >= d.nz || y >= d.ny) return;
  for (int x = blockIdx.z; x < d.nx; x += gridDim.z) {
    {
      const long long q = ((long long)x * d.ny + y) * d.nz + z;
      T r = T(0);
      if (d.inner(x, y, z)) {
        const T c2 = A::mul(T(2), f[q]);
        const T tx = div_const(A::add(A::sub(f[q + sx], c2), f[q - sx]), hx2);
        const T ty = div_const(A::add(A::sub(f[q + sy], c2), f[q - sy]), hy2);
        const T tz = div_const(A::add(A::sub(f[q + 1], c2), f[q - 1]), hz2);
        r = A::add(A::add(tx, ty), tz);
      }
      out[q] = r;
    }
  }
}

template <typename T>
__global__ void divergence_kernel(const T* __restrict__ fx, const T* __restrict__ fy,
                                  const T* __restrict__ fz, T* __restrict__ out, Dense d,
                                  ConstDiv<T> h2x, ConstDiv<T> h2y, ConstDiv<T> h2z) {
  using A = Ar<T>;
  const long long sx = (long long)d.ny * d.nz, sy = d.nz;
  const int z = blockIdx.x * kCellBlockZ + threadIdx.x, y = blockIdx.y * kCellBlockY + threadIdx.y;
  if (z >= d.nz || y >= d.ny) return;
  for (int x = blockIdx.z; x < d.nx; x += gridDim.z) {
    {
      const long long q = ((long long)x * d.ny + y) * d.nz + z;
      T r = T(0);
      if (d.inner(x, y, z)) {
        const T tx = div_const(A::sub(fx[q + sx], fx[q - sx]), h2x);
        const T ty = div_const(A::sub(fy[q + sy], fy[q - sy]), h2y);
        const T tz = div_const(A::sub(fz[q + 1], fz[q - 1]), h2z);
        r = A::add(A::add(tx, ty), tz);
      }
      out[q] = r;
    }
  }
}

template <typename T>
__global__ void gradient_kernel(const T* __restrict__ p, T* __restrict__ gx, T* __restrict__ gy,
                                T* __restrict__ gz, Dense d, ConstDiv<T> h2x,
                                ConstDiv<T> h2y, ConstDiv<T> h2z) {
  using A = Ar<T>;
  const long long sx = (long long)d.ny * d.nz, sy = d.nz;
  const int z = blockIdx.x * kCellBlockZ + threadIdx.x, y = blockIdx.y * kCellBlockY + threadIdx.y;
  if (z >= d.nz || y >= d.ny) return;
  for (int x = blockIdx.z; x < d.nx; x += gridDim.z) {
    {
      const long long q = ((long long)x * d.ny + y) * d.nz + z;
      T a = T(0), b = T(0), c = T(0);
      if (d.inner(x, y, z)) {
        a = div_const(A::sub(p[q + sx], p[q - sx]), h2x);
        b = div_const(A::sub(p[q + sy], p[q - sy]), h2y);
        c = div_const(A::sub(p[q + 1], p[q - 1]), h2z);
      }
      gx[q] = a;
      gy[q] = b;
      gz[q] = c;
    }
  }
}

// Invariants of one Voigt vector, in the reference's operation order
// (strain.py:110-128).  von Mises is float64: numpy multiplies the dtype
// `dev` by the float64 scalar sqrt(2/3) (`vm_c`).
template <typename T>
__device__ inline void invariants(const T e[6], const ConstDiv<T>& third, double vm_c, T& vol,
                                  T& dev, T& msh, double& vm) {
  using A = Ar<T>;
  vol = div_const(A::add(A::add(e[0], e[1]), e[2]), third);
  const T dxx = A::sub(e[0], vol), dyy = A::sub(e[1], vol), dzz = A::sub(e[2], vol);
  const T nrm = A::add(A::add(A::mul(dxx, dxx), A::mul(dyy, dyy)), A::mul(dzz, dzz));
  const T shr = A::mul(T(0.5), A::add(A::add(A::mul(e[3], e[3]), A::mul(e[4], e[4])),
                                      A::mul(e[5], e[5])));
  const T s = A::add(nrm, shr);
  dev = A::sqrt_(s);
  const T j2 = A::mul(T(0.5), s);
  msh = A::sqrt_(j2 > T(0) ? j2 : T(0));
  vm = __dmul_rn(vm_c, (double)dev);
}

// Pairs of elements, for whole-sector stores of the tensor.
template <typename T>
struct Pair;
template <>
struct Pair<float> {
  using type = float2;
};
template <>
struct Pair<double> {
  using type = double2;
};

// A warp owns a row of 32 cells and walks x over kStrainPlanes planes with
// its column in registers; the z neighbours come from the lanes either side,
// the rows either side from L1.  The tensor's six values per cell pass
// through shared memory and leave as whole rows (stored from the lanes, each
// 24-byte cell is six partial writes of its sectors).  What bounds it after
// that is instructions: the nine divisions per cell are multiply-adds with one
// range test (div_fast), a solver's displacement (AOS: the components next to
// each other) shares its addresses, and a call that wants the tensor and all
// invariants (ALL) tests no output pointer.  192^3 float fields: 107 us with
// divisions and a thread per cell, 93 with this walk (316 warp instructions per
// 32 cells; the bytes alone take 60).
constexpr int kStrainPlanes = 12;
template <typename T, bool PAIRS, bool AOS, bool ALL>
__global__ void __launch_bounds__(kCellBlockZ * kCellBlockY)
    strain_kernel(const T* __restrict__ ux, const T* __restrict__ uy, const T* __restrict__ uz,
                  long long sx, long long sy, long long sz, Dense d, ConstDiv<T> h2x,
                  ConstDiv<T> h2y, ConstDiv<T> h2z, ConstDiv<T> third, double vm_c, int planes,
                  T* __restrict__ eps, T* __restrict__ vol, T* __restrict__ dev,
                  T* __restrict__ msh, double* __restrict__ vm) {
  using A = Ar<T>;
  using P = typename Pair<T>::type;
  __shared__ P stage[kCellBlockY][kCellBlockZ * 3];
  const int lane = threadIdx.x;
  const int z0 = blockIdx.x * kCellBlockZ, z = z0 + lane;
  const int y = blockIdx.y * kCellBlockY + threadIdx.y;
  if (y >= d.ny) return;  // whole warps
  const int x0 = blockIdx.z * planes, x1 = min(x0 + planes, d.nx);
  const bool zin = z < d.nz, yin = y >= 1 && y <= d.ny - 2;
  const bool inner_zy = yin && z >= 1 && z <= d.nz - 2;
  const bool fast = h2x.fast && h2y.fast && h2z.fast;
  const long long i0 = x0 * sx + y * sy + z * sz;
  const T *cx = ux + i0, *cy = uy + i0, *cz = uz + i0;  // this cell; only read where zin
  auto at = [&](int a, long long off) -> T {
    return AOS ? (cx + off)[a] : (a == 0 ? cx : (a == 1 ? cy : cz))[off];
  };
  const unsigned plane = (unsigned)d.ny * (unsigned)d.nz;
  long long q = ((long long)x0 * d.ny + y) * d.nz + z;
  T m[3], c[3];  // this column at x - 1 and x
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    m[a] = zin && x0 > 0 ? at(a, -sx) : T(0);
    c[a] = zin ? at(a, 0) : T(0);
  }
  for (int x = x0; x < x1; ++x, q += plane) {
    T n[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) n[a] = zin && x + 1 < d.nx ? at(a, sx) : T(0);
    T e[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    if (yin && x >= 1 && x <= d.nx - 2) {  // uniform across the warp
      // g[a][b] = d u_a / d x_b, first its numerator
      T g[3][3];
      auto range = range_of(T(0));
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        T zl = __shfl_up_sync(0xffffffffu, c[a], 1), zr = __shfl_down_sync(0xffffffffu, c[a], 1);
        if (lane == 0 && inner_zy) zl = at(a, -sz);
        if (lane == 31 && inner_zy) zr = at(a, sz);
        const T yu = zin ? at(a, sy) : T(0), yd = zin ? at(a, -sy) : T(0);
        g[a][0] = A::sub(n[a], m[a]);
        g[a][1] = A::sub(yu, yd);
        g[a][2] = A::sub(zr, zl);
#pragma unroll
        for (int b = 0; b < 3; ++b) range.add(g[a][b]);
      }
      if (fast && range.ok()) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          g[a][0] = div_fast(g[a][0], h2x);
          g[a][1] = div_fast(g[a][1], h2y);
          g[a][2] = div_fast(g[a][2], h2z);
        }
      } else {
#pragma unroll 1
        for (int a = 0; a < 3; ++a) {
          g[a][0] = A::div(g[a][0], h2x.b);
          g[a][1] = A::div(g[a][1], h2y.b);
          g[a][2] = A::div(g[a][2], h2z.b);
        }
      }
      if (inner_zy) {
        e[0] = g[0][0];
        e[1] = g[1][1];
        e[2] = g[2][2];
        e[3] = A::add(g[1][2], g[2][1]);
        e[4] = A::add(g[0][2], g[2][0]);
        e[5] = A::add(g[0][1], g[1][0]);
      }
    }
    if (ALL || eps) {
      P* st = stage[threadIdx.y];
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 3; ++k) st[3 * lane + k] = P{e[2 * k], e[2 * k + 1]};
      __syncwarp();
      const int cells = min(kCellBlockZ, d.nz - z0);
      if (PAIRS) {
        P* row = reinterpret_cast<P*>(eps) + 3 * (q - lane) + lane;
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (lane + 32 * k < 3 * cells) row[32 * k] = st[lane + 32 * k];
      } else {  // a tensor that is aligned to its elements only
        T* row = eps + 6 * (q - lane) + lane;
#pragma unroll
        for (int k = 0; k < 6; ++k)
          if (lane + 32 * k < 6 * cells) row[32 * k] = reinterpret_cast<const T*>(st)[lane + 32 * k];
      }
    }
    if (zin && (ALL || vol || dev || msh || vm)) {
      T va, vb, vc;
      double v;
      invariants<T>(e, third, vm_c, va, vb, vc, v);
      if (ALL || vol) vol[q] = va;
      if (ALL || dev) dev[q] = vb;
      if (ALL || msh) msh[q] = vc;
      if (ALL || vm) vm[q] = v;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      m[a] = c[a];
      c[a] = n[a];
    }
    cx += sx;
    if (!AOS) {
      cy += sx;
      cz += sx;
    }
  }
}

template <typename T, bool PAIRS>
__global__ void invariants_kernel(const T* __restrict__ eps, long long n, ConstDiv<T> third,
                                  double vm_c, T* __restrict__ vol, T* __restrict__ dev,
                                  T* __restrict__ msh, double* __restrict__ vm) {
  using P = typename Pair<T>::type;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    T e[6];
    if (PAIRS) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const P w = reinterpret_cast<const P*>(eps)[3 * q + k];
        e[2 * k] = w.x;
        e[2 * k + 1] = w.y;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 6; ++k) e[k] = eps[6 * q + k];
    }
    T a, b, c;
    double v;
    invariants<T>(e, third, vm_c, a, b, c, v);
    if (vol) vol[q] = a;
    if (dev) dev[q] = b;
    if (msh) msh[q] = c;
    if (vm) vm[q] = v;
  }
}

static bool bad_grid(int nx, int ny, int nz) { return nx <= 0 || ny <= 0 || nz <= 0; }

}  // namespace sw

using namespace sw;

namespace {
// numpy's divisors: h**2 and 2.0*h computed in double, then cast to the dtype
template <typename T>
ConstDiv<T> sq(double h) {
  return const_div((T)(h * h));
}
template <typename T>
ConstDiv<T> twice(double h) {
  return const_div((T)(2.0 * h));
}
const double kVonMises = std::sqrt(2.0 / 3.0);
int blocks_for(long long n) { return grid_blocks(n, 256, 148 * 32); }
// planes per block: kStrainPlanes, more where they would take over 65535 blocks
int strain_planes(int nx) { return std::max(kStrainPlanes, (nx - 1) / 65535 + 1); }
dim3 strain_grid(int nx, int ny, int nz) {
  const int planes = strain_planes(nx);
  return dim3((unsigned)((nz + kCellBlockZ - 1) / kCellBlockZ),
              (unsigned)((ny + kCellBlockY - 1) / kCellBlockY),
              (unsigned)((nx - 1) / planes + 1));
}
// whether a tensor's six values per cell can be read or written in pairs
template <typename T>
bool pairs_ok(const void* eps) {
  return ((uintptr_t)eps & (2 * sizeof(T) - 1)) == 0;
}
// blocks of 32 (z) x 8 (y) threads, one x plane per block in z (up to 65535)
dim3 cell_grid(int nx, int ny, int nz) {
  return dim3((unsigned)((nz + kCellBlockZ - 1) / kCellBlockZ),
              (unsigned)((ny + kCellBlockY - 1) / kCellBlockY), (unsigned)std::min(nx, 65535));
}
const dim3 kCellBlock(kCellBlockZ, kCellBlockY);

template <typename T>
void launch_strain(const void* ux, const void* uy, const void* uz, int64_t sx, int64_t sy,
                   int64_t sz, const Dense& d, double dX, double dY, double dZ, void* eps,
                   void* vol, void* dev, void* msh, double* vm, cudaStream_t s) {
  using Fn = decltype(&strain_kernel<T, true, true, true>);
  const bool aos = (const T*)uy == (const T*)ux + 1 && (const T*)uz == (const T*)ux + 2;
  const bool all = eps && vol && dev && msh && vm;
  Fn fn;
  if (!pairs_ok<T>(eps)) fn = strain_kernel<T, false, false, false>;
  else if (aos && all) fn = strain_kernel<T, true, true, true>;
  else if (aos) fn = strain_kernel<T, true, true, false>;
  else if (all) fn = strain_kernel<T, true, false, true>;
  else fn = strain_kernel<T, true, false, false>;
  fn<<<strain_grid(d.nx, d.ny, d.nz), kCellBlock, 0, s>>>(
      (const T*)ux, (const T*)uy, (const T*)uz, sx, sy, sz, d, twice<T>(dX), twice<T>(dY),
      twice<T>(dZ), const_div(T(3)), kVonMises, strain_planes(d.nx), (T*)eps, (T*)vol, (T*)dev,
      (T*)msh, vm);
}

template <typename T>
void launch_invariants(const void* eps, int64_t n, void* vol, void* dev, void* msh, double* vm,
                       cudaStream_t s) {
  auto* fn = pairs_ok<T>(eps) ? invariants_kernel<T, true> : invariants_kernel<T, false>;
  fn<<<blocks_for(n), 256, 0, s>>>((const T*)eps, n, const_div(T(3)), kVonMises, (T*)vol, (T*)dev,
                                   (T*)msh, vm);
}
}  // namespace

extern "C" int sw_laplacian(int dtype, const void* f, void* out, int nx, int ny, int nz,
                            double dX, double dY, double dZ, void* stream) {
  if (bad_grid(nx, ny, nz) || !f || !out) {
    set_error("sw_laplacian: bad arguments");
    return SW_EINVAL;
  }
  Dense d{nx, ny, nz};
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == SW_F32)
    laplacian_kernel<float><<<cell_grid(nx, ny, nz), kCellBlock, 0, s>>>(
        (const float*)f, (float*)out, d, sq<float>(dX), sq<float>(dY), sq<float>(dZ));
  else if (dtype == SW_F64)
    laplacian_kernel<double><<<cell_grid(nx, ny, nz), kCellBlock, 0, s>>>(
        (const double*)f, (double*)out, d, sq<double>(dX), sq<double>(dY), sq<double>(dZ));
  else {
    set_error("sw_laplacian: unknown dtype");
    return SW_EINVAL;
  }
  count_launches(1);
  SW_CHECK_LAUNCH("laplacian");
  return SW_OK;
}

extern "C" int sw_divergence(int dtype, const void* fx, const void* fy, const void* fz, void* out,
                             int nx, int ny, int nz, double dX, double dY, double dZ,
                             void* stream) {
  if (bad_grid(nx, ny, nz) || !fx || !fy || !fz || !out) {
    set_error("sw_divergence: bad arguments");
    return SW_EINVAL;
  }
  Dense d{nx, ny, nz};
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == SW_F32)
    divergence_kernel<float><<<cell_grid(nx, ny, nz), kCellBlock, 0, s>>>(
        (const float*)fx, (const float*)fy, (const float*)fz, (float*)out, d, twice<float>(dX),
        twice<float>(dY), twice<float>(dZ));
  else if (dtype == SW_F64)
    divergence_kernel<double><<<cell_grid(nx, ny, nz), kCellBlock, 0, s>>>(
        (const double*)fx, (const double*)fy, (const double*)fz, (double*)out, d,
        twice<double>(dX), twice<double>(dY), twice<double>(dZ));
  else {
    set_error("sw_divergence: unknown dtype");
    return SW_EINVAL;
  }
  count_launches(1);
  SW_CHECK_LAUNCH("divergence");
  return SW_OK;
}

extern "C" int sw_gradient(int dtype, const void* phi, void* gx, void* gy, void* gz, int nx,
                           int ny, int nz, double dX, double dY, double dZ, void* stream) {
  if (bad_grid(nx, ny, nz) || !phi || !gx || !gy || !gz) {
    set_error("sw_gradient: bad arguments");
    return SW_EINVAL;
  }
  Dense d{nx, ny, nz};
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == SW_F32)
    gradient_kernel<float><<<cell_grid(nx, ny, nz), kCellBlock, 0, s>>>(
        (const float*)phi, (float*)gx, (float*)gy, (float*)gz, d, twice<float>(dX),
        twice<float>(dY), twice<float>(dZ));
  else if (dtype == SW_F64)
    gradient_kernel<double><<<cell_grid(nx, ny, nz), kCellBlock, 0, s>>>(
        (const double*)phi, (double*)gx, (double*)gy, (double*)gz, d, twice<double>(dX),
        twice<double>(dY), twice<double>(dZ));
  else {
    set_error("sw_gradient: unknown dtype");
    return SW_EINVAL;
  }
  count_launches(1);
  SW_CHECK_LAUNCH("gradient");
  return SW_OK;
}

extern "C" int sw_strain(int dtype, const void* ux, const void* uy, const void* uz, int64_t sx,
                         int64_t sy, int64_t sz, int nx, int ny, int nz, double dX, double dY,
                         double dZ, void* eps, void* vol, void* dev, void* max_shear,
                         double* von_mises, void* stream) {
  if (bad_grid(nx, ny, nz) || !ux || !uy || !uz) {
    set_error("sw_strain: bad arguments");
    return SW_EINVAL;
  }
  if (!(dX > 0 && dY > 0 && dZ > 0)) {
    set_error("sw_strain: grid spacing must be positive");
    return SW_EINVAL;
  }
  Dense d{nx, ny, nz};
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == SW_F32)
    launch_strain<float>(ux, uy, uz, sx, sy, sz, d, dX, dY, dZ, eps, vol, dev, max_shear, von_mises,
                         s);
  else if (dtype == SW_F64)
    launch_strain<double>(ux, uy, uz, sx, sy, sz, d, dX, dY, dZ, eps, vol, dev, max_shear, von_mises,
                          s);
  else {
    set_error("sw_strain: unknown dtype");
    return SW_EINVAL;
  }
  count_launches(1);
  SW_CHECK_LAUNCH("strain");
  return SW_OK;
}

extern "C" int sw_strain_invariants(int dtype, const void* eps, int64_t n, void* vol, void* dev,
                                    void* max_shear, double* von_mises, void* stream) {
  if (n < 0 || (n > 0 && !eps)) {
    set_error("sw_strain_invariants: bad arguments");
    return SW_EINVAL;
  }
  if (n == 0) return SW_OK;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == SW_F32)
    launch_invariants<float>(eps, n, vol, dev, max_shear, von_mises, s);
  else if (dtype == SW_F64)
    launch_invariants<double>(eps, n, vol, dev, max_shear, von_mises, s);
  else {
    set_error("sw_strain_invariants: unknown dtype");
    return SW_EINVAL;
  }
  count_launches(1);
  SW_CHECK_LAUNCH("strain invariants");
  return SW_OK;
}
