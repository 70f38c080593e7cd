// Helmholtz-Hodge projection and its FP64 conjugate-gradient Poisson solve.
//
// Reference: project_vector_field (src/shearwave/solver.py:644-683) and
// poisson_cg (src/shearwave/solver.py:1010-1050).
//
// The operator is A x = -div_c(grad_c x) with both 2h central differences
// zero on the shell, so per axis an interior row reads x at i-2, i, i+2 and
// drops the gradient term whose centre i+-1 lies on the shell.  One CG
// iteration is two phases of one persistent kernel (cg_ring):
//   apply  : p_k = r + beta p_{k-1} (written to the other p buffer), partial
//            p_k.A p_k
//   update : x += alpha p_k, r -= alpha A p_k (A p_k recomputed from the
//            stored p_k), partial r.r
// After the grid barrier that ends a phase every block sums the partials of
// its instances for itself, in a fixed order (deterministic), and follows the
// reference's stopping rule; the block with an instance's first tile records
// the instance's scalars.
// Every kernel works on a table of instances so that one launch can advance
// many independent solves (the batched path) as well as a single one.
#include <math.h>
#include <stdio.h>

#include <algorithm>
#include <vector>

#include "sw_common.cuh"
#include "sw_project.cuh"
#include "sw_tma.cuh"

namespace sw {

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------
__device__ inline int find_inst(const CgInst* __restrict__ tab, int ninst, int t) {
  int lo = 0, hi = ninst - 1;
  while (lo < hi) {  // last instance with tile_base <= t
    int mid = (lo + hi + 1) >> 1;
    if (tab[mid].tile_base <= t) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Take a ticket for instance `in`; returns true in every thread of the block
// that took the last ticket.  The caller has written its partial already.
__device__ inline bool last_block(const CgInst& in, unsigned int* flag_smem) {
  __syncthreads();
  if (flat_tid() == 0) {
    __threadfence();
    unsigned int t = atomicAdd(&in.st->ticket, 1u);
    *flag_smem = (t == (unsigned int)(in.ts.count - 1)) ? 1u : 0u;
  }
  __syncthreads();
  bool last = *flag_smem != 0u;
  if (last) __threadfence();
  return last;
}

// Sum (and max) of this instance's per-tile partials, fixed order.
__device__ inline double2 reduce_partials(const CgInst& in, double* red) {
  double s = 0.0, m = 0.0;
  const int tid = flat_tid(), nthr = blockDim.x * blockDim.y;
  for (int i = tid; i < in.ts.count; i += nthr) {
    double2 v = __ldcg(&in.partials[i]);
    s += v.x;
    m = fmax(m, v.y);
  }
  double2 out;
  out.x = block_sum(s, red);
  __syncthreads();
  out.y = block_max(m, red);
  return out;
}

template <typename T>
__device__ inline double ld_masked(const T* __restrict__ f, const CgInst& in, const InStride& s,
                                   int x, int y, int z) {
  if (f == nullptr || !interior(in.g, x, y, z)) return 0.0;
  return (double)f[(long long)x * s.sx + (long long)y * s.sy + (long long)z * s.sz];
}

// ---------------------------------------------------------------------------
// prep: rhs = -div_c(mask f), r = rhs, rs0, max|div|
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(TILE_THREADS) cg_prep(const CgInst* __restrict__ tab, int ninst,
                                                        int ntiles, const T* const* __restrict__ fin,
                                                        const InStride* __restrict__ fstride) {
  __shared__ double red[32];
  __shared__ unsigned int lastflag;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int ii = find_inst(tab, ninst, t);
    const CgInst& in = tab[ii];
    const Geom& g = in.g;
    const T* fx = fin[3 * ii + 0];
    const T* fy = fin[3 * ii + 1];
    const T* fz = fin[3 * ii + 2];
    const InStride s = fstride[ii];
    const int local = t - in.tile_base;
    const TileCoord tc = tile_coord(g, in.ts, local);
    const int z = tc.z0 + threadIdx.x, y = tc.y0 + threadIdx.y;
    double acc = 0.0, mx = 0.0;
    if (in.op == 1) {  // static elastic solve: r = p = mask b, mu to FP64
      const T* mu = fin[3 * ii + 1];
      for (int x = tc.x0; x < tc.x1; ++x) {
        if (!interior(g, x, y, z)) continue;
        const long long i = (long long)x * g.sxy + (long long)y * g.pz + z;
        const double b = ld_masked(fx, in, s, x, y, z);
        in.r[i] = b;
        if (mu) in.muf[i] = ld_masked(mu, in, s, x, y, z);
        acc += b * b;
      }
    }
    for (int x = tc.x0; x < tc.x1 && in.op == 0; ++x) {
      if (!interior(g, x, y, z)) continue;
      double tx = (ld_masked(fx, in, s, x + 1, y, z) - ld_masked(fx, in, s, x - 1, y, z)) * in.c2x;
      double ty = (ld_masked(fy, in, s, x, y + 1, z) - ld_masked(fy, in, s, x, y - 1, z)) * in.c2y;
      double tz = (ld_masked(fz, in, s, x, y, z + 1) - ld_masked(fz, in, s, x, y, z - 1)) * in.c2z;
      double div = (tx + ty) + tz;
      double rhs = -div;
      long long i = (long long)x * g.sxy + (long long)y * g.pz + z;
      in.r[i] = rhs;
      acc += rhs * rhs;
      mx = fmax(mx, fabs(div));
    }
    double bs = block_sum(acc, red);
    __syncthreads();
    double bm = block_max(mx, red);
    if (flat_tid() == 0) in.partials[local] = make_double2(bs, bm);
    if (last_block(in, &lastflag)) {
      double2 tot = reduce_partials(in, red);
      if (flat_tid() == 0) {
        CgState* st = in.st;
        st->ticket = 0u;
        st->rs[0] = tot.x;
        st->rs0 = fmax(tot.x, 2.220446049250313e-16);
        st->maxdiv = tot.y;
        st->iters = 0;
        st->brk = 0;
        st->rel = nan("");
        if (in.op == 0 && tot.y < 1e-12) st->reason = SW_CG_EARLY_EXIT;
        else if (st->max_iters <= 0) st->reason = SW_CG_MAXITERS;
        else st->reason = SW_CG_RUNNING;
        __threadfence();
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// the iterations: persistent TMA-ring kernel
// ---------------------------------------------------------------------------
// What bounds an iteration is DRAM: 64 bytes per cell (apply reads p and r
// and writes p; update reads p, x and r and writes x and r).  A block owns a
// 64 x 8 or 32 x 16 (z, y) tile (per solve, whichever covers its grid with
// fewer cells) and walks x: a producer warp streams the halo'd planes of p
// and r (68 x 12 or 36 x 20 boxes) and the point-wise planes of x and r into
// a shared-memory ring with TMA, eight consumer warps compute 32 z pairs
// each.  A thread keeps its own column in registers: the pair's value and the
// x gradient towards the plane behind, for the two interleaved sublattices
// (even and odd planes), so the gradient ahead of one plane is the one behind
// of the plane after next.  The rows y +- 2 and the pairs either side come
// from shared memory.  The update phase walks x the other way, starting with
// the planes the apply phase left in L2.  Two blocks per SM.  Measured against
// a walk with every stencil point from global memory: an iteration at 192^3
// takes 84 instead of 160 us (DRAM bytes alone 69; 6 TB/s while the tiles
// walk, the rest is the phases' ends), the 442 of a static solve at 121 x 121
// x 141, whose vectors fit L2, 13.0 instead of 31.6 ms.
// The walk goes by units of two planes (one barrier, and two independent
// stencils for a thread to overlap).  Stages: the unit in work and the one
// ahead held, two in flight.  A stage holds the boxes of p and r in the apply
// phase; in the update phase the same room holds a ring of p boxes and one of
// point-wise planes.
constexpr int CR_NA = 4, CR_NB = CR_NA - 1;
template <int LZ>
struct CrShape {
  static constexpr int LY = 512 / LZ;  // tile LZ x LY, a warp 64 / LZ rows of LZ / 2 pairs
  static constexpr int W = LZ + 4, H = LY + 4, BOX = W * H;
  static_assert(BOX * 8 % 128 == 0, "TMA destinations");
};
constexpr int CR_BOX = CrShape<64>::BOX > CrShape<32>::BOX ? CrShape<64>::BOX : CrShape<32>::BOX;
constexpr int CR_PT = 512;  // cells of a point box
constexpr int CR_WARPS = 8, CR_THREADS = 32 * (CR_WARPS + 1);
constexpr size_t CR_RINGS = sizeof(double) * (4 * CR_NA * CR_BOX);
static_assert(sizeof(double) * (2 * CR_NA * CR_BOX + 4 * CR_NB * CR_PT) <= CR_RINGS,
              "the update phase's rings take the apply phase's room");
constexpr size_t CR_SMEM = 128 + kRingOffset + CR_RINGS;
static_assert(2 * (CR_SMEM + 1024) <= 233472, "two blocks must fit one SM");
constexpr uint32_t kCgWaitBudget = 1u << 20;  // units of 1024 cycles (~0.5 s)

// The tensor maps and tiles of a solve's ring kernel, kept where the vector
// `ap` would be (A p is never stored).
struct CgRing {
  CUtensorMap ph[2], rh;  // halo boxes of p0, p1, r
  CUtensorMap rp, xp;     // point boxes of r, x
  TileSpace tr;
  int lz;                 // tile shape (CrShape)
};
static_assert(sizeof(CgRing) <= 768, "must fit the smallest vector of a grid with an interior");

__device__ __forceinline__ double2 ld2(const double* p) {
  return *reinterpret_cast<const double2*>(p);
}
__device__ __forceinline__ double2 fma2(double a, double2 b, double2 c) {
  return make_double2(fma(a, b.x, c.x), fma(a, b.y, c.y));
}

struct CgHeader {
  uint64_t full[CR_NA], empty[CR_NA];
  uint64_t sync;  // consumer_sync
};
static_assert(sizeof(CgHeader) <= kAbortFlagOffset, "header overlaps the abort flag");

// Shared-memory view and ring position of one thread's role in a block.
struct CgPipe {
  // apply: [stage][p box pair, r box pair]; update: [stage][p box pair], then
  // [stage][x pair, r pair]
  double* rings;
  CgHeader* hd;
  volatile int* abort_flag;
  RingPos<CR_NA> a;
  int b = 0;
  uint32_t sync_ph = 0;
  template <bool UPDATE>
  __device__ double* stage(int st) const {
    return rings + st * (UPDATE ? 2 * CR_BOX : 4 * CR_BOX);
  }
  __device__ double* points() const { return rings + CR_NA * 2 * CR_BOX + b * 4 * CR_PT; }
  __device__ void next_points() { b = b + 1 == CR_NB ? 0 : b + 1; }
};

// What a block keeps of the instance it works on (shared memory).  The scalars
// follow the iteration as the owner's record does (every block computes the
// same), so a block that stays with one instance reads the record once: with
// every warp of every block reading it in each phase, its few L2 lines were
// the longest part of a phase's start (6300 cycles of a 37000-cycle phase at
// 121 x 121 x 141; now 4100 that overlap the first loads).
struct CgCache {
  CgInst in;
  TileSpace tr;
  int lz;
  int inst;     // its table index
  int run;      // whether this phase works on it, and its beta or alpha
  double scal;
  double rs, rs0, tol;  // rs: r.r of the residual before the current iteration
  int reason, brk, max_iters;
};

// The producer's tile, looked up when it changes.
struct CgTile {
  const CgRing* rg;
  const CgState* st;
  TileCoord tc;
  int t, lz;
};

// Producer: the units of one tile in walk order: one behind, U = ceil(n / 2),
// one ahead (unit u holds planes 2u and 2u + 1 of the walk); in the update
// phase the point-wise planes of a unit, on the barrier of the unit ahead.
// (Their ring needs no barrier for its reuse: a free stage means that the unit
// CR_NA - 1 = CR_NB before the point-wise one being loaded is done, its points
// included: consumers release a unit's stage after they have read both.)  Of a
// last unit with one plane of the tile the other plane is loaded too and never
// used.  The tile's number goes with its first unit.
template <bool UPDATE>
__device__ __forceinline__ bool ring_load(const CgRing* __restrict__ rg, const TileCoord& tc,
                                          int t, int lz, int k, CgPipe& q, AbortLog* lg,
                                          volatile int* slots) {
  const CUtensorMap* pm = UPDATE ? &rg->ph[k & 1] : &rg->ph[(k & 1) ^ 1];
  const uint32_t box = 16u * (lz == 32 ? CrShape<32>::BOX : CrShape<64>::BOX);
  const int U = (tc.x1 - tc.x0 + 1) / 2;
  for (int u = -1; u <= U; ++u) {
    // lower plane of the pair
    const int x = UPDATE ? tc.x1 - 2 - 2 * u : tc.x0 + 2 * u;
    const int st = q.a.s;
    if (!ws_wait(&q.hd->empty[st], q.a.ph ^ 1u, q.abort_flag)) return false;
    double* A = q.stage<UPDATE>(st);
    uint64_t* full = &q.hd->full[st];
    const bool points = UPDATE && u >= 1;
    if (u == -1) slots[st] = t;
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(full, UPDATE ? box + (points ? 32u * CR_PT : 0u) : 2u * box);
    tma_load_3d(A, pm, full, tc.z0 - 2, tc.y0 - 2, x);
    if (!UPDATE) tma_load_3d(A + 2 * CR_BOX, &rg->rh, full, tc.z0 - 2, tc.y0 - 2, x);
    if (points) {
      double* B = q.points();
      tma_load_3d(B, &rg->xp, full, tc.z0, tc.y0, x + 2);
      tma_load_3d(B + 2 * CR_PT, &rg->rp, full, tc.z0, tc.y0, x + 2);
      q.next_points();
    }
    arm_record(lg->armedA, lg->parA, st, q.a.ph);
    q.a.next();
  }
  return true;
}

// Consumer: one tile for one warp; the first unit's barrier has been waited
// for.  `scal` is beta (apply) or alpha (update); acc receives the thread's
// partial of the phase's sum.
template <int LZ, int OP, bool UPDATE>
__device__ __forceinline__ bool ring_tile(const CgInst& in, const TileCoord& tc, int k,
                                          double scal, CgPipe& q, int w, int lane, double* acc) {
  using S = CrShape<LZ>;
  constexpr int W = S::W;
  // the walk's first and second plane of a unit in its boxes (halo, point)
  constexpr int I0 = UPDATE ? S::BOX : 0, I1 = UPDATE ? 0 : S::BOX;
  constexpr int B0 = UPDATE ? CR_PT : 0, B1 = UPDATE ? 0 : CR_PT;
  const int nx = in.g.nx, ny = in.g.ny, nz = in.g.nz;
  const long long sxy = in.g.sxy;
  const int row = LZ == 64 ? w : 2 * w + (lane >> 4), zl = LZ == 64 ? 2 * lane : 2 * (lane & 15);
  const int y = tc.y0 + row, z = tc.z0 + zl;
  const bool yin = y >= 1 && y <= ny - 2;
  const bool aa = yin && z >= 1 && z <= nz - 2, ab = yin && z + 1 <= nz - 2;
  const int o = (row + 2) * W + 2 + zl, ob = row * LZ + zl;
  const double cx = in.c2x, cy = in.c2y, cz = in.c2z;
  // a gradient whose centre lies on the shell is dropped: zero coefficients
  const double cyp = y + 1 <= ny - 2 ? cy : 0.0, cym = y - 1 >= 1 ? cy : 0.0;
  const double czpa = z + 1 <= nz - 2 ? cz : 0.0, czma = z - 1 >= 1 ? cz : 0.0;
  const double czpb = z + 2 <= nz - 2 ? cz : 0.0, czmb = z >= 1 ? cz : 0.0;
  double* __restrict__ X = UPDATE ? in.x : ((k & 1) ? in.p1 : in.p0);
  double* __restrict__ R = in.r;
  auto value = [&](const double* A, int i) -> double2 {  // p at a pair of a stage
    const double2 p = ld2(A + i);
    return UPDATE ? p : fma2(scal, p, ld2(A + 2 * CR_BOX + i));
  };
  auto release = [&](int st) {
    __syncwarp();
    if (lane == 0) mbar_arrive(&q.hd->empty[st]);
  };
  const int n = tc.x1 - tc.x0, xs = UPDATE ? tc.x1 - 1 : tc.x0;  // first plane of the walk
  const long long step = UPDATE ? -sxy : sxy;
  double2 g0, g1;  // the two planes behind the walk, then gradients towards them
  {
    const double* A = q.stage<UPDATE>(q.a.s);
    g0 = value(A, I0 + o);
    g1 = value(A, I1 + o);
    release(q.a.s);
    q.a.next();
  }
  int s0 = q.a.s;
  if (!ws_wait(&q.hd->full[s0], q.a.ph, q.abort_flag)) return false;
  q.a.next();
  double2 c0, c1;  // the unit's own pairs
  {
    const double* A = q.stage<UPDATE>(s0);
    c0 = value(A, I0 + o);
    c1 = value(A, I1 + o);
  }
  auto grad = [](double2 on, double2 back, double c) {
    return make_double2((on.x - back.x) * c, (on.y - back.y) * c);
  };
  const double2 behind = g1;  // op 1: the plane behind the walk
  if (OP == 0) {
    // centres: one plane behind xs, and xs itself (interior)
    const double cb = (UPDATE ? xs + 1 <= nx - 2 : xs - 1 >= 1) ? cx : 0.0;
    g0 = UPDATE ? grad(g0, c0, cb) : grad(c0, g0, cb);
    g1 = UPDATE ? grad(g1, c1, cx) : grad(c1, g1, cx);
  }
  double2 bk = behind;
  long long i = (long long)xs * sxy + (long long)y * in.g.pz + z;
  double sum = 0.0;
  // A p at one plane of op 0: gx the x gradient behind, go the one ahead
  auto stencil0 = [&](const double* A, double2 c, double2 gx, double2 go) -> double2 {
    const double2 N = value(A, o + 2 * W), Sv = value(A, o - 2 * W);
    const double2 L = value(A, o - 2), Rv = value(A, o + 2);
    double2 ap;
    {
      const double tx = (UPDATE ? gx.x - go.x : go.x - gx.x) * cx;
      const double ty = ((N.x - c.x) * cyp - (c.x - Sv.x) * cym) * cy;
      const double tz = ((Rv.x - c.x) * czpa - (c.x - L.x) * czma) * cz;
      ap.x = -((tx + ty) + tz);
    }
    {
      const double tx = (UPDATE ? gx.y - go.y : go.y - gx.y) * cx;
      const double ty = ((N.y - c.y) * cyp - (c.y - Sv.y) * cym) * cy;
      const double tz = ((Rv.y - c.y) * czpb - (c.y - L.y) * czmb) * cz;
      ap.y = -((tx + ty) + tz);
    }
    return ap;
  };
  // A p at one plane of op 1: xa, xb its x neighbours (either order)
  auto stencil1 = [&](const double* A, double2 c, double2 xa, double2 xb, long long at) -> double2 {
    const double hx = in.ihx2, hy = in.ihy2, hz = in.ihz2;
    double2 mu = make_double2(in.mu_s, in.mu_s);
    if (in.muf != nullptr && (aa || ab)) mu = ld2(in.muf + at);
    const double2 N = value(A, o + W), Sv = value(A, o - W);
    const double2 L = value(A, o - 2), Rv = value(A, o + 2);
    const double2 hi = UPDATE ? xa : xb, lo = UPDATE ? xb : xa;
    double2 ap;
    ap.x = -mu.x * (((hi.x - 2.0 * c.x) + lo.x) * hx + ((N.x - 2.0 * c.x) + Sv.x) * hy +
                    ((c.y - 2.0 * c.x) + L.y) * hz);
    ap.y = -mu.y * (((hi.y - 2.0 * c.y) + lo.y) * hx + ((N.y - 2.0 * c.y) + Sv.y) * hy +
                    ((Rv.x - 2.0 * c.y) + c.x) * hz);
    return ap;
  };
  // new x and r (update) or p (apply) of one plane, and its sum
  auto finish = [&](double2 c, double2 ap, const double* B, long long at, bool wa, bool wb) {
    double2 v, rn;
    if (UPDATE) {
      v = fma2(scal, c, ld2(B + ob));
      rn = fma2(-scal, ap, ld2(B + 2 * CR_PT + ob));
    } else {
      v = c;
    }
    if (wa && wb) {
      *reinterpret_cast<double2*>(X + at) = v;
      if (UPDATE) *reinterpret_cast<double2*>(R + at) = rn;
    } else if (wa) {
      X[at] = v.x;
      if (UPDATE) R[at] = rn.x;
    } else if (wb) {
      X[at + 1] = v.y;
      if (UPDATE) R[at + 1] = rn.y;
    }
    if (wa) sum = UPDATE ? fma(rn.x, rn.x, sum) : fma(c.x, ap.x, sum);
    if (wb) sum = UPDATE ? fma(rn.y, rn.y, sum) : fma(c.y, ap.y, sum);
  };
  for (int j = 0; j < n; j += 2, i += 2 * step) {
    const int s1 = q.a.s;  // the unit ahead
    if (!ws_wait(&q.hd->full[s1], q.a.ph, q.abort_flag)) return false;
    q.a.next();
    const bool two = j + 1 < n;
    const double* A = q.stage<UPDATE>(s0);
    const double* An = q.stage<UPDATE>(s1);
    const double2 f0 = value(An, I0 + o), f1 = value(An, I1 + o);
    double2 ap0, ap1;
    if (OP == 0) {
      const double ca0 = (UPDATE ? xs - j - 1 >= 1 : xs + j + 1 <= nx - 2) ? cx : 0.0;
      const double ca1 = (UPDATE ? xs - j - 2 >= 1 : xs + j + 2 <= nx - 2) ? cx : 0.0;
      const double2 go0 = UPDATE ? grad(c0, f0, ca0) : grad(f0, c0, ca0);
      const double2 go1 = UPDATE ? grad(c1, f1, ca1) : grad(f1, c1, ca1);
      ap0 = stencil0(A + I0, c0, g0, go0);
      ap1 = stencil0(A + I1, c1, g1, go1);
      g0 = go0;
      g1 = go1;
    } else {
      ap0 = stencil1(A + I0, c0, bk, c1, i);
      ap1 = stencil1(A + I1, c1, c0, f0, two ? i + step : i);
      bk = c1;
    }
    const double* B = q.points();
    finish(c0, ap0, B + B0, i, aa, ab);
    finish(c1, ap1, B + B1, i + step, aa && two, ab && two);
    if (UPDATE) q.next_points();
    release(s0);  // after the unit's points too: their room is reused on its word
    c0 = f0;
    c1 = f1;
    s0 = s1;
  }
  release(s0);  // the unit ahead of the walk
  *acc = sum;
  return true;
}

// Grid-wide barrier number n = 1, 2, ... (every block of the cooperative
// launch): arrivals are counted in one word, the last one raises the other,
// which the waiting blocks poll (on a line of its own, so the polls do not
// hold up the arrivals).  Bounded; an error raised by any block, or a wait
// that ran out in this one, ends it.  Returns whether the block goes on: with
// `run` (a single instance's, written by thread 0), only while *run holds.  It
// is read here, by its writer, because no warp can read it after the barrier:
// the consumers may be in the next phase by then and have changed it.
__device__ __forceinline__ bool cg_grid_sync(CgGrid b, unsigned int n, volatile int* abort_flag,
                                             const int* run, int* ok_s) {
  asm volatile("fence.proxy.async;" ::: "memory");  // this phase's stores, next phase's TMA reads
  __syncthreads();
  if (*abort_flag) return false;  // the same in every thread: set before the barrier, if at all
  if (threadIdx.x == 0) {
    int ok = 1;
    unsigned int v;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;"
                 : "=r"(v)
                 : "l"(b.count)
                 : "memory");
    if (v + 1u == n * gridDim.x) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(b.gen) : "memory");
    } else {
      const uint32_t t0 = (uint32_t)clock();
      while (true) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(b.gen) : "memory");
        if (v & kCgGridError) {
          ok = 0;
          break;
        }
        if ((int)((v << 1) - (n << 1)) >= 0) break;
        if ((((uint32_t)clock() - t0) >> 10) > kCgWaitBudget) {
          atomicOr(b.gen, kCgGridError);
          ok = 0;
          break;
        }
      }
    }
    *ok_s = ok && (run == nullptr || *run);
  }
  __syncthreads();
  asm volatile("fence.proxy.async;" ::: "memory");
  return *ok_s != 0;
}

// Barrier of the consumer warps; bounded, false once a wait of the block has
// run out.
constexpr int CR_CTHREADS = 32 * CR_WARPS;
__device__ __forceinline__ bool consumer_sync(CgPipe& q) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(&q.hd->sync);
  const bool ok = ws_wait(&q.hd->sync, q.sync_ph, q.abort_flag);
  q.sync_ph ^= 1u;
  return ok;
}

// Per-tile partials of a phase: p.Ap (apply), r.r (update).
__device__ __forceinline__ double* cg_partials(const CgInst& in, bool update) {
  return reinterpret_cast<double*>(in.partials) + (update ? in.ts.count : 0);
}

// Start of a phase for the cached instance, in every block that has one of its
// tiles (the consumer threads): sums the other phase's partials and applies
// the stopping rule; every block computes the same values.  Sets cc->run
// (whether the phase works on the instance) and cc->scal (its beta in apply
// phases, alpha in update phases).  The owner records the scalars: `reason`
// changes in apply phases only and `brk` in update phases only, so nobody
// reads a word in the phase that writes it except to reach the decision it
// holds.
__device__ __forceinline__ bool cg_phase_begin(CgCache* cc, bool update, int k, bool owner,
                                               double* red, CgPipe& q) {
  const CgInst& in = cc->in;
  CgState* st = in.st;
  double v = 0.0;
  if (update || k > 0) {
    const double* pp = cg_partials(in, !update);
    for (int i = threadIdx.x; i < cc->tr.count; i += CR_CTHREADS) v += __ldcg(pp + i);
  }
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  if (!consumer_sync(q)) return false;
  if (threadIdx.x == 0) {
    v = 0.0;
#pragma unroll
    for (int w = 0; w < CR_WARPS; ++w) v += red[w];
    int run = cc->reason == SW_CG_RUNNING;
    double scal = 0.0;
    if (run && update) {
      const bool stop = in.op == 1 ? v <= 0.0 : (!isfinite(v) || v <= 0.0);
      if (stop) {
        cc->brk = 1;
        if (owner) st->brk = 1;
        run = 0;
      } else {
        scal = cc->rs / v;
      }
    } else if (run) {
      int why = SW_CG_RUNNING;
      if (cc->brk) {
        why = SW_CG_BREAKDOWN;
      } else if (k > 0) {
        if (owner) st->iters = k;
        if (in.op == 0 && !isfinite(v)) {
          why = SW_CG_NONFINITE;
        } else {
          const double rel = sqrt(v / cc->rs0);
          scal = v / fmax(cc->rs, 2.220446049250313e-16);
          if (owner) st->rel = rel;
          if (rel < cc->tol) {
            why = SW_CG_CONVERGED;
          } else {
            if (owner) st->rs[k & 1] = v;
            cc->rs = v;
            if (k >= cc->max_iters) why = SW_CG_MAXITERS;
          }
        }
      }
      if (why != SW_CG_RUNNING) {
        cc->reason = why;
        if (owner) st->reason = why;
        run = 0;
      }
    }
    cc->run = run;
    cc->scal = scal;
  }
  return consumer_sync(q);
}

// Last instance whose first ring tile is <= t.
__device__ inline int find_ring(const CgInst* __restrict__ tab, int ninst, int t) {
  int lo = 0, hi = ninst - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tab[mid].ring_base <= t) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

template <int LZ>
__device__ __forceinline__ bool ring_any(const CgInst& in, const TileCoord& tc, int k, bool update,
                                         double scal, CgPipe& q, int w, int lane, double* acc) {
  if (in.op == 0)
    return update ? ring_tile<LZ, 0, true>(in, tc, k, scal, q, w, lane, acc)
                  : ring_tile<LZ, 0, false>(in, tc, k, scal, q, w, lane, acc);
  return update ? ring_tile<LZ, 1, true>(in, tc, k, scal, q, w, lane, acc)
                : ring_tile<LZ, 1, false>(in, tc, k, scal, q, w, lane, acc);
}

// All iterations (bar: cooperative launch), or the one phase `phase` (bar.count
// null: a device without cooperative launch).  Within a phase the producer
// only follows the ring, so its loads start while the consumers still sum the
// partials; it skips the tiles of instances that had ended before the phase,
// and the consumers drain those of an instance that ends at its start.
__global__ void __launch_bounds__(CR_THREADS, 2)
    cg_ring(const CgInst* __restrict__ tab, int ninst, int ntiles, CgGrid bar, int phase) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ double red[CR_WARPS], part[2][CR_WARPS];
  __shared__ CgCache cc;
  __shared__ CgTile pt;  // the producer's
  __shared__ int slots_s[CR_NA], ok_s;
  unsigned char* base = smem_raw + ((128u - (smem_addr(smem_raw) & 127u)) & 127u);
  volatile int* slots = slots_s;
  CgPipe q;
  q.hd = reinterpret_cast<CgHeader*>(base);
  q.abort_flag = reinterpret_cast<volatile int*>(base + kAbortFlagOffset);
  q.rings = reinterpret_cast<double*>(base + kRingOffset);
  AbortLog* lg = abort_log(base);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < CR_NA; ++s) {
      mbar_init(&q.hd->full[s], 1);
      mbar_init(&q.hd->empty[s], CR_WARPS);
    }
    mbar_init(&q.hd->sync, CR_WARPS);
    *q.abort_flag = 0;
    q.abort_flag[1] = (int)kCgWaitBudget;
    lg->armedA = lg->parA = lg->armedB = lg->parB = 0;
    cc.inst = -1;
    pt.t = -1;
    cc.run = 1;
    mbar_fence_init();
  }
  __syncthreads();
  const bool coop = bar.count != nullptr;
  int npart = 0;
  unsigned int nsync = 0;
  for (;; ++phase) {
    const bool update = phase & 1;
    const int k = phase >> 1;
    if (update && coop && ninst > 1) {
      // reasons change in apply phases only: the same answer in every block
      int any = 0;
      for (int i = threadIdx.x; i < ninst; i += CR_THREADS)
        any |= __ldcg(&tab[i].st->reason) == SW_CG_RUNNING;
      if (!__syncthreads_or(any)) break;
    }
    if (warp == CR_WARPS) {
      if (lane == 0) {
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles && ok && !*q.abort_flag; t += gridDim.x) {
          if (t != pt.t) {  // look the tile up
            const CgInst& in = tab[find_ring(tab, ninst, t)];
            const CgRing* rg = reinterpret_cast<const CgRing*>(in.ap);
            pt.rg = rg;
            pt.st = in.st;
            pt.t = t;
            pt.lz = rg->lz;
            pt.tc = tile_coord_t(in.g, rg->tr, t - in.ring_base, pt.lz, 512 / pt.lz);
            for (const CUtensorMap* m : {&rg->ph[0], &rg->ph[1], &rg->rh, &rg->rp, &rg->xp}) {
              tmap_acquire(m);
              prefetch_tmap(m);
            }
          }
          // (a single instance runs until every block leaves)
          if ((ninst > 1 || !coop) && __ldcg(&pt.st->reason) != SW_CG_RUNNING) continue;
          ok = update ? ring_load<true>(pt.rg, pt.tc, t, pt.lz, k, q, lg, slots)
                      : ring_load<false>(pt.rg, pt.tc, t, pt.lz, k, q, lg, slots);
        }
        // the end of the phase: one stage armed without a copy
        if (ok && ws_wait(&q.hd->empty[q.a.s], q.a.ph ^ 1u, q.abort_flag)) {
          slots[q.a.s] = -1;
          mbar_arrive(&q.hd->full[q.a.s]);
          q.a.next();
        }
      }
      __syncwarp();
    } else {
      bool fresh = false;  // cc.run and cc.scal are this phase's
      if (coop && ntiles <= (int)gridDim.x && cc.inst >= 0) {
        // the block stays with its tile: sum the partials while its first
        // unit is on the way
        if (cg_phase_begin(&cc, update, k,
                           cc.in.ring_base % (int)gridDim.x == (int)blockIdx.x, red, q))
          fresh = true;
      }
      while (true) {
        if (!ws_wait(&q.hd->full[q.a.s], q.a.ph, q.abort_flag)) break;
        const int t = slots[q.a.s];
        if (t < 0) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&q.hd->empty[q.a.s]);
          q.a.next();
          break;
        }
        const int ii = find_ring(tab, ninst, t);
        if (!fresh || ii != cc.inst) {
          if (!consumer_sync(q)) break;
          if (ii != cc.inst) {
            const CgRing* rg = reinterpret_cast<const CgRing*>(tab[ii].ap);
            constexpr int NW = (int)(sizeof(CgInst) / 4);
            for (int e = threadIdx.x; e < NW; e += CR_CTHREADS)
              reinterpret_cast<int*>(&cc.in)[e] = reinterpret_cast<const int*>(&tab[ii])[e];
            if (threadIdx.x == 0) {
              const CgState* st = tab[ii].st;
              cc.tr = rg->tr;
              cc.lz = rg->lz;
              // (in the first apply phase rs[0] stands in for the one before)
              cc.rs = __ldcg(&st->rs[update || k == 0 ? (k & 1) : ((k - 1) & 1)]);
              cc.rs0 = __ldcg(&st->rs0);
              cc.tol = __ldcg(&st->tol);
              cc.reason = __ldcg(&st->reason);
              cc.brk = __ldcg(&st->brk);
              cc.max_iters = __ldcg(&st->max_iters);
            }
            if (!consumer_sync(q)) break;
            if (threadIdx.x == 0) cc.inst = ii;
          }
          if (!cg_phase_begin(&cc, update, k,
                              cc.in.ring_base % (int)gridDim.x == (int)blockIdx.x, red, q))
            break;
          fresh = true;
        }
        const int lz = cc.lz, local = t - cc.in.ring_base;
        const TileCoord tc = tile_coord_t(cc.in.g, cc.tr, local, lz, 512 / lz);
        if (!cc.run) {  // ended at the start of this phase: drain the tile
          bool ok = true;
          for (int u = (tc.x1 - tc.x0 + 1) / 2 + 2; u > 0 && ok; --u) {
            ok = ws_wait(&q.hd->full[q.a.s], q.a.ph, q.abort_flag);
            if (!ok) break;
            __syncwarp();  // every lane has seen the stage's phase (and its tile)
            if (lane == 0) mbar_arrive(&q.hd->empty[q.a.s]);
            if (update && u <= (tc.x1 - tc.x0 + 1) / 2) q.next_points();
            q.a.next();
          }
          if (!ok) break;
          continue;
        }
        double acc = 0.0;
        const bool ok = lz == 32
                            ? ring_any<32>(cc.in, tc, k, update, cc.scal, q, warp, lane, &acc)
                            : ring_any<64>(cc.in, tc, k, update, cc.scal, q, warp, lane, &acc);
        if (!ok) break;
        acc = warp_sum(acc);
        if (lane == 0) part[npart & 1][warp] = acc;
        if (!consumer_sync(q)) break;
        if (threadIdx.x == 0) {
          double v = 0.0;
#pragma unroll
          for (int w = 0; w < CR_WARPS; ++w) v += part[npart & 1][w];
          cg_partials(cc.in, update)[local] = v;
        }
        ++npart;
      }
    }
    if (!coop) break;
    // a single instance ends in every block alike; the owner has recorded why
    // (a breakdown found in an update phase ends the next apply phase)
    const int* run = ninst == 1 && !update ? &cc.run : nullptr;
    if (!cg_grid_sync(bar, ++nsync, q.abort_flag, run, &ok_s)) break;
  }
  __syncthreads();
  if (*q.abort_flag && warp == CR_WARPS && lane == 0) {
    // let every copy still in flight land, then end the other blocks' waits
    drain_ring(q.hd->full, lg->armedA, lg->parA, CR_NA);
    if (coop) atomicOr(bar.gen, kCgGridError);
    else if (ninst > 0) atomicExch(&tab[0].st->brk, -1);
  }
}

// ---------------------------------------------------------------------------
// finish: out = (mask f - grad_c x), zero shell
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(TILE_THREADS) cg_finish(const CgInst* __restrict__ tab, int ninst,
                                                          int ntiles, const T* const* __restrict__ fin,
                                                          const InStride* __restrict__ fstride,
                                                          double* const* __restrict__ outs) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int ii = find_inst(tab, ninst, t);
    const CgInst& in = tab[ii];
    const Geom& g = in.g;
    const InStride s = fstride[ii];
    double* out = outs[ii];
    const int local = t - in.tile_base;
    const TileCoord tc = tile_coord(g, in.ts, local);
    const int z = tc.z0 + threadIdx.x, y = tc.y0 + threadIdx.y;
    for (int x = tc.x0; x < tc.x1; ++x) {
      if (!interior(g, x, y, z)) continue;
      const long long i = (long long)x * g.sxy + (long long)y * g.pz + z;
      const double gx = (in.x[i + g.sxy] - in.x[i - g.sxy]) * in.c2x;
      const double gy = (in.x[i + g.pz] - in.x[i - g.pz]) * in.c2y;
      const double gz = (in.x[i + 1] - in.x[i - 1]) * in.c2z;
      out[i] = ld_masked(fin[3 * ii + 0], in, s, x, y, z) - gx;
      out[i + g.ncell] = ld_masked(fin[3 * ii + 1], in, s, x, y, z) - gy;
      out[i + 2 * g.ncell] = ld_masked(fin[3 * ii + 2], in, s, x, y, z) - gz;
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

size_t cg_workspace_bytes(const Geom& g, const TileSpace& ts) {
  size_t vec = align_up((size_t)g.ncell * sizeof(double), 256);
  size_t b = 6 * vec;                                            // x r p0 p1 ap muf
  b += align_up((size_t)ts.count * sizeof(double2), 256);        // partials
  b += align_up(sizeof(CgState), 256);                           // state + grid barrier
  b += align_up(sizeof(CgInst), 256);                            // instance table
  // input and output pointers, and the room of align_workspace
  constexpr size_t ptrs = 3 * sizeof(void*) + sizeof(InStride) + sizeof(double*);
  static_assert(ptrs + kWorkspaceAlign - 1 <= 256, "no room for align_workspace");
  b += 256;
  return b;
}

TileSpace cg_tiles(const Geom& g) { return make_tiles(g, choose_xchunk(g, 4 * 148)); }

int cg_layout(const Geom& g, char* ws, size_t ws_bytes, CgInst* in, CgState** st,
              char** tail) {
  in->g = g;
  in->ts = cg_tiles(g);
  size_t need = cg_workspace_bytes(g, in->ts);
  if (ws == nullptr || ws_bytes < need) {
    set_error("workspace of %zu bytes is smaller than the %zu bytes required", ws_bytes, need);
    return SW_EWORKSPACE;
  }
  size_t vec = align_up((size_t)g.ncell * sizeof(double), 256);
  char* p = align_workspace(ws);
  in->x = (double*)p;
  p += vec;
  in->r = (double*)p;
  p += vec;
  in->p0 = (double*)p;
  p += vec;
  in->p1 = (double*)p;
  p += vec;
  in->ap = (double*)p;
  p += vec;
  in->muf = (double*)p;
  p += vec;
  in->partials = (double2*)p;
  p += align_up((size_t)in->ts.count * sizeof(double2), 256);
  *st = (CgState*)p;
  in->st = *st;
  p += align_up(sizeof(CgState), 256);
  *tail = p;
  in->tile_base = 0;
  return SW_OK;
}

// Tiles of cg_ring: x chunks that minimise waves x planes walked (a chunk's
// n planes, its four halo planes and the fill of the ring) on two blocks per
// SM, and no more tiles than the partials' room (cg_tiles, which has at least
// as many (z, y) columns).
static TileSpace ring_tiles(const Geom& g, int* lz) {
  TileSpace t{};
  const long long nxi = g.nx > 2 ? g.nx - 2 : 0;
  t.xc = 1;
  *lz = 64;
  if (nxi == 0 || g.ny <= 2 || g.nz <= 2) return t;
  // (z, y) tiles from 0 to the last interior cell
  auto count = [](int n, int len) { return (n - 2) / len + 1; };
  // fewer cells; equal: the wide one, whose boxes have less halo
  if (count(g.nz, 32) * 32 * count(g.ny, 16) * 16 < count(g.nz, 64) * 64 * count(g.ny, 8) * 8)
    *lz = 32;
  t.ntz = count(g.nz, *lz);
  t.nty = count(g.ny, 512 / *lz);
  const long long cols = (long long)t.ntz * t.nty, slots = 2 * kNumSMs, room = cg_tiles(g).count;
  long long best = -1;
  for (long long nc = 1; nc <= nxi && (nc == 1 || cols * nc <= room); ++nc) {
    const long long xc = (nxi + nc - 1) / nc, nch = (nxi + xc - 1) / xc;
    const long long cost = ((cols * nch + slots - 1) / slots) * (xc + 6);
    if (best < 0 || cost < best) {
      best = cost;
      t.xc = (int)xc;
      t.nxc = (int)nch;
    }
  }
  t.count = (int)(cols * t.nxc);
  return t;
}

// Clear the iteration's vectors and build the instance's CgRing in its place.
// `base`: tiles of the instances before it.
static int cg_begin(CgInst* in, int base, int* ntiles, cudaStream_t s) {
  const Geom& g = in->g;
  const size_t vec = align_up((size_t)g.ncell * sizeof(double), 256);
  // x r p0 p1 are consecutive 256-byte aligned vectors
  cudaError_t e = cudaMemsetAsync(in->x, 0, 4 * vec, s);
  if (e != cudaSuccess) return cuda_status(e, "CG setup");
  in->ring_base = base;
  CgRing rg;
  rg.tr = ring_tiles(g, &rg.lz);
  *ntiles = rg.tr.count;
  if (rg.tr.count == 0) return SW_OK;
  const uint64_t dims[3] = {(uint64_t)g.pz, (uint64_t)g.ny, (uint64_t)g.nx};
  const uint64_t strides[2] = {(uint64_t)g.pz * 8, (uint64_t)g.sxy * 8};
  const uint32_t lz = (uint32_t)rg.lz, ly = 512 / lz;
  const uint32_t halo[3] = {lz + 4, ly + 4, 2}, point[3] = {lz, ly, 2};
  struct {
    CUtensorMap* map;
    double* base;
    const uint32_t* box;
  } const maps[5] = {{&rg.ph[0], in->p0, halo},
                     {&rg.ph[1], in->p1, halo},
                     {&rg.rh, in->r, halo},
                     {&rg.rp, in->r, point},
                     {&rg.xp, in->x, point}};
  for (const auto& m : maps) {
    const int rc = encode_tmap_3d(m.map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, m.base, dims, strides,
                                  m.box);
    if (rc != SW_OK) return rc;
  }
  e = cudaMemcpyAsync(in->ap, &rg, sizeof(rg), cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return cuda_status(e, "CG setup");
  return SW_OK;
}

// Blocks of a cooperative cg_ring launch on the current device (all resident
// at once), or 0 when the device cannot launch one.
static int cg_coop_blocks() {
  int dev = 0, coop = 0, sms = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, cg_ring, CR_THREADS, CR_SMEM) !=
      cudaSuccess)
    return 0;
  return per * sms;
}

int cg_run(const CgInst* d_tab, int ninst, int ntiles, CgState* d_states, int nst,
           CgGrid grid_words, cudaStream_t s) {
  if (ntiles == 0) return SW_OK;  // no interior cell
  // One cooperative launch runs every iteration (grid barriers between the
  // phases); without cooperative launch support, phases are launched in
  // growing batches and the host polls the exit reasons between batches.
  cudaError_t e = cudaFuncSetAttribute(cg_ring, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)CR_SMEM);
  if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(CG smem)");
  const int coop = cg_coop_blocks();
  if (coop > 0) {
    const int grid = std::max(1, std::min(ntiles, coop));
    e = cudaMemsetAsync(grid_words.count, 0, sizeof(unsigned int), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(grid_words.gen, 0, sizeof(unsigned int), s);
    int phase = 0;
    void* args[] = {(void*)&d_tab, (void*)&ninst, (void*)&ntiles, (void*)&grid_words,
                    (void*)&phase};
    if (e == cudaSuccess)
      e = cudaLaunchCooperativeKernel((const void*)cg_ring, dim3(grid), dim3(CR_THREADS), args,
                                      CR_SMEM, s);
    if (e != cudaSuccess) return cuda_status(e, "cg_ring launch");
    count_launches(1);
    unsigned int gen = 0;
    e = cudaMemcpyAsync(&gen, grid_words.gen, sizeof(gen), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_status(e, "cg_ring readback");
    if (gen & kCgGridError) {
      set_error("CG: a bounded wait of the persistent kernel ran out");
      return SW_ETIMEOUT;
    }
    return SW_OK;
  }
  const int grid = std::max(1, std::min(ntiles, kNumSMs * 2));
  CgState local[4];  // a single solve polls without touching the heap
  std::vector<CgState> heap(nst > 4 ? nst : 0);
  CgState* h = nst > 4 ? heap.data() : local;
  int batch = 8;
  for (int phase = 0;;) {
    e = cudaMemcpyAsync(h, d_states, nst * sizeof(CgState), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_status(e, "cg state readback");
    bool running = false;
    for (int i = 0; i < nst; ++i) {
      running |= (h[i].reason == SW_CG_RUNNING);
      if (h[i].brk < 0) {
        set_error("CG: a bounded wait of the iteration kernel ran out");
        return SW_ETIMEOUT;
      }
    }
    if (!running) return SW_OK;
    for (int b = 0; b < batch; ++b, ++phase)
      cg_ring<<<grid, CR_THREADS, CR_SMEM, s>>>(d_tab, ninst, ntiles, CgGrid{}, phase);
    count_launches((unsigned long long)batch);
    SW_CHECK_LAUNCH("cg iteration");
    batch = std::min(batch * 2, 128);
  }
}

template <typename T>
int project_one(const void* fx, const void* fy, const void* fz, InStride fs, const Geom& g,
                double dX, double dY, double dZ, double tol, int max_iters, double* out, void* ws,
                size_t ws_bytes, sw_cg_stats* stats, cudaStream_t s) {
  CgInst in{};
  CgState* st = nullptr;
  char* tail = nullptr;
  int rc = cg_layout(g, (char*)ws, ws_bytes, &in, &st, &tail);
  if (rc != SW_OK) return rc;
  in.c2x = 1.0 / (2.0 * dX);
  in.c2y = 1.0 / (2.0 * dY);
  in.c2z = 1.0 / (2.0 * dZ);
  CgInst* d_tab = (CgInst*)tail;
  tail += align_up(sizeof(CgInst), 256);
  const T** d_fin = (const T**)tail;
  InStride* d_fs = (InStride*)(tail + 3 * sizeof(void*));
  double** d_out = (double**)(tail + 3 * sizeof(void*) + sizeof(InStride));

  struct {
    const T* f[3];
    InStride st;
    double* out;
  } hostargs;
  hostargs.f[0] = (const T*)fx;
  hostargs.f[1] = (const T*)fy;
  hostargs.f[2] = (const T*)fz;
  hostargs.st = fs;
  hostargs.out = out;

  CgState hst{};
  hst.tol = tol;
  hst.max_iters = max_iters;
  hst.reason = SW_CG_RUNNING;
  int nring = 0;
  rc = cg_begin(&in, 0, &nring, s);
  if (rc != SW_OK) return rc;
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = cudaMemcpyAsync(st, &hst, sizeof(hst), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_tab, &in, sizeof(in), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_fin, hostargs.f, 3 * sizeof(void*), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_fs, &fs, sizeof(fs), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_out, &out, sizeof(out), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(out, 0, (size_t)g.ncell * 3 * sizeof(double), s);
  if (e != cudaSuccess) return cuda_status(e, "projection setup");
  const int ntiles = in.ts.count;
  if (ntiles > 0) {
    const int grid = std::max(1, std::min(ntiles, 148 * 8));
    cg_prep<T><<<grid, dim3(TILE_Z, TILE_Y), 0, s>>>(d_tab, 1, ntiles, d_fin, d_fs);
    count_launches(1);
    SW_CHECK_LAUNCH("cg_prep");
    rc = cg_run(d_tab, 1, nring, st, 1, cg_grid_of(st), s);
    if (rc != SW_OK) return rc;
    cg_finish<T><<<grid, dim3(TILE_Z, TILE_Y), 0, s>>>(d_tab, 1, ntiles, d_fin, d_fs, d_out);
    count_launches(1);
    SW_CHECK_LAUNCH("cg_finish");
  }
  e = cudaMemcpyAsync(&hst, st, sizeof(hst), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_status(e, "projection readback");
  if (stats) {
    if (ntiles == 0) {
      hst.iters = 0;
      hst.reason = SW_CG_EARLY_EXIT;
      hst.rel = nan("");
      hst.maxdiv = 0.0;
    }
    stats->iters = hst.iters;
    stats->reason = hst.reason;
    stats->rel = hst.rel;
    stats->max_div = hst.maxdiv;
  }
  return SW_OK;
}

// Static elastic solve: CG on (-mu L7) u = b (solver.py:569-625) in FP64;
// u (padded FP64) is written to `out`.
template <typename T>
int static_one(const void* b, const void* mu, double mu_s, InStride fs, const Geom& g,
               double dX, double dY, double dZ, double tol, int max_iters, double* out,
               void* ws, size_t ws_bytes, sw_cg_stats* stats, cudaStream_t s) {
  CgInst in{};
  CgState* st = nullptr;
  char* tail = nullptr;
  int rc = cg_layout(g, (char*)ws, ws_bytes, &in, &st, &tail);
  if (rc != SW_OK) return rc;
  in.op = 1;
  in.ihx2 = 1.0 / (dX * dX);
  in.ihy2 = 1.0 / (dY * dY);
  in.ihz2 = 1.0 / (dZ * dZ);
  in.mu_s = mu_s;
  CgInst* d_tab = (CgInst*)tail;
  tail += align_up(sizeof(CgInst), 256);
  const T** d_fin = (const T**)tail;
  InStride* d_fs = (InStride*)(tail + 3 * sizeof(void*));
  const void* fin[3] = {b, mu, nullptr};
  CgState hst{};
  hst.tol = tol;
  hst.max_iters = max_iters;
  hst.reason = SW_CG_RUNNING;
  if (mu == nullptr) in.muf = nullptr;
  int nring = 0;
  rc = cg_begin(&in, 0, &nring, s);
  if (rc != SW_OK) return rc;
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = cudaMemcpyAsync(st, &hst, sizeof(hst), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_tab, &in, sizeof(in), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_fin, fin, 3 * sizeof(void*), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_fs, &fs, sizeof(fs), cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return cuda_status(e, "static solve setup");
  const int ntiles = in.ts.count;
  if (ntiles > 0) {
    const int grid = std::max(1, std::min(ntiles, 148 * 8));
    cg_prep<T><<<grid, dim3(TILE_Z, TILE_Y), 0, s>>>(d_tab, 1, ntiles, d_fin, d_fs);
    count_launches(1);
    SW_CHECK_LAUNCH("static cg_prep");
    rc = cg_run(d_tab, 1, nring, st, 1, cg_grid_of(st), s);
    if (rc != SW_OK) return rc;
  }
  e = cudaMemcpyAsync(out, in.x, (size_t)g.ncell * sizeof(double), cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&hst, st, sizeof(hst), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_status(e, "static solve readback");
  if (stats) {
    stats->iters = hst.iters;
    // a grid without an interior cell has p.Ap = 0 at once
    const int done = nring == 0 && hst.reason == SW_CG_RUNNING ? SW_CG_BREAKDOWN : hst.reason;
    stats->reason = ntiles > 0 ? done : SW_CG_MAXITERS;
    stats->rel = hst.rel;
    stats->max_div = 0.0;
  }
  return SW_OK;
}

int project_field(int dtype, const void* fx, const void* fy, const void* fz, InStride fs,
                  const Geom& g, double dX, double dY, double dZ, double tol, int max_iters,
                  double* out, void* ws, size_t ws_bytes, sw_cg_stats* stats, cudaStream_t s) {
  if (dtype == SW_F32)
    return project_one<float>(fx, fy, fz, fs, g, dX, dY, dZ, tol, max_iters, out, ws, ws_bytes,
                              stats, s);
  if (dtype == SW_F64)
    return project_one<double>(fx, fy, fz, fs, g, dX, dY, dZ, tol, max_iters, out, ws, ws_bytes,
                               stats, s);
  set_error("projection: unknown dtype %d", dtype);
  return SW_EINVAL;
}

}  // namespace sw

using namespace sw;

extern "C" size_t sw_project_workspace_bytes(int nx, int ny, int nz) {
  if (nx <= 0 || ny <= 0 || nz <= 0) return 0;
  Geom g = make_geom(nx, ny, nz, pad_pitch(nz));
  return cg_workspace_bytes(g, cg_tiles(g));
}

extern "C" int sw_project(int in_dtype, const void* fx, const void* fy, const void* fz,
                          int64_t in_sx, int64_t in_sy, int64_t in_sz, int nx, int ny, int nz,
                          double dX, double dY, double dZ, double tol, int max_iters, double* out,
                          void* workspace, size_t workspace_bytes, sw_cg_stats* stats,
                          void* stream) {
  if (nx <= 0 || ny <= 0 || nz <= 0 || out == nullptr) {
    set_error("sw_project: bad grid or null output");
    return SW_EINVAL;
  }
  if (!(dX > 0 && dY > 0 && dZ > 0)) {
    set_error("sw_project: grid spacing must be positive");
    return SW_EINVAL;
  }
  Geom g = make_geom(nx, ny, nz, pad_pitch(nz));
  InStride fs{in_sx, in_sy, in_sz};
  return project_field(in_dtype, fx, fy, fz, fs, g, dX, dY, dZ, tol, max_iters, out, workspace,
                       workspace_bytes, stats, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// batched projection: many independent solves advance together, one launch
// per CG phase over all their tiles
// ---------------------------------------------------------------------------
namespace {
struct BatchTableLayout {
  size_t inst, state, fin, strides, outs, grid, total;
};
BatchTableLayout batch_layout(int n) {
  BatchTableLayout L;
  size_t off = 0;
  L.inst = off;
  off += align_up((size_t)n * sizeof(CgInst), 256);
  L.state = off;
  off += align_up((size_t)n * sizeof(CgState), 256);
  L.fin = off;
  off += align_up((size_t)3 * n * sizeof(void*), 256);
  L.strides = off;
  off += align_up((size_t)n * sizeof(InStride), 256);
  L.outs = off;
  off += align_up((size_t)n * sizeof(double*), 256);
  L.grid = off;
  off += 256;  // cg_grid_at
  L.total = off;
  return L;
}

template <typename T>
int project_batch_t(const sw_project_job* jobs, int n, char* table, sw_cg_stats* stats,
                    cudaStream_t s) {
  const BatchTableLayout L = batch_layout(n);
  std::vector<CgInst> insts(n);
  std::vector<CgState> hst(n);
  std::vector<const void*> fin(3 * (size_t)n);
  std::vector<InStride> strides(n);
  std::vector<double*> outs(n);
  CgState* d_states = (CgState*)(table + L.state);
  int ntiles = 0, nring = 0;
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < n; ++i) {
    const sw_project_job& j = jobs[i];
    Geom g = make_geom(j.nx, j.ny, j.nz, pad_pitch(j.nz));
    CgState* st_unused = nullptr;
    char* tail = nullptr;
    int rc = cg_layout(g, (char*)j.workspace, j.workspace_bytes, &insts[i], &st_unused, &tail);
    if (rc != SW_OK) return rc;
    insts[i].st = d_states + i;
    insts[i].c2x = 1.0 / (2.0 * j.dX);
    insts[i].c2y = 1.0 / (2.0 * j.dY);
    insts[i].c2z = 1.0 / (2.0 * j.dZ);
    insts[i].tile_base = ntiles;
    ntiles += insts[i].ts.count;
    hst[i] = CgState{};
    hst[i].tol = j.tol;
    hst[i].max_iters = j.max_iters;
    hst[i].reason = insts[i].ts.count > 0 ? SW_CG_RUNNING : SW_CG_EARLY_EXIT;
    fin[3 * i + 0] = j.fx;
    fin[3 * i + 1] = j.fy;
    fin[3 * i + 2] = j.fz;
    strides[i] = InStride{j.sx, j.sy, j.sz};
    outs[i] = j.out;
    int cnt = 0;
    rc = cg_begin(&insts[i], nring, &cnt, s);
    if (rc != SW_OK) return rc;
    nring += cnt;
    if (e == cudaSuccess) e = cudaMemsetAsync(j.out, 0, (size_t)g.ncell * 3 * sizeof(double), s);
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(table + L.inst, insts.data(), n * sizeof(CgInst), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_states, hst.data(), n * sizeof(CgState), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(table + L.fin, fin.data(), fin.size() * sizeof(void*),
                        cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(table + L.strides, strides.data(), n * sizeof(InStride),
                        cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(table + L.outs, outs.data(), n * sizeof(double*), cudaMemcpyHostToDevice,
                        s);
  if (e != cudaSuccess) return cuda_status(e, "batched projection setup");
  const CgInst* d_tab = (const CgInst*)(table + L.inst);
  if (ntiles > 0) {
    const int grid = std::max(1, std::min(ntiles, 148 * 8));
    cg_prep<T><<<grid, dim3(TILE_Z, TILE_Y), 0, s>>>(d_tab, n, ntiles, (const T* const*)(table + L.fin),
                                                     (const InStride*)(table + L.strides));
    count_launches(1);
    SW_CHECK_LAUNCH("cg_prep (batch)");
    int rc = cg_run(d_tab, n, nring, d_states, n, cg_grid_at(table + L.grid), s);
    if (rc != SW_OK) return rc;
    cg_finish<T><<<grid, dim3(TILE_Z, TILE_Y), 0, s>>>(d_tab, n, ntiles,
                                                       (const T* const*)(table + L.fin),
                                                       (const InStride*)(table + L.strides),
                                                       (double* const*)(table + L.outs));
    count_launches(1);
    SW_CHECK_LAUNCH("cg_finish (batch)");
  }
  e = cudaMemcpyAsync(hst.data(), d_states, n * sizeof(CgState), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_status(e, "batched projection readback");
  if (stats)
    for (int i = 0; i < n; ++i) {
      stats[i].iters = hst[i].iters;
      stats[i].reason = hst[i].reason;
      stats[i].rel = hst[i].rel;
      stats[i].max_div = hst[i].maxdiv;
    }
  return SW_OK;
}
}  // namespace

extern "C" size_t sw_project_batch_table_bytes(int n) {
  return n > 0 ? batch_layout(n).total : 0;
}

extern "C" int sw_project_batch(const sw_project_job* jobs, int n, void* table,
                                size_t table_bytes, sw_cg_stats* stats, void* stream) {
  if (n <= 0 || jobs == nullptr || table == nullptr) {
    set_error("sw_project_batch: bad arguments");
    return SW_EINVAL;
  }
  if (table_bytes < batch_layout(n).total) {
    set_error("sw_project_batch: table of %zu bytes, %zu required", table_bytes,
              batch_layout(n).total);
    return SW_EWORKSPACE;
  }
  const int dt = jobs[0].in_dtype;
  for (int i = 0; i < n; ++i) {
    const sw_project_job& j = jobs[i];
    if (j.in_dtype != dt || j.nx <= 0 || j.ny <= 0 || j.nz <= 0 || j.out == nullptr ||
        !(j.dX > 0 && j.dY > 0 && j.dZ > 0)) {
      set_error("sw_project_batch: job %d is invalid (dtype, grid, output or spacing)", i);
      return SW_EINVAL;
    }
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (dt == SW_F32) return project_batch_t<float>(jobs, n, (char*)table, stats, s);
  if (dt == SW_F64) return project_batch_t<double>(jobs, n, (char*)table, stats, s);
  set_error("sw_project_batch: unknown dtype %d", dt);
  return SW_EINVAL;
}

extern "C" int sw_static_solve(int dtype, const void* b, const void* mu, double mu_s,
                               int64_t sx, int64_t sy, int64_t sz, int nx, int ny, int nz,
                               double dX, double dY, double dZ, double tol, int max_iters,
                               double* out, void* workspace, size_t workspace_bytes,
                               sw_cg_stats* stats, void* stream) {
  if (nx <= 0 || ny <= 0 || nz <= 0 || out == nullptr || b == nullptr ||
      !(dX > 0 && dY > 0 && dZ > 0)) {
    set_error("sw_static_solve: bad grid, spacing or null pointer");
    return SW_EINVAL;
  }
  Geom g = make_geom(nx, ny, nz, pad_pitch(nz));
  InStride fs{sx, sy, sz};
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == SW_F32)
    return static_one<float>(b, mu, mu_s, fs, g, dX, dY, dZ, tol, max_iters, out, workspace,
                             workspace_bytes, stats, s);
  if (dtype == SW_F64)
    return static_one<double>(b, mu, mu_s, fs, g, dX, dY, dZ, tol, max_iters, out, workspace,
                              workspace_bytes, stats, s);
  set_error("sw_static_solve: unknown dtype %d", dtype);
  return SW_EINVAL;
}
