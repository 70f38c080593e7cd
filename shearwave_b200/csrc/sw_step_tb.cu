// Mixed-form step kernel that advances two time steps per pass over HBM
// (the default of every mixed solve, batched or alone; runs without the
// compensated sum).
//
// Same per-cell update as the one-step kernels (src/shearwave/solver.py:
// 195-226 in increment form), applied twice in one pass.  For the 64-wide
// tile shape (TbShape<64>; the 32-wide shape has two rows of 16 pairs per
// warp and a 28 x 28 output tile):
//
//   level 0  the state at step t, streamed by TMA: u and d of a plane around
//            the 60 x 13 output tile (one 68 x 17 x 1 x 6 box per plane;
//            4-stage ring: planes q and q+1 held, two in flight) and the
//            material coefficients of the 64 x 15 level-1 region, which arrive
//            on the barrier of the next plane;
//   level 1  step t+1 on the 64 x 15 region (the tile, one cell of halo, one
//            more column each side in z so z pairs stay aligned), written to
//            a 4-slot shared-memory ring of planes;
//   level 2  step t+2 on the output tile, written to global memory.
//
// The CTA marches along x: when level-0 plane q+1 lands, level 1 computes
// plane q and level 2 plane q-1.  Fifteen consumer warps each own one
// level-1 row of 32 z pairs (packed .f32x2 arithmetic) and the same pairs at
// level 2.  A thread walks its own column in registers at both levels (level
// 0 of planes q-1 and q, level 1 of planes q-1 and q, the coefficients of
// q-1) and takes the z neighbours from the lanes either side, so shared
// memory serves only the rows either side, the column's next level-0 plane,
// its level 1 of plane q-2 and the coefficients: 38 eight-byte loads per pair
// and plane instead of the 76 of reading every stencil point.  Plane q-2 comes
// from the ring, where the thread itself wrote it, because with it in
// registers too the loop cannot be unrolled by two without spilling, and
// unrolled the planes of a column change names instead of registers (52 moves
// of 377 instructions a plane): 600 steps with a push's projection at 256 x
// 256 x 384 145.5 -> 139.5 ms, 500 steps at 64^3 3.65 -> 3.54 ms; 1000 steps
// at 192^3, where the power limit holds the clock, 54.7 -> 54.0 ms.
//
// Two waits per plane and warp.  The level-1 ring has one mbarrier per slot
// (one arrival per warp, when its row of the plane is written); level 2 of
// plane q-1 waits for that plane.  Four slots need no barrier for their
// reuse: a warp that has seen plane q-2 complete knows that every warp has
// left iteration q-3, the last to read the slot plane q goes to (a thread's
// own element of it is read once more, by that thread, in iteration q-2).  With a
// barrier of its own for the coefficients and one for the reuse of a slot
// (four waits per plane) a quarter of the kernel's instructions were waits.
// Columns in registers and two waits: 104 instead of 115 us per launch at
// 192^3, 1.12x on a batch of 24 solves of 64..160 x 64..160 x 64..224 cells.
// Every wait is bounded and an abort stops each warp on its own.  Force
// terms of push tiles come from a shared-memory term buffer the producer
// fills.
//
// It moves about 30 bytes of DRAM traffic per cell-step (u, d in and out
// once per two steps, coefficients once per two steps, halos), against 66
// for one-step launches.
#include <math.h>

#include <algorithm>

#include "sw_common.cuh"
#include "sw_step.cuh"
#include "sw_step_tma.cuh"
#include "sw_tma.cuh"

namespace sw {

namespace {

struct TbCoord {
  int z0, y0, x0, x1;  // output tile: z in [z0, z0+OZ), y in [y0, y0+OY), x in [x0, x1)
};

__host__ __device__ inline TileSpace make_tiles_tb(const Geom& g, int xc, int lz) {
  const int oz = lz == 32 ? TbShape<32>::OZ : TbShape<64>::OZ;
  const int oy = lz == 32 ? TbShape<32>::OY : TbShape<64>::OY;
  TileSpace t;
  // tiles [oz k, oz k + oz) and [oy k, oy k + oy) cover the interior 1..n-2
  t.ntz = g.nz > 2 ? (g.nz - 2) / oz + 1 : 0;
  t.nty = g.ny > 2 ? (g.ny - 2) / oy + 1 : 0;
  const int nxi = g.nx > 2 ? g.nx - 2 : 0;
  t.xc = xc < 1 ? 1 : xc;
  t.nxc = nxi > 0 ? (nxi + t.xc - 1) / t.xc : 0;
  t.count = t.ntz * t.nty * t.nxc;
  return t;
}

// Shape constants the producer needs per tile when a launch mixes shapes:
// the output tile, and the bytes of a level-0 box and cells of a point box.
struct TbDims {
  int oz, oy;
  uint32_t a_bytes, b_cells;
};
template <int LZ>
__device__ constexpr TbDims tb_dims() {
  using S = TbShape<LZ>;
  return TbDims{S::OZ, S::OY, (uint32_t)(S::W * S::H * 6 * 4), (uint32_t)(S::WB * S::HB)};
}

__device__ inline TbCoord tb_coord_rt(const Geom& g, const TileSpace& t, int local, int oz,
                                      int oy) {
  TbCoord c;
  const int zt = local % t.ntz;
  const int rest = local / t.ntz;
  const int yt = rest % t.nty;
  const int xt = rest / t.nty;
  c.z0 = oz * zt;
  c.y0 = oy * yt;
  c.x0 = 1 + xt * t.xc;
  c.x1 = min(c.x0 + t.xc, g.nx - 1);
  return c;
}

template <int OZ, int OY>
__device__ inline TbCoord tb_coord(const Geom& g, const TileSpace& t, int local) {
  TbCoord c;
  const int zt = local % t.ntz;
  const int rest = local / t.ntz;
  const int yt = rest % t.nty;
  const int xt = rest / t.nty;
  c.z0 = OZ * zt;
  c.y0 = OY * yt;
  c.x0 = 1 + xt * t.xc;
  c.x1 = min(c.x0 + t.xc, g.nx - 1);
  return c;
}

__device__ __forceinline__ float2 tb_ld2(const float* p) {
  return *reinterpret_cast<const float2*>(p);
}
__device__ __forceinline__ void tb_st2(float* p, float a, float b) {
  *reinterpret_cast<float2*>(p) = make_float2(a, b);
}

// The force terms of a push tile's two steps, written by the producer when
// it takes the tile and read by the consumers: each term's pattern (its
// component 0) and scale, for step lit (level 1) and lit+1 (level 2).  Two
// buffers, by the parity of the tile's ordinal in the CTA: the producer
// fills the one of tile n+2 only after every consumer warp has released a
// plane of tile n+1 (a tile spans at least NA planes), so no warp still
// reads it.  A pair of steps with more than kTbTermCap terms at one step
// runs in one-step launches instead (the solver keeps such solves out of
// this kernel; the producer refuses the tile if one gets here).
constexpr int kTbTermCap = 32;
struct TbTermRef {
  const float* base;
  float scale;
  int pad;
};
struct TbTermBuf {
  int n[2];
  int pad[2];
  TbTermRef t[2][kTbTermCap];
};

// The z neighbours of a pair come from the lanes either side: (left's .y,
// right's .x).  The first and last lane of a row get a value of another row
// (or their own) in the half that looks outside the region, which no cell
// that is used depends on: level 1 needs only the inner cell of the region's
// outermost pairs, and level 2 leaves those pairs out.
__device__ __forceinline__ float2 tb_zsum(float2 C) {
  const float l = __shfl_up_sync(0xffffffffu, C.y, 1);
  const float r = __shfl_down_sync(0xffffffffu, C.x, 1);
  return make_float2(__fadd_rn(C.y, l), __fadd_rn(r, C.x));
}

// New u and increment of one component of a z pair: C / Cd the pair's u and
// d, X / Xd and Xm / Xmd those of the planes after and before, (N, S) and
// (Nd, Sd) the rows either side, P the force increment's terms.
template <bool VISC, bool DAMP, bool PUSH>
__device__ __forceinline__ float2 tb_inc(float2 C, float2 Cd, float2 X, float2 Xd, float2 Xm,
                                         float2 Xmd, float2 N, float2 S, float2 Nd, float2 Sd,
                                         float2 M, float2 E, const Lap7Pair& lk, float damp,
                                         const TbTermRef* __restrict__ terms, int nterms,
                                         long long i, long long pf) {
  const float2 lu = lap7f2(fadd2(X, Xm), fadd2(N, S), tb_zsum(C), C, lk);
  float2 inc = ffma2(M, lu, Cd);
  if (VISC) {
    const float2 ld = lap7f2(fadd2(Xd, Xmd), fadd2(Nd, Sd), tb_zsum(Cd), Cd, lk);
    inc = ffma2(E, ld, inc);
  }
  if (PUSH) {
    for (int j = 0; j < nterms; ++j) {
      const TbTermRef r = terms[j];
      const float* pp = r.base + i;
      // the pattern is read with plain loads, outside the TMA ring: ask L2
      // for the next plane's now (pf: its offset, 0 when there is none)
      if (pf != 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(pp + pf));
      const float2 Pt = __ldg(reinterpret_cast<const float2*>(pp));
      inc = ffma2(Pt, splat2(r.scale), inc);
    }
  }
  if (DAMP) inc = fmul2(inc, splat2(damp));
  return inc;
}

// Where the two-step kernel's rings and barriers live.
struct TbRings {
  float* ringA;
  float* ringB;
  float* ringL;
  WsHeader* hd;
  uint64_t* Lfull;
  volatile int* abort_flag;
  const TbTermBuf* terms;  // the two term buffers
};

// A consumer warp's next stage of each ring (level-0 planes, point-wise
// planes, level-1 slots), and whether its waits have all succeeded.
struct TbPos {
  RingPos<TmaF32TB::NA> ca;
  RingPos<TmaF32TB::NB> cb;  // filled with ring A's next plane: no barrier of its own
  RingPos<TmaF32TB::NL> lw;
  // the level-1 slot before it (a wait on the slot before the very first
  // plane returns at once: parity 1 of a fresh barrier)
  RingPos<TmaF32TB::NL> lp{TmaF32TB::NL - 1, 1u};
  int ord = 0;  // tiles this warp has finished (picks the term buffer)
  bool ok = true;
};

// One tile of a consumer warp (level-1 row w): the tile's first plane x0-2
// (centres only; its full barrier waited on by the caller), then for every
// plane q = x0-1 .. x1 level 1 at q and level 2 at q-1.  Returns the ring
// positions after the tile, with ok = false when a wait gave up.
template <int LZ, bool VISC, bool DAMP, bool PUSH, bool SNAP>
__device__ __forceinline__ TbPos tb_tile(const TmaF32TB* __restrict__ in, int local, int lit,
                                         const TbRings& k, TbPos p, int w, int lane) {
  using T = TmaF32TB;
  using S = TbShape<LZ>;
  constexpr int W = S::W, H = S::H, WB = S::WB, HB = S::HB;
  constexpr int AF = T::A_STAGE / 4, BF = T::B_STAGE / 4, LF = T::L_STAGE / 4;
  constexpr int LP = LZ * S::LY;  // level-1 cells per component
  const Geom& g = in->g;
  const TbCoord tc = tb_coord<S::OZ, S::OY>(g, in->ts, local);
  float* __restrict__ D = in->state[(lit + 2) % 3];
  const unsigned nc = (unsigned)g.ncell;  // the host keeps ncell below 2^32
  const float damp = in->damp;
  const Lap7Pair lk =
      lap7_pair_coefs(in->hx, in->hy, in->hz, lap7_centre_coef(in->hx, in->hy, in->hz));
  // this thread: level-1 row r (y = y0-1+r), z pair zp, zp+1 (zp = z0-2+2 pl):
  // a warp owns one row of 32 pairs (LZ 64) or two rows of 16 (LZ 32)
  const int r = S::RPW == 1 ? w : 2 * w + (lane >> 4);
  const int pl = lane & (S::PAIRS - 1);
  const int y = tc.y0 - 1 + r, zp = tc.z0 - 2 + 2 * pl;
  const bool yin = y >= 1 && y <= g.ny - 2;
  const bool zin_a = zp >= 1 && zp <= g.nz - 2, zin_b = zp + 1 >= 1 && zp + 1 <= g.nz - 2;
  // a warp whose rows all lie outside the grid interior only writes zeros at
  // level 1 (the shell that level 2 reads)
  const bool warp_live = __any_sync(0xffffffffu, yin);
  // level 2: rows 1..OY and pairs 1..PAIRS-2 are the output tile
  const bool out_rc = r >= 1 && r <= S::OY && pl >= 1 && pl <= S::PAIRS - 2;
  const bool store = out_rc && yin && zp < g.pz;  // pz is even: the pair is in the row
  const bool warp_out = __any_sync(0xffffffffu, store);
  const int o = (r + 1) * W + 2 + 2 * pl, ob = r * WB + 2 + 2 * pl, ol = r * LZ + 2 * pl;
  const int ol2 = min(max(r, 1), S::OY) * LZ + 2 * pl;  // rows 0 and OY+1 read no neighbour rows
  // the force terms of steps lit (level 1) and lit+1 (level 2)
  const TbTermBuf& tbuf = k.terms[p.ord & 1];
  const int n1 = PUSH ? tbuf.n[0] : 0;
  const int n2 = PUSH ? tbuf.n[1] : 0;
  const bool snap1 = SNAP && ((lit + 1) % in->snap_stride) == 0;
  const bool snap2 = SNAP && ((lit + 2) % in->snap_stride) == 0;
  const int slot1 = snap1 ? (lit + 1) / in->snap_stride - 1 : 0;
  const int slot2 = snap2 ? (lit + 2) / in->snap_stride - 1 : 0;
  // Each thread walks its own column in registers: level 0 of planes q-1 and
  // q, level 1 of plane q-1 (u and d of three components).  Shared memory is
  // read for what other threads hold (the rows either side at both levels),
  // the column's next level-0 plane and its level 1 of plane q-2.
  float2 au[3], ad[3], bu[3], bd[3];  // level 0: planes q-1, q
  float2 fu[3], fd[3];                // level 1: plane q-1
  const float2 zero2 = make_float2(0.f, 0.f);
  float2 Mp = zero2, Ep = zero2;  // coefficients of the previous plane
  {
    const float* P0 = k.ringA + p.ca.s * AF + o;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      au[c] = tb_ld2(P0 + c * H * W);
      ad[c] = VISC ? tb_ld2(P0 + (3 + c) * H * W) : zero2;
      fu[c] = fd[c] = zero2;
    }
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(&k.hd->emptyA[p.ca.s]);
  p.ca.next();
  RingPos<T::NA> cur = p.ca;  // plane q
  if (!ws_wait(&k.hd->fullA[cur.s], cur.ph, k.abort_flag)) {
    p.ok = false;
    return p;
  }
  p.ca.next();
  {
    const float* P0 = k.ringA + cur.s * AF + o;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      bu[c] = tb_ld2(P0 + c * H * W);
      bd[c] = tb_ld2(P0 + (3 + c) * H * W);
    }
  }
#pragma unroll 2
  for (int q = tc.x0 - 1; q <= tc.x1; ++q) {
    const RingPos<T::NA> nxt = p.ca;  // plane q+1
    if (!ws_wait(&k.hd->fullA[nxt.s], nxt.ph, k.abort_flag)) {
      p.ok = false;
      return p;
    }
    p.ca.next();
    float* Lw = k.ringL + p.lw.s * LF + ol;
    // ---- level 1: step lit+1 at plane q on the level-1 region ----
    const float* Bm = k.ringB + p.cb.s * BF;
    p.cb.next();
    const float2 Mc = tb_ld2(Bm + ob);
    const float2 Ec = VISC ? tb_ld2(Bm + HB * WB + ob) : zero2;
    const bool xin = q >= 1 && q <= g.nx - 2;
    const float* P = k.ringA + cur.s * AF + o;
    const float* Pn = k.ringA + nxt.s * AF + o;
    float2 nu[3], nd[3];  // level 1 of plane q
    if (!(xin && warp_live)) {
      // every cell of the warp's rows is outside the interior: level 1 is the
      // zero shell
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        nu[c] = nd[c] = zero2;
        au[c] = bu[c];
        bu[c] = tb_ld2(Pn + c * H * W);
        if (VISC) ad[c] = bd[c];
        bd[c] = tb_ld2(Pn + (3 + c) * H * W);
      }
    } else {
      const bool aa = yin && zin_a, ab = yin && zin_b;
      long long i = 0;  // the pair's cell, for the force patterns
      int nl = 0;
      if (PUSH) {
        i = (long long)min(max(q, 0), g.nx - 1) * g.sxy +
            (long long)min(max(y, 0), g.ny - 1) * g.pz + max(zp, 0);
        nl = (aa || ab) ? n1 : 0;
      }
      float* sp = nullptr;
      if (SNAP && snap1 && store && q >= tc.x0 && q < tc.x1)
        sp = in->snaps + ((((long long)slot1 * g.nx + q) * g.ny + y) * g.nz + zp) * 3;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float* Pc = P + c * H * W;
        const float* Pd = P + (3 + c) * H * W;
        const float2 X = tb_ld2(Pn + c * H * W), Xd = tb_ld2(Pn + (3 + c) * H * W);
        const float2 inc = tb_inc<VISC, DAMP, PUSH>(
            bu[c], bd[c], X, Xd, au[c], ad[c], tb_ld2(Pc + W), tb_ld2(Pc - W),
            VISC ? tb_ld2(Pd + W) : zero2, VISC ? tb_ld2(Pd - W) : zero2, Mc, Ec, lk, damp,
            tbuf.t[0], nl, c * (long long)nc + i, PUSH && q + 1 <= g.nx - 2 ? g.sxy : 0);
        const float2 un = fadd2(bu[c], inc);
        nu[c] = make_float2(aa ? un.x : 0.f, ab ? un.y : 0.f);
        nd[c] = make_float2(aa ? inc.x : 0.f, ab ? inc.y : 0.f);
        if (SNAP && sp != nullptr) {
          if (aa) sp[c] = un.x;
          if (ab) sp[3 + c] = un.y;
        }
        au[c] = bu[c];
        bu[c] = X;
        if (VISC) ad[c] = bd[c];
        bd[c] = Xd;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      tb_st2(Lw + c * LP, nu[c].x, nu[c].y);
      tb_st2(Lw + (3 + c) * LP, nd[c].x, nd[c].y);
    }
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(&k.hd->emptyA[cur.s]);  // level-0 plane q is no longer needed
      mbar_arrive(&k.Lfull[p.lw.s]);      // this warp's row of level-1 plane q is written
    }
    // every warp has written plane q-1 (and has left iteration q-2, so the
    // slot after the next, plane q-3's, can be written again)
    if (!ws_wait(&k.Lfull[p.lp.s], p.lp.ph, k.abort_flag)) {
      p.ok = false;
      return p;
    }
    if (q > tc.x0 && warp_out) {
      // ---- level 2: step lit+2 at plane x = q-1 on the output tile ----
      const float* Lc = k.ringL + p.lp.s * LF + ol2;  // a row of the output tile
      const float* Le = k.ringL + ((p.lp.s + T::NL - 1) & (T::NL - 1)) * LF + ol;  // plane q-2
      const int x = q - 1;
      const long long i = (long long)x * g.sxy + (long long)y * g.pz + zp;
      float* sp = nullptr;
      if (SNAP && snap2 && store)
        sp = in->snaps + ((((long long)slot2 * g.nx + x) * g.ny + y) * g.nz + zp) * 3;
      float* out = D + i;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float* Pc = Lc + c * LP;
        const float* Pd = Lc + (3 + c) * LP;
        const float2 inc = tb_inc<VISC, DAMP, PUSH>(
            fu[c], fd[c], nu[c], nd[c], tb_ld2(Le + c * LP),
            VISC ? tb_ld2(Le + (3 + c) * LP) : zero2, tb_ld2(Pc + LZ), tb_ld2(Pc - LZ),
            VISC ? tb_ld2(Pd + LZ) : zero2, VISC ? tb_ld2(Pd - LZ) : zero2, Mp, Ep, lk, damp,
            tbuf.t[1], PUSH && store ? n2 : 0, c * (long long)nc + i, 0);
        const float2 un = fadd2(fu[c], inc);
        if (store) {
          tb_st2(out + (size_t)c * nc, zin_a ? un.x : 0.f, zin_b ? un.y : 0.f);
          tb_st2(out + (size_t)(3 + c) * nc, zin_a ? inc.x : 0.f, zin_b ? inc.y : 0.f);
        }
        if (SNAP && sp != nullptr) {
          if (zin_a) sp[c] = un.x;
          if (zin_b) sp[3 + c] = un.y;
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      fu[c] = nu[c];
      fd[c] = nd[c];
    }
    Mp = Mc;
    Ep = Ec;
    p.lp = p.lw;
    p.lw.next();
    cur = nxt;
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(&k.hd->emptyA[cur.s]);  // the closing halo plane x1+1
  return p;
}

// Whether the tile's pair of steps (lit+1, lit+2) adds force terms.
__device__ __forceinline__ bool tb_pushes(const TmaF32TB* __restrict__ in, int lit) {
  return in->term_off != nullptr && in->term_off[lit + 2] > in->term_off[lit];
}
// Whether the tile's pair of steps writes a snapshot.
__device__ __forceinline__ bool tb_snaps(const TmaF32TB* __restrict__ in, int lit) {
  return in->snap_stride > 0 && in->snaps != nullptr &&
         (((lit + 1) % in->snap_stride) == 0 || ((lit + 2) % in->snap_stride) == 0);
}

// The tile's switches (viscosity, damping, force terms, snapshot), resolved
// once per tile into a specialised loop, every path inlined.  Tiles of push
// or snapshot steps need more live values than the others; with their paths
// in called functions the common loop kept values on the stack around the
// calls (~3 local loads per warp and plane), and with the force terms read
// from the solve's tables inside the loop the push loop spilled (push tiles
// 4.9x slower).  With the terms in the shared term buffer the whole kernel
// fits 128 registers with one to three of them spilled.  (Running the push and snapshot
// tiles in a second launch of their own, which kept the first launch's
// variant at 102 registers, measured 1.4 % slower than this one launch.)
template <int LZ, bool VISC, bool DAMP>
__device__ __forceinline__ TbPos tb_tile_ps(bool push, bool snap, const TmaF32TB* __restrict__ in,
                                            int local, int lit, const TbRings& k, TbPos p, int w,
                                            int lane) {
  if (push) {
    if (snap) return tb_tile<LZ, VISC, DAMP, true, true>(in, local, lit, k, p, w, lane);
    return tb_tile<LZ, VISC, DAMP, true, false>(in, local, lit, k, p, w, lane);
  }
  if (snap) return tb_tile<LZ, VISC, DAMP, false, true>(in, local, lit, k, p, w, lane);
  return tb_tile<LZ, VISC, DAMP, false, false>(in, local, lit, k, p, w, lane);
}

template <int LZ>
__device__ __forceinline__ TbPos tb_tile_sw(const TmaF32TB* __restrict__ in, int local, int lit,
                                            const TbRings& k, TbPos p, int w, int lane) {
  const bool visc = in->ncoef > 1, damp = in->use_damp != 0;
  const bool push = tb_pushes(in, lit), snap = tb_snaps(in, lit);
  if (visc) {
    if (damp) return tb_tile_ps<LZ, true, true>(push, snap, in, local, lit, k, p, w, lane);
    return tb_tile_ps<LZ, true, false>(push, snap, in, local, lit, k, p, w, lane);
  }
  if (damp) return tb_tile_ps<LZ, false, true>(push, snap, in, local, lit, k, p, w, lane);
  return tb_tile_ps<LZ, false, false>(push, snap, in, local, lit, k, p, w, lane);
}


// Progress of a resident launch's tiles: `words` holds one count per tile,
// `stride` words apart, of the consumer warps that have finished it (15 per
// pair of steps).
struct TbProgress {
  int* words;
  int stride, npairs;
};

// End of a block of a resident launch (every thread): the last one to finish
// clears the progress words and the finish count.
__device__ __forceinline__ void tb_resident_done(int* queues, const TbProgress& pr, int ntiles) {
  __shared__ int last_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last_s = atomicAdd(queues + 1, 1) == (int)gridDim.x - 1;
    if (last_s) atomicExch(queues + 1, 0);
  }
  __syncthreads();
  if (last_s)
    for (int t = threadIdx.x; t < ntiles; t += blockDim.x) pr.words[t * pr.stride] = 0;
}

// Whole producer warp: wait until tile `t` and the tiles around it have
// finished `need` warps' work.  Bounded like ws_wait; gives up as soon as the
// solve is abandoned (returns false, the block ends its work).
__device__ __forceinline__ bool tb_wait_around(const TmaF32TB& in, const TbProgress& pr, int t,
                                               int need, volatile int* abort_flag, int lane) {
  const TileSpace& ts = in.ts;
  const int zt = t % ts.ntz + lane % 3 - 1, yt = t / ts.ntz % ts.nty + lane / 3 % 3 - 1,
            xt = t / ts.ntz / ts.nty + lane / 9 - 1;
  const bool mine = lane < 27 && zt >= 0 && zt < ts.ntz && yt >= 0 && yt < ts.nty && xt >= 0 &&
                    xt < ts.nxc;
  const int* w = pr.words + (mine ? ((xt * ts.nty + yt) * ts.ntz + zt) * pr.stride : 0);
  const uint32_t t0 = (uint32_t)clock();
  while (true) {
    int v = need;
    if (mine) asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(w) : "memory");
    if (__all_sync(0xffffffffu, v >= need)) {
      // votes do not order memory: every lane's acquire before the copies that
      // one lane issues for the warp
      __syncwarp();
      return true;
    }
    const bool late = (((uint32_t)clock() - t0) >> 10) > (uint32_t)abort_flag[1];
    if (late) *abort_flag = 1;
    if (__any_sync(0xffffffffu, late || *abort_flag != 0 || solve_abandoned(in.flags)))
      return false;
  }
}

// LZ 0 (batched launches): each solve's tiles have the solve's own shape
// (TmaF32TB::lz), the one that computes fewer cells on its grid.
//
// RES (a lone solve, cooperative launch): the blocks stay for pr.npairs pairs
// of steps, each with its own tiles, and a tile starts its next pair as soon
// as the tiles around it have finished the one before (their halos are
// written; with three state buffers nobody still reads the one it writes), so
// the launches, barrier set-ups and pipeline fills between pairs, and the wait
// for the slowest tile of the grid, are gone.
template <bool BATCH, int LZ, bool RES = false>
__global__ void __launch_bounds__(TmaF32TB::THREADS, 1)
    step_f32_fused2(const __grid_constant__ TmaF32TB one, const TmaF32TB* __restrict__ tab,
                    int ninst, int ntiles, int it, const int* __restrict__ it_dev, int* queues,
                    TbProgress pr) {
  static_assert(LZ != 0 || BATCH, "a single solve has one shape");
  static_assert(!RES || !BATCH, "a resident launch is a lone solve's");
  if (it_dev != nullptr) it += *it_dev;  // step counter kept on the device (graph replays)
  // batched launches take tiles from a launch-wide queue (see step_f32_tma)
  int* queue = queues;
  using T = TmaF32TB;
  constexpr int NA = T::NA, NB = T::NB, NL = T::NL;
  constexpr int AF = T::A_STAGE / 4, BF = T::B_STAGE / 4, LF = T::L_STAGE / 4;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((128u - (smem_addr(smem_raw) & 127u)) & 127u);
  WsHeader* hd = reinterpret_cast<WsHeader*>(base);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(base + kAbortFlagOffset);
  float* ringA = reinterpret_cast<float*>(base + kRingOffset);
  float* ringB = ringA + NA * AF;
  float* ringL = ringB + NB * BF;
  uint64_t* Lfull = reinterpret_cast<uint64_t*>(ringL + NL * LF);  // after the rings
  TbTermBuf* terms = reinterpret_cast<TbTermBuf*>(Lfull + NL);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto flags_of = [&](int k) -> int* { return BATCH ? tab[k].flags : one.flags; };
  if ((smem_addr(ringA) & 127u) != 0u) {
    if (threadIdx.x == 0)
      for (int k = 0; k < (BATCH ? ninst : 1); ++k)
        if (int* fl = flags_of(k)) atomicOr(fl, kFlagRefused);
    if (RES) tb_resident_done(queue, pr, ntiles);
    else queue_cta_done(queue);
    return;
  }
  AbortLog* lg = abort_log(base);
  if (threadIdx.x == 0) {
    for (int s = 0; s < NA; ++s) {
      mbar_init(&hd->fullA[s], 1);
      mbar_init(&hd->emptyA[s], T::CONSUMER_WARPS);
    }
    for (int s = 0; s < NL; ++s) mbar_init(&Lfull[s], T::CONSUMER_WARPS);
    *abort_flag = 0;
    abort_flag[1] = BATCH ? (ninst > 0 ? tab[0].wait_k : 1) : one.wait_k;
    lg->n_taken = 0;
    lg->armedA = lg->parA = lg->armedB = lg->parB = 0;
    for (int w = 0; w < 16; ++w) lg->done[w] = 0;
    mbar_fence_init();
  }
  __syncthreads();

  if (warp == T::CONSUMER_WARPS) {
    // ------------------------------- producer -----------------------------
    RingPos<NA> pa;
    RingPos<NB> pb;
    bool ok = true;
    int acquired = -1;  // the solve whose tensor maps are acquired
    // one lane: the planes of one tile (`tag` goes to the consumers with it)
    auto load_tile = [&](const T* in, int k, int tag, int t, int local, int lit, bool push) {
      const int ord = lg->n_taken;  // the tile's ordinal: its term buffer
      lg->solve[lg->n_taken & 7] = k;
      ++lg->n_taken;
      const Geom& g = in->g;
      const TbDims dm = LZ == 32 || (LZ == 0 && in->lz == 32) ? tb_dims<32>() : tb_dims<64>();
      const TbCoord tc = tb_coord_rt(g, in->ts, local, dm.oz, dm.oy);
      const CUtensorMap* tma = &in->tm[lit % 3];
      if (BATCH && k != acquired) {
        tmap_acquire(tma);
        tmap_acquire(&in->tmm);
        acquired = k;
      }
      const uint32_t bbytes = dm.b_cells * 4 * in->ncoef;
      bool first = true;
      // level-0 plane p, and from plane x0 on the coefficients of plane p-1
      // (what level 1 of plane p-1 reads) on the same barrier
      auto issue = [&](int p) {
        const int sa = pa.s;
        ok = ok && ws_wait(&hd->emptyA[sa], pa.ph ^ 1u, abort_flag);
        if (!ok) return;
        if (first) {
          first = false;
          if (in->stall_test) {  // the testing switch leaves the tile's first stage unarmed
            pa.next();
            return;
          }
          tile_slots(base)[sa] = t;
          solve_slots(base)[sa] = tag;
          if (push) {  // every warp has left tile ord-2, which used this buffer
            TbTermBuf& tb = terms[ord & 1];
            const unsigned nc = (unsigned)g.ncell;
            for (int lev = 0; lev < 2; ++lev) {
              const int j0 = in->term_off[lit + lev], j1 = in->term_off[lit + lev + 1];
              tb.n[lev] = j1 - j0;
              for (int j = j0; j < j1; ++j)
                tb.t[lev][j - j0] = TbTermRef{in->pat + (long long)in->term_pat[j] * 3 * nc,
                                              (float)in->term_scale[j], 0};
            }
          }
        }
        const int pl = min(max(p, 0), g.nx - 1);  // planes outside the grid feed only the shell
        fence_proxy_async_smem();
        const bool points = p >= tc.x0;
        mbar_arrive_expect_tx(&hd->fullA[sa], dm.a_bytes + (points ? bbytes : 0u));
        tma_load_4d(ringA + sa * AF, tma, &hd->fullA[sa], tc.z0 - 4, tc.y0 - 2, pl, 0);
        if (points) {
          const int ql = min(max(p - 1, 0), g.nx - 1);
          tma_load_4d(ringB + pb.s * BF, &in->tmm, &hd->fullA[sa], tc.z0 - 4, tc.y0 - 1, ql, 0);
          pb.next();
        }
        arm_record(lg->armedA, lg->parA, sa, pa.ph);
        pa.next();
      };
      for (int p = tc.x0 - 2; p <= tc.x1 + 1 && ok; ++p) issue(p);
    };
    // whether a pair's force terms fit the term buffer (see kTbTermCap)
    auto terms_fit = [&](const T* in, int lit) -> bool {
      return in->term_off[lit + 1] - in->term_off[lit] <= kTbTermCap &&
             in->term_off[lit + 2] - in->term_off[lit + 1] <= kTbTermCap;
    };
    auto end_work = [&]() {  // arm one stage without a copy
      if (!ws_wait(&hd->emptyA[pa.s], pa.ph ^ 1u, abort_flag)) return;
      tile_slots(base)[pa.s] = -1;
      mbar_arrive(&hd->fullA[pa.s]);
      pa.next();
    };
    if (RES) {
      bool go = true;
      for (int j = 0; j < pr.npairs && go; ++j) {
        const int lit = it + 2 * j;
        for (int t = blockIdx.x; t < ntiles && go; t += gridDim.x) {
          if (j > 0)
            go = tb_wait_around(one, pr, t, j * T::CONSUMER_WARPS, abort_flag, lane);
          else
            go = !solve_abandoned(one.flags);
          go = __all_sync(0xffffffffu, go);
          if (!go) break;
          if (lane == 0) {
            fence_proxy_async_all();  // the neighbours' stores before this tile's copies
            const bool push = tb_pushes(&one, lit);
            if (push && !terms_fit(&one, lit)) {
              if (one.flags != nullptr) atomicOr(one.flags, kFlagRefused);
              ok = false;
            } else {
              load_tile(&one, 0, j, t, t, lit, push);
            }
          }
          go = __all_sync(0xffffffffu, ok) && !*abort_flag;
        }
      }
      if (lane == 0 && !*abort_flag) end_work();
    } else if (lane == 0) {
      int stride_next = blockIdx.x;
      while (ok && !*abort_flag) {
        const int t = next_tile(queue, stride_next);
        if (t >= ntiles) {
          end_work();
          break;
        }
        const int k = BATCH ? find_solve(tab, ninst, t) : 0;
        const T* in = BATCH ? &tab[k] : &one;
        const int local = BATCH ? t - in->tile_base : t;
        const int lit = it - in->it_begin;
        if (lit < 0 || lit + 1 >= in->n_steps || solve_abandoned(in->flags)) continue;
        const bool push = tb_pushes(in, lit);
        if (push && !terms_fit(in, lit)) {
          if (in->flags != nullptr) atomicOr(in->flags, kFlagRefused);
          continue;
        }
        load_tile(in, k, k, t, local, lit, push);
      }
    }
  } else {
    // ------------------------------- consumers ----------------------------
    const TbRings k{ringA, ringB, ringL, hd, Lfull, abort_flag, terms};
    TbPos p;
    while (true) {
      // the tile's first plane, x0-2: centres only
      if (!ws_wait(&hd->fullA[p.ca.s], p.ca.ph, abort_flag)) break;
      const int t = tile_slots(base)[p.ca.s];
      if (t < 0) break;
      const T* in = BATCH ? &tab[solve_slots(base)[p.ca.s]] : &one;
      const int local = BATCH ? t - in->tile_base : t;
      const int lit = RES ? it + 2 * solve_slots(base)[p.ca.s] : it - in->it_begin;
      if (LZ == 0)
        p = in->lz == 32 ? tb_tile_sw<32>(in, local, lit, k, p, warp, lane)
                         : tb_tile_sw<64>(in, local, lit, k, p, warp, lane);
      else
        p = tb_tile_sw<LZ == 0 ? 64 : LZ>(in, local, lit, k, p, warp, lane);
      if (!p.ok) break;
      ++p.ord;
      if (lane == 0) ++lg->done[warp];
      if (RES) {  // this warp's rows of the tile are written
        fence_proxy_async_all();
        __syncwarp();
        if (lane == 0)
          asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(pr.words + t * pr.stride)
                       : "memory");
      }
    }
  }
  __syncthreads();
  if (*abort_flag && warp == T::CONSUMER_WARPS && lane == 0) {
    // let every copy still in flight land, then flag the abandoned tiles' solves
    drain_ring(hd->fullA, lg->armedA, lg->parA, NA);
    flag_unfinished(lg, T::CONSUMER_WARPS, BATCH ? ninst : 1, kFlagTimeout, flags_of);
    // (a wait for other tiles leaves none of this block's own unfinished)
    if (RES && one.flags != nullptr) atomicOr(one.flags, kFlagTimeout);
  }
  if (RES) tb_resident_done(queue, pr, ntiles);
  else queue_cta_done(queue);
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// alignment slack + header + rings + the level-1 ring's barriers + the two
// term buffers
size_t tb_smem_bytes() {
  return 128 + kRingOffset + (size_t)TmaF32TB::NA * TmaF32TB::A_STAGE +
         (size_t)TmaF32TB::NB * TmaF32TB::B_STAGE + (size_t)TmaF32TB::NL * TmaF32TB::L_STAGE +
         TmaF32TB::NL * sizeof(uint64_t) + 2 * sizeof(TbTermBuf);
}

static int tb_set_attr() {
  static bool done = false;
  if (done) return SW_OK;
  const int bytes = (int)tb_smem_bytes();
  const void* fns[7] = {(const void*)step_f32_fused2<false, 64>,
                        (const void*)step_f32_fused2<true, 64>,
                        (const void*)step_f32_fused2<false, 32>,
                        (const void*)step_f32_fused2<true, 32>,
                        (const void*)step_f32_fused2<true, 0>,
                        (const void*)step_f32_fused2<false, 64, true>,
                        (const void*)step_f32_fused2<false, 32, true>};
  for (const void* f : fns) {
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(fused step smem)");
  }
  done = true;
  return SW_OK;
}

// planes per x chunk: minimise waves x (level-1 planes per tile) on 148 SMs
static int tb_xchunk(const Geom& g, int lz) {
  const long long nxi = g.nx > 2 ? g.nx - 2 : 0;
  if (nxi == 0 || g.nz <= 2 || g.ny <= 2) return 1;
  const TileSpace one = make_tiles_tb(g, (int)nxi, lz);
  const long long cols = (long long)one.ntz * one.nty;
  const long long slots = kNumSMs;
  long long best_nc = 1, best = -1;
  for (long long nc = 1; nc <= nxi; ++nc) {
    const long long xc = (nxi + nc - 1) / nc;
    const long long nch = (nxi + xc - 1) / xc;
    const long long cost = ((cols * nch + slots - 1) / slots) * (xc + 2);
    if (best < 0 || cost < best) {
      best = cost;
      best_nc = nc;
    }
  }
  return (int)((nxi + best_nc - 1) / best_nc);
}

// Cells the two levels compute per interior plane for tile width lz: the
// tiles times (level-1 region + output tile).
long long tb_work(const Geom& g, int lz) {
  const TileSpace t = make_tiles_tb(g, 1, lz);
  const long long per = lz == 32
                            ? (long long)TbShape<32>::LZ * TbShape<32>::LY +
                                  (long long)TbShape<32>::OZ * TbShape<32>::OY
                            : (long long)TbShape<64>::LZ * TbShape<64>::LY +
                                  (long long)TbShape<64>::OZ * TbShape<64>::OY;
  return (long long)t.ntz * t.nty * per;
}

int tb_tile_width(const Geom& g) {
  const int knob = tune_get(SW_TUNE_TILE_SHAPE);
  if (knob == 1) return 64;
  if (knob == 2) return 32;
  return tb_work(g, 32) < tb_work(g, 64) ? 32 : 64;
}

int make_tma_f32_tb(const StepArgs& a, int xchunk, TmaF32TB* t, int lz) {
  *t = TmaF32TB{};
  if (a.g.ncell >= (1LL << 32)) {  // the kernel offsets components by a 32-bit cell count
    set_error("grid too large for the two-step kernel (%lld cells)", a.g.ncell);
    return SW_ERANGE;
  }
  t->lz = lz == 32 || lz == 64 ? lz : tb_tile_width(a.g);
  t->g = a.g;
  t->ts = make_tiles_tb(a.g, xchunk > 0 ? xchunk : tb_xchunk(a.g, t->lz), t->lz);
  if (a.coef_e == nullptr) {
    t->ncoef = 1;
  } else if ((const char*)a.coef_e == (const char*)a.coef_m + a.g.ncell * 4) {
    t->ncoef = 2;
  } else {
    set_error("the fused step kernel needs coef_e == coef_m + ncell");
    return SW_EINVAL;
  }
  if (a.kahan) {
    set_error("the two-steps-per-pass kernel runs without the compensated sum");
    return SW_EINVAL;
  }
  const bool n32 = t->lz == 32;
  const uint32_t W = n32 ? TbShape<32>::W : TbShape<64>::W;
  const uint32_t H = n32 ? TbShape<32>::H : TbShape<64>::H;
  const uint32_t WB = n32 ? TbShape<32>::WB : TbShape<64>::WB;
  const uint32_t HB = n32 ? TbShape<32>::HB : TbShape<64>::HB;
  const uint64_t dims[4] = {(uint64_t)a.g.pz, (uint64_t)a.g.ny, (uint64_t)a.g.nx, 9};
  const uint64_t strides[3] = {(uint64_t)a.g.pz * 4, (uint64_t)a.g.sxy * 4,
                               (uint64_t)a.g.ncell * 4};
  const uint32_t boxA[4] = {W, H, 1, 6};
  for (int b = 0; b < 3; ++b) {
    t->state[b] = (float*)a.state[b];
    int rc = encode_tmap_4d(&t->tm[b], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, a.state[b], dims, strides,
                            boxA);
    if (rc != SW_OK) return rc;
  }
  const uint64_t mdims[4] = {(uint64_t)a.g.pz, (uint64_t)a.g.ny, (uint64_t)a.g.nx,
                             (uint64_t)t->ncoef};
  const uint32_t boxM[4] = {WB, HB, 1, (uint32_t)t->ncoef};
  int rc = encode_tmap_4d(&t->tmm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (void*)a.coef_m, mdims,
                          strides, boxM);
  if (rc != SW_OK) return rc;
  t->pat = (const float*)a.patterns;
  t->term_off = a.term_off;
  t->term_pat = a.term_pat;
  t->term_scale = a.term_scale;
  t->hx = (float)a.ihx2;
  t->hy = (float)a.ihy2;
  t->hz = (float)a.ihz2;
  t->damp = (float)a.damp;
  t->use_damp = a.use_damp;
  t->n_steps = a.n_steps;
  t->snap_stride = a.snap_stride;
  t->snaps = (float*)a.snaps;
  t->flags = a.flags;
  t->it_begin = 0;
  t->tile_base = 0;
  t->wait_k = tune_get(SW_TUNE_WAIT_BUDGET);
  t->stall_test = a.stall_test;
  return SW_OK;
}

int launch_fused2_prepare() { return tb_set_attr(); }

const void* step_f32_fused2_ptr(int lz) {
  return lz == 32 ? reinterpret_cast<const void*>(step_f32_fused2<false, 32>)
                  : reinterpret_cast<const void*>(step_f32_fused2<false, 64>);
}

const void* step_f32_fused2_batch_ptr(int lz) {
  if (lz == 0) return reinterpret_cast<const void*>(step_f32_fused2<true, 0>);
  return lz == 32 ? reinterpret_cast<const void*>(step_f32_fused2<true, 32>)
                  : reinterpret_cast<const void*>(step_f32_fused2<true, 64>);
}

static void launch_tb(const void* fn, int grid, cudaStream_t s, const TmaF32TB& one,
                      const TmaF32TB* tab, int ninst, int ntiles, int it, int* queues) {
  const int* itd = nullptr;
  TbProgress none{};
  void* args[] = {(void*)&one, (void*)&tab, (void*)&ninst, (void*)&ntiles, (void*)&it,
                  (void*)&itd, (void*)&queues, (void*)&none};
  cudaLaunchKernel(fn, dim3(grid), dim3(TmaF32TB::THREADS), args, tb_smem_bytes(), s);
}

// SMs a cooperative launch of the resident kernel can use on the current
// device, or 0 when it cannot run one block per SM.
static int tb_resident_slots(int lz) {
  int dev = 0, coop = 0, sms = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  const void* fn = lz == 32 ? (const void*)step_f32_fused2<false, 32, true>
                            : (const void*)step_f32_fused2<false, 64, true>;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, TmaF32TB::THREADS,
                                                    tb_smem_bytes()) != cudaSuccess)
    return 0;
  return per * sms;
}

// Run pairs of a lone solve in resident launches (prepared: tb_set_attr).  The
// progress words lie in the shell plane x = 0 of the compensation component of
// state buffer 0, which is zero in every state and is cleared again, so the
// solve's own memory carries them: any number of solves, streams and threads.
// A launch holds every SM until it ends, and work on other streams waits for it,
// so it is bounded to about 2 ms, or one pair where that takes longer: 1 to 250
// pairs by the time of one (a pair measured 12 us at 64^3, 106 at 192^3, 0.42 ms
// at 256 x 256 x 384).  *done: steps enqueued, 0 when the solve's tiles do not
// allow it.
constexpr double kResidentUs = 2000.0;
inline double pair_us(long long cells) { return 8.0 + 1.55e-5 * (double)cells; }
int run_fused2_resident(const TmaF32TB& t, int* queue, int it0, int nsteps, cudaStream_t s,
                        int* done, unsigned long long* launches) {
  *done = 0;
  const int pairs = nsteps / 2, ntiles = t.ts.count;
  // (chunks of one plane would reach past their neighbours)
  if (queue == nullptr || pairs < 2 || ntiles == 0 || (t.ts.xc < 2 && t.ts.nxc > 1)) return SW_OK;
  const int stride = (int)std::min<long long>(8, t.g.sxy / ntiles);
  if (stride < 1) return SW_OK;
  const int most =
      std::max(1, (int)(kResidentUs / pair_us((long long)t.g.nx * t.g.ny * t.g.nz)));
  const int slots = tb_resident_slots(t.lz);
  if (slots == 0) return SW_OK;
  const int grid = std::min(ntiles, slots);
  TbProgress pr{reinterpret_cast<int*>(t.state[0] + 6 * t.g.ncell), stride, 0};
  const void* fn = t.lz == 32 ? (const void*)step_f32_fused2<false, 32, true>
                              : (const void*)step_f32_fused2<false, 64, true>;
  const TmaF32TB* tab = nullptr;
  const int* itd = nullptr;
  int ninst = 1, nt = ntiles;
  cudaError_t e = cudaMemsetAsync(pr.words, 0, sizeof(int) * (size_t)ntiles * stride, s);
  for (int left = pairs; left > 0 && e == cudaSuccess; left -= pr.npairs) {
    // equal launches
    const int n = (left + most - 1) / most;
    pr.npairs = (left + n - 1) / n;
    int it = it0 + *done;
    void* args[] = {(void*)&t,   (void*)&tab,   (void*)&ninst, (void*)&nt,
                    (void*)&it, (void*)&itd, (void*)&queue, (void*)&pr};
    e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(TmaF32TB::THREADS), args, tb_smem_bytes(),
                                    s);
    *done += 2 * pr.npairs;
    ++*launches;
  }
  if (e != cudaSuccess) return cuda_status(e, "resident two-step launch");
  return SW_OK;
}

void launch_fused2_raw(const TmaF32TB& t, int it, cudaStream_t s) {
  if (t.ts.count == 0) return;
  launch_tb(step_f32_fused2_ptr(t.lz), std::min(t.ts.count, kNumSMs), s, t, nullptr, 1,
            t.ts.count, it, nullptr);
}

int launch_fused2(const StepArgs& a, int xchunk, int it, cudaStream_t s) {
  int rc = tb_set_attr();
  if (rc != SW_OK) return rc;
  TmaF32TB t;
  rc = make_tma_f32_tb(a, xchunk, &t, 0);
  if (rc != SW_OK) return rc;
  if (t.ts.count == 0) return SW_OK;
  launch_fused2_raw(t, it, s);
  count_launches(1);
  SW_CHECK_LAUNCH("fused two-step kernel");
  return SW_OK;
}

int launch_fused2_batch(const void* d_tab, int ninst, int ntiles, int it, int* queues, int lz,
                        cudaStream_t s) {
  int rc = tb_set_attr();
  if (rc != SW_OK) return rc;
  if (ntiles == 0) return SW_OK;
  TmaF32TB dummy{};
  launch_tb(step_f32_fused2_batch_ptr(lz), std::min(ntiles, kNumSMs), s, dummy,
            (const TmaF32TB*)d_tab, ninst, ntiles, it, queues);
  count_launches(1);
  SW_CHECK_LAUNCH("fused two-step kernel (batch)");
  return SW_OK;
}

}  // namespace sw
