// Internal interface of the projection / CG stage (see sw_project.cu).
#pragma once

#include "sw_common.cuh"

namespace sw {

// Element strides of an input field: element (x, y, z) at x*sx + y*sy + z*sz.
struct InStride {
  long long sx, sy, sz;
};

// Scalar state of one CG solve, recorded on the device.
struct CgState {
  double rs[2];   // r.r of the residual before iteration k in rs[k & 1]
  double rs0;     // max(r0.r0, eps64)
  double rel;     // sqrt(rs_new / rs0) of the last update
  double maxdiv;  // max |div_c f| of the masked input
  double tol;
  int iters;      // completed x updates
  int reason;     // enum sw_cg_reason
  int max_iters;
  int brk;        // the last p.Ap ended the iteration (breakdown); -1: a wait ran out
  unsigned int ticket;
};

// Grid-wide barrier of the persistent CG kernel: a count of arrivals and the
// number of the last barrier passed, 128-byte lines apart, both zeroed before
// each launch.  The top bit of `gen` is set when a wait runs out.
struct CgGrid {
  unsigned int* count;
  unsigned int* gen;
};
constexpr unsigned int kCgGridError = 0x80000000u;
// In a 256-byte block of its own (a batch), or in a single solve's 256-byte
// state block: `gen` after the state, `count` in the second line.
inline CgGrid cg_grid_at(char* block) {
  return CgGrid{(unsigned int*)(block + 128), (unsigned int*)(block + 120)};
}
static_assert(sizeof(CgState) <= 120, "the grid barrier shares the state's 256-byte slot");
inline CgGrid cg_grid_of(CgState* st) { return cg_grid_at((char*)st); }

// One solve in a launch's instance table.
//   op 0: the projection's Poisson operator A = -div_c(grad_c .)
//         (src/shearwave/solver.py:1024-1026), rhs = -div_c(mask f);
//   op 1: the static elastic operator A = -mu L7(.) (solver.py:596-597),
//         rhs = mask b; no non-finite breaks and no early exit, like the
//         reference's elastic_solve_static loop (solver.py:605-623).
struct CgInst {
  Geom g;
  TileSpace ts;          // tiles of cg_prep and cg_finish
  int ring_base;         // first tile of this instance in cg_ring
  double c2x, c2y, c2z;  // 1 / (2 h)
  double ihx2, ihy2, ihz2;  // 1 / h^2 (op 1)
  double *x, *r, *p0, *p1;
  double* ap;            // holds the solve's CgRing (A p is recomputed, not stored)
  double* muf;           // mu on interior cells, FP64 (op 1; null: mu_s)
  double mu_s;           // scalar mu when no field is given (op 1)
  double2* partials;     // per tile: (sum, max)
  CgState* st;
  int tile_base;         // first global tile index of this instance
  int op;
};

size_t align_up(size_t v, size_t a);

// Callers' workspaces may lie on any address.  The kernels' vectors and tensor
// maps need 64-byte boundaries (TMA) and 16-byte ones (cp.async, pairs), so a
// workspace is used from its first 128-byte boundary on; the last 256 bytes of
// every workspace size leave the room for it.
constexpr size_t kWorkspaceAlign = 128;
inline char* align_workspace(char* ws) { return (char*)align_up((size_t)ws, kWorkspaceAlign); }
TileSpace cg_tiles(const Geom& g);
size_t cg_workspace_bytes(const Geom& g, const TileSpace& ts);

// Project one 3-component field (any dtype / strides) into `out`
// (3 padded FP64 components).  Synchronises `s`.
int project_field(int dtype, const void* fx, const void* fy, const void* fz, InStride fs,
                  const Geom& g, double dX, double dY, double dZ, double tol, int max_iters,
                  double* out, void* ws, size_t ws_bytes, sw_cg_stats* stats, cudaStream_t s);

}  // namespace sw
