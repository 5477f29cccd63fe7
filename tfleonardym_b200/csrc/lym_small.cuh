// Whole even-odd CG solves on small lattices, one cluster of thread blocks per
// right-hand side (lym_small.cu); called by the solvers of lym_solver.cu.
#pragma once

#include "lym_eo.cuh"

namespace lym {

struct SmallReport {
  double true_residual;
  int iterations, updates, done;
  int going;                              // stopped by the limit of the launch: the rest is where it goes on
  double bnorm2, prev_q2, rr, pause2;
  int pause_iter, pad;
};

// One lattice of a call: geometry, links, the fields of its workspace, and the system.
struct SmallLat {
  EoGeom g;
  HopGauge hg64, hgs;                     // FP64 and sloppy links (full N x N, boundary factor folded in)
  EoField be, bo, bp, x64, s64;           // FP64
  EoField r, p, t, s, xs;                 // sloppy (xs: the solution's accumulator; x64 itself in FP64)
  const double2* b;                       // sources and solutions, reference layout (nrhs, ns, N, V)
  double2* x;
  double kappa, tol, delta;
  int hermitian, max_iter;
  int sys0;                               // first right-hand side of this lattice in the launch
  SmallReport* rep;                       // of the lattice's right-hand sides
};

// Whether this form is the faster one for `systems` right-hand sides in all on `lattices`
// lattices of at most vh sites per parity.
bool small_applies(int nd, int nc, int sp, int64_t vh, int systems, int lattices);

// Launches the solves of nlat lattices with `systems` right-hand sides in all; `lats` is a
// device array, or null with one lattice passed by value.  A launch ends after a bounded
// number of iterations; right-hand sides whose report then says `going` go on from there in
// the launch of the next `round` (from 0), which leaves the others as they are.
int small_launch(int nd, int nc, int sp, int64_t vh, const SmallLat* lats, int nlat, const SmallLat& one, int systems,
                 int round, cudaStream_t st);

}  // namespace lym
