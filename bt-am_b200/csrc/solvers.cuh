// Device kernels of the relaxation and of the hydrogen master equation.
#pragma once

#include <cuda_runtime.h>

#include "topo_kernels.cuh"

namespace btam {

// relaxation (L-BFGS on occupancy-scaled z = (q, log sigma) of the real sites)
struct RelaxBounds {
  double ls_lo, ls_hi;  // log sigma bounds
  double x_min;         // sites with smaller occupancy are held fixed
};
// The periodic images that follow the real rows (n = 0: none).
struct RelaxImages {
  int n = 0;
  const int *owner = nullptr;  // real site of every row
  const char4 *image = nullptr;
  GhostBox box;
};
// z, g of the state and its evaluation; out[0] = F, out[1] = |R|^2, out[2] = the
// error bits, which are cleared.  part: 2 min(kRelaxParts, ceil(n / 128))
// doubles; count: zero before the first call and after each.
constexpr int kRelaxParts = 148;
cudaError_t relax_gather(int n, const double4 *pos, const double2 *xb, const double *V0,
                         const double *Rq, const double *Rs, const RelaxBounds &bd, double *z,
                         double *g, double *part, unsigned *count, int *err, double *out,
                         cudaStream_t st);
// Positions and widths at z0 + alpha p, alpha = scale times *alpha_dev (if
// given), of the real sites and their images.
cudaError_t relax_apply(int n, const double2 *xb, const double *z0, const double *p,
                        double scale, const double *alpha_dev, const RelaxBounds &bd,
                        double4 *pos, const RelaxImages &im, cudaStream_t st);
cudaError_t vec_dot(int n, const double *a, const double *b, double *out, cudaStream_t st);
// out = a x + b y (out may alias x or y)
cudaError_t vec_axpby(int n, double a, const double *x, double b, const double *y, double *out,
                      cudaStream_t st);
// One direction of the limited-memory BFGS iteration: p = -H g by the two-loop
// recursion over the pairs in `order` (newest last) and, when new_slot >= 0,
// the pair (z - z0, g - g0) put into that slot, which is the newest if its
// curvature s.y is above 1e-300; steepest descent if that is no descent
// direction.  z0, g0 then hold z, g.  out: [0] g.p, [1] the first trial's step
// length (a direction without history moves no q or log sigma by more than
// 0.05), [2] 1 if it fell back to steepest descent, [3] s.y of the new pair.
struct LbfgsStep {
  static constexpr int kMax = 16;
  int n4;
  const double *z, *g;
  double *z0, *g0;
  double *S, *Y;  // slot k at k n4
  double *rho;    // 1 / s.y by slot
  int order[kMax];
  int m_used, new_slot;
  const double2 *xb;
  double *p, *out;
};
cudaError_t lbfgs_step(const LbfgsStep &a, cudaStream_t st);

// master equation
constexpr double kDmdQuantum = 8.8817841970012523e-16;    // 2^-50
constexpr double kDmdInvQuantum = 1125899906842624.0;     // 2^50

struct DmdParams {
  double dt;      // time step
  double Df;      // diffusivity (Variables.hpp:71)
  double dr;      // diffusive distance (Variables.hpp:77)
  double min_dx;  // smallest occupancy moved across an edge (Variables.hpp:85)
  double max_x;   // largest occupancy a site may receive up to (Variables.hpp:92)
};

struct DmdArgs {
  int n, n_all;  // real sites; with their images
  double2 *xb;
  const int *code, *owner;
  const double *Rx, *gamma;
  const int *moffs, *midx;  // mechanical neighbours (real sites)
  const int *doffs, *didx;  // diffusive neighbours (real sites)
  long long *X, *X0;        // occupancy quanta, snapshot at the step's start
  long long *out, *in;      // quanta an edge of the site may give, take
  double *mu;
  int *active;
  // step-control counters: [0] the largest edge move over its room and [1]
  // the largest site change over max_dx of the last decision (non-negative
  // doubles as their bits), [2] edge moves clipped to a nonzero room
  unsigned long long *ctl = nullptr;
};

cudaError_t dmd_init(int n, const double2 *xb, const int *code, long long *X, cudaStream_t st);
// x of every H site and image from the quanta, which become the snapshot.
cudaError_t dmd_commit(const DmdArgs &a, cudaStream_t st);
// A step in its parts: chemical potentials, activity and rooms of the
// current state; then (optionally) the step-control decision for a step
// of prm.dt into ctl[0..1]; then the occupancy update of one step of
// prm.dt (edge moves, commit).
cudaError_t dmd_prepare(const DmdArgs &a, const DmdParams &prm, cudaStream_t st);
cudaError_t dmd_control(const DmdArgs &a, const DmdParams &prm, double max_dx, cudaStream_t st);
cudaError_t dmd_apply(const DmdArgs &a, const DmdParams &prm, cudaStream_t st);
cudaError_t dmd_total(int n, const int *code, const long long *X, long long *out2,
                      cudaStream_t st);

}  // namespace btam
