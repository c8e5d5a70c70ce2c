// Device-resident relaxation of (q, sigma) and the hydrogen master-equation
// step: the two consumers of the residual evaluation.
//
// The reference has neither (its only solver, mechanical_relaxation_bulk in
// Mechanical-Relaxation-bulk.cpp:123-437, relaxes three stretches of the
// deformation gradient; the master equation exists only as parameters,
// src/Variables.hpp:68-90, and the diffusive graph, Neighbors.cpp:139-275).
// Both are defined here and restated by the CPU oracle.
//
// Relaxation: minimise  F(q, s) = sum_i beta_i V0_i - 3 sum_u log sigma_u,
// s = log sigma, over the active real sites; dF/dq_u = beta_u R_q(u) and
// dF/ds_u = beta_u sigma_u R_sigma(u), so F is stationary exactly where the
// residuals vanish.  Limited-memory BFGS (m pairs) with a backtracking
// Armijo line search; the vectors stay on the device, the host only reads
// two scalars per line-search trial.  Converged when
// sqrt(sum |R_q|^2 + R_sigma^2) <= tol.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "solvers.cuh"
#include "topo_kernels.cuh"

namespace btam {

namespace {

constexpr int kRB = 1024;  // threads of the reduction blocks

// Sum (or maximum) over the block of each thread's v, in every thread: fixed
// shuffle trees, sh holds one value per warp.
template <bool MAX> __device__ __forceinline__ double block_reduce(double v, double *sh) {
  auto op = [](double a, double b) { return MAX ? fmax(a, b) : a + b; };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  v = sh[lane];  // kRB / 32 = 32 warps
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();  // sh is written again by the next reduction
  return v;
}

// A cluster's reductions: every block leaves its value in every block's
// shared memory and combines them in rank order.  Two sets of slots in turn,
// so that one cluster barrier per reduction suffices: a slot is written again
// two reductions later, past a barrier that every reader has reached.
struct ClusterReduce {
  static constexpr int kMax = 8;
  double (*slots)[kMax];  // [2][kMax], shared
  double *sh;             // 32, shared
  int rank, size, turn = 0;
  // every block runs before its slots are written, none leaves before that
  __device__ __forceinline__ void begin() const {
    if (size > 1) cooperative_groups::this_cluster().sync();
  }
  __device__ __forceinline__ void end() const { begin(); }
  template <bool MAX> __device__ __forceinline__ double reduce(double v) {
    v = block_reduce<MAX>(v, sh);
    if (size == 1) return v;
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    double *own = slots[turn];
    if ((int)threadIdx.x < size) cl.map_shared_rank(own, threadIdx.x)[rank] = v;
    cl.sync();
    double r = own[0];
    for (int k = 1; k < size; ++k) r = MAX ? fmax(r, own[k]) : r + own[k];
    turn ^= 1;
    return r;
  }
  __device__ __forceinline__ double sum(double v) { return reduce<false>(v); }
  __device__ __forceinline__ double max(double v) { return reduce<true>(v); }
};

// Blocks of a cluster for vectors of n values: one block holds up to four
// values a thread without the cluster's barriers; above that eight SMs read
// the vectors (one block streams about 0.1 TB/s: a dot product of 108,000
// values takes 13.5 us in one block).
inline int cluster_of(int n) { return n <= 4 * kRB ? 1 : ClusterReduce::kMax; }

template <class... KA, class... A>
cudaError_t launch_cluster(void (*k)(KA...), int size, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(size);
  cfg.blockDim = dim3(kRB);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = size;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, KA(args)...);
}

// Sum a[i] * b[i] over one cluster (fixed strides, fixed tree).
__global__ void __launch_bounds__(kRB) dot_kernel(int n, const double *a, const double *b,
                                                  double *out) {
  __shared__ double sh[32], slots[2][ClusterReduce::kMax];
  const int size = gridDim.x, rank = blockIdx.x;
  ClusterReduce R{slots, sh, rank, size};
  R.begin();
  double v = 0.0;
  for (int i = rank * kRB + threadIdx.x; i < n; i += size * kRB) v += a[i] * b[i];
  v = R.sum(v);
  if (rank == 0 && threadIdx.x == 0) *out = v;
  R.end();
}

// One L-BFGS direction (LbfgsStep): the newest pair from the last step, the
// two-loop recursion, and what the line search needs of p, in one launch of
// one cluster.  It replaces 7 launches per pair of the history and 6 more; each
// was a few microseconds of latency with one reduction in it.  What bounds it
// is the latency of its 2 m + 4 reductions, about a microsecond each over the
// cluster.  Relaxation calls with this, the images moved with their owners and
// the host reading once per trial, before and after: 15 iterations of 605
// sites 5.36 -> 2.33 ms, 10 of 27,000 sites 23.4 -> 20.4 ms.
__global__ void __launch_bounds__(kRB) lbfgs_step_kernel(const LbfgsStep a) {
  __shared__ double sh[32], slots[2][ClusterReduce::kMax];
  const int size = gridDim.x, rank = blockIdx.x, n4 = a.n4;
  const int i0 = rank * kRB + threadIdx.x, step = size * kRB;
  ClusterReduce R{slots, sh, rank, size};
  R.begin();
  auto S = [&](int k) { return a.S + (size_t)k * n4; };
  auto Y = [&](int k) { return a.Y + (size_t)k * n4; };
  // the pair of the last step; kept if its curvature is positive
  int used = a.m_used;
  int order[LbfgsStep::kMax + 1];
  for (int t = 0; t < used; ++t) order[t] = a.order[t];
  double sy = 0.0, yy = 0.0;
  bool fresh = false;  // sy and yy are those of the newest pair in use
  double rho_new = 0.0;
  if (a.new_slot >= 0) {
    double *s = S(a.new_slot), *y = Y(a.new_slot);
    double v = 0.0, w = 0.0;
    for (int i = i0; i < n4; i += step) {
      const double ds = a.z[i] - a.z0[i], dy = a.g[i] - a.g0[i];
      s[i] = ds;
      y[i] = dy;
      v += dy * ds;
      w += dy * dy;
    }
    sy = R.sum(v);
    yy = R.sum(w);
    if (sy > 1e-300) {
      rho_new = 1.0 / sy;
      order[used++] = a.new_slot;
      fresh = true;
    }
    if (rank == 0 && threadIdx.x == 0) {
      if (fresh) a.rho[a.new_slot] = rho_new;
      a.out[3] = sy;
    }
  }
  auto rho_of = [&](int k) { return fresh && k == a.new_slot ? rho_new : a.rho[k]; };
  double *q = a.p;  // the recursion runs in p's buffer, each thread on its own values
  double alpha[LbfgsStep::kMax + 1];
  {
    double v = 0.0;  // s . q of the newest pair
    const double *s = used > 0 ? S(order[used - 1]) : nullptr;
    for (int i = i0; i < n4; i += step) {
      const double gi = a.g[i];
      q[i] = gi;
      if (s) v += s[i] * gi;
    }
    for (int t = used - 1; t >= 0; --t) {
      const int k = order[t];
      const double al = rho_of(k) * R.sum(v);
      alpha[t] = al;
      const double *y = Y(k), *sn = t > 0 ? S(order[t - 1]) : nullptr;
      v = 0.0;
      for (int i = i0; i < n4; i += step) {
        const double qi = q[i] + -1.0 * al * y[i];
        q[i] = qi;
        if (sn) v += sn[i] * qi;
      }
    }
  }
  if (used > 0) {
    const int k = order[used - 1];
    if (!fresh) {  // H0 = (s.y)/(y.y) I of an older pair
      double v = 0.0, w = 0.0;
      const double *s = S(k), *y = Y(k);
      for (int i = i0; i < n4; i += step) {
        v += s[i] * y[i];
        w += y[i] * y[i];
      }
      sy = R.sum(v);
      yy = R.sum(w);
    }
    const double h0 = yy > 0.0 ? sy * (1.0 / yy) : 1.0;
    double v = 0.0;  // y . q of the oldest pair
    const double *y = Y(order[0]);
    for (int i = i0; i < n4; i += step) {
      const double qi = q[i] * h0;
      q[i] = qi;
      v += y[i] * qi;
    }
    for (int t = 0; t < used; ++t) {
      const int j = order[t];
      const double c = __dsub_rn(alpha[t], __dmul_rn(rho_of(j), R.sum(v)));
      const double *s = S(j), *yn = t + 1 < used ? Y(order[t + 1]) : nullptr;
      v = 0.0;
      for (int i = i0; i < n4; i += step) {
        const double qi = q[i] + 1.0 * c * s[i];
        q[i] = qi;
        if (yn) v += yn[i] * qi;
      }
    }
  }
  // p = -q, g.p, the largest move in unscaled units; the step's start
  double gp = 0.0, mx = 0.0;
  for (int i = i0; i < n4; i += step) {
    const double pi = -q[i], gi = a.g[i];
    q[i] = pi;
    gp += gi * pi;
    mx = fmax(mx, fabs(pi) / sqrt(fmax(a.xb[i >> 2].x, 1e-3)));
    a.z0[i] = a.z[i];
    a.g0[i] = gi;
  }
  gp = R.sum(gp);
  double restart = 0.0;
  if (!(gp < 0.0)) {  // not a descent direction: steepest descent
    restart = 1.0;
    used = 0;
    gp = mx = 0.0;
    for (int i = i0; i < n4; i += step) {
      const double gi = a.g[i];
      q[i] = -gi;
      gp += gi * -gi;
      mx = fmax(mx, fabs(gi) / sqrt(fmax(a.xb[i >> 2].x, 1e-3)));
    }
    gp = R.sum(gp);
  }
  // first step of a history: move no q (A) or log sigma by more than 0.05
  const double pmax = R.max(mx);
  if (rank == 0 && threadIdx.x == 0) {
    a.out[0] = gp;
    a.out[1] = used == 0 && pmax > 0.05 ? 0.05 / pmax : 1.0;
    a.out[2] = restart;
  }
  R.end();
}

// Per-site scale of the optimisation variables: a site's energy terms carry
// its occupancy, so its curvature does too; w = sqrt(max(x, 1e-3)) z puts
// weakly and fully occupied sites on a comparable footing.
__device__ __forceinline__ double occ_scale(double x) { return sqrt(fmax(x, 1e-3)); }

// w = scale (q, log sigma) of the real sites; gw = (beta R_q, beta sigma
// R_sigma) / scale on relaxed sites (x >= x_min), 0 elsewhere and on log
// sigma components pinned at a bound with the gradient pointing outwards;
// F = sum_active beta V0 - 3 sum_relaxed log sigma; the projected residual
// |R|^2 over the relaxed sites.
// The two sums: a partial per block, the last block to finish adds the
// partials in block order (fixed strides, fixed trees) and resets the count.
constexpr int kGB = 128;
__global__ void __launch_bounds__(kGB)
gather_kernel(int n, const double4 *pos, const double2 *xb, const double *V0, const double *Rq,
              const double *Rs, RelaxBounds bd, double *z, double *g, double *part,
              unsigned *count, int *err, double *out) {
  __shared__ double sh[2][kGB / 32];
  __shared__ bool last;
  double f = 0.0, r2 = 0.0;
  for (int i = blockIdx.x * kGB + threadIdx.x; i < n; i += gridDim.x * kGB) {
    double4 p = pos[i];
    double2 b = xb[i];
    bool act = b.x >= 5e-4;
    bool rel = act && b.x >= bd.x_min;
    double sc = occ_scale(b.x), ls = log(p.w), be = b.y;
    z[4 * i] = sc * p.x;
    z[4 * i + 1] = sc * p.y;
    z[4 * i + 2] = sc * p.z;
    z[4 * i + 3] = sc * ls;
    double gs = be * p.w * Rs[i];
    bool pin = (ls >= bd.ls_hi - 1e-12 && gs < 0.0) || (ls <= bd.ls_lo + 1e-12 && gs > 0.0);
    g[4 * i] = rel ? be * Rq[3 * i] / sc : 0.0;
    g[4 * i + 1] = rel ? be * Rq[3 * i + 1] / sc : 0.0;
    g[4 * i + 2] = rel ? be * Rq[3 * i + 2] / sc : 0.0;
    g[4 * i + 3] = (rel && !pin) ? gs / sc : 0.0;
    f += act ? be * V0[i] - (rel ? 3.0 * ls : 0.0) : 0.0;
    r2 += rel ? Rq[3 * i] * Rq[3 * i] + Rq[3 * i + 1] * Rq[3 * i + 1] +
                    Rq[3 * i + 2] * Rq[3 * i + 2] + (pin ? 0.0 : Rs[i] * Rs[i])
              : 0.0;
  }
  auto both = [&](double &a, double &b) {  // the block's sums, in thread 0
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
      sh[0][threadIdx.x >> 5] = a;
      sh[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      a = sh[0][0];
      b = sh[1][0];
      for (int w = 1; w < kGB / 32; ++w) {
        a += sh[0][w];
        b += sh[1][w];
      }
    }
  };
  both(f, r2);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = f;
    part[2 * blockIdx.x + 1] = r2;
    __threadfence();
    last = atomicAdd(count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  f = r2 = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kGB) {
    f += __ldcg(part + 2 * b);
    r2 += __ldcg(part + 2 * b + 1);
  }
  both(f, r2);
  if (threadIdx.x == 0) {
    out[0] = f;
    out[1] = r2;
    out[2] = (double)*err;  // the evaluation's error bits, read and cleared
    *err = 0;
    *count = 0;
  }
}

// Rows of the real sites, then of their images, from w = w0 + alpha p (sigma =
// exp(s), s kept in bounds); alpha = scale times *alpha_dev if given.  A site
// below x_min is held: its position is left untouched.  An image takes its
// owner's new position, formed again from the same operations, plus its shift.
__global__ void apply_kernel(int n, const double2 *xb, const double *z0, const double *p,
                             double scale, const double *alpha_dev, RelaxBounds bd, double4 *pos,
                             RelaxImages im) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= n + im.n) return;
  const double alpha = alpha_dev ? scale * *alpha_dev : scale;
  const int i = row < n ? row : im.owner[row];
  const double x = xb[i].x;
  if (!(x >= 5e-4 && x >= bd.x_min)) return;
  double sc = occ_scale(x);
  double4 q;
  q.x = (z0[4 * i] + alpha * p[4 * i]) / sc;
  q.y = (z0[4 * i + 1] + alpha * p[4 * i + 1]) / sc;
  q.z = (z0[4 * i + 2] + alpha * p[4 * i + 2]) / sc;
  double ls = (z0[4 * i + 3] + alpha * p[4 * i + 3]) / sc;
  q.w = exp(fmin(fmax(ls, bd.ls_lo), bd.ls_hi));
  if (row >= n) {
    const double qi[3] = {q.x, q.y, q.z};
    double s[3];
    image_position(im.box, im.image[row - n], qi, s);
    q.x = s[0];
    q.y = s[1];
    q.z = s[2];
  }
  pos[row] = q;
}

inline int nb(long long n) { return (int)((n + 255) / 256); }

}  // namespace

cudaError_t relax_gather(int n, const double4 *pos, const double2 *xb, const double *V0,
                         const double *Rq, const double *Rs, const RelaxBounds &bd, double *z,
                         double *g, double *part, unsigned *count, int *err, double *out,
                         cudaStream_t st) {
  const int need = (n + kGB - 1) / kGB, blocks = need < kRelaxParts ? need : kRelaxParts;
  gather_kernel<<<blocks, kGB, 0, st>>>(n, pos, xb, V0, Rq, Rs, bd, z, g, part, count, err, out);
  return cudaGetLastError();
}

cudaError_t relax_apply(int n, const double2 *xb, const double *z0, const double *p,
                        double scale, const double *alpha_dev, const RelaxBounds &bd,
                        double4 *pos, const RelaxImages &im, cudaStream_t st) {
  apply_kernel<<<nb((long long)n + im.n), 256, 0, st>>>(n, xb, z0, p, scale, alpha_dev, bd, pos,
                                                        im);
  return cudaGetLastError();
}

namespace {
__global__ void axpby_kernel(int n, double a, const double *x, double b, const double *y,
                             double *out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = a * x[i] + b * y[i];
}
}  // namespace

cudaError_t vec_axpby(int n, double a, const double *x, double b, const double *y, double *out,
                      cudaStream_t st) {
  if (n > 0) axpby_kernel<<<nb(n), 256, 0, st>>>(n, a, x, b, y, out);
  return cudaGetLastError();
}

cudaError_t vec_dot(int n, const double *a, const double *b, double *out, cudaStream_t st) {
  return launch_cluster(dot_kernel, cluster_of(n), st, n, a, b, out);
}

cudaError_t lbfgs_step(const LbfgsStep &a, cudaStream_t st) {
  return launch_cluster(lbfgs_step_kernel, cluster_of(a.n4), st, a);
}

}  // namespace btam

// ---------------------------------------------------------------------------
// Hydrogen master equation on the diffusive graph (H-H pairs within
// r_cutoff_Eb = 2.6 A, at most 50 per site: list_of_diffusive_neighs,
// Neighbors.cpp:139-275).  Occupancies are carried as int64 quanta of
// 2^-50, and every undirected edge moves +n quanta into one end and -n out
// of the other with integer atomics, so the total hydrogen is conserved
// exactly and the result does not depend on the order of the updates.
namespace btam {

namespace {

__global__ void dmd_init_kernel(int n, const double2 *xb, const int *code, long long *X) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  X[i] = code[i] == 1 ? llrint(xb[i].x * kDmdInvQuantum) : 0;
}

// chemical potential and diffusive activity (local H mass >= 0.01,
// Topology.cpp:202-364) of every real H site: one warp per site, its lanes over
// the list (a thread per site walked some 110 entries in turn: 34 us for 38,040
// sites, a warp 10.6).  Occupancies are multiples of 2^-50, so a mass below 8 is
// exact in any order of the sum and the test against 0.01 does not depend on
// it.
__global__ void dmd_mu_kernel(int n, const double2 *xb, const int *code, const double *Rx,
                              const double *gamma, const int *moffs, const int *midx,
                              const long long *X, double *mu, int *active) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= n) return;
  if (code[i] != 1) {
    if (lane == 0) {
      active[i] = 0;
      mu[i] = 0.0;
    }
    return;
  }
  double x = (double)X[i] * kDmdQuantum;
  double mass = lane == 0 ? x : 0.0;
  // past the threshold nothing more is needed (the terms are not negative)
  for (int base = moffs[i]; base < moffs[i + 1]; base += 32) {
    const int p = base + lane;
    if (p < moffs[i + 1]) {
      const int j = midx[p];
      if (code[j] == 1) mass += xb[j].x;
    }
    if (__any_sync(0xffffffffu, mass >= 0.01)) break;
  }
  for (int o = 16; o > 0; o >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
  if (lane != 0) return;
  active[i] = mass >= 0.01 ? 1 : 0;
  if (x >= 5e-4) {
    const double beta = xb[i].y;
    mu[i] = Rx[i] + (x < 0.9999 ? gamma[i] / beta : 0.0);
  } else {
    double xt = x > 1e-12 ? x : 1e-12;
    mu[i] = -(3.0 / (2.0 * xt) + 1.0 / (1.0 - xt)) / xb[i].y;
  }
}

// Active degree of every site, and the room one of its edges has under the
// degree split: out, what the site may give, and in, what it may take.
__global__ void dmd_degree_kernel(int n, const int *doffs, const int *didx, const int *owner,
                                  const int *active, const long long *X, long long xmax,
                                  long long *out, long long *in) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !active[i]) return;
  int d = 0;
  for (int p = doffs[i]; p < doffs[i + 1]; ++p) d += active[owner[didx[p]]];
  const long long di = d > 0 ? d : 1, x = X[i];
  out[i] = x / di;
  in[i] = xmax > x ? (xmax - x) / di : 0;
}

// Occupancy moved from i to o across an active edge in one step: dt J with
// J = Df/dr^2 (beta_i+beta_j)/2 xm (1-xm) (mu_i - mu_o), xm = (x_i+x_o)/2
// (exactly antisymmetric in i, o).
__device__ __forceinline__ double dmd_move(const double2 *xb, const double *mu,
                                           const long long *X, int i, int o,
                                           const DmdParams &prm) {
  const double xi = (double)X[i] * kDmdQuantum, xo = (double)X[o] * kDmdQuantum;
  const double xm = 0.5 * (xi + xo), bm = 0.5 * (xb[i].y + xb[o].y);
  const double J = prm.Df / (prm.dr * prm.dr) * bm * xm * (1.0 - xm) * (mu[i] - mu[o]);
  return prm.dt * J;
}

// A move in quanta, rounded to nearest from a value first held within
// +-4e18 (far outside any room, which is at most max_x in quanta), so that a
// move whose quanta overflow 64 bits (an empty site's chemical potential
// against an occupied one) is cut to the room like any other large move.
__device__ __forceinline__ long long dmd_quanta(double dlt) {
  return llrint(fmin(fmax(dlt * kDmdInvQuantum, -4e18), 4e18));
}

// The room of edge (i, o) in quanta: a move from i to o of at most hi, from o
// to i of at most -lo (lo <= 0).
__device__ __forceinline__ void dmd_room(const long long *out, const long long *in, int i, int o,
                                         long long &hi, long long &lo) {
  const long long out_i = out[i], out_o = out[o], in_i = in[i], in_o = in[o];
  hi = out_i < in_o ? out_i : in_o;
  lo = -(out_o < in_i ? out_o : in_i);
}

__global__ void dmd_flux_kernel(int n, const double2 *xb, const int *doffs, const int *didx,
                                const int *owner, const int *active, const long long *out,
                                const long long *in, const double *mu, const long long *X0,
                                long long *X, DmdParams prm, unsigned long long *ctl) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !active[i]) return;
  for (int p = doffs[i]; p < doffs[i + 1]; ++p) {
    int o = owner[didx[p]];
    if (o <= i || !active[o]) continue;  // each undirected edge once, from its lower end
    const double dlt = dmd_move(xb, mu, X0, i, o, prm);  // occupancy moved from i to o
    if (fabs(dlt) < prm.min_dx) continue;
    long long q = dmd_quanta(dlt);
    long long hi, lo;
    dmd_room(out, in, i, o, hi, lo);
    // a move cut to a nonzero room is counted; a zero room (empty giver,
    // full receiver) moves nothing and is not
    if (ctl && ((q > hi && hi > 0) || (q < lo && lo < 0))) atomicAdd(ctl + 2, 1ull);
    q = q > hi ? hi : (q < lo ? lo : q);
    if (q == 0) continue;
    atomicAdd((unsigned long long *)&X[i], (unsigned long long)(-q));
    atomicAdd((unsigned long long *)&X[o], (unsigned long long)q);
  }
}

// Step-control decision for a step of prm.dt at the current state: per
// site, its occupancy change over max_dx (moves below min_dx skipped, as in
// the update) and, over its edges to higher sites, each move over its
// nonzero room; the maxima go to ctl[1] and ctl[0] (a non-negative
// double's bits order as the double).
__global__ void dmd_control_kernel(int n, const double2 *xb, const int *doffs, const int *didx,
                                   const int *owner, const int *active, const long long *out,
                                   const long long *in, const double *mu, const long long *X,
                                   DmdParams prm, double max_dx, unsigned long long *ctl) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  double ratio = 0.0, dx = 0.0;
  if (i < n && active[i]) {
    for (int p = doffs[i]; p < doffs[i + 1]; ++p) {
      int o = owner[didx[p]];
      if (o == i || !active[o]) continue;
      const double dlt = dmd_move(xb, mu, X, i, o, prm);
      if (fabs(dlt) < prm.min_dx) continue;
      dx = __dsub_rn(dx, dlt);  // no contraction: the oracle rounds each term
      if (o < i) continue;  // the room of each edge once
      const long long q = dmd_quanta(dlt);
      long long hi, lo;
      dmd_room(out, in, i, o, hi, lo);
      if (q > hi && hi > 0) ratio = fmax(ratio, (double)q / (double)hi);
      if (q < lo && lo < 0) ratio = fmax(ratio, (double)q / (double)lo);
    }
  }
  double r = fabs(dx) / max_dx;
  // warp maxima (every lane of the block takes part), then one atomic per warp
  for (int off = 16; off > 0; off >>= 1) {
    ratio = fmax(ratio, __shfl_xor_sync(0xffffffffu, ratio, off));
    r = fmax(r, __shfl_xor_sync(0xffffffffu, r, off));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(ctl, (unsigned long long)__double_as_longlong(ratio));
    atomicMax(ctl + 1, (unsigned long long)__double_as_longlong(r));
  }
}

// x of every H row (real sites, then images) from its owner's quanta; the
// quanta themselves become the next step's snapshot.
__global__ void dmd_commit_kernel(int n, int n_all, const int *code, const int *owner,
                                  const long long *X, long long *X0, double2 *xb) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_all) return;
  const long long q = X[i < n ? i : owner[i]];
  if (i < n) X0[i] = q;
  if (code[i] == 1) xb[i].x = (double)q * kDmdQuantum;
}

// exact total of the quanta (128-bit), single block, fixed order
__global__ void __launch_bounds__(1024) dmd_total_kernel(int n, const int *code,
                                                        const long long *X, long long *out) {
  __shared__ __int128 sh[1024];
  __int128 v = 0;
  for (int i = threadIdx.x; i < n; i += 1024)
    if (code[i] == 1) v += (__int128)X[i];
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int s = 512; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    unsigned __int128 u = (unsigned __int128)sh[0];
    out[0] = (long long)(u >> 64);
    out[1] = (long long)(unsigned long long)(u & 0xffffffffffffffffull);
  }
}

inline int nbk(long long n) { return (int)((n + 255) / 256); }

}  // namespace

cudaError_t dmd_init(int n, const double2 *xb, const int *code, long long *X, cudaStream_t st) {
  dmd_init_kernel<<<nbk(n), 256, 0, st>>>(n, xb, code, X);
  return cudaGetLastError();
}

cudaError_t dmd_commit(const DmdArgs &a, cudaStream_t st) {
  dmd_commit_kernel<<<nbk(a.n_all), 256, 0, st>>>(a.n, a.n_all, a.code, a.owner, a.X, a.X0, a.xb);
  return cudaGetLastError();
}

cudaError_t dmd_prepare(const DmdArgs &a, const DmdParams &prm, cudaStream_t st) {
  dmd_mu_kernel<<<nbk((long long)a.n * 32), 256, 0, st>>>(a.n, a.xb, a.code, a.Rx, a.gamma,
                                                          a.moffs, a.midx, a.X, a.mu, a.active);
  dmd_degree_kernel<<<nbk(a.n), 256, 0, st>>>(a.n, a.doffs, a.didx, a.owner, a.active, a.X,
                                              std::llrint(prm.max_x * kDmdInvQuantum), a.out,
                                              a.in);
  return cudaGetLastError();
}

cudaError_t dmd_control(const DmdArgs &a, const DmdParams &prm, double max_dx,
                        cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(a.ctl, 0, 2 * sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  dmd_control_kernel<<<nbk(a.n), 256, 0, st>>>(a.n, a.xb, a.doffs, a.didx, a.owner, a.active,
                                               a.out, a.in, a.mu, a.X, prm, max_dx, a.ctl);
  return cudaGetLastError();
}

cudaError_t dmd_apply(const DmdArgs &a, const DmdParams &prm, cudaStream_t st) {
  dmd_flux_kernel<<<nbk(a.n), 256, 0, st>>>(a.n, a.xb, a.doffs, a.didx, a.owner, a.active,
                                            a.out, a.in, a.mu, a.X0, a.X, prm, a.ctl);
  return dmd_commit(a, st);
}

cudaError_t dmd_total(int n, const int *code, const long long *X, long long *out2,
                      cudaStream_t st) {
  dmd_total_kernel<<<1, 1024, 0, st>>>(n, code, X, out2);
  return cudaGetLastError();
}

}  // namespace btam
