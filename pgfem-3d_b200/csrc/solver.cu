// solver.cu -- linear solve and Newton-Raphson load step on the device.
//
// The consumer of the assembled operator.  The reference hands K and the
// residual to hypre (src/solvers/hypre/Hypre.cc:147-194) and iterates
// Newton-Raphson around it (src/Newton_Raphson.cc:931-1330).  Here:
//
//  - CSR SpMV, one warp per row: the row's values and column ids are read
//    contiguously (12 bytes per non-zero from HBM), the vector is gathered
//    through L2; the Krylov dot products that follow a product are fused into
//    it (per-block partial sums);
//  - restarted GMRES(kdim) (GMRes.cc, the reference's default solver) and
//    BiCGSTAB (BCGStab.cc), both right-preconditioned by diagonal scaling
//    (ScaleDiag.cc: 1/K_ii, or 1.1 where |K_ii| <= 1e-5) or not at all.  GMRES
//    orthogonalises by classical Gram-Schmidt applied twice and runs whole
//    restart cycles in one cooperative kernel (gmres_persistent.cuh), large
//    systems as a sequence of launches (launches_faster, kMostRows).  The
//    sequence and BiCGSTAB keep their scalars in device memory, so an iteration
//    is a fixed sequence of launches with no host round trip; every kernel
//    returns at once when the device-side `done` flag is set (converged, end of
//    a GMRES cycle, or broken down), so the host queues several iterations
//    between checks.  Reductions sum per-block
//    partials in a fixed order: the result does not depend on timing;
//  - pgfem_gpu_newton_step: full Newton (stiffness every iteration, FNR = 1)
//    for one load step through the public assembly entry point, converged
//    when ||R|| / ||R_0|| <= nor_min or ||R|| <= computer_zero (the
//    reference's nor / nor2 test, :1203-1217, 1323).  No line search.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>

#include "gmres_persistent.cuh"
#include "pgfem_gpu.h"

namespace {

constexpr int kBlk = 256;            // threads per block of every vector kernel
constexpr int kFin = 1024;           // threads of the one-block finalize kernels
constexpr int kBlocksPerSm = 8;      // grid-stride grids: 8 blocks per SM
constexpr double kDiagThresh = 1e-5, kDiagReplace = 1.1;  // ScaleDiag.cc constants

// Device-resident BiCGSTAB state.
struct Scalars {
  double rho, rho_new, alpha, omega;
  double bnorm2, rnorm2, tol2;
  int iter, done, breakdown, pad;
};

enum Stage { kInit = 0, kAlpha = 1, kOmega = 2, kRho = 3, kNorm = 4 };

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block sum of two values into part0/part1[blockIdx.x] (thread 0 writes).
__device__ __forceinline__ void block_partials(double d0, double d1, double *part0, double *part1) {
  __shared__ double s0[kBlk / 32], s1[kBlk / 32];
  d0 = warp_sum(d0);
  d1 = warp_sum(d1);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    s0[w] = d0;
    s1[w] = d1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int i = 0; i < kBlk / 32; i++) {
      a += s0[i];
      b += s1[i];
    }
    if (part0) part0[blockIdx.x] = a;
    if (part1) part1[blockIdx.x] = b;
  }
}

// y = K x; with w0: partial (w0, y); with self: partial (y, y).
// One warp per row, grid-stride over rows.
__global__ void __launch_bounds__(kBlk) k_spmv(long n, const int *__restrict__ Ap, const int *__restrict__ Ai,
                                               const double *__restrict__ K, const double *__restrict__ x,
                                               double *__restrict__ y, const double *__restrict__ w0, int self,
                                               double *part0, double *part1, const Scalars *S) {
  if (S && S->done) return;
  const int lane = threadIdx.x & 31;
  const long warp0 = ((long)blockIdx.x * kBlk + threadIdx.x) >> 5;
  const long nwarps = ((long)gridDim.x * kBlk) >> 5;
  double d0 = 0.0, d1 = 0.0;
  for (long i = warp0; i < n; i += nwarps) {
    const int b = Ap[i], e = Ap[i + 1];
    double acc = 0.0;
    for (int j = b + lane; j < e; j += 32) acc = fma(K[j], x[Ai[j]], acc);
    acc = warp_sum(acc);
    if (lane == 0) {
      y[i] = acc;
      if (w0) d0 = fma(w0[i], acc, d0);
      if (self) d1 = fma(acc, acc, d1);
    }
  }
  if (part0 || part1) block_partials(d0, d1, part0, part1);
}

// dinv[i] = 1 / K_ii (|K_ii| > thresh), else the replacement; 1 without
// preconditioning.
__global__ void k_diag_scale(long n, const long *__restrict__ dpos, const double *__restrict__ K, int precond,
                             double *__restrict__ dinv) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    double v = 1.0;
    if (precond == PGFEM_PRECOND_DIAG_SCALE) {
      const double d = dpos[i] >= 0 ? K[dpos[i]] : 0.0;
      v = fabs(d) > kDiagThresh ? 1.0 / d : kDiagReplace;
    }
    dinv[i] = v;
  }
}

// r = b - Ax (Ax in r on entry), rh = r, p = v = 0; partials (r, r), (b, b).
__global__ void __launch_bounds__(kBlk) k_init(long n, const double *__restrict__ b, double *__restrict__ r,
                                               double *__restrict__ rh, double *__restrict__ p,
                                               double *__restrict__ v, double *part0, double *part1) {
  double d0 = 0.0, d1 = 0.0;
  for (long i = blockIdx.x * (long)kBlk + threadIdx.x; i < n; i += (long)gridDim.x * kBlk) {
    const double ri = b[i] - r[i];
    r[i] = ri;
    rh[i] = ri;
    p[i] = 0.0;
    v[i] = 0.0;
    d0 = fma(ri, ri, d0);
    d1 = fma(b[i], b[i], d1);
  }
  block_partials(d0, d1, part0, part1);
}

// p = r + beta (p - omega v), ph = dinv p  (first iteration: p = r).
__global__ void __launch_bounds__(kBlk) k_update_p(long n, const double *__restrict__ r, double *__restrict__ p,
                                                   const double *__restrict__ v, const double *__restrict__ dinv,
                                                   double *__restrict__ ph, const Scalars *S) {
  if (S->done) return;
  const double beta = S->iter == 0 ? 0.0 : (S->rho_new / S->rho) * (S->alpha / S->omega);
  const double om = S->omega;
  for (long i = blockIdx.x * (long)kBlk + threadIdx.x; i < n; i += (long)gridDim.x * kBlk) {
    const double pi = S->iter == 0 ? r[i] : r[i] + beta * (p[i] - om * v[i]);
    p[i] = pi;
    ph[i] = dinv[i] * pi;
  }
}

// s = r - alpha v, sh = dinv s  (s stored in place of r).
__global__ void __launch_bounds__(kBlk) k_update_s(long n, double *__restrict__ r, const double *__restrict__ v,
                                                   const double *__restrict__ dinv, double *__restrict__ sh,
                                                   const Scalars *S) {
  if (S->done) return;
  const double al = S->alpha;
  for (long i = blockIdx.x * (long)kBlk + threadIdx.x; i < n; i += (long)gridDim.x * kBlk) {
    const double si = r[i] - al * v[i];
    r[i] = si;
    sh[i] = dinv[i] * si;
  }
}

// x += alpha ph + omega sh, r = s - omega t; partials (rh, r), (r, r).
__global__ void __launch_bounds__(kBlk) k_update_xr(long n, double *__restrict__ x, const double *__restrict__ ph,
                                                    const double *__restrict__ sh, double *__restrict__ r,
                                                    const double *__restrict__ t, const double *__restrict__ rh,
                                                    double *part0, double *part1, const Scalars *S) {
  if (S->done) return;
  const double al = S->alpha, om = S->omega;
  double d0 = 0.0, d1 = 0.0;
  for (long i = blockIdx.x * (long)kBlk + threadIdx.x; i < n; i += (long)gridDim.x * kBlk) {
    x[i] += al * ph[i] + om * sh[i];
    const double ri = r[i] - om * t[i];
    r[i] = ri;
    d0 = fma(rh[i], ri, d0);
    d1 = fma(ri, ri, d1);
  }
  block_partials(d0, d1, part0, part1);
}

// One block: sums the partials in a fixed order and advances the scalars.
__global__ void __launch_bounds__(kFin) k_finalize(int nblocks, const double *part0, const double *part1, int stage,
                                                   Scalars *S, double *out) {
  if (stage != kInit && stage != kNorm && S->done) return;
  __shared__ double s0[kFin], s1[kFin];
  double a = 0.0, b = 0.0;
  for (int i = threadIdx.x; i < nblocks; i += kFin) {
    a += part0[i];
    if (part1) b += part1[i];
  }
  s0[threadIdx.x] = a;
  s1[threadIdx.x] = b;
  __syncthreads();
  for (int o = kFin / 2; o; o >>= 1) {
    if (threadIdx.x < o) {
      s0[threadIdx.x] += s0[threadIdx.x + o];
      s1[threadIdx.x] += s1[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x) return;
  const double d0 = s0[0], d1 = s1[0];
  switch (stage) {
    case kInit:  // d0 = (r, r), d1 = (b, b)
      S->rho = S->alpha = S->omega = 1.0;
      S->rho_new = d0;
      S->rnorm2 = d0;
      S->bnorm2 = d1;
      S->iter = 0;
      S->breakdown = 0;
      S->done = (d0 <= S->tol2 * d1) ? 1 : 0;
      break;
    case kAlpha:  // d0 = (rh, v)
      if (d0 == 0.0 || !isfinite(d0)) {
        S->breakdown = 1;
        S->done = 1;
      } else {
        S->alpha = S->rho_new / d0;
      }
      break;
    case kOmega:  // d0 = (t, s), d1 = (t, t)
      if (d1 == 0.0 || !isfinite(d1)) {
        S->breakdown = 1;
        S->done = 1;
      } else {
        S->omega = d0 / d1;
      }
      break;
    case kRho:  // d0 = (rh, r), d1 = (r, r)
      S->rho = S->rho_new;
      S->rho_new = d0;
      S->rnorm2 = d1;
      S->iter += 1;
      if (!isfinite(d1)) {
        S->breakdown = 1;
        S->done = 1;
      } else if (d1 <= S->tol2 * S->bnorm2) {
        S->done = 1;
      } else if (d0 == 0.0 || S->omega == 0.0) {
        S->breakdown = 1;
        S->done = 1;
      }
      break;
    case kNorm:  // plain dot product into *out
      *out = d0;
      break;
  }
}

// y = a x + y  /  y = a x
__global__ void k_axpy(long n, double a, const double *__restrict__ x, double *__restrict__ y, int overwrite) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] = overwrite ? a * x[i] : fma(a, x[i], y[i]);
}

// x = -x
__global__ void k_negate(long n, double *x) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) x[i] = -x[i];
}

__global__ void __launch_bounds__(kBlk) k_dot(long n, const double *__restrict__ a, const double *__restrict__ b,
                                              double *part0) {
  double d = 0.0;
  for (long i = blockIdx.x * (long)kBlk + threadIdx.x; i < n; i += (long)gridDim.x * kBlk) d = fma(a[i], b[i], d);
  block_partials(d, 0.0, part0, nullptr);
}

// partials of ||b - w||^2 (true residual, w = K x)
__global__ void __launch_bounds__(kBlk) k_resid(long n, const double *__restrict__ b, const double *__restrict__ w,
                                                double *part0) {
  double d = 0.0;
  for (long i = blockIdx.x * (long)kBlk + threadIdx.x; i < n; i += (long)gridDim.x * kBlk) {
    const double r = b[i] - w[i];
    d = fma(r, r, d);
  }
  block_partials(d, 0.0, part0, nullptr);
}

// ---- GMRES as a launch sequence (large systems, see launches_faster) -----------
constexpr int kTile = 8;  // basis vectors per register tile of the dot products

struct GState {
  double beta0, bnorm, tol;
  int j;          // Arnoldi steps completed in this cycle
  int m;          // Krylov dimension
  int done, converged, breakdown, pad;
};

// w = K (dinv o V[j]), j = G->j (one warp per row)
__global__ void __launch_bounds__(kBlk) k_spmv_basis(long n, const int *__restrict__ Ap, const int *__restrict__ Ai,
                                                     const double *__restrict__ K, const double *__restrict__ dinv,
                                                     const double *__restrict__ V, double *__restrict__ w,
                                                     const GState *G) {
  if (G->done) return;
  const double *x = V + (long)G->j * n;
  const int lane = threadIdx.x & 31;
  const long warp0 = ((long)blockIdx.x * kBlk + threadIdx.x) >> 5;
  const long nwarps = ((long)gridDim.x * kBlk) >> 5;
  for (long i = warp0; i < n; i += nwarps) {
    const int b = Ap[i], e = Ap[i + 1];
    double acc = 0.0;
    for (int jj = b + lane; jj < e; jj += 32) {
      const int c = Ai[jj];
      acc = fma(K[jj], dinv[c] * x[c], acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) w[i] = acc;
  }
}

// partials part[t * nblk + block] = (V[t], w), t <= j.  Each warp walks its
// own slice of the block's rows through all tiles of kTile basis vectors and
// keeps its sums in shared memory, so warps never wait for each other between
// tiles; one barrier at the end combines the warps.
constexpr int kMdWarps = kBlk / 32;
__global__ void __launch_bounds__(kBlk) k_multidot(long n, const double *__restrict__ V, const double *__restrict__ w,
                                                   double *part, const GState *G) {
  if (G->done) return;
  extern __shared__ double smd[];  // [kMdWarps][nt]
  const int nt = G->j + 1;
  const int wp = threadIdx.x >> 5, l = threadIdx.x & 31;
  const long chunk = (n + gridDim.x - 1) / gridDim.x;
  const long i0 = (long)blockIdx.x * chunk, i1 = i0 + chunk < n ? i0 + chunk : n;
  for (int t0 = 0; t0 < nt; t0 += kTile) {
    double acc[kTile];
#pragma unroll
    for (int u = 0; u < kTile; u++) acc[u] = 0.0;
    // two rows per pass: sixteen loads in flight, same summation order
#pragma unroll 2
    for (long i = i0 + threadIdx.x; i < i1; i += kBlk) {
      const double wi = w[i];
#pragma unroll
      for (int u = 0; u < kTile; u++)
        if (t0 + u < nt) acc[u] = fma(V[(long)(t0 + u) * n + i], wi, acc[u]);
    }
#pragma unroll
    for (int u = 0; u < kTile; u++) {
      const double v = warp_sum(acc[u]);
      if (l == 0 && t0 + u < nt) smd[wp * nt + t0 + u] = v;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nt; t += kBlk) {
    double sum = 0.0;
    for (int q = 0; q < kMdWarps; q++) sum += smd[q * nt + t];
    part[(long)t * gridDim.x + blockIdx.x] = sum;
  }
}

inline size_t multidot_smem(int nt) { return sizeof(double) * kMdWarps * (size_t)nt; }

// h[t] = sum of the partials (one warp per t); column j of H gets h
// (accumulate: +=), htmp gets h for the following update of w.
__global__ void __launch_bounds__(kFin) k_multidot_fin(int nblk, const double *part, double *H, double *htmp,
                                                       int accumulate, const GState *G) {
  if (G->done) return;
  const int nt = G->j + 1, m1 = G->m + 1;
  const int wp = threadIdx.x >> 5, l = threadIdx.x & 31;
  for (int t = wp; t < nt; t += kFin / 32) {
    double sum = 0.0;
    for (int b = l; b < nblk; b += 32) sum += part[(long)t * nblk + b];
    sum = warp_sum(sum);
    if (l == 0) {
      htmp[t] = sum;
      double &h = H[(long)G->j * m1 + t];
      h = accumulate ? h + sum : sum;
    }
  }
}

// w -= sum_{t <= j} V[t] htmp[t]; with norm: partials of (w, w) of the result
// (the second Gram-Schmidt pass and ||w|| in one sweep)
__global__ void __launch_bounds__(kBlk) k_multiaxpy(long n, const double *__restrict__ V, double *__restrict__ w,
                                                    const double *__restrict__ htmp, double *part0,
                                                    const GState *G) {
  if (G->done) return;
  const int nt = G->j + 1;
  double d = 0.0;
  for (long i = blockIdx.x * (long)kBlk + threadIdx.x; i < n; i += (long)gridDim.x * kBlk) {
    double a0 = w[i], a1 = 0.0, a2 = 0.0, a3 = 0.0;
    int t = 0;
    // eight basis loads in flight per pass, same summation order
#pragma unroll 2
    for (; t + 4 <= nt; t += 4) {
      a0 = fma(-V[(long)t * n + i], htmp[t], a0);
      a1 = fma(-V[(long)(t + 1) * n + i], htmp[t + 1], a1);
      a2 = fma(-V[(long)(t + 2) * n + i], htmp[t + 2], a2);
      a3 = fma(-V[(long)(t + 3) * n + i], htmp[t + 3], a3);
    }
    for (; t < nt; t++) a0 = fma(-V[(long)t * n + i], htmp[t], a0);
    const double r = (a0 + a1) + (a2 + a3);
    w[i] = r;
    d = fma(r, r, d);
  }
  if (part0) block_partials(d, 0.0, part0, nullptr);
}

// H[j+1, j] = ||w|| (one block)
__global__ void __launch_bounds__(kFin) k_gnorm_fin(int nblk, const double *part0, double *H, const GState *G) {
  if (G->done) return;
  __shared__ double s0[kFin];
  double a = 0.0;
  for (int i = threadIdx.x; i < nblk; i += kFin) a += part0[i];
  s0[threadIdx.x] = a;
  __syncthreads();
  for (int o = kFin / 2; o; o >>= 1) {
    if (threadIdx.x < o) s0[threadIdx.x] += s0[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) H[(long)G->j * (G->m + 1) + G->j + 1] = sqrt(s0[0]);
}

// V[j+1] = w / H[j+1, j] (zero when the new direction vanished)
__global__ void k_gscale(long n, double *__restrict__ V, const double *__restrict__ w, const double *H,
                         const GState *G) {
  if (G->done) return;
  const double h = H[(long)G->j * (G->m + 1) + G->j + 1];
  const double inv = h > 0.0 ? 1.0 / h : 0.0;
  double *v = V + (long)(G->j + 1) * n;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    v[i] = w[i] * inv;
}

// One thread: apply the previous rotations to column j, form rotation j,
// update the residual estimate |g[j+1]|, advance j, end the cycle when it is
// converged, full, or broken down.
__global__ void k_givens(double *H, double *cs, double *sn, double *g, GState *G) {
  if (G->done) return;
  const int j = G->j, m1 = G->m + 1;
  double *h = H + (long)j * m1;
  for (int t = 0; t < j; t++) {
    const double a = cs[t] * h[t] + sn[t] * h[t + 1];
    h[t + 1] = -sn[t] * h[t] + cs[t] * h[t + 1];
    h[t] = a;
  }
  const double hn = h[j + 1];
  const double d = hypot(h[j], hn);
  if (!(d > 0.0) || !isfinite(d)) {
    G->breakdown = 1;
    G->done = 1;
    return;
  }
  cs[j] = h[j] / d;
  sn[j] = hn / d;
  h[j] = d;
  h[j + 1] = 0.0;
  g[j + 1] = -sn[j] * g[j];
  g[j] = cs[j] * g[j];
  G->j = j + 1;
  if (fabs(g[j + 1]) <= G->tol * G->bnorm || hn == 0.0) {
    G->converged = 1;
    G->done = 1;
  } else if (G->j >= G->m) {
    G->done = 1;
  }
}

// Cycle start: V[0] = b - w (w = K x), partials (r, r), (b, b).
__global__ void __launch_bounds__(kBlk) k_ginit(long n, const double *__restrict__ b, const double *__restrict__ w,
                                                double *__restrict__ V, double *part0, double *part1) {
  double d0 = 0.0, d1 = 0.0;
  for (long i = blockIdx.x * (long)kBlk + threadIdx.x; i < n; i += (long)gridDim.x * kBlk) {
    const double ri = b[i] - w[i];
    V[i] = ri;
    d0 = fma(ri, ri, d0);
    d1 = fma(b[i], b[i], d1);
  }
  block_partials(d0, d1, part0, part1);
}

// One block: beta0 = ||r0||, g = (beta0, 0, ...), j = 0.
__global__ void __launch_bounds__(kFin) k_ginit_fin(int nblk, const double *part0, const double *part1, double *g,
                                                    GState *G) {
  __shared__ double s0[kFin], s1[kFin];
  double a = 0.0, b = 0.0;
  for (int i = threadIdx.x; i < nblk; i += kFin) {
    a += part0[i];
    b += part1[i];
  }
  s0[threadIdx.x] = a;
  s1[threadIdx.x] = b;
  __syncthreads();
  for (int o = kFin / 2; o; o >>= 1) {
    if (threadIdx.x < o) {
      s0[threadIdx.x] += s0[threadIdx.x + o];
      s1[threadIdx.x] += s1[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x) return;
  G->beta0 = sqrt(s0[0]);
  G->bnorm = sqrt(s1[0]);
  G->j = 0;
  G->breakdown = 0;
  G->converged = (G->beta0 <= G->tol * G->bnorm) ? 1 : 0;
  G->done = G->converged || !isfinite(G->beta0);
  if (!isfinite(G->beta0)) G->breakdown = 1;
  g[0] = G->beta0;
}

// V[0] /= beta0
__global__ void k_gscale0(long n, double *V, const GState *G) {
  if (G->done) return;
  const double inv = 1.0 / G->beta0;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) V[i] *= inv;
}

// One thread: y = H(0:k, 0:k)^-1 g(0:k), k = j (upper triangular after the
// rotations).
__global__ void k_backsolve(const double *H, const double *g, double *y, const GState *G) {
  const int k = G->j, m1 = G->m + 1;
  for (int t = k - 1; t >= 0; t--) {
    double a = g[t];
    for (int q = t + 1; q < k; q++) a -= H[(long)q * m1 + t] * y[q];
    const double d = H[(long)t * m1 + t];
    y[t] = d != 0.0 ? a / d : 0.0;
  }
}

// x += dinv o (V y) over the cycle's k = j basis vectors
__global__ void k_gupdate_x(long n, const double *__restrict__ V, const double *__restrict__ y,
                            const double *__restrict__ dinv, double *__restrict__ x, const GState *G) {
  const int k = G->j;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int t = 0; t < k; t++) acc = fma(V[(long)t * n + i], y[t], acc);
    x[i] = fma(dinv[i], acc, x[i]);
  }
}

// Position of the diagonal entry of every row (-1 when the row has none).
void find_diagonal(const int *Ap, const int *Ai, long n, long *dpos) {
  for (long i = 0; i < n; i++) {
    dpos[i] = -1;
    int lo = Ap[i], hi = Ap[i + 1];
    while (lo < hi) {  // columns sorted ascending
      const int mid = (lo + hi) >> 1;
      if (Ai[mid] < i) lo = mid + 1;
      else hi = mid;
    }
    if (lo < Ap[i + 1] && Ai[lo] == i) dpos[i] = lo;
  }
}

int g_sms = 0;
int grid_size() {
  if (!g_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_sms <= 0) g_sms = 148;
  }
  return g_sms * kBlocksPerSm;
}

int device_ok() {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
    cudaGetLastError();
    return 0;
  }
  int dev = 0, major = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
  return major >= 10;
}

}  // namespace

struct pgfem_gpu_solver {
  long n = 0, nnz = 0;
  pgfem_solver_opts opts{};
  int grid = 0;
  int *Ap = nullptr, *Ai = nullptr;
  long *dpos = nullptr;
  double *dinv = nullptr, *r = nullptr, *rh = nullptr, *p = nullptr, *v = nullptr, *ph = nullptr, *sh = nullptr,
         *t = nullptr;
  double *part0 = nullptr, *part1 = nullptr, *dot_out = nullptr;
  Scalars *S = nullptr;
  Scalars *hS = nullptr;  // pinned host copy
  // GMRES
  double *V = nullptr, *H = nullptr, *g = nullptr, *y = nullptr, *w = nullptr, *z = nullptr;
  ulonglong2 *words = nullptr;      // tagged partial sums and sums
  unsigned long long seq = 0;       // sequence numbers used so far
  gmp::State *PS = nullptr, *hPS = nullptr;  // device state, pinned host copy
  unsigned *bar = nullptr;
  bool launches = false;  // GMRES by the launch sequence: its rotations, dot products and state
  double *cs = nullptr, *sn = nullptr, *htmp = nullptr, *gpart = nullptr;
  GState *G = nullptr, *hG = nullptr;
  int p_rows = 0, p_blocks = 0, p_ldv = 0, p_vs = 0, p_ks = 0, p_kcap = 0;  // row blocks of the persistent kernel
  size_t p_smem = 0;
  // Newton buffers (allocated by the first newton_step)
  double *R = nullptr, *K = nullptr, *du = nullptr;
  long bytes = 0;
};

namespace {

template <class T>
int salloc(pgfem_gpu_solver *s, T **p, size_t n) {
  if (cudaMalloc((void **)p, (n ? n : 1) * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return PGFEM_GPU_ENOMEM;
  }
  s->bytes += (long)((n ? n : 1) * sizeof(T));
  return PGFEM_GPU_OK;
}

void release(pgfem_gpu_solver *s) {
  void *ptrs[] = {s->Ap, s->Ai, s->dpos, s->dinv, s->r, s->rh, s->p, s->v, s->ph, s->sh, s->t,
                  s->part0, s->part1, s->dot_out, s->S, s->R, s->K, s->du, s->V, s->H,
                  s->g, s->y, s->w, s->words, s->PS, s->z, s->bar, s->cs, s->sn, s->htmp, s->gpart, s->G};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  if (s->hS) cudaFreeHost(s->hS);
  if (s->hPS) cudaFreeHost(s->hPS);
  if (s->hG) cudaFreeHost(s->hG);
}

#define SK(x)                         \
  do {                                \
    if ((x) != cudaSuccess) {         \
      cudaGetLastError();             \
      return PGFEM_GPU_ECUDA;         \
    }                                 \
  } while (0)

int ew_grid(const pgfem_gpu_solver *s) {
  const long need = (s->n + kBlk - 1) / kBlk;
  return (int)(need < s->grid ? (need > 0 ? need : 1) : s->grid);
}

// ||a||^2 or (a, b) on the stream into s->dot_out (device)
int dot_device(pgfem_gpu_solver *s, const double *a, const double *b, cudaStream_t st) {
  const int g = ew_grid(s);
  k_dot<<<g, kBlk, 0, st>>>(s->n, a, b, s->part0);
  k_finalize<<<1, kFin, 0, st>>>(g, s->part0, nullptr, kNorm, s->S, s->dot_out);
  SK(cudaGetLastError());
  return PGFEM_GPU_OK;
}

int bicg_impl(pgfem_gpu_solver *s, const double *K, const double *b, double *x, pgfem_solve_info *info,
              cudaStream_t st) {
  const long n = s->n;
  const int g = ew_grid(s);
  const int gs = s->grid;  // SpMV grid (warp per row, grid-stride)
  // tolerance into the device scalars, preconditioner, initial residual
  Scalars init{};
  init.tol2 = s->opts.tol * s->opts.tol;
  SK(cudaMemcpyAsync(s->S, &init, sizeof(Scalars), cudaMemcpyHostToDevice, st));
  k_diag_scale<<<g, kBlk, 0, st>>>(n, s->dpos, K, s->opts.precond, s->dinv);
  k_spmv<<<gs, kBlk, 0, st>>>(n, s->Ap, s->Ai, K, x, s->r, nullptr, 0, nullptr, nullptr, nullptr);
  k_init<<<g, kBlk, 0, st>>>(n, b, s->r, s->rh, s->p, s->v, s->part0, s->part1);
  k_finalize<<<1, kFin, 0, st>>>(g, s->part0, s->part1, kInit, s->S, nullptr);
  SK(cudaGetLastError());
  const int every = s->opts.check_every > 0 ? s->opts.check_every : 8;
  int queued = 0;
  for (;;) {
    const int k = (s->opts.maxit - queued) < every ? (s->opts.maxit - queued) : every;
    for (int it = 0; it < k; it++) {
      k_update_p<<<g, kBlk, 0, st>>>(n, s->r, s->p, s->v, s->dinv, s->ph, s->S);
      k_spmv<<<gs, kBlk, 0, st>>>(n, s->Ap, s->Ai, K, s->ph, s->v, s->rh, 0, s->part0, nullptr, s->S);
      k_finalize<<<1, kFin, 0, st>>>(gs, s->part0, nullptr, kAlpha, s->S, nullptr);
      k_update_s<<<g, kBlk, 0, st>>>(n, s->r, s->v, s->dinv, s->sh, s->S);
      k_spmv<<<gs, kBlk, 0, st>>>(n, s->Ap, s->Ai, K, s->sh, s->t, s->r, 1, s->part0, s->part1, s->S);
      k_finalize<<<1, kFin, 0, st>>>(gs, s->part0, s->part1, kOmega, s->S, nullptr);
      k_update_xr<<<g, kBlk, 0, st>>>(n, x, s->ph, s->sh, s->r, s->t, s->rh, s->part0, s->part1, s->S);
      k_finalize<<<1, kFin, 0, st>>>(g, s->part0, s->part1, kRho, s->S, nullptr);
    }
    SK(cudaGetLastError());
    queued += k;
    SK(cudaMemcpyAsync(s->hS, s->S, sizeof(Scalars), cudaMemcpyDeviceToHost, st));
    SK(cudaStreamSynchronize(st));
    if (s->hS->done || queued >= s->opts.maxit) break;
  }
  const Scalars &h = *s->hS;
  if (info) {
    info->iters = h.iter;
    info->res_norm = h.bnorm2 > 0.0 ? std::sqrt(h.rnorm2 / h.bnorm2) : std::sqrt(h.rnorm2);
    info->converged = (h.done && !h.breakdown && h.rnorm2 <= init.tol2 * h.bnorm2) ? 1 : 0;
    info->breakdown = h.breakdown;
  }
  return PGFEM_GPU_OK;
}

// tagged words of the persistent kernel: partial sums and sums
size_t words_of(const pgfem_gpu_solver *s) {
  return (size_t)(s->opts.kdim + 2) * s->p_blocks + s->opts.kdim + 3;
}

// Whether the launch sequence takes less time than the persistent kernel.  That
// one multiplies by K with a quarter to a third of the sequence's warps, which costs
// time per row (less where rows are long), reads the basis faster, and saves some
// 45 us of launches a step; the line is where the three cancel.  Measured, us per
// step, persistent / sequence.  J2 quadratic tets (85 entries a row): 345,744 rows, kdim
// 10: 185 / 185, kdim 100: 248 / 308; 545,832 rows, kdim 30: 296 / 288, kdim 100: 391 /
// 480; 888,822 rows, kdim 30: 493 / 418, kdim 100: 633 / 687; 1,574,640 rows, kdim 30:
// 923 / 786, kdim 100: 1156 / 1228; 3,060,300 rows, kdim 30: 1836 / 1576, kdim 100:
// 2301 / 2380.  Linear tets (43 entries a row): 86,490 rows, kdim 30: 34 / 73; 669,780
// rows, kdim 30: 348 / 285, kdim 100: 464 / 476; 1,574,640 rows, kdim 30: 831 / 617, kdim
// 100: 1078 / 1059.
bool launches_faster(long n, long nnz, int kdim) {
  return kdim + 25e6 / (double)n < 150.0 - 0.68 * (double)nnz / (double)n;
}

// Rows of a CTA up to which the persistent kernel is used: its slice of w takes 166 KB
// of shared memory, so that the fixed part fits at every restart length (4.07 M
// rows at kdim 100 would be the end of it).  3,060,300 rows are 20,678 a CTA, and
// there the two are within 4 % at kdim 100.
constexpr int kMostRows = 20736;
static_assert(gmp::smem_fixed(kMostRows, PGFEM_GMRES_MAX_KDIM) <= gmp::kSmemMost, "a plan for every restart length");

// Row blocks of the persistent kernel: one CTA per SM, at least 32 rows each,
// with the basis slice and the K rows in shared memory where they fit.  False when
// the blocks have too many rows: the launch sequence takes any number.
bool plan_persistent(pgfem_gpu_solver *s, const int *Ap) {
  const long n = s->n;
  const int m = s->opts.kdim;
  long nblk = (n + 31) / 32;
  if (nblk > g_sms) nblk = g_sms;
  const long rows = (((n + nblk - 1) / nblk) + 3) / 4 * 4;
  if (rows > kMostRows) return false;
  s->p_rows = (int)rows;
  s->p_blocks = (int)((n + s->p_rows - 1) / s->p_rows);
  long cap = 0;
  for (int b = 0; b < s->p_blocks; b++) {
    const long lo = (long)b * s->p_rows, hi = lo + s->p_rows < n ? lo + s->p_rows : n;
    if (Ap[hi] - Ap[lo] > cap) cap = Ap[hi] - Ap[lo];
  }
  cap = (cap + 1) / 2 * 2;
  const size_t most = gmp::kSmemMost, fixed = gmp::smem_fixed(s->p_rows, m);
  const int ldv = (s->p_rows + 7) / 16 * 16 + 8;
  const size_t vs = sizeof(double) * (size_t)ldv * (m + 1), ks = 12 * (size_t)cap + sizeof(int) * (s->p_rows + 1);
  s->p_vs = fixed + vs <= most;
  s->p_ks = fixed + (s->p_vs ? vs : 0) + ks <= most;
  s->p_ldv = s->p_vs ? ldv : (int)n;
  s->p_kcap = s->p_ks ? (int)cap : 0;
  s->p_smem = fixed + (s->p_vs ? vs : 0) + (s->p_ks ? ks : 0);
  return true;
}

int gmres_persistent(pgfem_gpu_solver *s, const double *K, const double *b, double *x, pgfem_solve_info *info,
                     cudaStream_t st) {
  const long n = s->n;
  const int g = ew_grid(s);
  k_diag_scale<<<g, kBlk, 0, st>>>(n, s->dpos, K, s->opts.precond, s->dinv);
  gmp::Args A{};
  A.n = n;
  A.rows = s->p_rows;
  A.ldv = s->p_ldv;
  A.m = s->opts.kdim;
  A.nblk = s->p_blocks;
  A.vs = s->p_vs;
  A.ks = s->p_ks;
  A.kcap = s->p_kcap;
  A.Ap = s->Ap;
  A.Ai = s->Ai;
  A.K = K;
  A.dinv = s->dinv;
  A.b = b;
  A.x = x;
  A.V = s->V;
  A.z = s->z;
  A.H = s->H;
  A.g = s->g;
  A.y = s->y;
  A.slot = s->words;
  A.res = s->words + (size_t)(s->opts.kdim + 2) * s->p_blocks;
  A.S = s->PS;
  A.bar = s->bar;
  A.maxit = s->opts.maxit;
  A.wait_ns = 2000000000ull;
  // cycles a launch: about 0.1 s of work at the rate of a step's reads
  const double step = 12.0 * s->nnz + 16.0 * (double)n * A.m;
  const double cyc = 2e11 / (A.m * (step + 5e7));
  A.max_cycles = cyc < 1.0 ? 1 : (cyc > 1000.0 ? 1000 : (int)cyc);
  gmp::State init{};
  init.tol = s->opts.tol;
  *s->hPS = init;
  SK(cudaMemcpyAsync(s->PS, s->hPS, sizeof(init), cudaMemcpyHostToDevice, st));
  do {
    SK(cudaMemsetAsync(s->bar, 0, sizeof(unsigned), st));
    A.seq0 = s->seq;
    s->seq += 1ull << 32;  // more than a launch uses
    void *args[] = {&A};
    SK(cudaLaunchCooperativeKernel((const void *)gmp::k_gmres_cycles, dim3(s->p_blocks), dim3(gmp::kThreads), args,
                                   s->p_smem, st));
    SK(cudaMemcpyAsync(s->hPS, s->PS, sizeof(init), cudaMemcpyDeviceToHost, st));
    SK(cudaStreamSynchronize(st));
    if (s->hPS->timeout) return PGFEM_GPU_ETIMEOUT;
  } while (!s->hPS->stop);
  const gmp::State h = *s->hPS;
  // true relative residual ||b - K x|| / ||b||
  k_spmv<<<s->grid, kBlk, 0, st>>>(n, s->Ap, s->Ai, K, x, s->w, nullptr, 0, nullptr, nullptr, nullptr);
  k_resid<<<g, kBlk, 0, st>>>(n, b, s->w, s->part0);
  k_finalize<<<1, kFin, 0, st>>>(g, s->part0, nullptr, kNorm, s->S, s->dot_out);
  SK(cudaGetLastError());
  double rr = 0.0;
  SK(cudaMemcpyAsync(&rr, s->dot_out, sizeof(double), cudaMemcpyDeviceToHost, st));
  SK(cudaStreamSynchronize(st));
  if (info) {
    info->iters = h.iters;
    info->res_norm = h.bnorm > 0.0 ? std::sqrt(rr) / h.bnorm : std::sqrt(rr);
    info->converged = h.converged;
    info->breakdown = h.breakdown;
  }
  return PGFEM_GPU_OK;
}

int gmres_launches(pgfem_gpu_solver *s, const double *K, const double *b, double *x, pgfem_solve_info *info,
                   cudaStream_t st) {
  const long n = s->n;
  const int g = ew_grid(s), gs = s->grid, m = s->opts.kdim;
  const int gm = g < g_sms * 4 ? g : g_sms * 4;  // one wave of the dot kernel
  const int every = s->opts.check_every > 0 ? s->opts.check_every : 8;
  k_diag_scale<<<g, kBlk, 0, st>>>(n, s->dpos, K, s->opts.precond, s->dinv);
  GState init{};
  init.tol = s->opts.tol;
  init.m = m;
  SK(cudaMemcpyAsync(s->G, &init, sizeof(GState), cudaMemcpyHostToDevice, st));
  int total = 0;
  bool converged = false, breakdown = false;
  while (true) {
    // cycle start from the current x
    k_spmv<<<gs, kBlk, 0, st>>>(n, s->Ap, s->Ai, K, x, s->w, nullptr, 0, nullptr, nullptr, nullptr);
    k_ginit<<<g, kBlk, 0, st>>>(n, b, s->w, s->V, s->part0, s->part1);
    k_ginit_fin<<<1, kFin, 0, st>>>(g, s->part0, s->part1, s->g, s->G);
    k_gscale0<<<g, kBlk, 0, st>>>(n, s->V, s->G);
    SK(cudaGetLastError());
    int steps = 0;
    for (;;) {
      int k = every;
      if (k > m - steps) k = m - steps;
      if (k > s->opts.maxit - total - steps) k = s->opts.maxit - total - steps;
      for (int it = 0; it < k; it++) {
        // the basis has steps + it + 1 vectors at this step (host-known count
        // sizes the dot kernel's shared memory; the kernels read j themselves)
        const int nt = steps + it + 1;
        k_spmv_basis<<<gs, kBlk, 0, st>>>(n, s->Ap, s->Ai, K, s->dinv, s->V, s->w, s->G);
        for (int pass = 0; pass < 2; pass++) {
          k_multidot<<<gm, kBlk, multidot_smem(nt), st>>>(n, s->V, s->w, s->gpart, s->G);
          k_multidot_fin<<<1, kFin, 0, st>>>(gm, s->gpart, s->H, s->htmp, pass, s->G);
          k_multiaxpy<<<g, kBlk, 0, st>>>(n, s->V, s->w, s->htmp, pass ? s->part0 : nullptr, s->G);
        }
        k_gnorm_fin<<<1, kFin, 0, st>>>(g, s->part0, s->H, s->G);
        k_gscale<<<g, kBlk, 0, st>>>(n, s->V, s->w, s->H, s->G);
        k_givens<<<1, 1, 0, st>>>(s->H, s->cs, s->sn, s->g, s->G);
      }
      SK(cudaGetLastError());
      steps += k;
      SK(cudaMemcpyAsync(s->hG, s->G, sizeof(GState), cudaMemcpyDeviceToHost, st));
      SK(cudaStreamSynchronize(st));
      if (s->hG->done || k <= 0 || steps >= m || total + steps >= s->opts.maxit) break;
    }
    // x += D V y over the steps of this cycle
    k_backsolve<<<1, 1, 0, st>>>(s->H, s->g, s->y, s->G);
    k_gupdate_x<<<g, kBlk, 0, st>>>(n, s->V, s->y, s->dinv, x, s->G);
    SK(cudaGetLastError());
    SK(cudaMemcpyAsync(s->hG, s->G, sizeof(GState), cudaMemcpyDeviceToHost, st));
    SK(cudaStreamSynchronize(st));
    total += s->hG->j;
    converged = s->hG->converged != 0;
    breakdown = s->hG->breakdown != 0;
    if (converged || breakdown || total >= s->opts.maxit || s->hG->j == 0) break;
  }
  // true relative residual ||b - K x|| / ||b||
  k_spmv<<<gs, kBlk, 0, st>>>(n, s->Ap, s->Ai, K, x, s->w, nullptr, 0, nullptr, nullptr, nullptr);
  k_resid<<<g, kBlk, 0, st>>>(n, b, s->w, s->part0);
  k_finalize<<<1, kFin, 0, st>>>(g, s->part0, nullptr, kNorm, s->S, s->dot_out);
  SK(cudaGetLastError());
  double rr = 0.0;
  SK(cudaMemcpyAsync(&rr, s->dot_out, sizeof(double), cudaMemcpyDeviceToHost, st));
  SK(cudaStreamSynchronize(st));
  if (info) {
    const double bn = s->hG->bnorm;
    info->iters = total;
    info->res_norm = bn > 0.0 ? std::sqrt(rr) / bn : std::sqrt(rr);
    info->converged = converged ? 1 : 0;
    info->breakdown = breakdown ? 1 : 0;
  }
  return PGFEM_GPU_OK;
}

int solve_impl(pgfem_gpu_solver *s, const double *K, const double *b, double *x, pgfem_solve_info *info,
               cudaStream_t st) {
  if (s->opts.solver != PGFEM_SOLVER_GMRES) return bicg_impl(s, K, b, x, info, st);
  return s->launches ? gmres_launches(s, K, b, x, info, st) : gmres_persistent(s, K, b, x, info, st);
}

}  // namespace

extern "C" {

int pgfem_gpu_solver_create(const int *Ap, const int *Ai, long nrows, const pgfem_solver_opts *opts,
                            pgfem_gpu_solver **out) {
  if (!out) return PGFEM_GPU_EINVAL;
  *out = nullptr;
  if (!Ap || !Ai || nrows <= 0 || !opts || opts->maxit <= 0 || !(opts->tol > 0.0) ||
      (opts->solver != PGFEM_SOLVER_BCG_STAB && opts->solver != PGFEM_SOLVER_GMRES) ||
      (opts->precond != PGFEM_PRECOND_NONE && opts->precond != PGFEM_PRECOND_DIAG_SCALE))
    return PGFEM_GPU_EINVAL;
  if (opts->solver == PGFEM_SOLVER_GMRES && opts->kdim <= 0) return PGFEM_GPU_EINVAL;
  if (opts->solver == PGFEM_SOLVER_GMRES && opts->kdim > PGFEM_GMRES_MAX_KDIM) return PGFEM_GPU_ELIMIT;
  if (Ap[0] != 0) return PGFEM_GPU_EINVAL;
  for (long i = 0; i < nrows; i++)
    if (Ap[i + 1] < Ap[i]) return PGFEM_GPU_EINVAL;
  const long nnz = Ap[nrows];
  for (long j = 0; j < nnz; j++)
    if (Ai[j] < 0 || Ai[j] >= nrows) return PGFEM_GPU_EPATTERN;
  if (!device_ok()) return PGFEM_GPU_ENODEV;
  if (opts->solver == PGFEM_SOLVER_GMRES &&
      (cudaFuncSetAttribute(gmp::k_gmres_cycles, cudaFuncAttributeMaxDynamicSharedMemorySize, gmp::kSmemMost) !=
           cudaSuccess ||
       cudaFuncSetAttribute(k_multidot, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)multidot_smem(PGFEM_GMRES_MAX_KDIM)) != cudaSuccess)) {
    cudaGetLastError();
    return PGFEM_GPU_ECUDA;
  }
  pgfem_gpu_solver *s = new pgfem_gpu_solver();
  s->n = nrows;
  s->nnz = nnz;
  s->opts = *opts;
  s->grid = grid_size();
  const bool gmres = opts->solver == PGFEM_SOLVER_GMRES;
  if (gmres) s->launches = !plan_persistent(s, Ap) || launches_faster(nrows, nnz, opts->kdim);
  long *hdpos = new long[nrows];
  find_diagonal(Ap, Ai, nrows, hdpos);
  int r = PGFEM_GPU_OK;
  if ((r = salloc(s, &s->Ap, nrows + 1)) || (r = salloc(s, &s->Ai, nnz)) || (r = salloc(s, &s->dpos, nrows)) ||
      (r = salloc(s, &s->dinv, nrows)) || (r = salloc(s, &s->r, nrows)) || (r = salloc(s, &s->rh, nrows)) ||
      (r = salloc(s, &s->p, nrows)) || (r = salloc(s, &s->v, nrows)) || (r = salloc(s, &s->ph, nrows)) ||
      (r = salloc(s, &s->sh, nrows)) || (r = salloc(s, &s->t, nrows)) || (r = salloc(s, &s->part0, s->grid)) ||
      (r = salloc(s, &s->part1, s->grid)) || (r = salloc(s, &s->dot_out, 1)) || (r = salloc(s, &s->S, 1)) ||
      (gmres && ((r = salloc(s, &s->V, (size_t)(opts->kdim + 1) * nrows)) ||
                 (r = salloc(s, &s->H, (size_t)(opts->kdim + 1) * opts->kdim)) ||
                 (r = salloc(s, &s->g, opts->kdim + 1)) || (r = salloc(s, &s->y, opts->kdim)) ||
                 (r = salloc(s, &s->w, nrows)))) ||
      (gmres && !s->launches && ((r = salloc(s, &s->words, words_of(s))) || (r = salloc(s, &s->PS, 1)) ||
                                 (r = salloc(s, &s->z, nrows)) || (r = salloc(s, &s->bar, 1)))) ||
      (s->launches && ((r = salloc(s, &s->cs, opts->kdim)) || (r = salloc(s, &s->sn, opts->kdim)) ||
                       (r = salloc(s, &s->htmp, opts->kdim + 1)) ||
                       (r = salloc(s, &s->gpart, (size_t)(opts->kdim + 1) * s->grid)) || (r = salloc(s, &s->G, 1))))) {
    delete[] hdpos;
    release(s);
    delete s;
    return r;
  }
  if (cudaMallocHost((void **)&s->hS, sizeof(Scalars)) != cudaSuccess ||
      (s->PS && cudaMallocHost((void **)&s->hPS, sizeof(gmp::State)) != cudaSuccess) ||
      (s->G && cudaMallocHost((void **)&s->hG, sizeof(GState)) != cudaSuccess) ||
      (s->words && cudaMemset(s->words, 0, sizeof(ulonglong2) * words_of(s)) != cudaSuccess) ||
      cudaMemcpy(s->Ap, Ap, sizeof(int) * (nrows + 1), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(s->Ai, Ai, sizeof(int) * nnz, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(s->dpos, hdpos, sizeof(long) * nrows, cudaMemcpyHostToDevice) != cudaSuccess) {
    cudaGetLastError();
    delete[] hdpos;
    release(s);
    delete s;
    return PGFEM_GPU_ECUDA;
  }
  delete[] hdpos;
  *out = s;
  return PGFEM_GPU_OK;
}

int pgfem_gpu_solver_destroy(pgfem_gpu_solver *s) {
  if (!s) return PGFEM_GPU_EINVAL;
  release(s);
  delete s;
  return PGFEM_GPU_OK;
}

long pgfem_gpu_solver_device_bytes(const pgfem_gpu_solver *s) { return s ? s->bytes : -1; }

int pgfem_gpu_spmv(pgfem_gpu_solver *s, const double *d_K, const double *d_x, double *d_y, void *stream) {
  if (!s || !d_K || !d_x || !d_y) return PGFEM_GPU_EINVAL;
  cudaStream_t st = (cudaStream_t)stream;
  k_spmv<<<s->grid, kBlk, 0, st>>>(s->n, s->Ap, s->Ai, d_K, d_x, d_y, nullptr, 0, nullptr, nullptr, nullptr);
  SK(cudaGetLastError());
  return PGFEM_GPU_OK;
}

int pgfem_gpu_solve(pgfem_gpu_solver *s, const double *d_K, const double *d_b, double *d_x,
                    pgfem_solve_info *info, void *stream) {
  if (!s || !d_K || !d_b || !d_x) return PGFEM_GPU_EINVAL;
  return solve_impl(s, d_K, d_b, d_x, info, (cudaStream_t)stream);
}

int pgfem_gpu_newton_step(pgfem_gpu_ctx *ctx, pgfem_gpu_solver *s, double *d_u, const double *d_u_presc,
                          double dt, const pgfem_newton_opts *o, pgfem_newton_info *info, void *stream) {
  if (!ctx || !s || !d_u || !o || !info || o->iter_max <= 0 || !(o->nor_min > 0.0)) return PGFEM_GPU_EINVAL;
  if (pgfem_gpu_nnz(ctx) != s->nnz) return PGFEM_GPU_EPATTERN;
  std::memset(info, 0, sizeof(*info));
  cudaStream_t st = (cudaStream_t)stream;
  int r;
  if (!s->R && ((r = salloc(s, &s->R, s->n)) || (r = salloc(s, &s->K, s->nnz)) || (r = salloc(s, &s->du, s->n))))
    return r;
  const int g = ew_grid(s);
  double NORM = 0.0;
  for (int iter = 0;; iter++) {
    if ((r = pgfem_gpu_assemble_RK_device(ctx, d_u, d_u_presc, dt, s->R, s->K, stream))) return r;
    if ((r = dot_device(s, s->R, s->R, st))) return r;
    double nrm2 = 0.0;
    SK(cudaMemcpyAsync(&nrm2, s->dot_out, sizeof(double), cudaMemcpyDeviceToHost, st));
    SK(cudaStreamSynchronize(st));
    pgfem_gpu_status es;
    if ((r = pgfem_gpu_read_status(ctx, &es, 1))) return r;
    info->elem_failures += es.inverted + es.nonconverged + es.bad_diagonal + es.other;
    const double nor2 = std::sqrt(nrm2);
    if (iter == 0) NORM = nor2 > o->computer_zero ? nor2 : (o->computer_zero > 0.0 ? o->computer_zero : 1.0);
    const double nor = nor2 / NORM;
    if (iter < PGFEM_NEWTON_HISTORY) info->nor_hist[iter] = nor;
    info->iters = iter;
    info->nor = nor;
    info->nor2 = nor2;
    if (!std::isfinite(nor) || info->elem_failures) {
      info->converged = 0;
      return PGFEM_GPU_OK;
    }
    if (nor <= o->nor_min || nor2 <= o->computer_zero) {
      info->converged = 1;
      return PGFEM_GPU_OK;
    }
    if (iter >= o->iter_max) {
      info->converged = 0;
      return PGFEM_GPU_OK;
    }
    // K du = -R, du from zero
    k_negate<<<g, kBlk, 0, st>>>(s->n, s->R);
    SK(cudaMemsetAsync(s->du, 0, sizeof(double) * s->n, st));
    SK(cudaGetLastError());
    pgfem_solve_info si{};
    if ((r = solve_impl(s, s->K, s->R, s->du, &si, st))) return r;
    info->lin_iters += si.iters;
    if (!si.converged) {
      info->lin_failed = 1;
      info->converged = 0;
      return PGFEM_GPU_OK;
    }
    // three-field element: the element pressure and volume follow du
    // (compute_d_theta_dP at the current u), then u += du
    if (pgfem_gpu_three_field_enabled(ctx) &&
        (r = pgfem_gpu_three_field_update_device(ctx, d_u, d_u_presc, s->du, nullptr, stream)))
      return r;
    k_axpy<<<g, kBlk, 0, st>>>(s->n, 1.0, s->du, d_u, 0);
    SK(cudaGetLastError());
  }
}

}  // extern "C"
