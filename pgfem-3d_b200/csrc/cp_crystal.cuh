// cp_crystal.cuh -- crystal plasticity in the crystal frame: the local Newton
// and the element stage for contexts whose crystal rotations are orthogonal.
//
// The same Newton iterates, line search, convergence test and consistent
// tangent as k_cp_update / k_cp_tangent / k_cp_element (cp_kernels.cuh), with
// the local problem reduced by two facts of this model:
//
//  - neo-Hookean + U_Common elasticity has the Mandel stress
//    Ce S = a dev(Ce) + kappa J (J - 1) 1, a = mu det(Ce)^-1/3, and the Schmid
//    tensors are traceless, so tau_a = a s_a . Ce n_a.  In the crystal frame
//    s and n have entries 0, +-1 (over sqrt 2, sqrt 3): with T = M^T Ce' M the
//    twelve numbers t_a = sqrt 6 s_a . T n_a are sums of three of the five
//    combinations (T11 - T33, T22 - T33, T23, T13, T12), and sum_a q_a P_a is
//    sums of the q_a.  No Schmid tensor is formed.
//  - d tau_a depends on dM only through those five combinations of
//    y = d(a T) = D dM, so the 10 x 10 Newton system J (dM, dg) = -Res becomes
//    (1 + D B) y + D c dg = -D Res_M (5 rows) and the hardening row, with
//    B y = dt sum_a dgd_a P_a t_a(y) / sqrt 6 and c = -(a / g) B T: six
//    unknowns, held in registers, then dM = -Res_M - B y - c dg.  det of the
//    reduced matrix is det J, so it is singular when J is.
//
// A point iteration takes about 1.3 k FP64 instructions and no shared-memory
// matrix.  Measured at 663,552 points, load step 10 (48^3 cells): cold local
// update 18.9 -> 1.19 ms, tangent 3.18 ms -> element records 0.22 ms, whole R+K
// iterate 23.2 -> 1.76 ms, from a guess (3.6 iterations) 12.5 -> 1.25 ms; 7,986
// points 0.99 -> 0.10 ms (R and K by the row owners, assemble_gather.cuh; the
// scatter below, for meshes without their lists, takes 0.1 ms more).  The update is bound by fixed-latency waits and the
// FP64 pipe (54 % busy) at 8 warps per SM: 254 registers hold a point's state
// and the reduced matrix; at 168 registers (12 warps) spills cost more than
// the warps gain (2.03 ms an iterate).
//
// Contexts with a matrix that is not orthogonal to 1e-12 keep the sample-frame
// kernels of cp_kernels.cuh, and so do the allocation-free point update (its
// rotations are on the device, unseen by the host) and the dM/dF tangent of the
// transient and element-level calls.
#pragma once
#include <cuda_runtime.h>

#include "cp_kernels.cuh"

namespace pgb {

constexpr double kIs6 = 0.40824829046386301637;  // 1 / sqrt 6

// sqrt 6 s_a . Y n_a of the twelve systems (order of c_slip_s / c_slip_n) from
// y = (Y11 - Y33, Y22 - Y33, Y23, Y13, Y12) of a symmetric Y.
__device__ __forceinline__ void cx_t(const double *y, double *t) {
  const double al = y[0], be = y[1], gm = al - be;
  const double m32 = y[4] - y[3], m31 = y[4] - y[2], m21 = y[3] - y[2];
  const double p32 = y[4] + y[3], p31 = y[4] + y[2], p21 = y[3] + y[2];
  t[0] = be + m32, t[1] = al + m31, t[2] = gm + m21;
  t[3] = be - m32, t[4] = p31 - al, t[5] = p21 - gm;
  t[6] = p32 - be, t[7] = al - m31, t[8] = p21 + gm;
  t[9] = p32 + be, t[10] = p31 + al, t[11] = gm - m21;
}

// e . t(y) as a row vector over y: the transpose of cx_t.
__device__ __forceinline__ void cx_tT(const double *e, double *r) {
  const double g = (e[2] + e[11]) + (e[8] - e[5]);
  r[0] = ((e[1] + e[7]) + (e[10] - e[4])) + g;
  r[1] = ((e[0] + e[3]) + (e[9] - e[6])) - g;
  r[2] = ((e[7] - e[1]) + (e[4] + e[10])) + ((e[11] - e[2]) + (e[5] + e[8]));
  r[3] = ((e[3] - e[0]) + (e[6] + e[9])) + ((e[2] - e[11]) + (e[5] + e[8]));
  r[4] = ((e[0] - e[3]) + (e[6] + e[9])) + ((e[1] - e[7]) + (e[4] + e[10]));
}

// 3x3 sum over the four slip planes of v_p n_p^T, n_p the unnormalised normals
// (1,1,1), (-1,1,1), (1,-1,1), (1,1,-1); v[p][i].
__device__ __forceinline__ void cx_planes(const double (*v)[3], double *G) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double p = v[0][i] + v[1][i], m = v[0][i] - v[1][i];
    const double q = v[2][i] + v[3][i], d = v[2][i] - v[3][i];
    G[i * 3 + 0] = m + q;
    G[i * 3 + 1] = p - d;
    G[i * 3 + 2] = p + d;
  }
}

// sqrt 6 sum_a q_a P_a
__device__ __forceinline__ void cx_gamma(const double *q, double *G) {
  const double v[4][3] = {{q[1] + q[2], q[0] - q[2], -(q[0] + q[1])},
                          {q[4] + q[5], q[3] + q[5], q[4] - q[3]},
                          {q[7] + q[8], q[6] + q[8], q[6] - q[7]},
                          {q[10] + q[11], q[9] - q[11], q[9] + q[10]}};
  cx_planes(v, G);
}

// sqrt 6 sum_a c_a P_a dt_a/dy_j: the columns of 6 B / dt for the weights c.
template <int COL>
__device__ __forceinline__ void cx_bcol(const double *c, double *G) {
  if (COL == 0) {
    const double v[4][3] = {{c[1] + c[2], -c[2], -c[1]},
                            {-(c[4] + c[5]), -c[5], -c[4]},
                            {c[7] + c[8], c[8], -c[7]},
                            {c[10] + c[11], -c[11], c[10]}};
    cx_planes(v, G);
  } else if (COL == 1) {
    const double v[4][3] = {{-c[2], c[0] + c[2], -c[0]},
                            {c[5], c[3] + c[5], -c[3]},
                            {-c[8], -(c[6] + c[8]), -c[6]},
                            {-c[11], c[9] + c[11], c[9]}};
    cx_planes(v, G);
  } else if (COL == 2) {
    const double v[4][3] = {{-(c[1] + c[2]), c[2], c[1]},
                            {c[4] + c[5], c[5], c[4]},
                            {c[7] + c[8], c[8], -c[7]},
                            {c[10] + c[11], -c[11], c[10]}};
    cx_planes(v, G);
  } else if (COL == 3) {
    const double v[4][3] = {{c[2], -(c[0] + c[2]), c[0]},
                            {c[5], c[3] + c[5], -c[3]},
                            {c[8], c[6] + c[8], c[6]},
                            {-c[11], c[9] + c[11], c[9]}};
    cx_planes(v, G);
  } else {
    const double v[4][3] = {{c[1], c[0], -(c[0] + c[1])},
                            {c[4], -c[3], c[3] + c[4]},
                            {-c[7], c[6], c[6] + c[7]},
                            {c[10], c[9], c[9] + c[10]}};
    cx_planes(v, G);
  }
}

// y = D X: the five combinations of d(a T) for dM = X, with G = Ce' M,
// Mi = M^-1 and the five combinations T5 of T.
__device__ __forceinline__ void cx_D(const double *G, const double *Mi, double a, const double *T5,
                                     const double *X, double *y) {
  double tr = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0, o1 = 0.0, o2 = 0.0, o3 = 0.0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double x0 = X[k * 3], x1 = X[k * 3 + 1], x2 = X[k * 3 + 2];
    const double g0 = G[k * 3], g1 = G[k * 3 + 1], g2 = G[k * 3 + 2];
    d1 = fma(x0, g0, d1), d2 = fma(x1, g1, d2), d3 = fma(x2, g2, d3);
    o1 = fma(x1, g2, fma(x2, g1, o1));
    o2 = fma(x0, g2, fma(x2, g0, o2));
    o3 = fma(x0, g1, fma(x1, g0, o3));
    tr = fma(Mi[k], x0, fma(Mi[3 + k], x1, fma(Mi[6 + k], x2, tr)));  // Mi_lk X_kl
  }
  const double f = (-2.0 / 3.0) * tr;
  y[0] = a * fma(f, T5[0], 2.0 * (d1 - d3));
  y[1] = a * fma(f, T5[1], 2.0 * (d2 - d3));
  y[2] = a * fma(f, T5[2], o1);
  y[3] = a * fma(f, T5[3], o2);
  y[4] = a * fma(f, T5[4], o3);
}

// |x|^e of the twelve systems (flow_pow's rule), non-integer exponents out of line
__device__ __noinline__ double cx_pow(double r, double e) { return pow(r, e); }

__device__ __forceinline__ void cx_flow(double *x, double e) {
  const int n = (int)e;
  if ((double)n == e && n >= 0 && n <= 64) {
    double y[kSlip];
#pragma unroll
    for (int a = 0; a < kSlip; a++) y[a] = 1.0;
    for (int k = n; k;) {
      if (k & 1)
#pragma unroll
        for (int a = 0; a < kSlip; a++) y[a] *= x[a];
      k >>= 1;
      if (k)
#pragma unroll
        for (int a = 0; a < kSlip; a++) x[a] *= x[a];
    }
#pragma unroll
    for (int a = 0; a < kSlip; a++) x[a] = y[a];
  } else {
#pragma unroll
    for (int a = 0; a < kSlip; a++) x[a] = cx_pow(x[a], e);
  }
}

// What the residual leaves for the Newton step: slopes d gamma_dot_a / d tau_a,
// the five combinations of T, a = mu det(Ce)^-1/3 and the total slip rate.
struct CxEval {
  double dgd[kSlip], T5[5], a, gdot;
};

// C = Ce' M products shared by the residual and the step
__device__ __forceinline__ void cx_sym_mul(const double *C6, const double *M, double *G) {  // G = C M
#pragma unroll
  for (int j = 0; j < 3; j++) {
    G[j] = C6[0] * M[j] + C6[5] * M[3 + j] + C6[4] * M[6 + j];
    G[3 + j] = C6[5] * M[j] + C6[1] * M[3 + j] + C6[3] * M[6 + j];
    G[6 + j] = C6[4] * M[j] + C6[3] * M[3 + j] + C6[2] * M[6 + j];
  }
}

// The residual at (M, g): Res (crystal frame) and Res[9]; false outside the
// domain (E untouched).  detC = det Ce'.
__device__ __forceinline__ bool cx_residual(const Mat &mat, const double *C6, double detC, double g_n, double dt,
                                            const double *M, double g, double *Res, CxEval &E) {
  const double dM = det3(M);
  const double dCe = detC * dM * dM;
  if (!(g > 0.0) || !(dCe > 0.0)) return false;
  double G[9], T5[5];
  cx_sym_mul(C6, M, G);
  auto T = [&](int i, int j) { return M[i] * G[j] + M[3 + i] * G[3 + j] + M[6 + i] * G[6 + j]; };
  const double T33 = T(2, 2);
  T5[0] = T(0, 0) - T33, T5[1] = T(1, 1) - T33, T5[2] = T(1, 2), T5[3] = T(0, 2), T5[4] = T(0, 1);
  const double a = mat.mu / cbrt(dCe), im = 1.0 / mat.m, ig = 1.0 / g;
  double x[kSlip], pw[kSlip];
  cx_t(T5, x);
  const double ag = a * ig * kIs6;
#pragma unroll
  for (int k = 0; k < kSlip; k++) {
    x[k] *= ag;  // tau / g
    pw[k] = fabs(x[k]);
  }
  cx_flow(pw, im - 1.0);
  const double cd = mat.gdot0 * im * ig;
  double gdot = 0.0;
#pragma unroll
  for (int k = 0; k < kSlip; k++) {
    E.dgd[k] = cd * pw[k];
    x[k] *= mat.gdot0 * pw[k];  // slip rate
    gdot += fabs(x[k]);
  }
  double Gm[9];
  cx_gamma(x, Gm);
  const double c = dt * kIs6;
#pragma unroll
  for (int i = 0; i < 9; i++) Res[i] = fma(c, Gm[i], M[i] - (i % 4 == 0 ? 1.0 : 0.0));
  const double gs = cp_hardening(mat, gdot, g, dt).gs;
  Res[9] = g - g_n - dt * mat.G0 * gdot * (gs - g) / (gs - mat.g0);
#pragma unroll
  for (int i = 0; i < 5; i++) E.T5[i] = T5[i];
  E.a = a;
  E.gdot = gdot;
  return true;
}

// LU of the reduced matrix in registers, rows 0..4 the combinations y, row 5
// the hardening equation.  A row swap is taken when a later pivot is more than
// four times the current one (the matrix is near 1 + a positive semidefinite
// one for the small elastic strains of the model, so it is rare).  NR right-hand
// sides, rhs[row][j].  false when a pivot vanishes or is not a number.
template <int NR>
__device__ __forceinline__ bool cx_solve(double (*A)[6], double (*b)[NR]) {
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    if (k < 5) {
      double best = 0.0;
#pragma unroll
      for (int i = k + 1; i < 6; i++) best = fmax(best, fabs(A[i][k]));
      if (best > 4.0 * fabs(A[k][k])) {
#pragma unroll
        for (int i = k + 1; i < 6; i++)
          if (fabs(A[i][k]) > fabs(A[k][k])) {
#pragma unroll
            for (int j = 0; j < 6; j++) {
              const double t = A[k][j];
              A[k][j] = A[i][j];
              A[i][j] = t;
            }
#pragma unroll
            for (int j = 0; j < NR; j++) {
              const double t = b[k][j];
              b[k][j] = b[i][j];
              b[i][j] = t;
            }
          }
      }
    }
    ok = ok && fabs(A[k][k]) > 0.0;
    const double inv = 1.0 / A[k][k];
    A[k][k] = inv;  // the reciprocal pivot is kept for the back substitution
#pragma unroll
    for (int i = k + 1; i < 6; i++) {
      const double f = A[i][k] * inv;
#pragma unroll
      for (int j = k + 1; j < 6; j++) A[i][j] = fma(-f, A[k][j], A[i][j]);
#pragma unroll
      for (int j = 0; j < NR; j++) b[i][j] = fma(-f, b[k][j], b[i][j]);
    }
  }
#pragma unroll
  for (int k = 5; k >= 0; k--) {
#pragma unroll
    for (int j = 0; j < NR; j++) {
      double v = b[k][j];
#pragma unroll
      for (int i = k + 1; i < 6; i++) v = fma(-A[k][i], b[i][j], v);
      b[k][j] = v * A[k][k];
    }
  }
  return ok;
}

// The reduced matrix: columns D B (scaled dt / 6), the hardening column
// -(a / g) (D B) T and the hardening row.
__device__ __forceinline__ void cx_matrix(const Mat &mat, double dt, double g, const double *G, const double *Mi,
                                          const CxEval &E, double (*A)[6]) {
  const double c6 = dt * (1.0 / 6.0), rg = -E.a / g;
  double X[9], y[5], cg[5] = {0, 0, 0, 0, 0};
#define PGB_CX_COL(J)                        \
  cx_bcol<J>(E.dgd, X);                      \
  cx_D(G, Mi, E.a, E.T5, X, y);              \
  _Pragma("unroll") for (int i = 0; i < 5; i++) { \
    const double v = c6 * y[i];              \
    cg[i] = fma(v, E.T5[J], cg[i]);          \
    A[i][J] = i == J ? 1.0 + v : v;          \
  }
  PGB_CX_COL(0)
  PGB_CX_COL(1)
  PGB_CX_COL(2)
  PGB_CX_COL(3)
  PGB_CX_COL(4)
#undef PGB_CX_COL
#pragma unroll
  for (int i = 0; i < 5; i++) A[i][5] = rg * cg[i];
  const CpHard hd = cp_hardening(mat, E.gdot, g, dt);
  double t[kSlip], r[5];
  cx_t(E.T5, t);  // the slip rate's sign is that of t (a > 0)
#pragma unroll
  for (int k = 0; k < kSlip; k++) t[k] = t[k] < 0.0 ? -E.dgd[k] : E.dgd[k];
  cx_tT(t, r);
#pragma unroll
  for (int j = 0; j < 5; j++) A[5][j] = hd.dRg * kIs6 * r[j];
  A[5][5] = 1.0 + dt * mat.G0 / (hd.gs - mat.g0) * E.gdot - hd.dRg * E.gdot / (mat.m * g);
}

// dt sum_a P_a d gamma_dot_a for the solution (y, dg): (dt / 6) sqrt 6 sum_a P_a
// sqrt 6 dgd_a t_a(y - (a dg / g) T).
__device__ __forceinline__ void cx_slip(double dt, double g, const double *y, double dg, const CxEval &E,
                                        double *dM) {
  const double f = -E.a * dg / g;
  double z[5], q[kSlip];
#pragma unroll
  for (int i = 0; i < 5; i++) z[i] = fma(f, E.T5[i], y[i]);
  cx_t(z, q);
#pragma unroll
  for (int k = 0; k < kSlip; k++) q[k] *= E.dgd[k];
  cx_gamma(q, dM);
  const double c = dt * (1.0 / 6.0);
#pragma unroll
  for (int i = 0; i < 9; i++) dM[i] *= c;
}

// Lane-strided shared memory of a point: crystal rotation (9), Ce' (6).
constexpr int kCxLane = 15;
constexpr int kCxWarps = 4;  // warps per CTA

// max |R Res R^T| and |Res[9]| / g0: the convergence measure of cp_norm, in the
// sample frame.
__device__ __forceinline__ double cx_norm(const double *sR, const double *Res, double g0) {
  double m = fabs(Res[9]) / g0;
  double t[9];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double a = sR[(i * 3) * 32], b = sR[(i * 3 + 1) * 32], c = sR[(i * 3 + 2) * 32];
#pragma unroll
    for (int j = 0; j < 3; j++) t[i * 3 + j] = a * Res[j] + b * Res[3 + j] + c * Res[6 + j];
  }
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const double a = sR[(j * 3) * 32], b = sR[(j * 3 + 1) * 32], c = sR[(j * 3 + 2) * 32];
#pragma unroll
    for (int i = 0; i < 3; i++) m = fmax(m, fabs(t[i * 3] * a + t[i * 3 + 1] * b + t[i * 3 + 2] * c));
  }
  return m;
}

// The local Newton, one point per lane, persistent over a ticket counter.
// Lanes that finish wait until REFILL lanes of the warp are idle (or none is
// active); results are then written and new points set up together, so that
// this code runs with many lanes.  28 was chosen: whole iterate at 48^3 cells,
// cold / from a guess, 8: 2.09 / 1.73, 16: 2.05 / 1.53, 24: 1.93 / 1.39, 32: 1.88 /
// 1.37 ms; 32 would let one slow point hold a warp.
template <int REFILL>
__global__ void __launch_bounds__(32 * kCxWarps, 2) k_cp_update_cx(const CpArgs A) {
  __shared__ double smem_cx[kCxWarps * kCxLane * 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double *sR = smem_cx + warp * kCxLane * 32 + lane, *sC = sR + 9 * 32;
  const unsigned FULL = 0xffffffffu;
  const long S = A.nqp;
  const double tol = A.mat.tol;
  long qp = -1;
  bool fin = true, done = false;  // fin: no running point (qp >= 0: results to write)
  double M[9], Res[10], g = 0.0, g_n = 0.0, detC = 0.0, nr = 0.0;
  CxEval E;
  int it = 0, it0 = 0;
  bool warm = false;
  for (;;) {
    const unsigned idle = __ballot_sync(FULL, fin && !done);
    const unsigned act = __ballot_sync(FULL, !fin);
    if (!idle && !act) break;
    if (idle && (__popc(idle) >= REFILL || !act)) {
      if (fin && !done) {
        if (qp >= 0) {  // results: M and pF_{n+1} = M^-1 pF_n in the sample frame
          double t[9], Ms[9], R[9], Mi[9], pFn[9];
#pragma unroll
          for (int i = 0; i < 9; i++) R[i] = sR[i * 32];
          mm3(R, M, t);
          mm3nt(t, R, Ms);
          const bool okM = inv3(Ms, Mi), conv = nr <= tol;
#pragma unroll
          for (int i = 0; i < 9; i++) {
            A.out[i * S + qp] = Ms[i];
            pFn[i] = A.state_n[i * S + qp];
          }
          mm3(Mi, pFn, t);
#pragma unroll
          for (int i = 0; i < 9; i++) A.state_np1[i * S + qp] = okM ? t[i] : pFn[i];
          A.state_np1[9 * S + qp] = g;
          A.out[90 * S + qp] = g;
          double x[kSlip];
          cx_t(E.T5, x);
          const double c = A.dt * A.mat.m * E.a * kIs6;  // gamma_dot = m tau d gamma_dot / d tau
#pragma unroll
          for (int k = 0; k < kSlip; k++) A.out[(91 + k) * S + qp] = c * x[k] * E.dgd[k];
          if (A.iters) A.iters[qp] = it;
          if (A.conv) A.conv[qp] = (conv && okM) ? 1 : 0;
          if (!conv) atomicAdd(&A.status[1], 1ull);
          qp = -1;
        }
      }
      unsigned base = 0;
      const int leader = __ffs(idle) - 1;
      if (lane == leader) base = atomicAdd(A.counter, (unsigned)__popc(idle));
      base = __shfl_sync(FULL, base, leader);
      if (fin && !done) {
        const long cand = (long)base + __popc(idle & ((1u << lane) - 1u));
        if (cand < S) {
          qp = cand;
          const long e = qp / A.nqp_e;
          double F[9], R[9], P[9], t[9];
#pragma unroll
          for (int i = 0; i < 9; i++) {
            F[i] = A.F[i * S + qp];
            P[i] = A.state_n[i * S + qp];
            R[i] = A.Rcp[i * A.ne + e];
            sR[i * 32] = R[i];
          }
          g_n = A.state_n[9 * S + qp];
          double Pi[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, C6[6];
          inv3(P, Pi);
          mm3(F, Pi, t);
          mm3(t, R, F);  // F pF_n^-1 R: Ce' = its square in the crystal frame
          auto cc = [&](int i, int j) { return F[i] * F[j] + F[3 + i] * F[3 + j] + F[6 + i] * F[6 + j]; };
          C6[0] = cc(0, 0), C6[1] = cc(1, 1), C6[2] = cc(2, 2), C6[3] = cc(1, 2), C6[4] = cc(0, 2), C6[5] = cc(0, 1);
#pragma unroll
          for (int i = 0; i < 6; i++) sC[i * 32] = C6[i];
          const double dF = det3(F);
          detC = dF * dF;
          warm = A.guess != nullptr;
          if (warm) {
#pragma unroll
            for (int i = 0; i < 9; i++) P[i] = A.guess[i * S + qp];
            mm3(P, R, t);
            mm3tn(R, t, M);
            g = A.guess[9 * S + qp];
          } else {
#pragma unroll
            for (int i = 0; i < 9; i++) M[i] = (i % 4 == 0) ? 1.0 : 0.0;
            g = g_n;
          }
          it = it0 = 0;
#pragma unroll
          for (int k = 0; k < kSlip; k++) E.dgd[k] = 0.0;
#pragma unroll
          for (int i = 0; i < 5; i++) E.T5[i] = 0.0;
          E.a = E.gdot = 0.0;
          nr = cx_residual(A.mat, C6, detC, g_n, A.dt, M, g, Res, E) ? cx_norm(sR, Res, A.mat.g0) : 1e300;
          fin = false;
        } else {
          done = true;
        }
      }
    }
    if (!fin) {
      // one Newton step (or finish)
      const int cap = warm && A.warm_k > 0 ? A.warm_k : A.mat.max_iter;
      fin = !(nr > tol) || it - it0 >= cap || !(nr < 1e299);
      if (!fin) {
        double C6[6], dM[9], dg;
#pragma unroll
        for (int i = 0; i < 6; i++) C6[i] = sC[i * 32];
        bool ok;
        {
          double G[9], Mi[9], Am[6][6], b[6][1], y[5];
          cx_sym_mul(C6, M, G);
          const double rd = 1.0 / det3(M);
          Mi[0] = rd * (M[4] * M[8] - M[5] * M[7]);
          Mi[1] = rd * (M[2] * M[7] - M[1] * M[8]);
          Mi[2] = rd * (M[1] * M[5] - M[2] * M[4]);
          Mi[3] = rd * (M[5] * M[6] - M[3] * M[8]);
          Mi[4] = rd * (M[0] * M[8] - M[2] * M[6]);
          Mi[5] = rd * (M[2] * M[3] - M[0] * M[5]);
          Mi[6] = rd * (M[3] * M[7] - M[4] * M[6]);
          Mi[7] = rd * (M[1] * M[6] - M[0] * M[7]);
          Mi[8] = rd * (M[0] * M[4] - M[1] * M[3]);
          cx_D(G, Mi, E.a, E.T5, Res, y);
#pragma unroll
          for (int i = 0; i < 5; i++) b[i][0] = -y[i];
          b[5][0] = -Res[9];
          cx_matrix(A.mat, A.dt, g, G, Mi, E, Am);
          ok = cx_solve<1>(Am, b);
          dg = b[5][0];
#pragma unroll
          for (int i = 0; i < 5; i++) y[i] = b[i][0];
          cx_slip(A.dt, g, y, dg, E, dM);
#pragma unroll
          for (int i = 0; i < 9; i++) dM[i] = -(Res[i] + dM[i]);
        }
        if (!ok) {
          nr = 1e300;
          fin = true;
        } else {
          double lam = 1.0, nt = 1e300, Mt[9], gt = g;
          for (int ls = 0; ls < 8; ls++) {
#pragma unroll
            for (int i = 0; i < 9; i++) Mt[i] = fma(lam, dM[i], M[i]);
            gt = fma(lam, dg, g);
            if (cx_residual(A.mat, C6, detC, g_n, A.dt, Mt, gt, Res, E)) {
              nt = cx_norm(sR, Res, A.mat.g0);
              if (nt < nr || ls == 7) break;
            }
            lam *= 0.5;
          }
#pragma unroll
          for (int i = 0; i < 9; i++) M[i] = Mt[i];
          g = gt;
          nr = nt;
          it++;
        }
      }
      if (fin && warm && !(nr <= tol)) {
        // the guess did not converge in cap iterations (or left the domain):
        // restart from the elastic predictor with the full iteration budget
        warm = false;
        it0 = it;
        if (A.fallbacks) atomicAdd(A.fallbacks, 1ull);
        double C6[6];
#pragma unroll
        for (int i = 0; i < 6; i++) C6[i] = sC[i * 32];
#pragma unroll
        for (int i = 0; i < 9; i++) M[i] = (i % 4 == 0) ? 1.0 : 0.0;
        g = g_n;
        nr = cx_residual(A.mat, C6, detC, g_n, A.dt, M, g, Res, E) ? cx_norm(sR, Res, A.mat.g0) : 1e300;
        fin = false;
      }
    }
  }
}

// ---- element stage ---------------------------------------------------------

// Element record: G = (dX/dxi)^-1 F^-1 (p_a = G^T dN_a/dxi), w tau (Voigt) and
// the 36 numbers w c_(kl)(ij) of the spatial tangent, c : d = d tau - d tau -
// tau d for symmetric d (columns kl of d, rows ij); zeros for an element without
// contribution.  Contiguous per element, padded to 16 bytes; turned in shared
// memory so that a CTA writes its records in whole lines.
constexpr int kCxRec = 52;
constexpr int kCxT = 9, kCxC = 15;
constexpr int kCxRecThreads = 64;
constexpr int kCxTile = 32;  // elements per CTA of the scatter

struct CxElemArgs {
  CpElemArgs e;
  const double *Rcp;
  const uint8_t *conv;
  double dt;
  double *rec;  // kCxRec * ne
};

// Kirchhoff stress tau = pJ (a dev(be) + kappa J (J - 1) 1), be = Fe Fe^T, and
// its consistent spatial tangent from the converged local state: for a
// symmetric d the reduced system of the Newton step with right-hand side
// d(a T) at fixed M (dT = 2 H^T d H, H = Fe R) gives dM, and
//   c : d = pJ (a (2/3 (tr be d - (be : d) 1) + dev(H (l + l^T) H^T))
//               - 2/3 a x dev(be) + (kappa (2J - 1) J x) 1 - 2 kappa J (J - 1) d)
//           - tr(l) tau,     l = M^-1 dM, x = tr d + tr l.
// Six right-hand sides instead of the nine of dM/dF and 36 numbers per element
// instead of 81: the update is objective, so only symmetric d count.  Points
// that did not converge, or whose system is singular (counted in status[3]),
// keep l = 0.
__device__ __forceinline__ void cx_record(const CxElemArgs &B, long e, double *rec) {
  const CpElemArgs &A = B.e;
  const long S = A.ne;
  rec[kCxRec - 1] = 0.0;
  const double w = A.detJw[e];
  double H[9], Mu[9], be[6], tau[6];
  double Gc[9], Mi[9], E6[6][6];  // E6: right-hand sides, then solutions
  double a = 0.0, pJ = 0.0, Je = 0.0, g = 0.0;
  CxEval E;
  bool ok = w > 0.0, plast = false;
  if (ok) {
    double F[9], pF[9], pFi[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, R[9], t[9], Fp[9];
#pragma unroll
    for (int i = 0; i < 9; i++) {
      F[i] = A.F[i * S + e];
      Mu[i] = A.out[i * S + e];
      pF[i] = A.state_n[i * S + e];
      R[i] = B.Rcp[i * S + e];
    }
    inv3(pF, pFi);
    pJ = det3(pF) / det3(Mu);
    mm3(F, pFi, Fp);
    mm3(Fp, Mu, t);  // Fe
    be[0] = t[0] * t[0] + t[1] * t[1] + t[2] * t[2];
    be[1] = t[3] * t[3] + t[4] * t[4] + t[5] * t[5];
    be[2] = t[6] * t[6] + t[7] * t[7] + t[8] * t[8];
    be[3] = t[3] * t[6] + t[4] * t[7] + t[5] * t[8];
    be[4] = t[0] * t[6] + t[1] * t[7] + t[2] * t[8];
    be[5] = t[0] * t[3] + t[1] * t[4] + t[2] * t[5];
    mm3(t, R, H);
    const double dFe = det3(t), dC = dFe * dFe;
    ok = dC > 0.0;
    Je = fabs(dFe);
    a = A.mat.mu / cbrt(dC);
    g = A.out[90 * S + e];
    plast = ok && B.conv[e] != 0 && g > 0.0;
    if (plast) {
      double Mc[9], C6[6];
      mm3(Mu, R, t);
      mm3tn(R, t, Mc);
      mm3(Fp, R, t);
      auto cc = [&](int i, int j) { return t[i] * t[j] + t[3 + i] * t[3 + j] + t[6 + i] * t[6 + j]; };
      C6[0] = cc(0, 0), C6[1] = cc(1, 1), C6[2] = cc(2, 2), C6[3] = cc(1, 2), C6[4] = cc(0, 2), C6[5] = cc(0, 1);
      cx_sym_mul(C6, Mc, Gc);
      inv3(Mc, Mi);
      // slopes at the converged state
      auto hh = [&](int i, int j) { return H[i] * H[j] + H[3 + i] * H[3 + j] + H[6 + i] * H[6 + j]; };
      const double T33 = hh(2, 2);
      E.T5[0] = hh(0, 0) - T33, E.T5[1] = hh(1, 1) - T33, E.T5[2] = hh(1, 2), E.T5[3] = hh(0, 2), E.T5[4] = hh(0, 1);
      E.a = a;
      E.gdot = 0.0;
      const double im = 1.0 / A.mat.m, ig = 1.0 / g;
      double x[kSlip];
      cx_t(E.T5, x);
#pragma unroll
      for (int k = 0; k < kSlip; k++) {
        x[k] = fabs(x[k] * (a * ig * kIs6));
        E.dgd[k] = x[k];
      }
      cx_flow(E.dgd, im - 1.0);
#pragma unroll
      for (int k = 0; k < kSlip; k++) {
        E.gdot += A.mat.gdot0 * x[k] * E.dgd[k];
        E.dgd[k] *= A.mat.gdot0 * im * ig;
      }
    }
  }
  if (!ok) {
    for (int i = 0; i < kCxRec; i++) rec[i] = 0.0;
    return;
  }
  const int vk[6] = {0, 1, 2, 1, 0, 0}, vl[6] = {0, 1, 2, 2, 2, 1};
  if (plast) {
    double Am[6][6];
    cx_matrix(A.mat, B.dt, g, Gc, Mi, E, Am);
#pragma unroll
    for (int q = 0; q < 6; q++) {  // d(a T) of the unit d_kl at fixed M
      const double *hk = H + 3 * vk[q], *hl = H + 3 * vl[q];
      const double f = q < 3 ? -2.0 / 3.0 : 0.0;
      const double t33 = 2.0 * hk[2] * hl[2];
      E6[0][q] = a * fma(f, E.T5[0], 2.0 * hk[0] * hl[0] - t33);
      E6[1][q] = a * fma(f, E.T5[1], 2.0 * hk[1] * hl[1] - t33);
      E6[2][q] = a * fma(f, E.T5[2], hk[1] * hl[2] + hl[1] * hk[2]);
      E6[3][q] = a * fma(f, E.T5[3], hk[0] * hl[2] + hl[0] * hk[2]);
      E6[4][q] = a * fma(f, E.T5[4], hk[0] * hl[1] + hl[0] * hk[1]);
      E6[5][q] = 0.0;
    }
    if (!cx_solve<6>(Am, E6)) {
      atomicAdd(&A.status[3], 1ull);
      plast = false;
    }
  }
  const double trb = be[0] + be[1] + be[2], tb3 = trb * (1.0 / 3.0), pv = A.mat.kappa * Je * (Je - 1.0);
  const double dpv = A.mat.kappa * (2.0 * Je - 1.0) * Je, wp = w * pJ;
#pragma unroll
  for (int v = 0; v < 6; v++) tau[v] = a * (v < 3 ? be[v] - tb3 : be[v]) + (v < 3 ? pv : 0.0);
#pragma unroll
  for (int q = 0; q < 6; q++) {
    double Sl[6] = {0, 0, 0, 0, 0, 0}, trl = 0.0;
    if (plast) {
      double y[5], dM[9], N[9];
#pragma unroll
      for (int i = 0; i < 5; i++) y[i] = E6[i][q];
      cx_slip(B.dt, g, y, E6[5][q], E, dM);  // dM = -(B y + c dg)
#pragma unroll
      for (int i = 0; i < 9; i++) dM[i] = -dM[i];
      double l[9];
      mm3(Mi, dM, l);
      trl = l[0] + l[4] + l[8];
      mm3(H, l, N);
      auto sy = [&](int i, int j) {
        return N[i * 3] * H[j * 3] + N[i * 3 + 1] * H[j * 3 + 1] + N[i * 3 + 2] * H[j * 3 + 2];
      };
      Sl[0] = 2.0 * sy(0, 0), Sl[1] = 2.0 * sy(1, 1), Sl[2] = 2.0 * sy(2, 2);
      Sl[3] = sy(1, 2) + sy(2, 1), Sl[4] = sy(0, 2) + sy(2, 0), Sl[5] = sy(0, 1) + sy(1, 0);
    }
    const double x = (q < 3 ? 1.0 : 0.0) + trl, s3 = (Sl[0] + Sl[1] + Sl[2]) * (1.0 / 3.0);
    const double dq = q < 3 ? 1.0 : 0.5;  // the nonzero entry of d in Voigt form
#pragma unroll
    for (int v = 0; v < 6; v++) {
      const double dev_be = v < 3 ? be[v] - tb3 : be[v];
      double z = a * ((v < 3 ? Sl[v] - s3 : Sl[v]) - (2.0 / 3.0) * (v < 3 ? be[q] : 0.0) - (2.0 / 3.0) * x * dev_be);
      if (v == q) z += dq * ((2.0 / 3.0) * a * trb - 2.0 * pv);
      if (v < 3) z += dpv * x;
      rec[kCxC + q * 6 + v] = wp * (z - trl * tau[v]);
    }
  }
#pragma unroll
  for (int v = 0; v < 6; v++) rec[kCxT + v] = wp * tau[v];
  // G = (dX/dxi)^-1 F^-1
  double x[4][3], dX[9], dXi[9], F[9], Fi[9], G[9];
#pragma unroll
  for (int n = 0; n < 4; n++) {
    const int nd = A.conn[(long)n * A.ne + e];
#pragma unroll
    for (int i = 0; i < 3; i++) x[n][i] = A.X[i * A.nn + nd];
  }
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int c = 0; c < 3; c++) dX[i * 3 + c] = x[c + 1][i] - x[0][i];
  inv3(dX, dXi);
#pragma unroll
  for (int i = 0; i < 9; i++) F[i] = A.F[i * S + e];
  inv3(F, Fi);
  mm3(dXi, Fi, G);
#pragma unroll
  for (int i = 0; i < 9; i++) rec[i] = G[i];
}

__global__ void __launch_bounds__(kCxRecThreads) k_cp_record_cx(const CxElemArgs B) {
  __shared__ double srow[kCxRecThreads * (kCxRec + 1)];
  const long e0 = blockIdx.x * (long)kCxRecThreads, e = e0 + threadIdx.x;
  if (e < B.e.ne) cx_record(B, e, srow + threadIdx.x * (kCxRec + 1));
  __syncthreads();
  const int cnt = (int)(B.e.ne - e0 < kCxRecThreads ? B.e.ne - e0 : kCxRecThreads) * kCxRec;
  for (int i = threadIdx.x; i < cnt; i += kCxRecThreads)
    B.rec[e0 * kCxRec + i] = srow[(i / kCxRec) * (kCxRec + 1) + i % kCxRec];
}

// R and K from the element records: K_ab[i][k] = p_a[j] c_(ij)(kl) p_b[l] +
// d_ik p_a . tau p_b, R_a = tau p_a.  Thread (element, row node a, column
// component k); the three k of an (element, a) are adjacent lanes, so a
// reduction instruction writes runs of three doubles of a CSR row.
constexpr int kCxElemThreads = 12 * kCxTile;
__global__ void __launch_bounds__(kCxElemThreads) k_cp_scatter_cx(const CxElemArgs B) {
  const CpElemArgs &A = B.e;
  __shared__ double sm[kCxTile * (kCxRec + 1)];
  const long e0 = (long)blockIdx.x * kCxTile;
  const int tid = threadIdx.x;
  const int nel = (int)(A.ne - e0 < kCxTile ? A.ne - e0 : kCxTile);
  for (int i = tid; i < nel * kCxRec; i += kCxElemThreads)
    sm[(i / kCxRec) * (kCxRec + 1) + i % kCxRec] = B.rec[e0 * kCxRec + i];
  __syncthreads();
  const int el = tid / 12, r = tid - el * 12, a = r / 3, k = r - a * 3;
  if (el >= nel) return;
  const long e = e0 + el;
  auto rec = [&](int f) { return sm[el * (kCxRec + 1) + f]; };
  const int na = A.conn[(long)a * A.ne + e];
  const unsigned ma = A.mask[na];
  if (!ma) return;
  auto node = [&](int n, double *p) {  // rows of G; node 0: minus their sum
#pragma unroll
    for (int j = 0; j < 3; j++)
      p[j] = n == 0 ? -(rec(j) + rec(3 + j) + rec(6 + j)) : rec((n - 1) * 3 + j);
  };
  double pa[3], tp[3], s6[6];
  node(a, pa);
#pragma unroll
  for (int v = 0; v < 6; v++) s6[v] = rec(kCxT + v);
  smv(s6, pa, tp);
  {
    const int id = A.dof[k * A.nn + na];
    if (id > 0) atomicAdd(A.R + (id - 1), k == 0 ? tp[0] : (k == 1 ? tp[1] : tp[2]));
  }
  if (!A.K) return;
  // L[i][l] = sum_j p_a[j] c_(ij)(kl) for the own k
  const int row[9] = {0, 5, 4, 5, 1, 3, 4, 3, 2};
  double L[9];
#pragma unroll
  for (int l = 0; l < 3; l++) {
    const int col = k == 0 ? row[l] : (k == 1 ? row[3 + l] : row[6 + l]);
    double y[3];
#pragma unroll
    for (int v = 0; v < 6; v++) s6[v] = rec(kCxC + col * 6 + v);
    smv(s6, pa, y);
#pragma unroll
    for (int i = 0; i < 3; i++) L[i * 3 + l] = y[i];
  }
  const long base = A.rowptr0[na];
  const long rl = A.rowlen[na];
#pragma unroll 1
  for (int b = 0; b < 4; b++) {
    const int nb = A.conn[(long)b * A.ne + e];
    const unsigned mb = A.mask[nb];
    if (!((mb >> k) & 1u)) continue;
    double pb[3];
    node(b, pb);
    const double gg = tp[0] * pb[0] + tp[1] * pb[1] + tp[2] * pb[2];
    const long col = base + A.pos[(e * 4 + a) * 4 + b] + rank_of(mb, k);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      if (!((ma >> i) & 1u)) continue;
      const double v = L[i * 3] * pb[0] + L[i * 3 + 1] * pb[1] + L[i * 3 + 2] * pb[2] + (i == k ? gg : 0.0);
      atomicAdd(A.K + col + (long)rank_of(ma, i) * rl, v);
    }
  }
}

}  // namespace pgb
