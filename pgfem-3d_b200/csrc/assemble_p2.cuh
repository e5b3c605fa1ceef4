// assemble_p2.cuh -- FP64 R+K assembly of quadratic tets from point records, one
// warp per element.
//
// Same operation as the other assembly kernels (fd_residuals_MP +
// stiffmat_fd_MP for the constitutive-model element, src/fd_residuals.cc:
// 468-636, src/stiffmat_fd.cc:831-993), in two kernels:
//
//  k_qp_update<..., YREC = true>  one thread per quadrature point: F, the
//      constitutive update (run_integration_algorithm,
//      src/constitutive_model.cc:1100-1129; state n -> n+1) and a 26-double
//      point record from which the assembly forms the matrices of the element
//      contraction:
//        G = (dX/dxi)^-1 F^-1      (p_a = G^T dN_a/dxi = F^-T grad_X N_a)
//        T' = a1 w/2 1 + w tau,  s'' = -2/3 w s,  U' = w a2 1 + s'',
//        W' = w (a4 n + a5 dev(n^2)),  h = a1 w / 2
//      for the spatial tangent c = a1 I + a2 1(x)1 - 2/3 (s(x)1 + 1(x)s)
//      + a4 n(x)n + a5 n(x)dev(n^2) (cm_models.cuh) and w = det(dX/dxi) x weight.
//      At a plastic point s = |s| n (radial return), so the record holds
//      V = n and s'' = c V with c = -2/3 w (s : n); elsewhere V = s,
//      c = -2/3 w and a4 = a5 = 0.  A warp's records are contiguous: staged in
//      shared memory and written by one bulk copy.
//
//  k_assemble_p2r  persistent grid, one element per warp at a time.  With p of node
//      b at point q, T = T'p, U = U'p, W = W'p, the element block K_ab[i][k]
//      (compute_stiffness_matrix, src/constitutive_model.cc:1520-1616, in spatial
//      form) is
//        K_ab[i][k] = sum_q sum_j p_a[j] Y_q[j][i],
//        Y_q[j][i] = d_jk h p_b[i] + d_ij U_b[k] + s''_ij p_b[k] + n_ij W_b[k] + d_ik T_b[j]
//      for lane (b, k), and lane 30 holds the residual R_a[i] with Y = w tau
//      (compute_residual_vector, :1628-1662).  A lane builds its Y in registers
//      and Z_q = G_q Y_q, the derivatives by the corners' barycentric coordinates
//      (Z of corner 0 = -sum of the others).  dN_a is linear in those, lambda_l(q)
//      = B + (A - B) d_lq by the rule, so the sum over a point's ten nodes reduces
//      to S_l = sum_q Z_q,l, the corner's own Z, and one sum per edge: 24 FP64
//      operations per point and lane where the plain contraction takes 90.
//      The columns of one row (node a, component i) then are the warp's lanes: one
//      reduction instruction writes the element's 30 entries of a row, so that
//      neighbouring column nodes share the 32-byte sectors (340 sectors per
//      element, against 440 for eight columns of four rows), through the
//      node-block map (fd_res_assemble, src/fd_residuals.cc:58-73; PLoc_Sparse,
//      src/PLoc_Sparse.cc:15-175).
//      What bounds it is the rate of FP64 reductions in L2 (about 300e9 per second
//      measured, whatever the sectors), so a warp takes runs of up to eight consecutive
//      elements and hands the entries of two nodes that the next element has too
//      to that element through shared memory (930 -> about 680 reductions per
//      element with the face-chained processing order).
//      Against the earlier kernel (Y through shared memory, the contraction on the
//      FP64 tensor cores at 96 x 16 x 12 padded, a scatter of eight columns of four
//      rows): J2, 1.57 M elements, whole call 6003 -> 5224 us; three-field, 146,334
//      elements, 612 -> 502 us; J2, 2,058 elements, 28.9 -> 26.7 us.
#pragma once
#include <cstdint>

#include "assemble.cuh"
#include "assemble_p1.cuh"  // bounded mbarrier waits

namespace pgb {

constexpr int kQRec = kRec;  // point record of the linear-tet path: G 9, w, tau 6, s 6, n 6, dev(n^2) 6, a1 a2 a4 a5
// point record of the quadratic-tet path, one point after the other in processing
// order: T' 6, V 6, G 9, w a2, c, w a4, w a5, h
constexpr int kYT = 0, kYV = 6, kYG = 12, kYWa2 = 21, kYC = 22, kYW4 = 23, kYW5 = 24, kYH = 25;
constexpr int kYRec = 26;
// the three-field (CM3F) element adds w J, w and the element's theta and P
constexpr int kYWJ = 26, kYW = 27, kYTheta = 28, kYP = 29;
constexpr int kYRecTF = 30;
__host__ __device__ constexpr int yrec_fields(bool tf) { return tf ? kYRecTF : kYRec; }

struct QpArgs {
  const double *X;      // 3*nn
  const double *unode;  // 3*nn
  const int *conn;      // NNE*ne (SoA)
  long nn, ne, nqp;
  const double *F0;
  const int *elem_group;  // FE2 batches: element -> group (or nullptr)
  const double *F0_tab;   // group -> macro deformation (9)
  const double *state_n;
  double *state_np1;
  double *qrec;         // kQRec*nqp (SoA) or, for 10-node elements, kYRec (kYRecTF) doubles per point
  unsigned long long *status;
  // processing order: record slot e' holds element perm[e'] (nullptr: e' = e);
  // the state stays in element order
  const int *perm;
  Mat mat;
  ShapeTable shp;
  // three-field element (10-node records, hyperelastic and J2 models): the
  // pressure and the volume of each element (element order)
  const double *tf_P, *tf_theta;
  double wscale;  // factor of every record's point weight (the transient's factor of K)
};

// One point: rec is its record (YREC: NRF doubles, 16-byte aligned) or the first
// field's array (SoA of nqp).
template <int NNE, int NQP, int MODEL, bool YREC, bool TF>
__device__ __forceinline__ void qp_point(const QpArgs &A, long qs, double *rec) {
  constexpr bool PLASTIC = (MODEL == 1);
  constexpr int NRF = yrec_fields(TF);
  constexpr int NR = YREC ? NRF : kQRec;
  const long es = qs / NQP;
  const int q = (int)(qs - es * NQP);
  const long e = A.perm ? (long)A.perm[es] : es;
  const long qp = e * NQP + q;  // state index
  double dX[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, dU[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int b = 0; b < NNE; b++) {
    const int n = A.conn[(long)b * A.ne + e];
    const double g0 = A.shp.dNxi[q][b][0], g1 = A.shp.dNxi[q][b][1], g2 = A.shp.dNxi[q][b][2];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double x = A.X[i * A.nn + n], u = A.unode[i * A.nn + n];
      dX[i * 3 + 0] += g0 * x;
      dX[i * 3 + 1] += g1 * x;
      dX[i * 3 + 2] += g2 * x;
      dU[i * 3 + 0] += g0 * u;
      dU[i * 3 + 1] += g1 * u;
      dU[i * 3 + 2] += g2 * u;
    }
  }
  const long S = A.nqp;
  const double detJ = det3(dX);
  double dXi[9], F[9], Fi[9];
  bool ok = detJ > 0.0 && inv3(dX, dXi);
  if (ok) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++)
        F[i * 3 + j] = (i == j ? 1.0 : 0.0) + dU[i * 3 + 0] * dXi[0 * 3 + j] + dU[i * 3 + 1] * dXi[1 * 3 + j] +
                       dU[i * 3 + 2] * dXi[2 * 3 + j];
    const double *F0 = A.elem_group ? A.F0_tab + 9 * (long)A.elem_group[e] : A.F0;
    if (F0)
#pragma unroll
      for (int i = 0; i < 9; i++) F[i] += F0[i];
  }
  const double J = ok ? det3(F) : -1.0;
  if (ok) ok = J > 0.0 && inv3(F, Fi);
  if (!ok) {
    atomicAdd(&A.status[0], 1ull);
#pragma unroll
    for (int c = 0; c < NR; c++) rec[YREC ? c : c * S + qs] = 0.0;
    return;
  }
  double Ast[6] = {1, 1, 1, 0, 0, 0}, alpha = 0.0;
  if (PLASTIC) {
#pragma unroll
    for (int c = 0; c < 6; c++) Ast[c] = A.state_n[c * S + qp];
    alpha = A.state_n[6 * S + qp];
  }
  QpTangent t;
  double Anp1[6], alpha_np1;
  spatial_update<PLASTIC>(A.mat, F, J, Ast, alpha, t, Anp1, &alpha_np1);
  double tfP = 0.0, tfTh = 0.0;
  if (TF) {
    // three-field element: the volumetric stress is the element pressure,
    // P J 1, at fixed P (no kappa J^2 U'' term in the tangent)
    tfP = A.tf_P[e];
    tfTh = A.tf_theta[e];
    double dU, d2U;
    vol_derivs(A.mat.vol_pot, J, dU, d2U);
    const double pJ = A.mat.kappa * J * dU, PJ = tfP * J;
#pragma unroll
    for (int c = 0; c < 3; c++) t.tau[c] += PJ - pJ;
    t.a1 += 2.0 * (pJ - PJ);
    t.a2 += PJ - A.mat.kappa * (J * dU + J * J * d2U);
  }
  if (PLASTIC && A.state_np1) {
#pragma unroll
    for (int c = 0; c < 6; c++) A.state_np1[c * S + qp] = Anp1[c];
    A.state_np1[6 * S + qp] = alpha_np1;
  }
  double G[9];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      G[i * 3 + j] = dXi[i * 3 + 0] * Fi[0 * 3 + j] + dXi[i * 3 + 1] * Fi[1 * 3 + j] + dXi[i * 3 + 2] * Fi[2 * 3 + j];
  const double w = detJ * A.shp.w[q] * A.wscale;
  if (YREC) {
    const double h = 0.5 * t.a1 * w, c23 = (2.0 / 3.0) * w;
    // plastic point: n != 0 (the unit flow direction, s = (s : n) n)
    const bool pl = PLASTIC && (t.n[0] != 0.0 || t.n[1] != 0.0 || t.n[2] != 0.0 || t.n[3] != 0.0 ||
                                t.n[4] != 0.0 || t.n[5] != 0.0);
    double r[NRF];
#pragma unroll
    for (int c = 0; c < 6; c++) {
      r[kYT + c] = h * (c < 3 ? 1.0 : 0.0) + w * t.tau[c];
      r[kYV + c] = pl ? t.n[c] : t.s[c];
    }
#pragma unroll
    for (int c = 0; c < 9; c++) r[kYG + c] = G[c];
    r[kYWa2] = w * t.a2;
    r[kYC] = pl ? -c23 * sdot(t.s, t.n) : -c23;
    r[kYW4] = w * t.a4;
    r[kYW5] = w * t.a5;
    r[kYH] = h;
    if (TF) {
      r[kYWJ] = w * J;
      r[kYW] = w;
      r[kYTheta] = tfTh;
      r[kYP] = tfP;
    }
#pragma unroll
    for (int c = 0; c < NRF; c += 2) *reinterpret_cast<double2 *>(rec + c) = make_double2(r[c], r[c + 1]);
  } else {
#pragma unroll
    for (int c = 0; c < 9; c++) rec[c * S + qs] = G[c];
    rec[9 * S + qs] = w;
#pragma unroll
    for (int c = 0; c < 6; c++) {
      rec[(10 + c) * S + qs] = t.tau[c];
      rec[(16 + c) * S + qs] = t.s[c];
      rec[(22 + c) * S + qs] = t.n[c];
      rec[(28 + c) * S + qs] = t.D[c];
    }
    rec[34 * S + qs] = t.a1;
    rec[35 * S + qs] = t.a2;
    rec[36 * S + qs] = t.a4;
    rec[37 * S + qs] = t.a5;
  }
}

template <int NNE, int NQP, int MODEL, bool YREC = false, bool TF = false>
__global__ void __launch_bounds__(128) k_qp_update(const QpArgs A) {
  if (YREC) {
    pdl_wait();
    pdl_release();
  }
  const long qs = blockIdx.x * (long)blockDim.x + threadIdx.x;  // record slot
  if (!YREC) {
    if (qs < A.nqp) qp_point<NNE, NQP, MODEL, YREC, TF>(A, qs, A.qrec);
    return;
  }
  // the warp's records are contiguous: staged in shared memory, written by one bulk copy
  constexpr int NRF = YREC ? yrec_fields(TF) : 2;
  __shared__ __align__(16) double stage[4][32 * NRF];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (qs < A.nqp) qp_point<NNE, NQP, MODEL, YREC, TF>(A, qs, stage[warp] + lane * NRF);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  const long q0 = qs - lane;
  if (lane == 0 && q0 < A.nqp) {
    const long n = A.nqp - q0 < 32 ? A.nqp - q0 : 32;
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(A.qrec + q0 * NRF),
                 "r"((unsigned)__cvta_generic_to_shared(stage[warp])), "r"((unsigned)(n * NRF * sizeof(double)))
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group 0;" ::: "memory");
  }
}

// ---- element assembly -------------------------------------------------------

constexpr int kP2Threads = 128;
// Longest run of elements: longer ones hand over more entries, but spread the
// warps over more of the mesh than L2 holds the rows of (1.57 M elements, call time
// for 4, 8, 16, 32: 5.72, 5.16, 6.08, 6.72 ms).
constexpr int kP2Run = 8;
// Per-element scatter block (int32 words, 480 bytes so that it copies in 16-byte chunks):
//   [0, 30)    row base of (node a, component i): CSR offset of the row, -1 if not free
//   [32, 62)   residual index of (a, i): free DOF id - 1, -1 if not free
//   [64, 114)  node-pair positions pos[a][b] (uint16, column offset of b's block in a's rows)
//   [114, 117) free-component masks of the ten nodes (bytes)
//   [117, 119) 4 bits per node: its local number in the previous element of the
//              processing order, 15 when not there (or when either holds it twice)
//   [119]      bit a: node a is in the next element too (once in both)
constexpr int kEBW = 120;
constexpr int kEBRes = 32, kEBPos = 64, kEBMask = 114, kEBPrev = 117, kEBNext = 119;
// the four-point rule: point q has barycentric coordinate A at corner (q + 1) mod 4, B at the others
constexpr double kP2RuleA = 0.58541020, kP2RuleB = 0.13819660;

constexpr int kP2Stage = 30 * 32;  // doubles of the values an element hands to the next one: [row 3 a + i][lane]

// bytes of one element's copies: its point records and its scatter block
__host__ __device__ constexpr unsigned p2r_elem_bytes(bool tf) {
  return (unsigned)(4 * sizeof(double) * yrec_fields(tf) + sizeof(int) * kEBW);
}
inline size_t p2r_smem_bytes(bool tf) {
  return (size_t)(kP2Threads / 32) * 2 *
         (p2r_elem_bytes(tf) + kP2Stage * sizeof(double) + sizeof(uint64_t));
}

// one-dimensional bulk copy global -> shared through the tensor memory
// accelerator, completing on an mbarrier (16-byte aligned, size a multiple of 16)
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          (unsigned)__cvta_generic_to_shared(dst)),
      "l"(src), "r"(bytes), "r"((unsigned)__cvta_generic_to_shared(bar))
      : "memory");
}
__device__ __forceinline__ void mb_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)),
               "r"(bytes)
               : "memory");
}

// Builds the scatter blocks of all 10-node elements from the node arrays and
// the element->CSR node-block map (thread per element).
// Block slot e' holds element perm[e'] (the processing order).
__global__ void k_build_eblock(const int *conn, long ne, const int *dof, long nn, const int *rowptr0,
                               const int *rowlen, const uint8_t *mask, const uint16_t *pos, const int *perm,
                               int *eb) {
  const long es = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (es >= ne) return;
  const long e = perm ? (long)perm[es] : es;
  int *o = eb + es * kEBW;
  uint16_t *o16 = reinterpret_cast<uint16_t *>(o + kEBPos);
  uint8_t *o8 = reinterpret_cast<uint8_t *>(o + kEBMask);
  const long ep = es > 0 ? (perm ? (long)perm[es - 1] : es - 1) : -1;
  const long en = es + 1 < ne ? (perm ? (long)perm[es + 1] : es + 1) : -1;
  unsigned long long prev = 0;
  int next = 0, ne_[10], np_[10], nn_[10];
  for (int a = 0; a < 10; a++) {
    ne_[a] = conn[(long)a * ne + e];
    np_[a] = ep >= 0 ? conn[(long)a * ne + ep] : -1;
    nn_[a] = en >= 0 ? conn[(long)a * ne + en] : -1;
  }
  for (int a = 0; a < 10; a++) {
    const int n = ne_[a];
    const unsigned mk = mask[n];
    // handed on only when the node stands once in either element (a mid-side node may
    // coincide with its corner): an entry then has one place in both
    int own = 0, inp = 0, inn = 0;
    unsigned long long pa = 15;
    for (int x = 0; x < 10; x++) {
      own += ne_[x] == n;
      inn += nn_[x] == n;
      if (np_[x] == n) {
        inp++;
        pa = x;
      }
    }
    prev |= (own == 1 && inp == 1 ? pa : 15ull) << (4 * a);
    next |= (own == 1 && inn == 1 ? 1 : 0) << a;
    for (int i = 0; i < 3; i++) {
      const bool fr = (mk >> i) & 1u;
      o[a * 3 + i] = fr ? rowptr0[n] + __popc(mk & ((1u << i) - 1u)) * rowlen[n] : -1;
      o[kEBRes + a * 3 + i] = fr ? dof[i * nn + n] - 1 : -1;
    }
    for (int b = 0; b < 10; b++) o16[a * 10 + b] = pos[(e * 10 + a) * 10 + b];
    o8[a] = (uint8_t)mk;
  }
  o8[10] = o8[11] = 0;
  o[30] = o[31] = o[62] = o[63] = -1;
  o[kEBPrev] = (int)(prev & 0xffffffffull);
  o[kEBPrev + 1] = (int)(prev >> 32);
  o[kEBNext] = next;
}

// predicated shared accesses and reduction, without branches around them
__device__ __forceinline__ double lds_if(unsigned a, bool on) {
  double v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t@q ld.shared.f64 %0, [%1];\n\t}"
               : "=d"(v)
               : "r"(a), "r"((unsigned)on)
               : "memory");
  return v;
}
__device__ __forceinline__ void sts_if(unsigned a, double v, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.shared.f64 [%0], %1;\n\t}" ::"r"(a), "d"(v),
               "r"((unsigned)on)
               : "memory");
}
__device__ __forceinline__ void red_if(double *p, double v, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q red.relaxed.gpu.global.add.f64 [%0], %1;\n\t}" ::"l"(p),
               "d"(v), "r"((unsigned)on)
               : "memory");
}

// edge node (less four) between two corners: 01 12 02 03 13 23
__host__ __device__ __forceinline__ constexpr int p2_edge(int c, int d) {
  const int lo = c < d ? c : d, hi = c < d ? d : c;
  return lo == 0 ? (hi == 1 ? 0 : hi) : lo == 1 ? (hi == 2 ? 1 : 4) : 5;
}

// Three CTAs per SM, 168 registers (16 spilled words): two CTAs without spills
// measured 15 % slower at 82,944 elements, four with more spills 8 % slower than two.
template <int MODEL, bool TF = false>
__global__ void __launch_bounds__(kP2Threads, 3) k_assemble_p2r(const AsmArgs args, int run) {
  constexpr bool PLASTIC = (MODEL == 1);
  constexpr int NRF = yrec_fields(TF);
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char p2sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr unsigned kElem = p2r_elem_bytes(TF), kRecB = 4u * NRF * (unsigned)sizeof(double);
  constexpr int NW = kP2Threads / 32;
  unsigned char *wb = p2sm + (size_t)warp * 2 * kElem;
  double *stage = reinterpret_cast<double *>(p2sm + (size_t)NW * 2 * kElem) + (size_t)warp * 2 * kP2Stage;
  uint64_t *mbar = reinterpret_cast<uint64_t *>(p2sm + (size_t)NW * 2 *
                                                           (kElem + kP2Stage * sizeof(double))) +
                   2 * warp;
  const long ne = args.ne;
  // lane (b, k): column k of node b in the element's rows; lane 30: the residual
  const bool isK = lane < 30, isR = lane == 30;
  const int b = isK ? lane / 3 : 0, k = isK ? lane - 3 * b : 0;
  double dn[4][3], e[3];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int c = 0; c < 3; c++) dn[q][c] = isK ? args.shp.dNxi[q][b][c] : 0.0;
#pragma unroll
  for (int c = 0; c < 3; c++) e[c] = c == k ? 1.0 : 0.0;
  auto pick = [&](double x0, double x1, double x2) { return k == 0 ? x0 : (k == 1 ? x1 : x2); };
  double *const out = isR ? args.R : args.K;
  if (lane == 0) {
    w_mb_init(&mbar[0], 1);
    w_mb_init(&mbar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  auto load = [&](int buf, long el) {  // lane 0: the copies of element slot el
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // after the generic reads of the buffer
    unsigned char *dst = wb + (size_t)buf * kElem;
    mb_expect_tx(&mbar[buf], kElem);
    bulk_g2s(dst, args.qrec + el * (4 * NRF), kRecB, &mbar[buf]);
    bulk_g2s(dst + kRecB, args.eblk + el * kEBW, kElem - kRecB, &mbar[buf]);
  };
  // Runs of `run` elements: one per warp when that covers the mesh, else claimed in
  // order from one counter (zeroed before the launch; a claim takes about 7 ns of it), so that all warps work on
  // neighbouring elements of the processing order and the CSR rows they reduce
  // into stay in L2 between neighbouring elements' contributions.
  const bool claims = (long)gridDim.x * NW * run < ne;
  pdl_wait();
  long el = ((long)blockIdx.x * NW + warp) * run, next = ne;  // next: lane 0's claim
  if (claims) {
    if (lane == 0) el = (long)atomicAdd(args.ticket, 1u) * run;
    el = __shfl_sync(FULL, el, 0);
  }
  if (lane == 0 && el < ne) load(0, el);
  for (int it = 0, x = 0; el < ne; it++) {
    const int buf = it & 1;
    // bounded wait; one that runs out is counted in status[3] and the warp leaves,
    // after waiting -- again bounded -- for the copies in flight
    const bool landed = w_mb_wait(&mbar[buf], (unsigned)((it >> 1) & 1), args.wait_ns);
    if (!__all_sync(FULL, landed)) {
      if (lane == 0) {
        atomicAdd(&args.status[3], 1ull);
        w_mb_wait(&mbar[buf], (unsigned)((it >> 1) & 1), args.wait_ns);
      }
      break;
    }
    const bool more = x + 1 < run && el + 1 < ne;  // this run goes on
    if (lane == 0) {
      if (x == 0 && claims) next = (long)atomicAdd(args.ticket, 1u) * run;
      if (more) load(buf ^ 1, el + 1);
    }
    {
      const double *rec = reinterpret_cast<const double *>(wb + (size_t)buf * kElem);
      const int *eb = reinterpret_cast<const int *>(wb + (size_t)buf * kElem + kRecB);
      double tfc = 0.0, tfs = 0.0, vk = 0.0;
      if (TF) {
        double W = 0.0, SJ = 0.0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const double *r = rec + q * NRF;
          const double wJ = r[kYWJ];
          SJ += wJ;
          W += r[kYW];
          vk = fma(wJ, r[kYG + k] * dn[q][0] + r[kYG + 3 + k] * dn[q][1] + r[kYG + 6 + k] * dn[q][2], vk);
        }
        const double th = rec[kYTheta], Pe = rec[kYP];
        double dU, d2U;
        vol_derivs(args.mat.vol_pot, th, dU, d2U);
        tfc = args.mat.kappa * d2U / W;
        tfs = tfc * (SJ - th * W) + args.mat.kappa * dU - Pe;
        vk *= tfc;
      }
      double S[3][3], C[4][3], E[6][3];
#pragma unroll
      for (int l = 0; l < 3; l++)
#pragma unroll
        for (int i = 0; i < 3; i++) S[l][i] = 0.0;
#pragma unroll
      for (int l = 0; l < 6; l++)
#pragma unroll
        for (int i = 0; i < 3; i++) E[l][i] = 0.0;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const double2 *r2 = reinterpret_cast<const double2 *>(rec + q * NRF);
        const double2 *v2 = r2 + (isR ? kYT / 2 : kYV / 2);
        double Tm[6], V[6], G[10];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const double2 t = r2[kYT / 2 + c], v = v2[c];
          Tm[2 * c] = t.x, Tm[2 * c + 1] = t.y, V[2 * c] = v.x, V[2 * c + 1] = v.y;
        }
#pragma unroll
        for (int c = 0; c < 5; c++) {
          const double2 g = r2[kYG / 2 + c];
          G[2 * c] = g.x, G[2 * c + 1] = g.y;
        }
        const double2 c4 = r2[kYC / 2], c5h = r2[kYW5 / 2];
        double p[3], np[3], T[3];
#pragma unroll
        for (int j = 0; j < 3; j++) p[j] = G[j] * dn[q][0] + G[3 + j] * dn[q][1] + G[6 + j] * dn[q][2];
        smv(V, p, np);
        smv(Tm, p, T);
        const double pk = pick(p[0], p[1], p[2]), npk = pick(np[0], np[1], np[2]);
        double U = G[9] * pk + c4.x * npk, m = c4.x * pk;
        if (PLASTIC) {
          // (w a4 n + w a5 dev(n^2)) p, n a unit tensor (zero weights at elastic points)
          const double nnp = pick(V[0], V[5], V[4]) * np[0] + pick(V[5], V[1], V[3]) * np[1] +
                             pick(V[4], V[3], V[2]) * np[2];
          m += c4.y * npk + c5h.x * (nnp - (1.0 / 3.0) * pk);
        }
        const double wJ = TF ? rec[q * NRF + kYWJ] : 0.0;
        if (TF) U = fma(wJ, vk, U);
        m = isR ? args.rscale : m;
        U = isR ? -args.rscale * (TF ? c5h.y - wJ * tfs : c5h.y) : U;
        double Y[3][3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
          const double hej = c5h.y * e[j];
#pragma unroll
          for (int i = 0; i < 3; i++) {
            double y = fma(e[i], T[j], i == j ? fma(V[i], m, U) : V[6 - i - j] * m);
            Y[j][i] = fma(hej, p[i], y);
          }
        }
        double Z[4][3];  // by corner
#pragma unroll
        for (int i = 0; i < 3; i++) {
#pragma unroll
          for (int l = 0; l < 3; l++) {
            Z[l + 1][i] = G[3 * l] * Y[0][i] + G[3 * l + 1] * Y[1][i] + G[3 * l + 2] * Y[2][i];
            S[l][i] += Z[l + 1][i];
          }
          Z[0][i] = -(Z[1][i] + Z[2][i] + Z[3][i]);
          // edges 01 12 02 03 13 23
          const int cq = (q + 1) & 3;
          C[cq][i] = Z[cq][i];
#pragma unroll
          for (int o = 0; o < 4; o++)
            if (o != cq) E[p2_edge(o, cq)][i] += Z[o][i];
        }
      }
      // ---- rows: node a's three rows, 30 consecutive columns of the element per reduction ----
      constexpr double kC = 4.0 * kP2RuleB - 1.0, kE = 4.0 * kP2RuleB, kG = 4.0 * (kP2RuleA - kP2RuleB);
      const int *rows = eb + (isR ? kEBRes : 0);
      const uint16_t *pos16 = reinterpret_cast<const uint16_t *>(eb + kEBPos);
      const unsigned maskB = reinterpret_cast<const uint8_t *>(eb + kEBMask)[b];
      const bool live = isR || (isK && ((maskB >> k) & 1u));
      const int rank = isR ? 0 : rank_of(maskB, k);
      double S0[3];
#pragma unroll
      for (int i = 0; i < 3; i++) S0[i] = -(S[0][i] + S[1][i] + S[2][i]);
      auto SS = [&](int l, int i) { return l == 0 ? S0[i] : S[l - 1][i]; };
      int rw[32];
#pragma unroll
      for (int c = 0; c < 8; c++) {
        const int4 v = reinterpret_cast<const int4 *>(rows)[c];
        rw[4 * c] = v.x, rw[4 * c + 1] = v.y, rw[4 * c + 2] = v.z, rw[4 * c + 3] = v.w;
      }
      // entries of two nodes that the next element of the run has too are handed to
      // it, not reduced
      const unsigned long long prev = (unsigned)eb[kEBPrev] | (unsigned long long)(unsigned)eb[kEBPrev + 1] << 32;
      const unsigned nextm = more ? (unsigned)eb[kEBNext] : 0u;
      const int pb = (int)(prev >> (4 * b)) & 15;
      const bool take = x > 0 && live && (isR || pb < 10), hand = isR || ((nextm >> b) & 1u);
      const unsigned st0 = (unsigned)__cvta_generic_to_shared(stage);
      const unsigned sin = st0 + 8u * (((x + 1) & 1) * kP2Stage + (isR ? lane : 3 * pb + k));
      const unsigned sout = st0 + 8u * ((x & 1) * kP2Stage + lane);
      constexpr int el0[6] = {0, 1, 0, 0, 1, 2}, el1[6] = {1, 2, 2, 3, 3, 3};
#pragma unroll
      for (int a = 0; a < 10; a++) {
        const int col = isR ? 0 : (int)pos16[a * 10 + b] + rank;
        const int pa = (int)(prev >> (4 * a)) & 15;
        const bool ta = take && pa < 10, ha = hand && ((nextm >> a) & 1u);
#pragma unroll
        for (int i = 0; i < 3; i++) {
          double v = a < 4 ? fma(kC, SS(a, i), kG * C[a][i])
                                 : fma(kE, SS(el0[a < 4 ? 0 : a - 4], i) + SS(el1[a < 4 ? 0 : a - 4], i),
                                       kG * E[a < 4 ? 0 : a - 4][i]);
          const int rb = rw[3 * a + i];
          v += lds_if(sin + (unsigned)(3 * pa + i) * 256u, ta);
          sts_if(sout + (unsigned)(3 * a + i) * 256u, v, ha);
          red_if(out + (rb + col), v, live && !ha && rb >= 0);
        }
      }
    }
    __syncwarp();
    if (more) {
      el++;
      x++;
    } else {
      if (lane == 0 && next < ne) load(buf ^ 1, next);
      el = __shfl_sync(FULL, next, 0);
      x = 0;
    }
  }
}

// Three-field element (one pressure P and one volume theta per element,
// quadratic tets, hyperelastic and J2 models): the local update after a displacement
// increment du (compute_d_theta_dP, src/constitutive_model_3f.cc:494-549, with
// the blocks at u; thread per element): with W = sum_q w, fp = sum_q w J -
// theta W and Kpu du = sum_q w J tr(Grad(du) F^-1),
//   d_theta = (Kpu du + fp) / W,  dP = kappa U'(theta) - P + kappa U''(theta) d_theta.
// An element with an inverted point gets zero increments and is counted.
__global__ void k_tf_update(const QpArgs A, const double *dunode, double *dP, double *dtheta) {
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e >= A.ne) return;
  double W = 0.0, SJ = 0.0, Kdu = 0.0;
  bool ok = true;
  for (int q = 0; q < 4 && ok; q++) {
    double dX[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, dU[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0},
           dD[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int b = 0; b < 10; b++) {
      const int n = A.conn[(long)b * A.ne + e];
      const double g0 = A.shp.dNxi[q][b][0], g1 = A.shp.dNxi[q][b][1], g2 = A.shp.dNxi[q][b][2];
      for (int i = 0; i < 3; i++) {
        const double x = A.X[i * A.nn + n], u = A.unode[i * A.nn + n], d = dunode[i * A.nn + n];
        dX[i * 3 + 0] += g0 * x;
        dX[i * 3 + 1] += g1 * x;
        dX[i * 3 + 2] += g2 * x;
        dU[i * 3 + 0] += g0 * u;
        dU[i * 3 + 1] += g1 * u;
        dU[i * 3 + 2] += g2 * u;
        dD[i * 3 + 0] += g0 * d;
        dD[i * 3 + 1] += g1 * d;
        dD[i * 3 + 2] += g2 * d;
      }
    }
    const double detJ = det3(dX);
    double dXi[9], F[9], Fi[9], L[9];
    ok = detJ > 0.0 && inv3(dX, dXi);
    if (!ok) break;
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) {
        F[i * 3 + j] = (i == j ? 1.0 : 0.0) + dU[i * 3 + 0] * dXi[0 * 3 + j] + dU[i * 3 + 1] * dXi[1 * 3 + j] +
                       dU[i * 3 + 2] * dXi[2 * 3 + j];
        L[i * 3 + j] = dD[i * 3 + 0] * dXi[0 * 3 + j] + dD[i * 3 + 1] * dXi[1 * 3 + j] + dD[i * 3 + 2] * dXi[2 * 3 + j];
      }
    if (A.F0)
      for (int i = 0; i < 9; i++) F[i] += A.F0[i];
    const double J = det3(F);
    ok = J > 0.0 && inv3(F, Fi);
    if (!ok) break;
    const double w = detJ * A.shp.w[q];
    double tr = 0.0;
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) tr += L[i * 3 + j] * Fi[j * 3 + i];
    W += w;
    SJ += w * J;
    Kdu += w * J * tr;
  }
  if (!ok) {
    atomicAdd(&A.status[0], 1ull);
    dP[e] = dtheta[e] = 0.0;
    return;
  }
  const double th = A.tf_theta[e], P = A.tf_P[e];
  double dUv, d2U;
  vol_derivs(A.mat.vol_pot, th, dUv, d2U);
  const double dth = (Kdu + SJ - th * W) / W;
  dtheta[e] = dth;
  dP[e] = A.mat.kappa * dUv - P + A.mat.kappa * d2U * dth;
}

// The three-field element in the transient (quadratic tets, hyperelastic):
// the corrections that turn the two condensed quasi-static assemblies at the
// mid points into the reference's transient condensation
// (residuals_el_constitutive_model_w_inertia_3f, src/constitutive_model.cc:
// 2960-3229).  With the blocks of the newer mid point a scaled by
// kK = -dt_np1 alpha (1 - alpha) and the residuals combined as
// R_x = cA R_x(a) + cB R_x(b), the condensed residual is
//   f = cA (fu_a + s_a Kup_a) + cB (fu_b + s_b Kup_b) - cB s_b Kup_b + d Kup_a,
//   d = cB (c_a fp_b + kappa U'(theta_b) - P_b),
// c = kappa U''(theta) / W, fp = sum w J - theta W, s = c fp + kappa U'(theta) - P
// (the first two terms are the condensed assemblies at a and at b): this
// kernel adds d Kup_a - cB s_b Kup_b into R.  With dunode set it instead
// forms the local update (compute_d_theta_dP with the combined blocks,
// :3880-3898): d_theta = (kK Kup_a du + Rp) / (kK W),
// dP = (Rt + kK W kappa U''(theta_a) d_theta) / (kK W).
struct TfTrArgs {
  QpArgs A;               // X, conn, shp, mat, status; unode = u_{n+alpha}
  const double *unode_b;  // u_{n-1+alpha} at the nodes (SoA 3*nn)
  const double *mid;      // 4*ne: P_a, theta_a, P_b, theta_b
  const int *dof;         // 3*nn SoA, 1-based free DOF ids
  double *R;
  const double *dunode;   // update mode: du at the nodes
  double *dP, *dtheta;
  double cA, cB, kK;
};

__global__ void k_tf_transient(const TfTrArgs T) {
  const QpArgs &A = T.A;
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e >= A.ne) return;
  const bool upd = T.dunode != nullptr;
  int nd[10];
  for (int b = 0; b < 10; b++) nd[b] = A.conn[(long)b * A.ne + e];
  // point q: reference gradient inverse, w, and F, F^-1, J at both mid points
  auto point = [&](int q, double *dXi, double &w, double *Fa, double *Fia, double &Ja, double *Fb, double *Fib,
                   double &Jb, double *Ld) -> bool {
    double dX[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, da[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0},
           db[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, dd[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int b = 0; b < 10; b++) {
      const int n = nd[b];
      const double g[3] = {A.shp.dNxi[q][b][0], A.shp.dNxi[q][b][1], A.shp.dNxi[q][b][2]};
      for (int i = 0; i < 3; i++) {
        const double x = A.X[i * A.nn + n], ua = A.unode[i * A.nn + n], ub = T.unode_b[i * A.nn + n];
        const double d = upd ? T.dunode[i * A.nn + n] : 0.0;
        for (int c = 0; c < 3; c++) {
          dX[i * 3 + c] += g[c] * x;
          da[i * 3 + c] += g[c] * ua;
          db[i * 3 + c] += g[c] * ub;
          dd[i * 3 + c] += g[c] * d;
        }
      }
    }
    const double detJ = det3(dX);
    if (!(detJ > 0.0) || !inv3(dX, dXi)) return false;
    w = detJ * A.shp.w[q];
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) {
        double fa = (i == j ? 1.0 : 0.0), fb = fa, l = 0.0;
        for (int c = 0; c < 3; c++) {
          fa += da[i * 3 + c] * dXi[c * 3 + j];
          fb += db[i * 3 + c] * dXi[c * 3 + j];
          l += dd[i * 3 + c] * dXi[c * 3 + j];
        }
        Fa[i * 3 + j] = fa;
        Fb[i * 3 + j] = fb;
        Ld[i * 3 + j] = l;
      }
    Ja = det3(Fa);
    Jb = det3(Fb);
    return Ja > 0.0 && Jb > 0.0 && inv3(Fa, Fia) && inv3(Fb, Fib);
  };
  double W = 0.0, SJa = 0.0, SJb = 0.0, Kdu = 0.0;
  bool ok = true;
  for (int q = 0; q < 4 && ok; q++) {
    double dXi[9], w, Fa[9], Fia[9], Ja, Fb[9], Fib[9], Jb, Ld[9];
    ok = point(q, dXi, w, Fa, Fia, Ja, Fb, Fib, Jb, Ld);
    if (!ok) break;
    W += w;
    SJa += w * Ja;
    SJb += w * Jb;
    if (upd) {
      double tr = 0.0;
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) tr += Ld[i * 3 + j] * Fia[j * 3 + i];
      Kdu += w * Ja * tr;
    }
  }
  if (!ok) {
    atomicAdd(&A.status[0], 1ull);
    if (upd) T.dP[e] = T.dtheta[e] = 0.0;
    return;
  }
  const double Pa = T.mid[e], tha = T.mid[A.ne + e], Pb = T.mid[2 * A.ne + e], thb = T.mid[3 * A.ne + e];
  const double kap = A.mat.kappa;
  double dUa, d2Ua, dUb, d2Ub;
  vol_derivs(A.mat.vol_pot, tha, dUa, d2Ua);
  vol_derivs(A.mat.vol_pot, thb, dUb, d2Ub);
  if (upd) {
    const double Rp = T.cA * (SJa - tha * W) + T.cB * (SJb - thb * W);
    const double Rt = W * (T.cA * (kap * dUa - Pa) + T.cB * (kap * dUb - Pb));
    const double dth = (T.kK * Kdu + Rp) / (T.kK * W);
    T.dtheta[e] = dth;
    T.dP[e] = (Rt + T.kK * W * kap * d2Ua * dth) / (T.kK * W);
    return;
  }
  const double ca = kap * d2Ua / W, cb = kap * d2Ub / W, fpb = SJb - thb * W;
  const double sb = cb * fpb + kap * dUb - Pb;
  const double da_ = T.cB * (ca * fpb + kap * dUb - Pb), db_ = -T.cB * sb;
  double out[10][3];
  for (int b = 0; b < 10; b++) out[b][0] = out[b][1] = out[b][2] = 0.0;
  for (int q = 0; q < 4; q++) {
    double dXi[9], w, Fa[9], Fia[9], Ja, Fb[9], Fib[9], Jb, Ld[9];
    point(q, dXi, w, Fa, Fia, Ja, Fb, Fib, Jb, Ld);
    for (int b = 0; b < 10; b++) {
      double gX[3];  // dN_b / dX
      for (int j = 0; j < 3; j++)
        gX[j] = A.shp.dNxi[q][b][0] * dXi[0 * 3 + j] + A.shp.dNxi[q][b][1] * dXi[1 * 3 + j] +
                A.shp.dNxi[q][b][2] * dXi[2 * 3 + j];
      for (int k = 0; k < 3; k++) {
        const double ta = gX[0] * Fia[0 * 3 + k] + gX[1] * Fia[1 * 3 + k] + gX[2] * Fia[2 * 3 + k];
        const double tb = gX[0] * Fib[0 * 3 + k] + gX[1] * Fib[1 * 3 + k] + gX[2] * Fib[2 * 3 + k];
        out[b][k] += w * (da_ * Ja * ta + db_ * Jb * tb);
      }
    }
  }
  for (int b = 0; b < 10; b++)
    for (int k = 0; k < 3; k++) {
      const int id = T.dof[k * A.nn + nd[b]];
      if (id > 0) atomicAdd(T.R + (id - 1), out[b][k]);
    }
}

// Residual of the condensed three-field element from its point records alone
// (quadratic tets; the residual part of k_assemble_p2r without its stiffness):
// R_bi = sum_q sum_j (w tau_ij + w J s delta_ij) p_qb,j with p_qb = G_q^T dN_b/dxi,
// s = c (sum w J - theta W) + kappa U'(theta) - P, c = kappa U''(theta) / W;
// w tau = T' minus the geometric term h on the diagonal.
// One thread per record slot (element perm[es]); inverted elements have zeroed
// records (W = 0) and are skipped, as the assembly skips them.
__global__ void k_tf_residual(const QpArgs A, const int *dof, double *R) {
  constexpr int NRF = kYRecTF;
  const long es = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (es >= A.ne) return;
  const long e = A.perm ? (long)A.perm[es] : es;
  const double *rec = A.qrec;
  double W = 0.0, SJ = 0.0;
  for (int q = 0; q < 4; q++) {
    SJ += rec[(es * 4 + q) * NRF + kYWJ];
    W += rec[(es * 4 + q) * NRF + kYW];
  }
  if (!(W > 0.0)) return;
  const double th = rec[es * 4 * NRF + kYTheta], Pe = rec[es * 4 * NRF + kYP];
  double dU, d2U;
  vol_derivs(A.mat.vol_pot, th, dU, d2U);
  const double c = A.mat.kappa * d2U / W;
  const double sc = c * (SJ - th * W) + A.mat.kappa * dU - Pe;
  double out[10][3];
  for (int b = 0; b < 10; b++) out[b][0] = out[b][1] = out[b][2] = 0.0;
  for (int q = 0; q < 4; q++) {
    const long qs = es * 4 + q;
    double G[9], T[3][3];
    for (int k = 0; k < 9; k++) G[k] = rec[qs * NRF + kYG + k];
    const double h = rec[qs * NRF + kYH], wJs = rec[qs * NRF + kYWJ] * sc;
    double wt[6];
    for (int k = 0; k < 6; k++) wt[k] = rec[qs * NRF + kYT + k] - (k < 3 ? h : 0.0);
    // Voigt order xx yy zz yz xz xy
    T[0][0] = wt[0] + wJs; T[1][1] = wt[1] + wJs; T[2][2] = wt[2] + wJs;
    T[1][2] = T[2][1] = wt[3];
    T[0][2] = T[2][0] = wt[4];
    T[0][1] = T[1][0] = wt[5];
    for (int b = 0; b < 10; b++) {
      const double g0 = A.shp.dNxi[q][b][0], g1 = A.shp.dNxi[q][b][1], g2 = A.shp.dNxi[q][b][2];
      double p[3];
      for (int j = 0; j < 3; j++) p[j] = G[j] * g0 + G[3 + j] * g1 + G[6 + j] * g2;
      for (int i = 0; i < 3; i++) out[b][i] += T[i][0] * p[0] + T[i][1] * p[1] + T[i][2] * p[2];
    }
  }
  for (int b = 0; b < 10; b++) {
    const int n = A.conn[(long)b * A.ne + e];
    for (int i = 0; i < 3; i++) {
      const int id = dof[i * A.nn + n];
      if (id > 0) atomicAdd(R + (id - 1), out[b][i]);
    }
  }
}

// ---- three-field transient: all terms beside the newer point's assembly -------
//
// The transient's condensed residual is cA (fu_a + s_a Kup_a) -- the assembly at the
// newer mid point -- plus cB fu_b + d Kup_a - f_i with d as in k_tf_transient (the
// s_b Kup_b terms of the older point cancel) and the inertia force f_i.  One
// thread per point forms its part of the three from the nodal fields:
//   out_b = M dN_b/dxi - N_b e,  M_ic = cB w tau_ij G_b,cj + d w J_a G_a,ci,
//   e = rho / (dt_np1 dt_n) w sum_C N_C v_C,  G = (dX/dxi)^-1 F^-1,
// and the four lanes of an element add their 30 values by halving exchanges, so
// that each ends with eight sums and their reductions.  257 us at 384,000 elements,
// bound by the L1 wavefronts of the node loads (67 % of their peak); 96-byte node
// records read by the lanes instead measured 326 us, as neighbouring elements no
// longer share the sectors.
struct TfTrResArgs {
  const double *X, *ua, *ub, *v;  // 3*nn SoA: coordinates, u_{n+a}, u_{n-1+a}, inertia combination
  const int *conn, *dof, *perm;
  long nn, ne;
  const double *mid;  // 4*ne: P_a, theta_a, P_b, theta_b
  double *R;
  unsigned long long *status;
  Mat mat;
  ShapeTable shp;
  double cB, cR;
};

__global__ void __launch_bounds__(128, 4) k_tf_transient_terms(const TfTrResArgs A) {
  __shared__ double sdN[4][10][3], sN[4][10], sw[4];
  for (int i = threadIdx.x; i < 120; i += 128) (&sdN[0][0][0])[i] = A.shp.dNxi[i / 30][(i / 3) % 10][i % 3];
  if (threadIdx.x < 40) sN[threadIdx.x / 10][threadIdx.x % 10] = A.shp.N[threadIdx.x / 10][threadIdx.x % 10];
  if (threadIdx.x < 4) sw[threadIdx.x] = A.shp.w[threadIdx.x];
  __syncthreads();
  const unsigned FULL = 0xffffffffu;
  const long t = blockIdx.x * 128L + threadIdx.x, es = t >> 2;
  const int q = (int)(t & 3);
  const bool in = es < A.ne;
  const long e = in ? (A.perm ? (long)A.perm[es] : es) : 0;
  double out[32];
#pragma unroll
  for (int i = 0; i < 32; i++) out[i] = 0.0;
  double dX[9], da[9], db[9], du[3] = {0, 0, 0};
#pragma unroll
  for (int i = 0; i < 9; i++) dX[i] = da[i] = db[i] = 0.0;
#pragma unroll
  for (int b = 0; b < 10; b++) {
    const int n = A.conn[(long)b * A.ne + e];
    const double g0 = sdN[q][b][0], g1 = sdN[q][b][1], g2 = sdN[q][b][2], N = sN[q][b];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double x = A.X[i * A.nn + n], ya = A.ua[i * A.nn + n], yb = A.ub[i * A.nn + n];
      dX[i * 3] = fma(g0, x, dX[i * 3]), dX[i * 3 + 1] = fma(g1, x, dX[i * 3 + 1]), dX[i * 3 + 2] = fma(g2, x, dX[i * 3 + 2]);
      da[i * 3] = fma(g0, ya, da[i * 3]), da[i * 3 + 1] = fma(g1, ya, da[i * 3 + 1]), da[i * 3 + 2] = fma(g2, ya, da[i * 3 + 2]);
      db[i * 3] = fma(g0, yb, db[i * 3]), db[i * 3 + 1] = fma(g1, yb, db[i * 3 + 1]), db[i * 3 + 2] = fma(g2, yb, db[i * 3 + 2]);
      du[i] = fma(N, A.v[i * A.nn + n], du[i]);
    }
  }
  const double detJ = det3(dX);
  double dXi[9], Fa[9], Fb[9], Fia[9], Fib[9], Ja = 0.0, Jb = 0.0;
  const bool geo = detJ > 0.0 && inv3(dX, dXi);
  bool oka = geo, okb = geo;
  if (geo) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const double one = i == j ? 1.0 : 0.0;
        Fa[i * 3 + j] = one + da[i * 3] * dXi[j] + da[i * 3 + 1] * dXi[3 + j] + da[i * 3 + 2] * dXi[6 + j];
        Fb[i * 3 + j] = one + db[i * 3] * dXi[j] + db[i * 3 + 1] * dXi[3 + j] + db[i * 3 + 2] * dXi[6 + j];
      }
    Ja = det3(Fa);
    Jb = det3(Fb);
    oka = Ja > 0.0 && inv3(Fa, Fia);
    okb = Jb > 0.0 && inv3(Fb, Fib);
  }
  const double w = geo ? detJ * sw[q] : 0.0;
  double W = w, SJb = w * Jb;
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    W += __shfl_xor_sync(FULL, W, o);
    SJb += __shfl_xor_sync(FULL, SJb, o);
  }
  const unsigned quad = 0xFu << (threadIdx.x & 28);
  const bool geo_all = (__ballot_sync(FULL, geo) & quad) == quad;
  const bool ok_all = (__ballot_sync(FULL, oka && okb) & quad) == quad;
  if (in && !okb) atomicAdd(&A.status[0], 1ull);               // a point inverted at the older mid point
  if (in && q == 0 && !ok_all) atomicAdd(&A.status[0], 1ull);  // an element inverted at either
  double M[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, f[3] = {0, 0, 0};
  if (geo_all)
#pragma unroll
    for (int i = 0; i < 3; i++) f[i] = A.cR * w * du[i];
  if (ok_all) {
    const double tha = A.mid[A.ne + e], Pb = A.mid[2 * A.ne + e], thb = A.mid[3 * A.ne + e], kap = A.mat.kappa;
    double dUa, d2Ua, dUb, d2Ub, dUj, d2Uj;
    vol_derivs(A.mat.vol_pot, tha, dUa, d2Ua);
    vol_derivs(A.mat.vol_pot, thb, dUb, d2Ub);
    vol_derivs(A.mat.vol_pot, Jb, dUj, d2Uj);
    const double d = A.cB * (kap * d2Ua / W * (SJb - thb * W) + kap * dUb - Pb);
    const double I6[6] = {1, 1, 1, 0, 0, 0};
    QpTangent tg;
    spatial_update<false>(A.mat, Fb, Jb, I6, 0.0, tg, nullptr, nullptr);
    const double dp = Pb * Jb - kap * Jb * dUj, cw = A.cB * w, dw = d * w * Ja;
    double T[6];
#pragma unroll
    for (int v = 0; v < 6; v++) T[v] = cw * (tg.tau[v] + (v < 3 ? dp : 0.0));
#pragma unroll
    for (int c = 0; c < 3; c++) {
      double ga[3], gb[3], y[3];
#pragma unroll
      for (int j = 0; j < 3; j++) {
        ga[j] = dXi[c * 3] * Fia[j] + dXi[c * 3 + 1] * Fia[3 + j] + dXi[c * 3 + 2] * Fia[6 + j];
        gb[j] = dXi[c * 3] * Fib[j] + dXi[c * 3 + 1] * Fib[3 + j] + dXi[c * 3 + 2] * Fib[6 + j];
      }
      smv(T, gb, y);
#pragma unroll
      for (int i = 0; i < 3; i++) M[i * 3 + c] = fma(dw, ga[i], y[i]);
    }
  }
#pragma unroll
  for (int b = 0; b < 10; b++)
#pragma unroll
    for (int i = 0; i < 3; i++)
      out[3 * b + i] = M[i * 3] * sdN[q][b][0] + M[i * 3 + 1] * sdN[q][b][1] + M[i * 3 + 2] * sdN[q][b][2] - sN[q][b] * f[i];
  // lane q ends with the sums of values 8 q .. 8 q + 7
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const double give = (q & 2) ? out[i] : out[16 + i], keep = (q & 2) ? out[16 + i] : out[i];
    out[i] = keep + __shfl_xor_sync(FULL, give, 2);
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const double give = (q & 1) ? out[i] : out[8 + i], keep = (q & 1) ? out[8 + i] : out[i];
    out[i] = keep + __shfl_xor_sync(FULL, give, 1);
  }
  if (!in) return;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int k = 8 * q + i;
    if (k >= 30) continue;
    const int b = k / 3, c = k - 3 * b;
    const int id = A.dof[c * A.nn + A.conn[(long)b * A.ne + e]];
    if (id > 0) atomicAdd(A.R + (id - 1), out[i]);
  }
}

}  // namespace pgb
