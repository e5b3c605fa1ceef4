// assemble_gather.cuh -- R+K assembly of linear tets by the owners of the rows.
//
// Same operation as k_assemble (fd_residuals_MP + stiffmat_fd_MP for the
// constitutive-model element, src/fd_residuals.cc:468-636,
// src/stiffmat_fd.cc:831-993), organised so that no reduction reaches L2: one
// warp owns the one to three CSR rows of a node (of all nodes that share their
// free DOFs: the images of a periodic node), one lane takes one incident
// element, forms the node's three rows of the element block in closed form and
// puts them in shared memory, and the warp then adds the incident elements'
// values column by column and writes each row once, in order.  R and K need no
// zero fill and K is never read.
//
// The scatter (k_assemble_p1ws: twelve lanes per element, FP64 reductions into the
// CSR) issues 144 + 12 reductions per element in 78 L2 sectors and is bound by the
// L1 data pipe and the L2 atomic unit.  Measured, 256 periodic cells (7.9 M
// elements, J2): whole iterate 5.59 -> 4.66 ms, 384,000 elements (40^3 cells) 0.23
// ms; 6,000 elements (HE) 21.2 -> 14.3 us, two launches instead of six; crystal
// plasticity records at 663,552 elements 0.44 -> 0.35 ms.  The gather is bound by
// the latency of its phases at 16 warps per SM (128 registers; 20 warps spill and
// take 5.6 ms, 12 warps 4.9) and the L1 pipe (59 %): records in, 31 values per
// incidence out and back.  The scatter stays for contexts whose lists cannot be
// built and for the failure-path test of its hand-off waits.
//
// The lists (incident elements of a row owner, its columns, the contributions
// of every column) are built on the device when the context is created, in an
// order that does not depend on timing, so the sums are deterministic.
#pragma once
#include <cstdint>

#include "assemble.cuh"

namespace pgb {

constexpr int kGatherMost = 128;  // incident elements of a row owner that the lists allow
constexpr int kGatherSmem = 227 * 1024;
constexpr int kGVal = 31;         // doubles per incidence: three 3x3 blocks and the residual (odd: no bank conflicts)
// place of nine zeros in a warp's values, after those of cap incidences
__host__ __device__ constexpr int gather_zero(int most) { return (most + 31) / 32 * 32 * kGVal; }
// record of HE and J2: G 9, V 6, w a2, c, w a4, w a5, h, h + w p_J (p_J the volumetric
// stress; s'' = c V = -2/3 w s), one pad: the 26 numbers of the quadratic tets'
// record (assemble_p2.cuh) without T' = (h + w p_J) 1 + w s
constexpr int kP1Rec = 22;

// Lists of the row owners (groups), in order of their first row.
//   head   two words per group: {incidences from, lists from, packs from, CSR
//          offset of the first row}, {incidences | lists << 8 | packs << 16 | free
//          mask << 28, row length, first DOF, own column's offset in the row}
//   inc    incidences: element * 4 + local node
//   slot   lists: {offset in the row | free mask << 16, first pack | packs << 16}: the
//          residual, the columns other than the owner's own ascending, and, free mask
//          0, the columns of fixed nodes together
//   ent    packs of four entries: where an incidence's block (or residual) starts in
//          its warp's values, incidence * kGVal + 9 j for the j-th of its nodes other
//          than the owner (27: residual); filled up with the place of nine zeros
// The own column needs no list: the p_b of an element sum to zero and every term
// of K_ab is linear in p_b, so it is minus the sum of the others.
struct GatherLists {
  long ng = 0;
  int most = 0;    // largest number of incidences
  int slots = 0;   // largest number of lists
  int packs = 0;   // largest number of packs
  int width = 0;   // largest row length
  const int4 *head = nullptr;
  const int *inc = nullptr;
  const uint2 *slot = nullptr;
  const uint2 *ent = nullptr;
};

// ---- construction -----------------------------------------------------------

__global__ void k_gather_count(const int *conn, long ne, const int *grp, int *cnt) {
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= 4 * ne) return;
  const int g = grp[conn[(t & 3) * ne + (t >> 2)]];
  if (g >= 0) atomicAdd(cnt + g, 1);
}

__global__ void k_gather_fill(const int *conn, long ne, const int *grp, const int *off, int *cursor, int *inc) {
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= 4 * ne) return;
  const int g = grp[conn[(t & 3) * ne + (t >> 2)]];
  if (g >= 0) inc[off[g] + atomicAdd(cursor + g, 1)] = (int)t;
}

// Sorts a group's incidences and counts its lists and packs into two[g],
// two[ng + g] and the own column's offset into two[2 ng + g] (fill = 0), or writes the lists and packs (fill = 1).  err: a group
// whose columns do not make up its row, or too many of them.
__global__ void k_gather_columns(long ng, const int *conn, long ne, const uint8_t *mask, const uint16_t *pos,
                                 const int *inc_off, int *inc, const int4 *row, int fill, const int4 *head,
                                 int *two, uint2 *slot, uint2 *ent, int zero, int *err) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g >= ng) return;
  int *I = inc + inc_off[g];
  const int n = inc_off[g + 1] - inc_off[g];
  if (!fill)
    for (int i = 1; i < n; i++) {  // lists of some 24
      const int v = I[i];
      int j = i - 1;
      for (; j >= 0 && I[j] > v; j--) I[j + 1] = I[j];
      I[j + 1] = v;
    }
  uint16_t col[kGatherMost], cnt[kGatherMost];
  uint8_t cm[kGatherMost];
  int nc = 0, width = 0, fixed = 0, own = -1;
  bool bad = n == 0;
  for (int i = 0; i < n && !bad; i++) {
    const long e = I[i] >> 2;
    const int a = I[i] & 3;
    const int o = pos[(e * 4 + a) * 4 + a];
    bad = own >= 0 && o != own;
    own = o;
    for (int b = 0; b < 4; b++) {
      const unsigned mb = mask[conn[(long)b * ne + e]];
      const uint16_t p = pos[(e * 4 + a) * 4 + b];
      if (b == a || (mb && p == o)) continue;  // the own column (of a periodic neighbour too)
      if (!mb) {
        fixed++;
        continue;
      }
      int s = 0;
      while (s < nc && col[s] < p) s++;
      if (s < nc && col[s] == p) {
        cnt[s]++;
        bad = bad || cm[s] != mb;
        continue;
      }
      if (nc == kGatherMost) {
        bad = true;
        break;
      }
      for (int k = nc++; k > s; k--) {
        col[k] = col[k - 1];
        cm[k] = cm[k - 1];
        cnt[k] = cnt[k - 1];
      }
      col[s] = p;
      cm[s] = (uint8_t)mb;
      cnt[s] = 1;
      width += __popc(mb);
    }
  }
  const int nl = 1 + nc + (fixed ? 1 : 0);
  if (!fill) {
    int packs = (n + 3) / 4 + (fixed + 3) / 4;
    for (int s = 0; s < nc; s++) packs += (cnt[s] + 3) / 4;
    two[g] = nl;
    two[ng + g] = packs;
    two[2 * ng + g] = own;
    if (bad || nl > kGatherMost || width + __popc((unsigned)row[g].w) != row[g].y) atomicAdd(err, 1);
    return;
  }
  uint2 *S = slot + head[2 * g].y;
  uint16_t *E = reinterpret_cast<uint16_t *>(ent + head[2 * g].z);
  int k = 0;
  auto close = [&](int s, unsigned what, int from) {
    while (k & 3) E[k++] = (uint16_t)zero;
    S[s] = make_uint2(what, (unsigned)(from >> 2) | ((unsigned)((k - from) >> 2) << 16));
  };
  for (int i = 0; i < n; i++) E[k++] = (uint16_t)(i * kGVal + 27);
  close(0, 0u, 0);
  for (int s = 0; s < nl - 1; s++) {
    const int from = k;
    for (int i = 0; i < n; i++) {
      const long e = I[i] >> 2;
      const int a = I[i] & 3;
      for (int b = 0; b < 4; b++) {
        if (b == a) continue;
        const bool free = mask[conn[(long)b * ne + e]] != 0;
        if (s < nc ? free && pos[(e * 4 + a) * 4 + b] == col[s] : !free)
          E[k++] = (uint16_t)(i * kGVal + 9 * (b - (b > a ? 1 : 0)));
      }
    }
    close(s + 1, s < nc ? (unsigned)col[s] | ((unsigned)cm[s] << 16) : 0u, from);
  }
}

// ---- point update of HE and J2, one thread per element ----------------------

struct P1PointArgs {
  const double *X;
  const int *conn, *dof;
  long nn, ne;
  const double *u, *presc;
  const double *F0;
  const int *elem_group;
  const double *F0_tab;
  const double *state_n;
  double *state_np1, *rec;  // rec: kP1Rec doubles per element, contiguous
  unsigned long long *status;
  Mat mat;
};

// Displacements are read through the DOF ids (no expanded copy).  Records are
// turned in shared memory so that a CTA writes its 128 in whole lines.  Bound by
// load latency: with the loads in order of use 64 us for 384,000 elements (J2),
// issued up front 47 us; five CTAs per SM (96 registers, some spills) against the
// three of 142 registers take 0.15 ms off 7.9 M elements.
template <int MODEL>
__global__ void __launch_bounds__(128, 5) k_p1_points(const P1PointArgs A) {
  constexpr bool PLASTIC = MODEL == 1;
  pdl_release();
  __shared__ double srow[128 * (kP1Rec + 1)];
  const long e0 = blockIdx.x * 128L, e = e0 + threadIdx.x;
  double *r = srow + threadIdx.x * (kP1Rec + 1);
  if (e < A.ne) {
    // loads first, in three dependent rounds: nodes, state and group; coordinates,
    // DOF ids and macro deformation; displacements
    int nd[4], id[4][3];
    double x[4][3], u[4][3], Ast[6] = {1, 1, 1, 0, 0, 0}, alpha = 0.0, M0[9];
#pragma unroll
    for (int a = 0; a < 4; a++) nd[a] = A.conn[(long)a * A.ne + e];
    const double *F0 = A.elem_group ? A.F0_tab + 9 * (long)A.elem_group[e] : A.F0;
    if (PLASTIC) {
#pragma unroll
      for (int c = 0; c < 6; c++) Ast[c] = A.state_n[c * A.ne + e];
      alpha = A.state_n[6 * A.ne + e];
    }
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int i = 0; i < 3; i++) {
        id[a][i] = A.dof[i * A.nn + nd[a]];
        x[a][i] = A.X[i * A.nn + nd[a]];
      }
#pragma unroll
    for (int i = 0; i < 9; i++) M0[i] = F0 ? F0[i] : 0.0;
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int i = 0; i < 3; i++)
        u[a][i] = id[a][i] > 0 ? A.u[id[a][i] - 1] : (id[a][i] < 0 && A.presc ? A.presc[-id[a][i] - 1] : 0.0);
    double dX[9], dU[9], dXi[9], F[9], Fi[9];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int c = 0; c < 3; c++) {
        dX[i * 3 + c] = x[c + 1][i] - x[0][i];
        dU[i * 3 + c] = u[c + 1][i] - u[0][i];
      }
    const double detJ = det3(dX);
    bool ok = detJ > 0.0 && inv3(dX, dXi);
    if (ok) {
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
          F[i * 3 + j] = (i == j ? 1.0 : 0.0) + dU[i * 3] * dXi[j] + dU[i * 3 + 1] * dXi[3 + j] +
                         dU[i * 3 + 2] * dXi[6 + j] + M0[i * 3 + j];
    }
    const double J = ok ? det3(F) : -1.0;
    ok = ok && J > 0.0 && inv3(F, Fi);
    if (!ok) {
      atomicAdd(&A.status[0], 1ull);
#pragma unroll
      for (int c = 0; c < kP1Rec; c++) r[c] = 0.0;
    } else {
      QpTangent t;
      double Anp1[6], alpha_np1;
      spatial_update<PLASTIC>(A.mat, F, J, Ast, alpha, t, Anp1, &alpha_np1);
      if (PLASTIC && A.state_np1) {
#pragma unroll
        for (int c = 0; c < 6; c++) A.state_np1[c * A.ne + e] = Anp1[c];
        A.state_np1[6 * A.ne + e] = alpha_np1;
      }
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
          r[i * 3 + j] = dXi[i * 3] * Fi[j] + dXi[i * 3 + 1] * Fi[3 + j] + dXi[i * 3 + 2] * Fi[6 + j];
      const double w = detJ * (1.0 / 6.0), h = 0.5 * t.a1 * w, c23 = (2.0 / 3.0) * w;
      const bool pl = PLASTIC && (t.n[0] != 0.0 || t.n[1] != 0.0 || t.n[2] != 0.0 || t.n[3] != 0.0 ||
                                  t.n[4] != 0.0 || t.n[5] != 0.0);
#pragma unroll
      for (int c = 0; c < 6; c++) r[9 + c] = pl ? t.n[c] : t.s[c];
      r[15] = w * t.a2;
      r[16] = pl ? -c23 * sdot(t.s, t.n) : -c23;
      r[17] = w * t.a4;
      r[18] = w * t.a5;
      r[19] = h;
      r[20] = h + w * (t.tau[0] - t.s[0]);
      r[21] = 0.0;
    }
  }
  __syncthreads();
  const int cnt = (int)(A.ne - e0 < 128 ? A.ne - e0 : 128) * kP1Rec;
  for (int i = threadIdx.x; i < cnt; i += 128)
    A.rec[e0 * kP1Rec + i] = srow[(i / kP1Rec) * (kP1Rec + 1) + i % kP1Rec];
}

// ---- gather -------------------------------------------------------------------

// p of local node a and x of the other three, ascending: rows of G for nodes 1..3,
// minus their sum for node 0.  The lane functions below fill the three rows (i) of
// node a in the element block, columns of those three nodes, and its residual:
// val[j * 9 + i * 3 + k] and val[27 + i].
__device__ __forceinline__ void gather_nodes(const double *G, int a, double *p, double *x) {
  double p0[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    p0[j] = -(G[j] + G[3 + j] + G[6 + j]);
    p[j] = a == 0 ? p0[j] : (a == 1 ? G[j] : (a == 2 ? G[3 + j] : G[6 + j]));
    x[j] = a == 0 ? G[j] : p0[j];
    x[3 + j] = a <= 1 ? G[3 + j] : G[j];
    x[6 + j] = a == 3 ? G[3 + j] : G[6 + j];
  }
}

// HE, J2: K_ab[i][k] = h p_b[i] p_a[k] + p_a[i] U_b[k] + (s'' p_a)[i] p_b[k]
// + (n p_a)[i] W_b[k] + d_ik p_a . T' p_b (compute_stiffness_matrix,
// src/constitutive_model.cc:1520-1616, in spatial form), R_a = w tau p_a.
template <bool PLASTIC>
__device__ __forceinline__ void gather_lane(const double *r, int a, double *val) {
  double p[3], x[9], T[3], s6[6], sp[3], np[3] = {0, 0, 0}, Wm[6];
  gather_nodes(r, a, p, x);
  const double *n = r + 9;
  const double cs = r[16], wa2 = r[15], h = r[19], t0 = r[20];
#pragma unroll
  for (int c = 0; c < 6; c++) s6[c] = cs * n[c];
  smv(s6, p, sp);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    T[i] = fma(t0, p[i], -1.5 * sp[i]);
    val[27 + i] = fma(-h, p[i], T[i]);
  }
  if (PLASTIC) {
    const double w4 = r[17], w5 = r[18];
    double n2[6];
    n2[0] = n[0] * n[0] + n[5] * n[5] + n[4] * n[4];
    n2[1] = n[5] * n[5] + n[1] * n[1] + n[3] * n[3];
    n2[2] = n[4] * n[4] + n[3] * n[3] + n[2] * n[2];
    n2[3] = n[5] * n[4] + n[1] * n[3] + n[3] * n[2];
    n2[4] = n[0] * n[4] + n[5] * n[3] + n[4] * n[2];
    n2[5] = n[0] * n[5] + n[5] * n[1] + n[4] * n[3];
    const double t3 = (n2[0] + n2[1] + n2[2]) * (1.0 / 3.0);
#pragma unroll
    for (int c = 0; c < 6; c++) Wm[c] = w4 * n[c] + w5 * (n2[c] - (c < 3 ? t3 : 0.0));
    smv(n, p, np);
  }
#pragma unroll
  for (int b = 0; b < 3; b++) {
    const double *pb = x + 3 * b;
    double U[3], W[3];
    smv(s6, pb, U);
#pragma unroll
    for (int j = 0; j < 3; j++) U[j] = fma(wa2, pb[j], U[j]);
    if (PLASTIC) smv(Wm, pb, W);
    const double g = T[0] * pb[0] + T[1] * pb[1] + T[2] * pb[2];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double hp = h * pb[i];
#pragma unroll
      for (int j = 0; j < 3; j++) {
        double v = i == j ? fma(hp, p[j], g) : hp * p[j];
        v = fma(p[i], U[j], v);
        v = fma(sp[i], pb[j], v);
        val[b * 9 + i * 3 + j] = PLASTIC ? fma(np[i], W[j], v) : v;
      }
    }
  }
}

// Crystal plasticity (cp_crystal.cuh records: G 9, w tau 6, w c 36): K_ab[i][k] =
// p_a[j] c_(ij)(kl) p_b[l] + d_ik p_a . tau p_b, R_a = tau p_a.
__device__ __forceinline__ void gather_lane_c(const double *r, int a, double *val) {
  const int vo[9] = {0, 5, 4, 5, 1, 3, 4, 3, 2};
  double p[3], x[9], T[3], L[6][3];
  gather_nodes(r, a, p, x);
  smv(r + 9, p, T);
#pragma unroll
  for (int q = 0; q < 6; q++) smv(r + 15 + 6 * q, p, L[q]);
#pragma unroll
  for (int i = 0; i < 3; i++) val[27 + i] = T[i];
#pragma unroll
  for (int b = 0; b < 3; b++) {
    const double *pb = x + 3 * b;
    const double g = T[0] * pb[0] + T[1] * pb[1] + T[2] * pb[2];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        double v = i == j ? g : 0.0;
#pragma unroll
        for (int l = 0; l < 3; l++) v = fma(L[vo[j * 3 + l]][i], pb[l], v);
        val[b * 9 + i * 3 + j] = v;
      }
  }
}

struct GatherArgs {
  GatherLists L;
  const double *rec;
  double *R, *K;     // K may be null
  unsigned *ticket;  // groups claimed `grab` at a time, or nullptr: grid-stride
  int grab;
};

// record doubles of model 0, 1 (HE, J2) and 2 (crystal plasticity), and the
// stride of a staged record: an odd number of 16-byte words
__host__ __device__ constexpr int gather_rec(int model) { return model == 2 ? 52 : kP1Rec; }
__host__ __device__ constexpr int gather_stride(int model) { return model == 2 ? 54 : kP1Rec; }

// shared memory of a warp: values and nine zeros, staged records (over the values
// while a group has one round of 32 incidences), the rows, the columns' sums, lists,
// packs
struct GatherPlan {
  int stg, out, acc, slot, ent, bytes;  // byte offsets
};
__host__ __device__ inline GatherPlan gather_plan(int model, int most, int slots, int packs, int width) {
  GatherPlan p;
  const int cap = (most + 31) / 32 * 32, v = (gather_zero(most) + 9) * 8, st = 32 * gather_stride(model) * 8;
  p.stg = cap == 32 ? 0 : (v + 15) / 16 * 16;
  p.out = ((cap == 32 ? (v > st ? v : st) : p.stg + st) + 15) / 16 * 16;
  p.acc = p.out + 3 * width * 8;
  p.slot = p.acc + slots * 9 * 8;
  p.ent = p.slot + slots * 8;
  p.bytes = (p.ent + packs * 8 + 15) / 16 * 16;
  return p;
}

// One warp per group.  Output: a lane task is three adjacent values (k = 0..2) of
// one row of one list -- the residual as four partial sums (lanes 0..3), then the
// columns row by row -- so a task adds some six contributions; the own column is
// minus the sum of the others; the finished rows go through shared memory and leave
// as one contiguous run.
template <int MODEL>
__global__ void __launch_bounds__(128, MODEL == 2 ? 3 : 4) k_gather_p1(const GatherArgs A) {
  constexpr int NR = gather_rec(MODEL), ST = gather_stride(MODEL), NC = NR / 2;
  constexpr int PER = 32 / NC;  // records a copy instruction moves
  extern __shared__ __align__(16) unsigned char gsm[];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const GatherPlan pl = gather_plan(MODEL, A.L.most, A.L.slots, A.L.packs, A.L.width);
  unsigned char *mine = gsm + warp * pl.bytes;
  double *val = reinterpret_cast<double *>(mine), *stg = reinterpret_cast<double *>(mine + pl.stg);
  double *out = reinterpret_cast<double *>(mine + pl.out), *acc = reinterpret_cast<double *>(mine + pl.acc);
  uint2 *sslot = reinterpret_cast<uint2 *>(mine + pl.slot);
  uint2 *sent = reinterpret_cast<uint2 *>(mine + pl.ent);
  const int zero = gather_zero(A.L.most);
  const int crec = lane / NC, cch = lane - crec * NC;  // record and 16-byte word this lane copies
  const unsigned sdst = (unsigned)__cvta_generic_to_shared(stg + crec * ST + 2 * cch);
  pdl_wait();
  const long step = (long)gridDim.x * nw;
  long gn = A.ticket ? 0 : (long)blockIdx.x * nw + warp, ge = 0;
  auto next = [&]() -> long {
    if (!A.ticket) {
      const long g = gn;
      gn += step;
      return g;
    }
    if (gn >= ge) {
      unsigned c = 0;
      if (lane == 0) c = atomicAdd(A.ticket, (unsigned)A.grab);
      gn = __shfl_sync(FULL, c, 0);
      ge = gn + A.grab;
    }
    return gn++;
  };
  long g = next();
  int4 h0 = make_int4(0, 0, 0, 0), h1 = h0;
  int id = 0;
  if (g < A.L.ng) {
    h0 = A.L.head[2 * g];
    h1 = A.L.head[2 * g + 1];
    id = lane < (h1.x & 0xff) ? A.L.inc[h0.x + lane] : 0;
  }
  while (g < A.L.ng) {
    const int n = h1.x & 0xff, ns = (h1.x >> 8) & 0xff, npk = (h1.x >> 16) & 0xfff, w = h1.y;
    const unsigned mr = (unsigned)h1.x >> 28;
    const long gnext = next();
    int4 n0 = h0, n1 = h1;
    for (int r0 = 0; r0 < n; r0 += 32) {
      const int m = n - r0 < 32 ? n - r0 : 32;
      if (r0) id = lane < m ? A.L.inc[h0.x + r0 + lane] : 0;
      // the elements' records, PER a copy instruction
      for (int q = 0; q < m; q += PER) {
        const int it = q + crec;
        const int e = __shfl_sync(FULL, id, it & 31) >> 2;
        if (crec < PER && it < m)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(sdst + q * ST * 8),
                       "l"(A.rec + (long)e * NR + 2 * cch)
                       : "memory");
      }
      if (!r0) {  // beside the copies: the lists, and the next group's head
        for (int i = lane; i < ns; i += 32) sslot[i] = A.L.slot[h0.y + i];
        for (int i = lane; i < npk; i += 32) sent[i] = A.L.ent[h0.z + i];
        if (gnext < A.L.ng) {
          n0 = A.L.head[2 * gnext];
          n1 = A.L.head[2 * gnext + 1];
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      double r[NR];
#pragma unroll
      for (int f = 0; f < NC; f++) {
        const double2 v = *reinterpret_cast<const double2 *>(stg + lane * ST + 2 * f);
        r[2 * f] = v.x;
        r[2 * f + 1] = v.y;
      }
      __syncwarp();
      if (lane < m) {
        double *v = val + (r0 + lane) * kGVal;
        if (MODEL == 2) gather_lane_c(r, id & 3, v);
        else gather_lane<MODEL == 1>(r, id & 3, v);
      }
      __syncwarp();
    }
    if (gnext < A.L.ng) id = lane < (n1.x & 0xff) ? A.L.inc[n0.x + lane] : 0;
    if (lane < 9) val[zero + lane] = 0.0;
    __syncwarp();
    const int nl = ns - 1, tasks = A.K ? 4 + 3 * nl : 4;
    for (int t0 = 0; t0 < tasks; t0 += 32) {
      const int t = t0 + lane, q = t - 4;
      const bool quad = t < 4;
      const int i = quad || q < nl ? 0 : (q < 2 * nl ? 1 : 2), list = quad ? 0 : 1 + q - i * nl;
      double a0 = 0.0, a1 = 0.0, a2 = 0.0;
      uint2 sl = make_uint2(0u, 0u);
      if (t < tasks) sl = sslot[list];
      const uint2 *en = sent + (sl.y & 0xffff);
      const double *vi = val + 3 * i;
      for (int p = quad ? t : 0, np = sl.y >> 16; p < np; p += quad ? 4 : 1) {
        const uint2 e = en[p];
        const double *v0 = vi + (e.x & 0xffff), *v1 = vi + (e.x >> 16), *v2 = vi + (e.y & 0xffff),
                     *v3 = vi + (e.y >> 16);
        a0 += (v0[0] + v1[0]) + (v2[0] + v3[0]);
        a1 += (v0[1] + v1[1]) + (v2[1] + v3[1]);
        a2 += (v0[2] + v1[2]) + (v2[2] + v3[2]);
      }
      if (t0 == 0) {  // the residual's four partial sums
        double s0 = a0, s1 = a1, s2 = a2;
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
          s0 += __shfl_xor_sync(FULL, s0, o);
          s1 += __shfl_xor_sync(FULL, s1, o);
          s2 += __shfl_xor_sync(FULL, s2, o);
        }
        if (lane < 3 && ((mr >> lane) & 1u)) A.R[h1.z + rank_of(mr, lane)] = lane == 0 ? s0 : (lane == 1 ? s1 : s2);
      }
      if (!quad && t < tasks) {
        double *c = acc + list * 9 + 3 * i;
        c[0] = a0;
        c[1] = a1;
        c[2] = a2;
        const unsigned mb = (sl.x >> 16) & 7u;
        if ((mr >> i) & 1u) {
          double *o = out + rank_of(mr, i) * w + (sl.x & 0xffff);
          if (mb & 1u) *o++ = a0;
          if (mb & 2u) *o++ = a1;
          if (mb & 4u) *o = a2;
        }
      }
    }
    __syncwarp();
    if (A.K) {  // the own column, three partial sums each
      const int ik = lane % 9, i = ik / 3, k = ik - 3 * i;
      double s = 0.0;
      if (lane < 27)
        for (int l = 1 + lane / 9; l <= nl; l += 3) s += acc[l * 9 + ik];
      s += __shfl_down_sync(FULL, s, 9) + __shfl_down_sync(FULL, s, 18);
      if (lane < 9 && ((mr >> i) & 1u) && ((mr >> k) & 1u)) out[rank_of(mr, i) * w + h1.w + rank_of(mr, k)] = -s;
    }
    __syncwarp();
    if (A.K) {
      const int cnt = __popc(mr) * w;
      for (int o = lane; o < cnt; o += 32) A.K[(long)h0.w + o] = out[o];
    }
    __syncwarp();
    g = gnext;
    h0 = n0;
    h1 = n1;
  }
}

}  // namespace pgb
