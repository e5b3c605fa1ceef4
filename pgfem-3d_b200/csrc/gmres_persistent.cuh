// gmres_persistent.cuh -- whole GMRES cycles in one cooperative kernel.
//
// Each CTA owns a contiguous block of rows: their slice of the Krylov basis
// and, where it fits, their rows of K stay in its shared memory for the whole
// launch, so an Arnoldi step reads only the vector it multiplies through L2.
//
// A step has one grid-wide wait (the product's input is written) and two
// all-reduces of j + 1 dot products (the two Gram-Schmidt passes).  An
// all-reduce is two one-way messages and no barrier: a partial sum travels as a
// 16-byte word {value, sequence number} to the CTA that owns its entry, which
// adds the partials in a fixed order and publishes {sum, sequence number}; the
// readers poll the words themselves.  A barrier and every CTA adding all
// partials took 7 k cycles, the messages 3 k.  Sums are the same bits in every
// CTA, so all take the same decisions, and they do not depend on timing.
//
// The norm of the new direction needs no reduction of its own: ||w - V h||^2 =
// ||w||^2 - ||h||^2 for an orthonormal V, with the explicit sum when the two
// terms cancel.  The Givens rotations of a column run in one warp of CTA 0
// beside the next product.
//
// Measured, us per step, against the launch sequence that takes the large systems
// (ten launches a step, rotations and back substitution in one-thread kernels;
// solver.cu has the line between the two), J2 quadratic tets, kdim 100: 1,863 rows
// 70.5 -> 12.7, 13,583 rows 75.5 -> 14.2, 44,375 rows 86 -> 27, 103,455 rows 122 -> 71,
// 343,343 rows 294 -> 238; kdim 500, 13,583 rows 165 -> 28.  Up to some 30 k rows at kdim 100 (basis slice in shared memory) it
// is bound by the five one-way messages of a step, about 1.3 us each between
// SMs; above, by reading the basis four times a step from L2 and HBM.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace gmp {

constexpr int kThreads = 1024, kWarps = kThreads / 32;
constexpr int kSmemMost = 227 * 1024;

struct State {
  double bnorm, tol;
  int iters;  // Arnoldi steps over all cycles
  int converged, breakdown, stop, timeout;
};

struct Args {
  long n;
  int rows, ldv, m, nblk;  // rows per CTA, leading dimension of the basis slice
  int vs, ks, kcap;        // basis / K rows in shared memory; entries of the K buffer
  const int *Ap, *Ai;
  const double *K, *dinv, *b;
  double *x, *V, *z, *H, *g, *y;
  ulonglong2 *slot, *res;  // partials [m + 2][nblk], sums [m + 3] (the last: the stop code)
  unsigned long long seq0;
  State *S;
  unsigned *bar;
  int maxit, max_cycles;
  unsigned long long wait_ns;
};

constexpr size_t smem_fixed(int rows, int m) {  // w, two columns of sums, rotations, the own Hessenberg column
  return sizeof(double) * ((size_t)rows + 2 * (m + 2) + 3 * (size_t)(m + 2) + kWarps + 1 + kThreads);
}

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ unsigned long long timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid-wide wait, bounded: false in every CTA that saw it run out (the others'
// next wait runs out too).  The launch is cooperative, so all CTAs are resident.
__device__ __forceinline__ bool grid_wait(const Args &A, unsigned &epoch) {
  __syncthreads();
  bool ok = true;
  if (threadIdx.x == 0) {
    epoch += (unsigned)A.nblk;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(A.bar) : "memory");
    const unsigned long long t0 = timer_ns();
    for (int spin = 0;; spin++) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(A.bar) : "memory");
      if ((int)(v - epoch) >= 0) break;
      if ((spin & 1023) == 1023 && timer_ns() - t0 > A.wait_ns) {
        ok = false;
        A.S->timeout = 1;
        break;
      }
    }
  }
  return __syncthreads_and(ok) != 0;
}

// y[r] = K z over the own rows into sw, by nwarps warps of the CTA, LPR lanes a
// row.  With K in shared memory eight lanes a row put all rows of a small block
// in flight at once; from global memory a whole warp reads a row in full lines.
template <int LPR>
__device__ __forceinline__ void product(const double *Kp, const int *Ip, const int *ap, int nr, const double *zin,
                                        double *sw, int warp, int nwarps) {
  const int sub = threadIdx.x & (LPR - 1);
  const int grp = (warp * 32 + (threadIdx.x & 31)) / LPR, ngrp = nwarps * 32 / LPR;
  constexpr int U = LPR == 8 ? 12 : 4;  // entries a lane loads at once
  for (int r0 = 0; r0 < nr; r0 += ngrp) {
    const int r = r0 + grp;
    double s = 0.0;
    if (r < nr) {
      const int e = ap[r + 1];
      for (int j = ap[r] + sub; j < e; j += U * LPR) {
        double x[U];
#pragma unroll
        for (int u = 0; u < U; u++) x[u] = j + u * LPR < e ? zin[Ip[j + u * LPR]] : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++)
          if (j + u * LPR < e) s = fma(Kp[j + u * LPR], x[u], s);
      }
    }
#pragma unroll
    for (int o = LPR / 2; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (r < nr && sub == 0) sw[r] = s;
  }
}

__device__ __forceinline__ void product_any(const Args &A, const double *Kp, const int *Ip, const int *ap, int nr,
                                            const double *zin, double *sw, int warp, int nwarps) {
  if (A.ks) product<8>(Kp, Ip, ap, nr, zin, sw, warp, nwarps);
  else product<32>(Kp, Ip, ap, nr, zin, sw, warp, nwarps);
}

// ---- all-reduce by tagged words ----
__device__ __forceinline__ void put(ulonglong2 *p, double v, unsigned long long seq) {
  asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(seq)
               : "memory");
}
__device__ __forceinline__ bool get(const ulonglong2 *p, double &v, unsigned long long seq) {
  unsigned long long a, b;
  asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
               : "=l"(a), "=l"(b)
               : "l"(p)
               : "memory");
  v = __longlong_as_double((long long)a);
  return b == seq;
}

// The own partials (V[t], w), t < nt, and with ww (w, w) as entry nt, sent to
// their owners.  LPV lanes a vector: eight (four vectors a warp, few shuffles) for
// a slice in shared memory, ld = 8 mod 16 doubles, free of bank conflicts; a
// whole warp, full lines, for one in global memory.
template <int LPV>
__device__ __forceinline__ void dots(const Args &A, const double *Vs, int ld, int nr, const double *sw, int nt, int ww,
                                     unsigned long long seq) {
  const int sub = threadIdx.x & (LPV - 1), cnt = nt + ww;
  for (int t0 = 0; t0 < cnt; t0 += kThreads / LPV) {
    const int t = t0 + threadIdx.x / LPV;
    double a0 = 0.0, a1 = 0.0;
    if (t < cnt) {
      const double *v = t < nt ? Vs + (long)t * ld : sw;
      int r = sub;
#pragma unroll 4
      for (; r + LPV < nr; r += 2 * LPV) {
        a0 = fma(v[r], sw[r], a0);
        a1 = fma(v[r + LPV], sw[r + LPV], a1);
      }
      if (r < nr) a0 = fma(v[r], sw[r], a0);
    }
    double s = a0 + a1;
#pragma unroll
    for (int o = LPV / 2; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (t < cnt && sub == 0) put(A.slot + (long)t * A.nblk + blockIdx.x, s, seq);
  }
}

// The sums of cnt entries whose partials every CTA has sent with this sequence
// number, into out; with code (may be null) the stop code of CTA 0.  A CTA sends
// the next all-reduce's partials only after it has every sum of this one, so one
// set of words is enough.  Bounded like grid_wait.
__device__ __forceinline__ bool allreduce(const Args &A, int cnt, unsigned long long seq, double *out, int *code) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long t0 = timer_ns();
  bool ok = true;
  auto late = [&](int &spin) {
    if ((++spin & 255) == 0 && timer_ns() - t0 > A.wait_ns) {
      A.S->timeout = 1;
      ok = false;
    }
    return !ok;
  };
  for (int t = blockIdx.x + A.nblk * warp; t < cnt; t += A.nblk * kWarps) {  // entries this CTA owns
    const ulonglong2 *p = A.slot + (long)t * A.nblk;
    double s = 0.0;
    for (int q0 = lane; q0 < A.nblk; q0 += 160) {
      double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
      for (int spin = 0;;) {
        bool all = true;
#pragma unroll
        for (int u = 0; u < 5; u++)
          if (q0 + 32 * u < A.nblk) all = get(p + q0 + 32 * u, v[u], seq) && all;
        if (all || late(spin)) break;
      }
#pragma unroll
      for (int u = 0; u < 5; u++) s += v[u];
    }
    __syncwarp();
    s = wsum(s);
    if (lane == 0) put(A.res + t, s, seq);
  }
  for (int t = tid; t < cnt + (code ? 1 : 0); t += kThreads) {
    double v = 0.0;
    const ulonglong2 *p = A.res + (t < cnt ? t : A.m + 2);
    for (int spin = 0; !get(p, v, seq) && !late(spin);) {
    }
    if (t < cnt) out[t] = v;
    else *code = (int)v;
  }
  return __syncthreads_and(ok) != 0;
}

// w - V h over the own rows, handed to done(row, value) once per row: eight groups
// of 128 threads, a row a thread
template <class F>
__device__ __forceinline__ void subtract(const double *Vs, int ld, int nr, const double *sw, int nt, const double *h,
                                         double *tmp, F done) {
  const int tid = threadIdx.x, gr = tid >> 7;
  for (int r0 = 0; r0 < nr; r0 += 128) {
    const int r = r0 + (tid & 127);
    double a0 = 0.0, a1 = 0.0;
    if (r < nr) {
      int t = gr;
#pragma unroll 4
      for (; t + 8 < nt; t += 16) {
        a0 = fma(Vs[(long)t * ld + r], h[t], a0);
        a1 = fma(Vs[(long)(t + 8) * ld + r], h[t + 8], a1);
      }
      if (t < nt) a0 = fma(Vs[(long)t * ld + r], h[t], a0);
    }
    tmp[tid] = a0 + a1;
    __syncthreads();
    if (tid < 128 && r < nr) {
      double s = 0.0;
#pragma unroll
      for (int u = 0; u < 8; u++) s += tmp[u * 128 + tid];
      done(r, sw[r] - s);
    }
    __syncthreads();
  }
}

// One warp: the previous rotations on column j (hc, j + 2 entries), rotation j,
// the residual estimate; returns the stop code of the step (0: go on).  The
// running entry h <- c_t h_{t+1} - s_t h is an affine recurrence, so 32 rotations
// are one scan over the lanes (a serial lane took longer than the product it
// runs beside from some 60 columns on).
__device__ __forceinline__ int givens(const Args &A, int j, double *hc, double *cs, double *sn) {
  const int lane = threadIdx.x & 31;
  double h0 = hc[0];
  double *col = A.H + (long)j * (A.m + 1);
  for (int t0 = 0; t0 < j; t0 += 32) {
    const int t = t0 + lane;
    const bool in = t < j;
    const double c = in ? cs[t] : 1.0, s = in ? sn[t] : 0.0, h1 = in ? hc[t + 1] : 0.0;
    double f = in ? -s : 1.0, p = in ? c * h1 : 0.0;  // h -> f h + p, composed over the lanes below
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double fo = __shfl_up_sync(0xffffffffu, f, o), po = __shfl_up_sync(0xffffffffu, p, o);
      if (lane >= o) {
        p = fma(f, po, p);
        f *= fo;
      }
    }
    const double after = fma(f, h0, p);
    double before = __shfl_up_sync(0xffffffffu, after, 1);
    if (lane == 0) before = h0;
    if (in) col[t] = c * before + s * h1;
    h0 = __shfl_sync(0xffffffffu, after, 31);
  }
  const double hn = hc[j + 1];
  const double d = hypot(h0, hn);
  if (!(d > 0.0) || !isfinite(d)) return 2;
  const double gj = A.g[j], c = h0 / d, s = hn / d, gn = -s * gj;
  __syncwarp();
  if (lane == 0) {
    cs[j] = c;
    sn[j] = s;
    col[j] = d;
    A.g[j + 1] = gn;
    A.g[j] = c * gj;
  }
  return fabs(gn) <= A.S->tol * A.S->bnorm || hn == 0.0 ? 1 : 0;
}

__device__ __forceinline__ void dots_any(const Args &A, const double *Vs, int ld, int nr, const double *sw, int nt,
                                         int ww, unsigned long long seq) {
  if (A.vs) dots<8>(A, Vs, ld, nr, sw, nt, ww, seq);
  else dots<32>(A, Vs, ld, nr, sw, nt, ww, seq);
}

__global__ void __launch_bounds__(kThreads, 1) k_gmres_cycles(const Args A) {
  extern __shared__ double sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blk = blockIdx.x, m = A.m;
  const long r0 = (long)blk * A.rows;
  const int nr = (int)(A.n - r0 < A.rows ? A.n - r0 : A.rows);
  double *sw = sm, *h1 = sw + A.rows, *h2 = h1 + m + 2, *cs = h2 + m + 2, *sn = cs + m + 2, *hc = sn + m + 2;
  double *sred = hc + m + 2;
  int *scode = reinterpret_cast<int *>(sred + kWarps);
  double *tmp = sred + kWarps + 1;
  unsigned long long seq = A.seq0;
  double *Vs = A.vs ? tmp + kThreads : A.V + r0;
  const int ld = A.ldv;
  double *Kb = tmp + kThreads + (A.vs ? (size_t)ld * (m + 1) : 0);
  int *Ib = reinterpret_cast<int *>(Kb + A.kcap), *ab = Ib + A.kcap;
  unsigned epoch = 0;
  // the own rows of K
  const double *Kp = A.K;
  const int *Ip = A.Ai, *ap = A.Ap + r0;
  if (A.ks) {
    const int b0 = A.Ap[r0], cnt = A.Ap[r0 + nr] - b0;
    for (int i = tid; i < cnt; i += kThreads) {
      Kb[i] = A.K[b0 + i];
      Ib[i] = A.Ai[b0 + i];
    }
    for (int i = tid; i <= nr; i += kThreads) ab[i] = A.Ap[r0 + i] - b0;
    Kp = Kb;
    Ip = Ib;
    ap = ab;
    __syncthreads();
  }
  for (int cycle = 0; cycle < A.max_cycles; cycle++) {
    // r = b - K x, its norm and b's
    product_any(A, Kp, Ip, ap, nr, A.x, sw, warp, kWarps);
    __syncthreads();
    double d0 = 0.0, d1 = 0.0;
    for (int r = tid; r < nr; r += kThreads) {
      const double bi = A.b[r0 + r], ri = bi - sw[r];
      sw[r] = ri;
      d0 = fma(ri, ri, d0);
      d1 = fma(bi, bi, d1);
    }
    seq++;
    d0 = wsum(d0);
    d1 = wsum(d1);
    if (lane == 0) {
      sred[warp] = d0;
      tmp[warp] = d1;
    }
    __syncthreads();
    if (warp < 2) {
      const double s = wsum(warp == 0 ? sred[lane] : tmp[lane]);
      if (lane == 0) put(A.slot + (long)warp * A.nblk + blk, s, seq);
    }
    if (!allreduce(A, 2, seq, h1, nullptr)) return;
    const double beta = sqrt(h1[0]), bnorm = sqrt(h1[1]);
    const bool conv0 = beta <= A.S->tol * bnorm;
    if (conv0 || !isfinite(beta)) {
      if (blk == 0 && tid == 0) {
        A.S->bnorm = bnorm;
        A.S->converged = conv0 ? 1 : 0;
        A.S->breakdown = conv0 ? 0 : 1;
        A.S->stop = 1;
      }
      return;
    }
    const int it0 = A.S->iters;
    const int jmax = A.maxit - it0 < m ? A.maxit - it0 : m;
    if (blk == 0 && tid == 0) {
      A.S->bnorm = bnorm;
      A.g[0] = beta;
    }
    const double ib = 1.0 / beta;
    for (int r = tid; r < nr; r += kThreads) {
      const double v = sw[r] * ib;
      Vs[r] = v;
      __stcg(A.z + r0 + r, A.dinv[r0 + r] * v);
    }
    if (!grid_wait(A, epoch)) return;
    int j = 0, code = 0;
    for (;; j++) {
      // product; CTA 0's last warp finishes the previous column meanwhile
      if (blk == 0 && warp == kWarps - 1 && j > 0) {
        const int c = givens(A, j - 1, hc, cs, sn);
        if (lane == 0) put(A.res + m + 2, (double)c, seq + 1);
      } else if (j < jmax) {
        product_any(A, Kp, Ip, ap, nr, A.z, sw, warp, blk == 0 && j > 0 ? kWarps - 1 : kWarps);
      }
      __syncthreads();
      seq++;
      if (j < jmax) dots_any(A, Vs, ld, nr, sw, j + 1, 0, seq);
      if (!allreduce(A, j < jmax ? j + 1 : 0, seq, h1, j > 0 ? scode : nullptr)) return;
      code = j > 0 ? *scode : 0;
      if (code || j >= jmax) break;
      subtract(Vs, ld, nr, sw, j + 1, h1, tmp, [&](int r, double v) { sw[r] = v; });
      seq++;
      dots_any(A, Vs, ld, nr, sw, j + 1, 1, seq);
      if (!allreduce(A, j + 2, seq, h2, nullptr)) return;
      const double ww = h2[j + 1];
      double hh = 0.0;
      for (int t = lane; t <= j; t += 32) hh = fma(h2[t], h2[t], hh);
      hh = wsum(hh);
      double nn = ww - hh;
      double *Vn = Vs + (long)(j + 1) * ld;
      double hn;
      if (nn > 0.25 * ww) {  // the same decision in every CTA
        hn = sqrt(nn);
        const double inv = 1.0 / hn;
        subtract(Vs, ld, nr, sw, j + 1, h2, tmp, [&](int r, double w) {
          const double v = w * inv;
          Vn[r] = v;
          __stcg(A.z + r0 + r, A.dinv[r0 + r] * v);
        });
      } else {  // cancellation: the explicit sum
        subtract(Vs, ld, nr, sw, j + 1, h2, tmp, [&](int r, double v) { sw[r] = v; });
        double d = 0.0;
        for (int r = tid; r < nr; r += kThreads) d = fma(sw[r], sw[r], d);
        d = wsum(d);
        if (lane == 0) sred[warp] = d;
        __syncthreads();
        seq++;
        if (warp == 0) {
          const double s = wsum(sred[lane]);
          if (lane == 0) put(A.slot + blk, s, seq);
        }
        if (!allreduce(A, 1, seq, tmp, nullptr)) return;
        hn = sqrt(tmp[0]);
        const double inv = hn > 0.0 ? 1.0 / hn : 0.0;
        for (int r = tid; r < nr; r += kThreads) {
          const double v = sw[r] * inv;
          Vn[r] = v;
          __stcg(A.z + r0 + r, A.dinv[r0 + r] * v);
        }
      }
      if (blk == 0) {
        for (int t = tid; t <= j; t += kThreads) hc[t] = h1[t] + h2[t];
        if (tid == 0) hc[j + 1] = hn;
      }
      if (!grid_wait(A, epoch)) return;
    }
    // k steps of this cycle count; y = H(0:k, 0:k)^-1 g (CTA 0, one warp, by columns)
    const int k = code == 2 ? j - 1 : j;
    if (blk == 0 && warp == 0) {
      for (int t = lane; t < k; t += 32) hc[t] = A.g[t];
      __syncwarp();
      for (int t = k - 1; t >= 0; t--) {
        const double *col = A.H + (long)t * (m + 1);
        const double d = col[t], yt = d != 0.0 ? hc[t] / d : 0.0;
        if (lane == 0) __stcg(A.y + t, yt);
        for (int i = lane; i < t; i += 32) hc[i] = fma(-col[i], yt, hc[i]);
        __syncwarp();
      }
      if (lane == 0) A.S->iters = it0 + k;
    }
    if (!grid_wait(A, epoch)) return;
    // x += D V y over the own rows
    for (int t = tid; t < k; t += kThreads) h1[t] = -__ldcg(A.y + t);
    for (int r = tid; r < nr; r += kThreads) sw[r] = 0.0;
    __syncthreads();
    subtract(Vs, ld, nr, sw, k, h1, tmp, [&](int r, double v) {
      const long i = r0 + r;
      A.x[i] = fma(A.dinv[i], v, A.x[i]);
    });
    const bool stop = code != 0 || it0 + k >= A.maxit || k == 0;
    if (blk == 0 && tid == 0) {
      A.S->converged = code == 1 ? 1 : 0;
      A.S->breakdown = code == 2 ? 1 : 0;
      A.S->stop = stop ? 1 : 0;
    }
    if (stop) return;
    if (!grid_wait(A, epoch)) return;
  }
}

}  // namespace gmp
