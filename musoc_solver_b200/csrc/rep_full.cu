// Reference-faithful SEVP drop-ins on the GPU: the full-width and strip
// marching solves (REP1, REP, REPBIR, REPBIR_PERIOD, M/sevp.f90:11-438), the
// influence precompute (PRE1, PRE, P/prep_GLOBAL.f90:327-513), the
// no-pivoting Gauss-Jordan inverse (MATINV, P/prep_GLOBAL.f90:516-568) and the
// overlapping-strip sweeps of FS_SOLVER (M/fs_GLOBAL.f90:1904-1966).
//
// Every floating-point step uses explicitly rounded intrinsics (__dmul_rn,
// __dadd_rn, __dsub_rn, __ddiv_rn: no contraction into fused multiply-adds)
// and the reference's evaluation order, including the serial order of the
// mat-vec and GEMM sums, so the results are bit-identical to an IEEE-754
// double evaluation of the Fortran (the CPU oracle is that evaluation).
// Parallelism is across columns (marching), across unit responses (PRE) and
// across matrix elements (MATINV, GEMM); the sequential structure of the
// method (rows, blocks) is kept.
#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include <cooperative_groups.h>

#include "common.cuh"
#include "dropin.cuh"

namespace sevp {

#define IXD(ld, i, j) ((size_t)((j) - 1) * (size_t)(ld) + (size_t)((i) - 1))

__device__ __forceinline__ double c64(const float *a, int ld, int i, int j) {
  return (double)a[IXD(ld, i, j)];
}
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }

// (F - AX*V_W - AY*V_S - BB*V_C - CX*V_E) / CY   (M/sevp.f90:29-30)
__device__ __forceinline__ double march_val(const MarchArgs &a, const double *v, int ldv, int i,
                                            int j, double f) {
  double t = sub(f, mul(c64(a.ax, a.ldc, i, j), v[IXD(ldv, i, j + 1)]));
  t = sub(t, mul(c64(a.ay, a.ldc, i, j), v[IXD(ldv, i + 1, j)]));
  t = sub(t, mul(c64(a.bb, a.ldc, i, j), v[IXD(ldv, i + 1, j + 1)]));
  t = sub(t, mul(c64(a.cx, a.ldc, i, j), v[IXD(ldv, i + 2, j + 1)]));
  return dvd(t, c64(a.cy, a.ldc, i, j));
}

// residual of equation row j (M/sevp.f90:37-38)
__device__ __forceinline__ double resid_val(const MarchArgs &a, int i, int j) {
  const double *x = a.x;
  const int ld = a.ldx;
  double t = sub((double)a.f[IXD(a.ldf, i, j)], mul(c64(a.ax, a.ldc, i, j), x[IXD(ld, i, j + 1)]));
  t = sub(t, mul(c64(a.ay, a.ldc, i, j), x[IXD(ld, i + 1, j)]));
  t = sub(t, mul(c64(a.bb, a.ldc, i, j), x[IXD(ld, i + 1, j + 1)]));
  t = sub(t, mul(c64(a.cx, a.ldc, i, j), x[IXD(ld, i + 2, j + 1)]));
  t = sub(t, mul(c64(a.cy, a.ldc, i, j), x[IXD(ld, i + 1, j + 2)]));
  return t;
}

__device__ __forceinline__ void ghost_row(double *v, int ld, int gi0, int j) {
  if (threadIdx.x == 0) {
    v[IXD(ld, 1, j)] = v[IXD(ld, gi0 - 1, j)];
    v[IXD(ld, gi0, j)] = v[IXD(ld, 2, j)];
  }
}

// out(n) = sum_m in(m) * R(m, n), serial in m, one thread per n.  The
// column's elements are loaded kVecmatBatch at a time before they are
// summed (one memory round trip per batch instead of per element); the sum
// keeps the reference's order.
constexpr int kVecmatBatch = 16;
__device__ __forceinline__ void vecmat_serial(const double *in, const double *R, int m2,
                                              double *out) {
  for (int n = threadIdx.x; n < m2; n += blockDim.x) {
    const double *col = R + (size_t)n * m2;
    double s = 0.0;
    int k = 0;
    for (; k + kVecmatBatch <= m2; k += kVecmatBatch) {
      double c[kVecmatBatch], v[kVecmatBatch];
#pragma unroll
      for (int q = 0; q < kVecmatBatch; ++q) {
        c[q] = col[k + q];
        v[q] = in[k + q];
      }
#pragma unroll
      for (int q = 0; q < kVecmatBatch; ++q) s = add(s, mul(v[q], c[q]));
    }
    for (; k < m2; ++k) s = add(s, mul(in[k], col[k]));
    out[n] = s;
  }
}

// One CTA runs the whole marching solve (forward and backward sweeps).
__global__ void __launch_bounds__(1024) k_march_solve(MarchArgs a) {
  const int m2 = a.m2;
  const size_t msz = (size_t)m2 * m2;
  double *X = a.x, *H = a.h;
  const int ldx = a.ldx, ldh = a.ldh;
  const int tid = threadIdx.x, nt = blockDim.x;
  int js = 1;
  for (int nb = 1; nb <= a.nblk; ++nb) {
    const int jf = a.ie[nb - 1] - 2;
    for (int j = js; j <= jf; ++j) {
      if (a.periodic) ghost_row(X, ldx, a.gi0, j + 1);
      __syncthreads();
      for (int i = 1 + tid; i <= m2; i += nt)
        X[IXD(ldx, i + 1, j + 2)] = march_val(a, X, ldx, i, j, (double)a.f[IXD(a.ldf, i, j)]);
      __syncthreads();
    }
    if (a.periodic) ghost_row(X, ldx, a.gi0, jf + 2);
    __syncthreads();
    if (nb != a.nblk) {
      int j = a.ie[nb - 1] - 1;
      for (int i = 1 + tid; i <= m2; i += nt) a.dum1[i - 1] = resid_val(a, i, j);
      __syncthreads();
      j = a.ie[nb - 1];
      vecmat_serial(a.dum1, a.rinv1 + (size_t)(nb - 1) * msz, m2, a.dum2);
      __syncthreads();
      for (int n = 1 + tid; n <= m2; n += nt) {
        a.dum0[IXD(m2, n, nb)] = X[IXD(ldx, n + 1, j)];
        X[IXD(ldx, n + 1, j)] = sub(X[IXD(ldx, n + 1, j)], a.dum2[n - 1]);
      }
      __syncthreads();
      if (a.periodic) ghost_row(X, ldx, a.gi0, j);
      __syncthreads();
    }
    js = a.ie[nb - 1];
  }
  for (int nbs = 1; nbs <= a.nblk; ++nbs) {
    const int nb = a.nblk - nbs + 1;
    js = (nb != 1) ? a.ie[nb - 2] : 1;
    const int jf = a.ie[nb - 1] - 2;
    if (nb != a.nblk) {
      const int j = a.ie[nb - 1];
      for (int n = 1 + tid; n <= m2; n += nt) X[IXD(ldx, n + 1, j)] = a.dum0[IXD(m2, n, nb)];
    }
    for (int j = js; j <= a.ie[nb - 1]; ++j)
      for (int i = 1 + tid; i <= a.hzero; i += nt) H[IXD(ldh, i, j)] = 0.0;
    __syncthreads();
    int j = a.ie[nb - 1] - 1;
    if (a.periodic) ghost_row(X, ldx, a.gi0, j + 1);
    __syncthreads();
    for (int i = 1 + tid; i <= m2; i += nt) a.dum1[i - 1] = resid_val(a, i, j);
    __syncthreads();
    vecmat_serial(a.dum1, a.rinv + (size_t)(nb - 1) * msz, m2, a.dum2);
    __syncthreads();
    for (int n = 1 + tid; n <= m2; n += nt) {
      H[IXD(ldh, n + 1, js + 1)] = a.dum2[n - 1];
      X[IXD(ldx, n + 1, js + 1)] = add(X[IXD(ldx, n + 1, js + 1)], a.dum2[n - 1]);
    }
    __syncthreads();
    if (a.periodic) {
      ghost_row(H, ldh, a.gi0, js + 1);
      ghost_row(X, ldx, a.gi0, js + 1);
    }
    __syncthreads();
    if (nb != 1) {
      for (int k = 1 + tid; k <= m2; k += nt)
        a.dum1[k - 1] = mul(H[IXD(ldh, k + 1, js + 1)], c64(a.cy, a.ldc, k, js - 1));
      __syncthreads();
      j = a.ie[nb - 2];
      vecmat_serial(a.dum1, a.rinv1 + (size_t)(nb - 2) * msz, m2, a.dum2);
      __syncthreads();
      for (int n = 1 + tid; n <= m2; n += nt) H[IXD(ldh, n + 1, j)] = a.dum2[n - 1];
      __syncthreads();
      if (a.periodic) ghost_row(H, ldh, a.gi0, j);
      __syncthreads();
    }
    for (j = js; j <= jf; ++j) {
      if (a.periodic) ghost_row(H, ldh, a.gi0, j + 1);
      __syncthreads();
      for (int i = 1 + tid; i <= m2; i += nt) {
        double hv = march_val(a, H, ldh, i, j, 0.0);
        H[IXD(ldh, i + 1, j + 2)] = hv;
        X[IXD(ldx, i + 1, j + 2)] = add(X[IXD(ldx, i + 1, j + 2)], hv);
      }
      __syncthreads();
      if (a.periodic) ghost_row(X, ldx, a.gi0, j + 2);
      __syncthreads();
    }
  }
  if (a.periodic) {
    for (int j = 2 + tid; j <= a.ie[a.nblk - 1]; j += nt) {
      X[IXD(ldx, 1, j)] = X[IXD(ldx, a.gi0 - 1, j)];
      X[IXD(ldx, a.gi0, j)] = X[IXD(ldx, 2, j)];
    }
  }
}

// The marching solve on a cluster of kMarchCtas CTAs, for grids whose blocks'
// rows fit their shared memory.
//
// k_march_solve is one CTA that reads each influence matrix (m2 x m2) for one
// serial mat-vec: 44 of them at 180 x 90 with 15 blocks, each 259 KB through
// one SM in dependent batches, and every marched row goes through global
// memory; 655 us.  Here the mat-vecs' output columns are split over the
// cluster: a CTA copies its columns of the next two matrices to shared memory
// while the rows march (cp.async), sums its outputs in the reference's serial
// order from there (two instructions' latency per term), and writes them to
// every CTA of the cluster.  All CTAs march all rows themselves, one column
// per thread, on rows in shared memory with the coefficients two rows ahead
// in registers, so the mat-vec results are all that is exchanged.  CTA 0
// writes the outputs; the other CTAs read of X only input rows that it has
// not written yet (the guess rows, in the forward sweep).
// The arithmetic of every value is that of k_march_solve, so the results are
// bit-identical.
constexpr int kMarchCtas = 8;
constexpr int kMarchMaxCols = 512;  // one thread per column

struct MarchCoef {
  float ax, ay, bb, cx, cy, f;
  double e;  // forward: row j + 2's ghost cell (closed grids); backward: X(., j + 2)
};

// Doubles of shared memory: saved rows (ie - 1, ie, guess) per block, two
// matrix slices, three rows, the mat-vec input and two outputs.
__host__ __device__ inline size_t march_smem_doubles(int m2, int nblk, int nper) {
  return (size_t)3 * nblk * m2 + (size_t)2 * nper * (m2 | 1) + (size_t)3 * (m2 + 2) +
         (size_t)3 * m2;
}

__global__ void __cluster_dims__(kMarchCtas, 1, 1) __launch_bounds__(kMarchMaxCols, 1)
    k_march_cluster(MarchArgs a, int nper) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) double msm[];
  const int rank = (int)cl.block_rank();
  const int m2 = a.m2, nblk = a.nblk, ldr = m2 | 1, ld = m2 + 2;
  const int tid = threadIdx.x, i = tid + 1, nt = blockDim.x;
  const bool act = tid < m2, lead = rank == 0, per = a.periodic != 0;
  const size_t msz = (size_t)m2 * m2;
  double *SA = msm, *D0 = SA + (size_t)nblk * m2, *G = D0 + (size_t)nblk * m2;
  double *Rb = G + (size_t)nblk * m2, *rows = Rb + (size_t)2 * nper * ldr;
  double *vin = rows + 3 * ld, *vout = vin + m2;
  const int n0 = rank * nper, cnt = max(0, min(nper, m2 - n0));
  const int last = a.ie[nblk - 1], crows = last - 1;

  // ---- the mat-vecs, in the order of the sweeps
  auto matrix = [&](int q) -> const double * {
    if (q < nblk - 1) return a.rinv1 + (size_t)q * msz;
    const int p = q - (nblk - 1), nb = nblk - p / 2;
    return (p & 1) ? a.rinv1 + (size_t)(nb - 2) * msz : a.rinv + (size_t)(nb - 1) * msz;
  };
  const int nq = 3 * nblk - 2;
  auto prefetch = [&](int q) {
    if (q < nq) {
      const double *R = matrix(q) + (size_t)n0 * m2;
      double *dst = Rb + (size_t)(q & 1) * nper * ldr;
      for (int c = tid >> 5; c < cnt; c += nt >> 5)
        for (int k = tid & 31; k < m2; k += 32) {
          const unsigned d = (unsigned)__cvta_generic_to_shared(dst + (size_t)c * ldr + k);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d),
                       "l"(R + (size_t)c * m2 + k)
                       : "memory");
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  int q = 0;
  prefetch(0);
  prefetch(1);
  cl.sync();  // every CTA runs before any writes to another's shared memory
  // out(n) = sum_k vin(k) R(k, n) for all n, on every CTA (vin is written by
  // the caller's threads just before)
  auto matvec = [&]() -> const double * {
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    double *out = vout + (size_t)(q & 1) * m2;
    if (tid < cnt) {
      const double *col = Rb + (size_t)(q & 1) * nper * ldr + (size_t)tid * ldr;
      double s = 0.0;
      int k = 0;
      for (; k + kVecmatBatch <= m2; k += kVecmatBatch) {
        double c[kVecmatBatch], v[kVecmatBatch];
#pragma unroll
        for (int u = 0; u < kVecmatBatch; ++u) c[u] = col[k + u], v[u] = vin[k + u];
#pragma unroll
        for (int u = 0; u < kVecmatBatch; ++u) s = add(s, mul(v[u], c[u]));
      }
      for (; k < m2; ++k) s = add(s, mul(vin[k], col[k]));
      for (int r = 0; r < kMarchCtas; ++r) cl.map_shared_rank(out, r)[n0 + tid] = s;
    }
    // the other output buffer is not written before every CTA has passed the
    // next barrier, so this one stays whole until all have read it
    cl.sync();
    prefetch(q + 2);
    ++q;
    return out;
  };
  auto coef = [&](int j, bool back) {
    MarchCoef c{};
    if (!act || j < 1 || j > crows) return c;
    const size_t o = IXD(a.ldc, i, j);
    c.ax = __ldg(a.ax + o), c.ay = __ldg(a.ay + o), c.bb = __ldg(a.bb + o);
    c.cx = __ldg(a.cx + o), c.cy = __ldg(a.cy + o);
    if (!back) {
      c.f = __ldg(a.f + IXD(a.ldf, i, j));
      if (!per && (tid == 0 || tid == m2 - 1))
        c.e = a.x[IXD(a.ldx, tid == 0 ? 1 : m2 + 2, j + 2)];
    } else if (lead) {
      c.e = a.x[IXD(a.ldx, i + 1, j + 2)];
    }
    return c;
  };
  // the five-point terms of a row, in march_val's and resid_val's order
  auto terms = [&](const MarchCoef &c, double f, double w, double s, double m, double e) {
    double t = sub(f, mul((double)c.ax, w));
    t = sub(t, mul((double)c.ay, s));
    t = sub(t, mul((double)c.bb, m));
    return sub(t, mul((double)c.cx, e));
  };
  // a value into a row in shared memory, with the row's ghost cells: periodic
  // copies, or gh (the cell next to the first and last column)
  auto put = [&](double *row, double v, double gh) {
    if (!act) return;
    row[i] = v;
    if (tid == m2 - 1) row[per ? 0 : m2 + 1] = per ? v : gh;
    if (tid == 0) row[per ? m2 + 1 : 0] = per ? v : gh;
  };
  auto xval = [&](int j) { return act ? a.x[IXD(a.ldx, i + 1, j)] : 0.0; };
  auto xghost = [&](int j) {
    return (!per && act && (tid == 0 || tid == m2 - 1))
               ? a.x[IXD(a.ldx, tid == 0 ? 1 : m2 + 2, j)]
               : 0.0;
  };
  double *S = rows, *C = rows + ld, *N = rows + 2 * ld;
  auto rotate = [&]() {
    double *t = S;
    S = C, C = N, N = t;
  };

  // ---- forward sweep
  put(S, xval(1), xghost(1));
  put(C, xval(2), xghost(2));
  MarchCoef p0 = coef(1, false), p1 = coef(2, false);
  int js = 1;
  double north = 0.0;
  __syncthreads();
  for (int nb = 1; nb <= nblk; ++nb) {
    const int ie = a.ie[nb - 1], jf = ie - 2;
    // the row above the block: its guess row above, or the north boundary
    north = xval(ie + 1);
    const double north_gh = xghost(ie + 1);
    if (act) G[(size_t)(nb - 1) * m2 + tid] = C[i];
    for (int j = js; j <= jf; ++j) {
      const MarchCoef c = p0;
      p0 = p1;
      p1 = coef(j + 2, false);
      if (act) {
        const double v = dvd(terms(c, (double)c.f, C[i - 1], S[i], C[i], C[i + 1]), (double)c.cy);
        put(N, v, c.e);
        if (lead) a.x[IXD(a.ldx, i + 1, j + 2)] = v;
      }
      __syncthreads();
      rotate();
    }
    if (act) {
      SA[(size_t)(nb - 1) * m2 + tid] = S[i];
      D0[(size_t)(nb - 1) * m2 + tid] = C[i];
    }
    if (nb != nblk) {
      const MarchCoef c = p0;
      p0 = p1;
      p1 = coef(ie + 1, false);
      if (act) {
        const double t = terms(c, (double)c.f, C[i - 1], S[i], C[i], C[i + 1]);
        vin[tid] = sub(t, mul((double)c.cy, north));
      }
      const double *o = matvec();
      if (act) {
        const double d = C[i];
        if (lead) a.dum0[IXD(m2, i, nb)] = d;
        put(N, sub(d, o[tid]), 0.0);  // the corrected row: the next block's south row
        put(S, north, north_gh);      // its guess row
      }
      double *t = S;  // (S, C, N) = (corrected, guess, free)
      S = N, N = C, C = t;
      __syncthreads();
    }
    js = ie;
  }
  // ---- backward sweep
  MarchCoef rc = coef(last - 1, false);
  double res = 0.0;
  const double *o = nullptr;
  for (int nb = nblk; nb >= 1; --nb) {
    const int ie = a.ie[nb - 1], jf = ie - 2;
    js = nb != 1 ? a.ie[nb - 2] : 1;
    const double *d0 = D0 + (size_t)(nb - 1) * m2;
    if (lead)
      for (int j = js; j <= ie; ++j)
        for (int k = 1 + tid; k <= a.hzero; k += nt) a.h[IXD(a.ldh, k, j)] = 0.0;
    if (act) {
      double w, e;
      if (per) {
        w = d0[tid > 0 ? tid - 1 : m2 - 1];
        e = d0[tid < m2 - 1 ? tid + 1 : 0];
      } else {
        w = tid > 0 ? d0[tid - 1] : a.x[IXD(a.ldx, 1, ie)];
        e = tid < m2 - 1 ? d0[tid + 1] : a.x[IXD(a.ldx, m2 + 2, ie)];
      }
      const double t = terms(rc, (double)rc.f, w, SA[(size_t)(nb - 1) * m2 + tid], d0[tid], e);
      res = sub(t, mul((double)rc.cy, north));
      vin[tid] = res;
    }
    const float cy_s = nb != 1 && act ? __ldg(a.cy + IXD(a.ldc, i, js - 1)) : 0.f;
    p0 = coef(js, true), p1 = coef(js + 1, true);
    o = matvec();
    const double v = act ? o[tid] : 0.0;
    if (act) {
      north = add(G[(size_t)(nb - 1) * m2 + tid], v);
      put(C, v, 0.0);
      S[i] = 0.0;
      if (lead) {
        a.h[IXD(a.ldh, i + 1, js + 1)] = v;
        a.x[IXD(a.ldx, i + 1, js + 1)] = north;
        if (per && tid == m2 - 1) a.h[IXD(a.ldh, 1, js + 1)] = v;
        if (per && tid == 0) a.h[IXD(a.ldh, a.gi0, js + 1)] = v;
      }
    }
    if (nb != 1) {
      if (act) vin[tid] = mul(v, (double)cy_s);
      o = matvec();
      if (act) {
        const double hv = o[tid];
        S[i] = hv;
        if (lead) {
          a.h[IXD(a.ldh, i + 1, js)] = hv;
          if (per && tid == m2 - 1) a.h[IXD(a.ldh, 1, js)] = hv;
          if (per && tid == 0) a.h[IXD(a.ldh, a.gi0, js)] = hv;
        }
      }
      rc = coef(js - 1, false);
    }
    __syncthreads();
    for (int j = js; j <= jf; ++j) {
      const MarchCoef c = p0;
      p0 = p1;
      p1 = coef(j + 2, true);
      if (act) {
        const double hv = dvd(terms(c, 0.0, C[i - 1], S[i], C[i], C[i + 1]), (double)c.cy);
        put(N, hv, 0.0);
        if (lead) {
          a.h[IXD(a.ldh, i + 1, j + 2)] = hv;
          a.x[IXD(a.ldx, i + 1, j + 2)] = add(c.e, hv);
          if (per && j < jf) {
            if (tid == m2 - 1) a.h[IXD(a.ldh, 1, j + 2)] = hv;
            if (tid == 0) a.h[IXD(a.ldh, a.gi0, j + 2)] = hv;
          }
        }
      }
      __syncthreads();
      rotate();
    }
  }
  if (lead) {
    if (act) a.dum1[tid] = res, a.dum2[tid] = o[tid];
    __syncthreads();
    if (per)
      for (int j = 2 + tid; j <= last; j += nt) {
        a.x[IXD(a.ldx, 1, j)] = a.x[IXD(a.ldx, a.gi0 - 1, j)];
        a.x[IXD(a.ldx, a.gi0, j)] = a.x[IXD(a.ldx, 2, j)];
      }
  }
}

// ---------------------------------------------------------------- PRE
// One CTA per unit response NG of block nb.  Its H slice has leading
// dimension ldh and holds padded rows jl .. jhp (local row = row - jl).
__device__ __forceinline__ double lhs4(const PreArgs &p, const double *H, int i, int j, int jl) {
  const int ld = p.ldh;
  double t = mul(c64(p.ax, p.ldc, i, j), H[IXD(ld, i, j + 1 - jl + 1)]);
  t = add(t, mul(c64(p.ay, p.ldc, i, j), H[IXD(ld, i + 1, j - jl + 1)]));
  t = add(t, mul(c64(p.bb, p.ldc, i, j), H[IXD(ld, i + 1, j + 1 - jl + 1)]));
  t = add(t, mul(c64(p.cx, p.ldc, i, j), H[IXD(ld, i + 2, j + 1 - jl + 1)]));
  return t;
}

__device__ __forceinline__ void ghost_local(double *H, int ld, int gi0, int row_local) {
  if (threadIdx.x == 0) {
    H[IXD(ld, 1, row_local)] = H[IXD(ld, gi0 - 1, row_local)];
    H[IXD(ld, gi0, row_local)] = H[IXD(ld, 2, row_local)];
  }
}

__global__ void __launch_bounds__(256) k_pre_units(PreArgs p, int nb, int jl) {
  const int ng = blockIdx.x + 1;
  const int m2 = p.m2;
  const size_t msz = (size_t)m2 * m2;
  const int jh = p.ie[nb - 1], jhp = jh + 1, jhm = jh - 2, jg = jl + 1, ig = ng + 1;
  const int rows = jhp - jl + 1;
  double *H = p.hwork + (size_t)blockIdx.x * p.ldh * rows;  // local rows 1..rows
  const int tid = threadIdx.x, nt = blockDim.x;
  double *R = p.rinv + (size_t)(nb - 1) * msz;
  double *Rs = p.rinv + (size_t)(p.nblk - 1) * msz;
  // local row index of padded row r is r - jl + 1
#define LR(r) ((r) - jl + 1)
  for (int e = tid; e < p.hzero * rows; e += nt) H[e % p.hzero + (size_t)(e / p.hzero) * p.ldh] = 0.0;
  __syncthreads();
  if (tid == 0) H[IXD(p.ldh, ig, LR(jg))] = 1.0;
  __syncthreads();
  if (p.periodic) ghost_local(H, p.ldh, p.gi0, LR(jg));
  __syncthreads();
  if (nb != 1) {
    const double *R1p = p.rinv1 + (size_t)(nb - 2) * msz;
    const double cyv = c64(p.cy, p.ldc, ig - 1, jg - 2);
    for (int n = 1 + tid; n <= m2; n += nt) H[IXD(p.ldh, n + 1, LR(jl))] = mul(R1p[IXD(m2, ng, n)], cyv);
    __syncthreads();
  }
  for (int j = jl; j <= jhm; ++j) {
    if (p.periodic) ghost_local(H, p.ldh, p.gi0, LR(j + 1));
    __syncthreads();
    for (int i = 1 + tid; i <= m2; i += nt) {
      double t = lhs4(p, H, i, j, jl);
      H[IXD(p.ldh, i + 1, LR(j + 2))] = -dvd(t, c64(p.cy, p.ldc, i, j));
    }
    __syncthreads();
  }
  int j = jh - 1;
  if (p.periodic) ghost_local(H, p.ldh, p.gi0, LR(j + 1));
  __syncthreads();
  for (int i = 1 + tid; i <= m2; i += nt) R[IXD(m2, ng, i)] = lhs4(p, H, i, j, jl);
  if (nb != p.nblk) {
    j = p.ie[nb - 1];
    for (int n = 1 + tid; n <= m2; n += nt) Rs[IXD(m2, ng, n)] = H[IXD(p.ldh, n + 1, LR(j))];
    __syncthreads();
    if (p.periodic && tid == 0) {
      H[IXD(p.ldh, 1, LR(jg))] = 0.0;
      H[IXD(p.ldh, p.gi0, LR(jg))] = 0.0;
    }
  }
  __syncthreads();
  if (tid == 0) H[IXD(p.ldh, ig, LR(jg))] = 0.0;
#undef LR
}

// RINV1(I,J) = -sum_K RINV(I,K) * S(K,J), serial in K (P/prep_GLOBAL.f90:379-383)
__global__ void k_rinv1_gemm(const double *R, const double *S, double *R1, int m2) {
  const int i = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int j = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > m2 || j > m2) return;
  double s = 0.0;
  for (int k = 1; k <= m2; ++k) s = sub(s, mul(R[IXD(m2, i, k)], S[IXD(m2, k, j)]));
  R1[IXD(m2, i, j)] = s;
}

// ------------------------------------------------------------- MATINV
// Small matrices: whole inverse in one CTA.
__global__ void __launch_bounds__(1024) k_matinv_cta(double *B, int n, double *b1, double *b2,
                                                   int *bad) {
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i = 1; i <= n - 1; ++i) {
    const double piv = B[IXD(n, i, i)];
    if (tid == 0 && piv == 0.0) *bad = 1;
    const double r = dvd(1.0, piv);
    __syncthreads();
    if (tid == 0) B[IXD(n, i, i)] = 1.0;
    __syncthreads();
    for (int j = 1 + tid; j <= n; j += nt) B[IXD(n, i, j)] = mul(B[IXD(n, i, j)], r);
    for (int ia = i + 1 + tid; ia <= n; ia += nt) b1[ia] = B[IXD(n, ia, i)];
    __syncthreads();
    for (int ia = i + 1 + tid; ia <= n; ia += nt) B[IXD(n, ia, i)] = 0.0;
    for (int j = 1 + tid; j <= n; j += nt) b2[j] = B[IXD(n, i, j)];
    __syncthreads();
    const int rows = n - i;
    for (int e = tid; e < rows * n; e += nt) {
      const int ia = i + 1 + e % rows, j = 1 + e / rows;
      B[IXD(n, ia, j)] = sub(B[IXD(n, ia, j)], mul(b1[ia], b2[j]));
    }
    __syncthreads();
  }
  {
    const double piv = B[IXD(n, n, n)];
    if (tid == 0 && piv == 0.0) *bad = 1;
    const double r = dvd(1.0, piv);
    __syncthreads();
    if (tid == 0) B[IXD(n, n, n)] = 1.0;
    __syncthreads();
    for (int j = 1 + tid; j <= n; j += nt) B[IXD(n, n, j)] = mul(B[IXD(n, n, j)], r);
    __syncthreads();
  }
  for (int i = 2; i <= n; ++i) {
    for (int ib = 1 + tid; ib <= i; ib += nt) b1[ib] = B[IXD(n, ib, i)];
    __syncthreads();
    for (int ib = 1 + tid; ib <= i - 1; ib += nt) B[IXD(n, ib, i)] = 0.0;
    for (int j = 1 + tid; j <= n; j += nt) b2[j] = B[IXD(n, i, j)];
    __syncthreads();
    const int rows = i - 1;
    for (int e = tid; e < rows * n; e += nt) {
      const int ib = 1 + e % rows, j = 1 + e / rows;
      B[IXD(n, ib, j)] = sub(B[IXD(n, ib, j)], mul(b1[ib], b2[j]));
    }
    __syncthreads();
  }
}

// Large matrices: one launch per elimination step.
__global__ void k_mi_pivot_row(double *B, int n, int i, double *b1, double *b2, int *bad) {
  // row i scaled by 1/B(i,i) with B(i,i) first set to 1; column below saved
  const double piv = B[IXD(n, i, i)];
  const double r = dvd(1.0, piv);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (piv == 0.0) *bad = 1;
    B[IXD(n, i, i)] = 1.0;
  }
  __syncthreads();
  for (int j = 1 + threadIdx.x; j <= n; j += blockDim.x) {
    double v = mul(B[IXD(n, i, j)], r);
    B[IXD(n, i, j)] = v;
    b2[j] = v;
  }
  for (int ia = i + 1 + threadIdx.x; ia <= n; ia += blockDim.x) {
    b1[ia] = B[IXD(n, ia, i)];
    B[IXD(n, ia, i)] = 0.0;
  }
}
__global__ void k_mi_update(double *B, int n, int r0, int r1, const double *b1, const double *b2) {
  const int rows = r1 - r0 + 1;
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (size_t)rows * n) return;
  const int ia = r0 + (int)(e % rows), j = 1 + (int)(e / rows);
  B[IXD(n, ia, j)] = sub(B[IXD(n, ia, j)], mul(b1[ia], b2[j]));
}
__global__ void k_mi_back_prep(double *B, int n, int i, double *b1, double *b2) {
  for (int ib = 1 + threadIdx.x; ib <= i; ib += blockDim.x) b1[ib] = B[IXD(n, ib, i)];
  __syncthreads();
  for (int ib = 1 + threadIdx.x; ib <= i - 1; ib += blockDim.x) B[IXD(n, ib, i)] = 0.0;
  for (int j = 1 + threadIdx.x; j <= n; j += blockDim.x) b2[j] = B[IXD(n, i, j)];
}

// ------------------------------------------------------- strip copies
// Extracts the wrapped last BIR strip (M/fs_GLOBAL.f90:1924-1944) or a plain
// strip source (:1910-1915).  mode 0: SRC only; mode 1: SRC, CL..CT, XX sides.
__global__ void k_strip_extract(StripArgs s, int il, int mode) {
  const int ibir = s.ibir, inc = ibir / 2, i2 = s.i2, i0 = i2 + 2;
  const int ir = il + inc, ir2 = il + ibir - 1;
  const size_t total = (size_t)ibir * s.j2;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const int ii = 1 + (int)(e % ibir), j = 1 + (int)(e / ibir);
    if (mode == 0) {
      s.src[IXD(ibir, ii, j)] = s.s[IXD(i2, il + ii - 1, j)];
      continue;
    }
    const int i = il + ii - 1;
    const int is = (i <= ir - 1) ? i : i - ir + 1;
    if (s.s) s.src[IXD(ibir, ii, j)] = s.s[IXD(i2, is, j)];
    s.cl[IXD(ibir, ii, j)] = s.al[IXD(i2, is, j)];
    s.cr[IXD(ibir, ii, j)] = s.ar[IXD(i2, is, j)];
    s.cb[IXD(ibir, ii, j)] = s.ab[IXD(i2, is, j)];
    s.ct[IXD(ibir, ii, j)] = s.at[IXD(i2, is, j)];
    s.cc[IXD(ibir, ii, j)] = s.ac[IXD(i2, is, j)];
    if (ii == 1 && s.x) {
      s.xx[IXD(ibir + 2, 1, j)] = s.x[IXD(i0, il, j)];
      s.xx[IXD(ibir + 2, ibir + 2, j)] = s.x[IXD(i0, inc + 2, j)];
    }
    (void)ir2;
  }
  if (mode == 1 && s.x && blockIdx.x == 0 && threadIdx.x == 0)
    for (int j = s.j2 + 1; j <= s.side_rows; ++j) {
      s.xx[IXD(ibir + 2, 1, j)] = s.x[IXD(i0, il, j)];
      s.xx[IXD(ibir + 2, ibir + 2, j)] = s.x[IXD(i0, inc + 2, j)];
    }
}

// Copies the solved wrapped strip back (M/fs_GLOBAL.f90:1947-1962).
__global__ void k_strip_scatter(StripArgs s, int il, int periodic) {
  const int ibir = s.ibir, inc = ibir / 2, i2 = s.i2, i0 = i2 + 2, j1 = s.j2 + 1;
  const int ir = il + inc, ir2 = il + ibir - 1;
  const size_t total = (size_t)ibir * (j1 - 1);
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const int i = il + (int)(e % ibir), j = 2 + (int)(e / ibir);
    if (i <= ir - 1)
      s.x[IXD(i0, i + 1, j)] = s.xx[IXD(ibir + 2, i - il + 2, j)];
    else if (i <= ir2)
      s.x[IXD(i0, i - ir + 2, j)] = s.xx[IXD(ibir + 2, i - il + 2, j)];
  }
}
__global__ void k_periodic_cols(double *x, int i2, int j2) {
  const int i0 = i2 + 2;
  for (int j = 2 + blockIdx.x * blockDim.x + threadIdx.x; j <= j2 + 1; j += gridDim.x * blockDim.x) {
    x[IXD(i0, 1, j)] = x[IXD(i0, i2 + 1, j)];
    x[IXD(i0, i0, j)] = x[IXD(i0, 2, j)];
  }
}

// ------------------------------------------------------------ host side
// Whether the current device can hold the marching cluster (a device may
// have fewer SMs free in one cluster than it takes).  The shared-memory
// opt-in and the answer belong to the device; the last shape is kept.
static int march_cluster_fits(size_t smem, int threads, bool &fits) {
  struct Fit {
    size_t smem = 0;
    int threads = 0;
    bool fits = false;
  };
  static std::mutex mu;
  static std::map<int, Fit> by_device;
  int dev = 0;
  SEVP_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  Fit &f = by_device[dev];
  if (f.threads == 0)
    SEVP_CUDA_TRY(cudaFuncSetAttribute(
        k_march_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
  if (f.threads != threads || f.smem != smem) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kMarchCtas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    int n = 0;
    SEVP_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, k_march_cluster, &cfg));
    f.smem = smem, f.threads = threads, f.fits = n > 0;
  }
  fits = f.fits;
  return SEVP_OK;
}

int dev_march_solve(const MarchArgs &a, cudaStream_t st) {
  // the cluster where a column has a thread, the blocks' rows fit its shared
  // memory, and H's zeroed columns cover the ghosts (the reference's shapes)
  const int nper = ceil_div(a.m2, kMarchCtas);
  const size_t smem = march_smem_doubles(a.m2, a.nblk, nper) * sizeof(double);
  if (a.m2 >= 2 && a.m2 <= kMarchMaxCols && a.hzero >= a.m2 + 2 &&
      (!a.periodic || a.gi0 == a.m2 + 2) && smem <= (size_t)220 * 1024) {
    const int threads = ceil_div(a.m2, 32) * 32;
    bool fits = false;
    const int s = march_cluster_fits(smem, threads, fits);
    if (s) return s;
    if (fits) {
      k_march_cluster<<<kMarchCtas, threads, smem, st>>>(a, nper);
      SEVP_CUDA_TRY(cudaGetLastError());
      return SEVP_OK;
    }
  }
  int threads = std::min(1024, std::max(32, ((a.m2 + 31) / 32) * 32));
  k_march_solve<<<1, threads, 0, st>>>(a);
  SEVP_CUDA_TRY(cudaGetLastError());
  return SEVP_OK;
}

int dev_matinv(double *B, int n, double *b1, double *b2, int *bad, cudaStream_t st) {
  if (n <= 320) {
    k_matinv_cta<<<1, 1024, 0, st>>>(B, n, b1, b2, bad);
    SEVP_CUDA_TRY(cudaGetLastError());
    return SEVP_OK;
  }
  const int T = 256;
  for (int i = 1; i <= n - 1; ++i) {
    k_mi_pivot_row<<<1, 1024, 0, st>>>(B, n, i, b1, b2, bad);
    size_t e = (size_t)(n - i) * n;
    k_mi_update<<<(unsigned)((e + T - 1) / T), T, 0, st>>>(B, n, i + 1, n, b1, b2);
  }
  k_mi_pivot_row<<<1, 1024, 0, st>>>(B, n, n, b1, b2, bad);
  for (int i = 2; i <= n; ++i) {
    k_mi_back_prep<<<1, 1024, 0, st>>>(B, n, i, b1, b2);
    size_t e = (size_t)(i - 1) * n;
    k_mi_update<<<(unsigned)((e + T - 1) / T), T, 0, st>>>(B, n, 1, i - 1, b1, b2);
  }
  SEVP_CUDA_TRY(cudaGetLastError());
  return SEVP_OK;
}

// PRE1 / PRE: blocks in sequence; per block all unit responses in parallel,
// then MATINV and the RINV1 product.  hfinal (ldh x J0) receives the H rows
// the reference leaves behind (the last unit response of each block).
int dev_pre(const PreArgs &p, double *hfinal, int *bad, cudaStream_t st) {
  const int m2 = p.m2;
  const size_t msz = (size_t)m2 * m2;
  int jl = 1;
  for (int nb = 1; nb <= p.nblk; ++nb) {
    const int jh = p.ie_host[nb - 1];
    const int rows = jh + 1 - jl + 1;
    k_pre_units<<<m2, 256, 0, st>>>(p, nb, jl);
    SEVP_CUDA_TRY(cudaGetLastError());
    if (hfinal) {
      // last unit response's rows jl .. jh+1
      const double *src = p.hwork + (size_t)(m2 - 1) * p.ldh * rows;
      SEVP_CUDA_TRY(cudaMemcpyAsync(hfinal + (size_t)(jl - 1) * p.ldh, src,
                                    sizeof(double) * p.ldh * rows, cudaMemcpyDeviceToDevice, st));
    }
    int s = dev_matinv(p.rinv + (size_t)(nb - 1) * msz, m2, p.b1, p.b2, bad, st);
    if (s) return s;
    if (nb == p.nblk) break;
    dim3 blk(16, 16), grd((m2 + 15) / 16, (m2 + 15) / 16);
    k_rinv1_gemm<<<grd, blk, 0, st>>>(p.rinv + (size_t)(nb - 1) * msz,
                                      p.rinv + (size_t)(p.nblk - 1) * msz,
                                      p.rinv1 + (size_t)(nb - 1) * msz, m2);
    SEVP_CUDA_TRY(cudaGetLastError());
    jl = jh;
  }
  return SEVP_OK;
}

int dev_strip_extract(const StripArgs &s, int il, int mode, cudaStream_t st) {
  k_strip_extract<<<128, 256, 0, st>>>(s, il, mode);
  SEVP_CUDA_TRY(cudaGetLastError());
  return SEVP_OK;
}
int dev_strip_scatter(const StripArgs &s, int il, int periodic, cudaStream_t st) {
  k_strip_scatter<<<128, 256, 0, st>>>(s, il, periodic);
  if (periodic) k_periodic_cols<<<8, 128, 0, st>>>(s.x, s.i2, s.j2);
  SEVP_CUDA_TRY(cudaGetLastError());
  return SEVP_OK;
}

}  // namespace sevp
