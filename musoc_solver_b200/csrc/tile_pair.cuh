// Block-Jacobi tile pass with two columns per lane: r -= alpha q (UPDATE),
// z = M^-1 r by tile SEVP, r.z and r.r and the finish of the PCG iteration
// (DOTS).  Symmetric operator (three planes), FP64 influence data, tiles of
// at most HM rows; the pass of k_tile_apply / k_tile_short in solver.cu with
// the same sub-blocks and influence matrices.
//
// What bounds it: the tile pass moves 28 B (FP32 vectors) or 44 B (FP64) per
// point plus the influence data (24.5 B per point at 3600 x 2400 with 16 x 6
// tiles).  With one column per lane it was bound by issue and by a task's
// latency (two memory round trips and 2 x HM dependent rows).  Here:
//   - a warp covers 64 columns (two of the tiling's warp groups), lane l of a
//     tile holding columns 2 l and 2 l + 1: half the shuffles, address
//     arithmetic and loads per point, two independent row chains per lane
//     (49 -> 31 M warp instructions per pass);
//   - the next task's rows are copied to a shared-memory stage of the warp
//     while it marches this one (cp.async; 16-byte copies past L1 where the
//     grid allows, since smaller ones allocate L1 lines), and the influence
//     matrices through one slot per lane, each copied as soon as the one
//     before it has been read;
//   - the west/east couplings across a tile edge are zeroed in the
//     coefficients, and the neighbour shuffles are confined to the tile's
//     lanes (shuffle width), so no select sits on the row recurrence;
//   - full tiles (the tiling's width, HM rows, one sub-block) run straight
//     code; the others run rolled loops on the staged rows, and come first in
//     the task order, so that they spread over the warps (131 -> 103 us);
//   - the backward sweep marches the rows again from the guess row the
//     influence matrix gives (z_{k+1} from r_k, z_{k-1}, z_k) instead of
//     marching a homogeneous correction and adding it to stored rows: the
//     same error (that of the guess row times the growth), no stored rows.
//     FP64 quotients are rounded as a division's (march_quot).  Error of z in
//     FP64 against refined dense solves of up to 6000 tiles, as a part of the
//     one-column pass's (geometric mean over the tiles; rms): 16 x 6 tiles of
//     1440 x 720 0.99; 0.98, 16 x 16 of 1203 x 601 0.99; 0.94, 32 x 8, 8 x 8
//     and 16 x 4 of 600 x 300 1.01; 1.05, 1.02; 1.04 and 1.00; 0.96.
// Two CTAs of four warps per SM: three spill, and the loads in flight already
// fill the memory (one SM's warps move 6.2 TB/s / 148 between their first and
// last task; the slowest SM ends 18 % after the median one, and handing out
// the last tasks from a counter cost more in their sums than it gained).
// Measured at 3600 x 2400, 16 x 6 tiles, one B200: FP32 138 -> 101 us (481 MB,
// 4.8 TB/s), FP64 179 -> 128 us; 1440 x 720 FP64 35.6 -> 28.3 us (of which
// the rounded quotients 1 us and 0.5 us).
#pragma once
#include "solver_core.cuh"

namespace sevp {

constexpr int kPairWarps = 4;  // warps per CTA (at most)

template <typename V>
struct Vec2;
template <>
struct Vec2<float> {
  using T = float2;
};
template <>
struct Vec2<double> {
  using T = double2;
};

template <int BYTES>
__device__ __forceinline__ void cp_async(unsigned dst, const void *src) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
  else if constexpr (BYTES == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Copies two neighbouring points into the lane's stage slot: one copy (the
// pair is 2 sizeof(V) aligned), or one per column (d1 is the second one's
// offset from the first, 0 when it is outside the tile).
template <typename V>
__device__ __forceinline__ void fetch_pair(unsigned dst, const V *p, size_t id, long long d1,
                                           bool vec) {
  if (vec) {
    cp_async<2 * sizeof(V)>(dst, p + id);
  } else {
    cp_async<sizeof(V)>(dst, p + id);
    cp_async<sizeof(V)>(dst + (unsigned)sizeof(V), p + id + d1);
  }
}
template <typename V>
__device__ __forceinline__ void stage_pair(const unsigned char *st, bool c0, bool c1, V &a, V &b) {
  const typename Vec2<V>::T t = *reinterpret_cast<const typename Vec2<V>::T *>(st);
  a = c0 ? t.x : V(0);
  b = c1 ? t.y : V(0);
}
template <typename V>
__device__ __forceinline__ void store_pair(V *p, size_t id, long long d1, bool vec, bool c0,
                                           bool c1, V a, V b) {
  if (vec) {
    if (c0) *reinterpret_cast<typename Vec2<V>::T *>(p + id) = typename Vec2<V>::T{a, b};
  } else {
    if (c0) p[id] = a;
    if (c1) p[id + d1] = b;
  }
}

// Shared memory of one warp, in bytes: the staged rows (r, q, three planes),
// one influence matrix per tile, the sub-blocks' residuals and entry rows of
// the general path, and the mat-vec inputs.
template <typename V, int W, int HM>
__host__ __device__ constexpr size_t pair_rows_bytes() {
  return (size_t)HM * 64 * (2 * sizeof(V) + 3 * sizeof(float));
}
template <typename V, int W, int HM>
__host__ __device__ constexpr size_t pair_smem_per_warp(int nbmax) {
  return pair_rows_bytes<V, W, HM>() + (size_t)W * 512 + (size_t)nbmax * 1024 +
         (size_t)(64 / W) * (W + 2) * 8;
}

// W: lane segment width of the tiling (8, 16 or 32 columns).
template <typename V, int W, int HM, bool UPDATE, bool DOTS>
__global__ void __launch_bounds__(kPairWarps * 32, 2)
    k_tile_pair(TileGeom tg, const float *__restrict__ ac, const float *__restrict__ ar,
                const float *__restrict__ at, const double *__restrict__ mats, V *r, const V *q,
                V *z, SolveState *st, double *partials, unsigned *ticket, int vec_ok) {
  pdl_trigger();
  constexpr int LPT = W / 2;   // lanes per tile
  constexpr int TPW = 64 / W;  // tiles per warp
  constexpr int DVS = W + 2;   // doubles between the tiles' mat-vec inputs (bank shift)
  constexpr unsigned kV = 64 * sizeof(V), kF = 64 * sizeof(float);  // a staged row
  constexpr bool kReg = HM <= kPairRegRows;  // full tiles in registers
  extern __shared__ __align__(16) unsigned char psm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  unsigned char *base = psm + pair_smem_per_warp<V, W, HM>(tg.nbmax) * wib;
  // the lane's own slots: rows r, q, AC, AR, AT; matrix; rho and zin
  const unsigned char *sr = base + lane * 2 * sizeof(V), *sq = sr + HM * kV;
  const unsigned char *sc = base + 2 * HM * kV + lane * 8, *se = sc + HM * kF, *sn = se + HM * kF;
  const unsigned ur = (unsigned)__cvta_generic_to_shared(sr),
                 uc = (unsigned)__cvta_generic_to_shared(sc);
  const double2 *stg =
      reinterpret_cast<const double2 *>(base + pair_rows_bytes<V, W, HM>()) + lane;
  const unsigned um = (unsigned)__cvta_generic_to_shared(stg);
  double2 *rho = reinterpret_cast<double2 *>(base + pair_rows_bytes<V, W, HM>() + W * 512) + lane;
  double2 *zin = rho + (size_t)tg.nbmax * 32;
  const int half = lane >> 4, seg = lane / LPT, n = 2 * (lane % LPT);
  double *dv = reinterpret_cast<double *>(base + pair_rows_bytes<V, W, HM>() + W * 512 +
                                          (size_t)tg.nbmax * 1024) +
               seg * DVS;
  double2 *dv2 = reinterpret_cast<double2 *>(dv + n);
  const bool vec = vec_ok != 0, quad = vec_ok == 2;
  // FP32 rows as 16-byte copies past L1 (a half warp per row): the 8-byte
  // copies allocate L1 lines, of which too few are left beside the stages
  constexpr bool kQuadV = sizeof(V) == 4;
  const unsigned uq = (unsigned)__cvta_generic_to_shared(base) + (lane >> 4) * kF +
                      (lane & 15) * 16;
  const int nx = tg.nx;
  const int ntasks = tg.ty * pair_cols(tg);
  const int nw = blockDim.x >> 5, stride = gridDim.x * nw;
  double acc_rz = 0.0, acc_rr = 0.0;

  // a task's columns in this lane (tile a = g2 TPW + seg of tile row b)
  struct Geo {
    int b, g2, mw, nb, hh;
    bool c0, c1;
    long long d1, moff;
    size_t id0;
  };
  auto locate = [&](Geo &g, int2 t) {
    g.b = t.x, g.g2 = t.y;
    const int a = g.g2 * TPW + seg, grp = 2 * g.g2 + half;
    g.mw = (a < tg.tx) ? tile_width(tg, a) : 0;
    g.nb = grp < tg.txg ? __ldg(tg.grp_nb + (size_t)g.b * tg.txg + grp) : 1;
    g.moff = g.mw > 0 ? __ldg(tg.moff + (size_t)g.b * tg.tx + a) : 0;
  };
  auto geo = [&](Geo &g) {
    const int a = g.g2 * TPW + seg;
    g.c0 = n < g.mw, g.c1 = n + 1 < g.mw;
    g.hh = tile_height(tg, g.b);
    const int i0 = tile_col(tg, a, n);
    g.d1 = g.c1 ? tile_col(tg, a, n + 1) - i0 : 0;
    g.id0 = (size_t)g.b * tg.th * nx + i0;
  };
  // The copies take no predicate (a branch each, otherwise): lanes and rows
  // outside the tile copy a clamped place of the grid, and stage_pair masks
  // what they brought.  VEC: the vectors r and q; else the three planes.
  auto fetch = [&](const Geo &g, auto is_vec) {
    constexpr bool VEC = decltype(is_vec)::value;
    if (quad && (!VEC || kQuadV)) {
      // a half warp per row, 16 bytes per lane
      const int col = min(g.g2 * 64 + (lane & 15) * 4, nx - 4);
      const size_t row0 = (size_t)g.b * tg.th * nx + col;
      constexpr unsigned kC = 2 * HM * kV;  // the planes follow r and q
#pragma unroll(kReg ? HM / 2 : 2)
      for (int k = 0; k < HM; k += 2) {
        if (!kReg && k >= g.hh) break;
        const size_t e = row0 + (size_t)((unsigned)min(k + (lane >> 4), g.hh - 1)) * (unsigned)nx;
        if constexpr (VEC) {
          if constexpr (kQuadV) {
            cp_async<16>(uq + k * kF, r + e);
            if (UPDATE) cp_async<16>(uq + (HM + k) * kF, q + e);
          }
        } else {
          cp_async<16>(uq + kC + k * kF, ac + e);
          cp_async<16>(uq + kC + (HM + k) * kF, ar + e);
          cp_async<16>(uq + kC + (2 * HM + k) * kF, at + e);
        }
      }
      return;
    }
#pragma unroll(kReg ? HM : 2)
    for (int k = 0; k < HM; ++k) {
      if (!kReg && k >= g.hh) break;
      const size_t id = g.id0 + (size_t)((unsigned)min(k, g.hh - 1)) * (unsigned)nx;
      if constexpr (VEC) {
        fetch_pair<V>(ur + k * kV, r, id, g.d1, vec);
        if (UPDATE) fetch_pair<V>(ur + (HM + k) * kV, q, id, g.d1, vec);
      } else {
        fetch_pair<float>(uc + k * kF, ac, id, g.d1, vec);
        fetch_pair<float>(uc + (HM + k) * kF, ar, id, g.d1, vec);
        fetch_pair<float>(uc + (2 * HM + k) * kF, at, id, g.d1, vec);
      }
    }
  };
  auto fetch_planes = [&](const Geo &g) { fetch(g, std::false_type{}); };
  auto fetch_vectors = [&](const Geo &g) { fetch(g, std::true_type{}); };
  // the lane's two columns of a matrix M (mw x mw)
  auto fetch_mat = [&](const double *M, int mw, bool c0, bool c1) {
    if (mw == W) {
#pragma unroll
      for (int k = 0; k < W; ++k) cp_async<16>(um + k * 512, M + k * W + n);
    } else if ((mw & 1) == 0) {
      if (c0) {
        const double *p = M + n;
#pragma unroll 8
        for (int k = 0; k < mw; ++k, p += mw) cp_async<16>(um + k * 512, p);
      }
    } else {
      for (int k = 0; k < mw; ++k) {
        if (c0) cp_async<8>(um + k * 512, M + k * mw + n);
        if (c1) cp_async<8>(um + k * 512 + 8, M + k * mw + n + 1);
      }
    }
  };
  // first matrix a task reads: R1_0 when it has sub-blocks, else Sinv_0
  auto fetch_first = [&](const Geo &g) {
    if (g.c0)
      fetch_mat(mats + g.moff + (g.nb > 1 ? (size_t)g.nb * g.mw * g.mw : 0), g.mw, g.c0, g.c1);
  };
  // out(n) = sum_k dv[k] M[k][n] from the staged matrix
  auto matvec = [&](int mw, bool c0, bool c1, double &o0, double &o1) {
    double s0 = 0.0, s1 = 0.0;
    if (c0) {
      if (mw == W) {
#pragma unroll
        for (int k = 0; k < W; k += 2) {
          const double2 d = *reinterpret_cast<const double2 *>(dv + k);
          const double2 ma = stg[k * 32], mb = stg[(k + 1) * 32];
          s0 += d.x * ma.x;
          s1 += d.x * ma.y;
          s0 += d.y * mb.x;
          s1 += d.y * mb.y;
        }
      } else {
#pragma unroll 8
        for (int k = 0; k < mw; ++k) {
          const double2 mk = stg[k * 32];
          s0 += dv[k] * mk.x;
          s1 += dv[k] * mk.y;
        }
      }
    }
    o0 = s0, o1 = c1 ? s1 : 0.0;
  };

  // The warp's tasks are strided entries of the order.  Everything a task
  // needs is asked for one task ahead of its use, behind the march: its entry,
  // its sub-blocks and matrix offset, then its rows and first matrix.
  auto entry = [&](int p) { return p < ntasks ? __ldg(tg.pair_order + p) : make_int2(0, 0); };
  int pos = blockIdx.x * nw + wib;             // the staged task
  int2 task2 = entry(pos + 2 * stride);        // two tasks on
  Geo nxt{}, nx1{};                            // the staged task, the one after it
  if (pos < ntasks) {
    locate(nxt, entry(pos));
    if (pos + stride < ntasks) locate(nx1, entry(pos + stride));
    geo(nxt);
    // the planes and the influence data do not change during a solve
    fetch_planes(nxt);
    fetch_first(nxt);
  }
  pdl_wait();
  // a finished run's launches, and the start pass of a run that resumes, end
  // here (tested once the first copies are under way)
  const int done = st ? st->done || (!UPDATE && st->resumed) : 0;
  const V alpha = UPDATE ? (V)st->alpha : V(0);
  if (pos < ntasks) {
    fetch_vectors(nxt);
    cp_commit();
    cp_commit();
  }
  if (done) {
    cp_wait<0>();
    return;
  }
  for (; pos < ntasks; pos += stride) {
    const Geo cur = nxt;
    const int mw = cur.mw, nb = cur.nb, hh = cur.hh;
    const bool c0 = cur.c0, c1 = cur.c1, more = pos + stride < ntasks;
    const long long d1 = cur.d1;
    const size_t id0 = cur.id0;
    const double *mt = mats + cur.moff;

    const bool full =
        kReg && __all_sync(0xffffffffu, hh == HM && nb == 1 && (mw == W || mw == 0));
    // the task after this one enters the stage's rows, and the ones behind it
    // move up
    auto stage_next = [&]() {
      __syncwarp();
      if (more) {
        nxt = nx1;
        geo(nxt);
        fetch_planes(nxt);
        fetch_vectors(nxt);
      }
      cp_commit();
      if (pos + 2 * stride < ntasks) {
        locate(nx1, task2);
        task2 = entry(pos + 3 * stride);
      }
    };
    // the staged rows (16-byte row copies serve two lanes)
    cp_wait<1>();
    __syncwarp();
    bool ran = false;
    if constexpr (kReg) {
      if (full) {
        V r0[HM], r1[HM];
        float cc0[HM], cc1[HM], ce0[HM], ce1[HM], cn0[HM], cn1[HM], cw0[HM];
#pragma unroll
        for (int k = 0; k < HM; ++k) {
          stage_pair<V>(sr + k * kV, c0, c0, r0[k], r1[k]);
          if (UPDATE) {
            V q0, q1;
            stage_pair<V>(sq + k * kV, c0, c0, q0, q1);
            r0[k] = fma_rn(-alpha, q0, r0[k]);
            r1[k] = fma_rn(-alpha, q1, r1[k]);
          }
          stage_pair<float>(sc + k * kF, c0, c0, cc0[k], cc1[k]);
          stage_pair<float>(se + k * kF, c0, c0, ce0[k], ce1[k]);
          stage_pair<float>(sn + k * kF, c0, c0, cn0[k], cn1[k]);
        }
        stage_next();
        if (UPDATE) {
#pragma unroll
          for (int k = 0; k < HM; ++k)
            store_pair<V>(r, id0 + (size_t)k * nx, d1, vec, c0, c0, r0[k], r1[k]);
        }
        // couplings across the tile's edges are dropped; lanes without a tile
        // march zeros (their north coefficient is one)
#pragma unroll
        for (int k = 0; k < HM; ++k) {
          if (n + 2 >= W) ce1[k] = 0.f;
          if (!c0) cn0[k] = cn1[k] = 1.f;
          cw0[k] = __shfl_up_sync(0xffffffffu, ce1[k], 1, LPT);
          if (n == 0) cw0[k] = 0.f;
        }
        auto emit = [&](int k, double z0, double z1) {
          const V v0 = (V)z0, v1 = (V)z1;
          store_pair<V>(z, id0 + (size_t)k * nx, d1, vec, c0, c0, v0, v1);
          if (DOTS) {
            acc_rz += (double)r0[k] * (double)v0;
            acc_rz += (double)r1[k] * (double)v1;
          }
        };
        if (DOTS) {
#pragma unroll
          for (int k = 0; k < HM; ++k) {
            const double a0 = (double)r0[k], a1 = (double)r1[k];
            acc_rr += a0 * a0;
            acc_rr += a1 * a1;
          }
        }
        // row k's equation residual with the rows below (zb, zc): two of the
        // three neighbours before the centre, which has the other sign, so
        // that the partial sums stay as small as they do from west to east
        // (8 x 8 tiles of 600 x 300, FP64: error of z 1.06 times as large
        // with the centre ahead of both columns); the term that waits on the
        // neighbour shuffles last
        auto row = [&](int k, bool first, bool second, double zb0, double zb1, double zc0,
                       double zc1, double &q0, double &q1) {
          double p0 = (double)r0[k], p1 = (double)r1[k];
          if (!first) {
            const double zw = __shfl_up_sync(0xffffffffu, zc1, 1, LPT);
            const double ze = __shfl_down_sync(0xffffffffu, zc0, 1, LPT);
            if (!second) {
              p0 -= (double)cn0[k > 0 ? k - 1 : 0] * zb0;
              p1 -= (double)cn1[k > 0 ? k - 1 : 0] * zb1;
            }
            const double e0 = (double)ce0[k];
            p0 -= e0 * zc1;
            p1 -= e0 * zc0;
            p0 -= (double)cc0[k] * zc0;
            p1 -= (double)cc1[k] * zc1;
            p0 -= (double)cw0[k] * zw;
            p1 -= (double)ce1[k] * ze;
          }
          q0 = p0, q1 = p1;
        };
        double zb0 = 0.0, zb1 = 0.0, zc0 = 0.0, zc1 = 0.0, q0, q1;
#pragma unroll
        for (int k = 0; k < HM; ++k) {
          row(k, k == 0, k == 1, zb0, zb1, zc0, zc1, q0, q1);
          if (k < HM - 1) {
            zb0 = zc0, zb1 = zc1;
            zc0 = march_quot<V>(q0, (double)cn0[k], march_rcp((double)cn0[k]));
            zc1 = march_quot<V>(q1, (double)cn1[k], march_rcp((double)cn1[k]));
          }
        }
        __syncwarp();
        *dv2 = make_double2(q0, q1);
        __syncwarp();
        double v0, v1;
        cp_wait<1>();
        matvec(W, c0, c0, v0, v1);
        if (more) fetch_first(nxt);
        cp_commit();
        zb0 = 0.0, zb1 = 0.0, zc0 = v0, zc1 = v1;
        emit(0, zc0, zc1);
#pragma unroll
        for (int k = 0; k < HM - 1; ++k) {
          row(k, false, k == 0, zb0, zb1, zc0, zc1, q0, q1);
          zb0 = zc0, zb1 = zc1;
          zc0 = march_quot<V>(q0, (double)cn0[k], march_rcp((double)cn0[k]));
          zc1 = march_quot<V>(q1, (double)cn1[k], march_rcp((double)cn1[k]));
          emit(k + 1, zc0, zc1);
        }
        ran = true;
      }
    }
    if (!ran) {
      // ---- general path: sub-blocks (the two halves of the warp may have
      // different counts), short tiles, narrow last tiles.  Rolled loops on
      // the staged rows (unrolled, its code ran out of the instruction cache
      // and a task took six times a full one); the stage takes the next rows
      // at the end.  The matrix slot holds the next matrix the lane's tile
      // reads: R1_0 .. R1_{nb-2} in the forward sweep, then Sinv_{nb-1},
      // R1_{nb-2}, .., R1_0, Sinv_0.
      V *wr = reinterpret_cast<V *>(const_cast<unsigned char *>(sr));
      constexpr int kR = 64;  // values per staged row
      const size_t msz = (size_t)mw * mw;
#pragma unroll 2
      for (int k = 0; k < hh; ++k) {
        V a, bv;
        stage_pair<V>(sr + k * kV, c0, c1, a, bv);
        if (UPDATE) {
          V q0, q1;
          stage_pair<V>(sq + k * kV, c0, c1, q0, q1);
          a = fma_rn(-alpha, q0, a);
          bv = fma_rn(-alpha, q1, bv);
          store_pair<V>(r, id0 + (size_t)k * nx, d1, vec, c0, c1, a, bv);
        }
        wr[k * kR] = a, wr[k * kR + 1] = bv;
        if (DOTS) {
          acc_rr += (double)a * (double)a;
          acc_rr += (double)bv * (double)bv;
        }
      }
      // Row k's coefficients and right-hand side, converted, and its
      // reciprocals of AT.  Taken at the row's use: one row ahead, the copies
      // they made cost more than the shorter chain gained at every height
      // (FP32 pass, 64 x 720 x 360 members, 16 x 6 tiles: 277 against 262 us; 24
      // x 24 tiles at 2400 x 1500: 236 against 218 us).
      struct RowC {
        double s0, s1, f0, f1, e0, e1, w0, n0, n1, i0, i1, p0, p1;
      };
      auto take = [&](int k) {
        RowC c;
        float f0, f1, s0 = 0.f, s1 = 0.f, n0, n1, e0, e1;
        stage_pair<float>(sc + k * kF, c0, c1, f0, f1);
        stage_pair<float>(se + k * kF, c1, n + 2 < mw, e0, e1);
        stage_pair<float>(sn + k * kF, c0, c1, n0, n1);
        if (k > 0) stage_pair<float>(sn + (k - 1) * kF, c0, c1, s0, s1);
        float w0 = __shfl_up_sync(0xffffffffu, e1, 1, LPT);
        if (n == 0) w0 = 0.f;
        c.s0 = (double)s0, c.s1 = (double)s1, c.f0 = (double)f0, c.f1 = (double)f1;
        c.e0 = (double)e0, c.e1 = (double)e1, c.w0 = (double)w0;
        c.p0 = (double)wr[k * kR], c.p1 = (double)wr[k * kR + 1];
        c.n0 = c0 ? (double)n0 : 1.0, c.n1 = c1 ? (double)n1 : 1.0;
        c.i0 = march_rcp(c.n0), c.i1 = march_rcp(c.n1);
        return c;
      };
      auto row = [&](const RowC &c, double zb0, double zb1, double zc0, double zc1, double &q0,
                     double &q1) {
        const double zw = __shfl_up_sync(0xffffffffu, zc1, 1, LPT);
        const double ze = __shfl_down_sync(0xffffffffu, zc0, 1, LPT);
        double p0 = c.p0 - c.s0 * zb0, p1 = c.p1 - c.s1 * zb1;
        p0 -= c.e0 * zc1;
        p1 -= c.e0 * zc0;
        p0 -= c.f0 * zc0;
        p1 -= c.f1 * zc1;
        p0 -= c.w0 * zw;
        p1 -= c.e1 * ze;
        q0 = p0, q1 = p1;
      };
      {
        double zb0 = 0.0, zb1 = 0.0, zc0 = 0.0, zc1 = 0.0, q0, q1;
        int t = 0, kb = 0, ke = sub_start(1, hh, nb) - 1;
#pragma unroll 1
        for (int k = 0; k < hh; ++k) {
          const RowC c = take(k);
          if (k == kb) {
            zc0 = zc1 = 0.0;
            zin[t * 32] = make_double2(zb0, zb1);
          }
          row(c, zb0, zb1, zc0, zc1, q0, q1);
          const bool last = k == ke, fix = last && t < nb - 1;
          if (last) rho[t * 32] = make_double2(q0, q1);
          zb0 = zc0, zb1 = zc1;
          if (!last) zc0 = march_quot<V>(q0, c.n0, c.i0), zc1 = march_quot<V>(q1, c.n1, c.i1);
          if (__any_sync(0xffffffffu, fix)) {
            __syncwarp();
            *dv2 = make_double2(q0, q1);
            __syncwarp();
            cp_wait<0>();
            if (fix) {
              double s0, s1;
              matvec(mw, c0, c1, s0, s1);
              fetch_mat(mt + (t + 1 < nb - 1 ? nb + t + 1 : nb - 1) * msz, c0 ? mw : 0, c0, c1);
              zb0 -= s0, zb1 -= s1;
            }
            cp_commit();
          }
          if (last) {
            ++t;
            kb = k + 1;
            ke = sub_start(t + 1, hh, nb) - 1;
          }
        }
      }
      const int nbm = max(nb, __shfl_xor_sync(0xffffffffu, nb, 16));
      double vn0 = 0.0, vn1 = 0.0;
#pragma unroll 1
      for (int s = 0; s < nbm; ++s) {
        const int t = nb - 1 - s;
        const bool on = t >= 0;
        const int kb = on ? sub_start(t, hh, nb) : hh, ke = on ? sub_start(t + 1, hh, nb) - 1 : 0;
        double2 d = make_double2(0.0, 0.0);
        if (on) {
          float k0, k1;
          stage_pair<float>(sn + ke * kF, c0, c1, k0, k1);
          d = rho[t * 32];
          d.x -= (double)k0 * vn0;
          d.y -= (double)k1 * vn1;
        }
        __syncwarp();
        *dv2 = d;
        __syncwarp();
        double v0 = 0.0, v1 = 0.0;
        cp_wait<0>();
        if (on) {
          matvec(mw, c0, c1, v0, v1);
          if (t > 0) fetch_mat(mt + (nb + t - 1) * msz, c0 ? mw : 0, c0, c1);
        }
        cp_commit();
        double zb0 = 0.0, zb1 = 0.0;
        if (__any_sync(0xffffffffu, t > 0)) {
          float k0 = 0.f, k1 = 0.f;
          if (t > 0) stage_pair<float>(sn + (kb - 1) * kF, c0, c1, k0, k1);
          __syncwarp();
          *dv2 = make_double2(v0 * (double)k0, v1 * (double)k1);
          __syncwarp();
          cp_wait<0>();
          if (t > 0) {
            double h0, h1;
            matvec(mw, c0, c1, h0, h1);
            fetch_mat(mt + (t - 1) * msz, c0 ? mw : 0, c0, c1);
            const double2 e = zin[t * 32];
            zb0 = e.x + h0, zb1 = e.y + h1;
          }
          cp_commit();
        }
        double zc0 = v0, zc1 = v1, q0, q1;
        const int k_lo = __reduce_min_sync(0xffffffffu, kb), k_hi = __reduce_max_sync(0xffffffffu, ke);
#pragma unroll 1
        for (int k = k_lo; k <= k_hi; ++k) {
          const RowC c = take(k);
          const bool in = on && k >= kb && k <= ke;
          if (in) {
            const V u0 = (V)zc0, u1 = (V)zc1;
            store_pair<V>(z, id0 + (size_t)k * nx, d1, vec, c0, c1, u0, u1);
            if (DOTS) {
              acc_rz += (double)wr[k * kR] * (double)u0;
              acc_rz += (double)wr[k * kR + 1] * (double)u1;
            }
          }
          row(c, zb0, zb1, zc0, zc1, q0, q1);
          if (in && k < ke) {
            zb0 = zc0, zb1 = zc1;
            zc0 = march_quot<V>(q0, c.n0, c.i0), zc1 = march_quot<V>(q1, c.n1, c.i1);
          }
        }
        vn0 = v0, vn1 = v1;
      }
      stage_next();
      if (more) fetch_first(nxt);
      cp_commit();
    }
  }
  cp_wait<0>();
  if (DOTS) {
    double v2[2] = {acc_rz, acc_rr};
    TileFin fin{st};
    reduce_and_finish<2>(v2, partials, ticket, fin);
  }
}

// Resident CTAs by CTA size (in warps), and the size with the most resident
// warps (0: not asked yet).
struct PairFit {
  int slots[kPairWarps + 1] = {};
  int best = 0, sms = 0;
};
// Of one kernel on the current device, per sub-block count (its shared memory
// depends on nothing else).
template <typename V, int W, int HM, bool UPDATE, bool DOTS>
int pair_fit(int nbmax, PairFit &fit) {
  auto kern = k_tile_pair<V, W, HM, UPDATE, DOTS>;
  static std::mutex mu;
  static std::map<int, std::array<PairFit, kPairMaxRows + 1>> fits;
  int dev = 0;
  SEVP_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  PairFit &f = fits[dev][nbmax];
  if (!f.best) {
    const size_t per_warp = pair_smem_per_warp<V, W, HM>(nbmax);
    PairFit found;
    int optin = 0;
    SEVP_CUDA_TRY(cudaDeviceGetAttribute(&found.sms, cudaDevAttrMultiProcessorCount, dev));
    SEVP_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const size_t room = (size_t)optin - 1024;  // static shared memory of the sums
    SEVP_CUDA_TRY(
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
    for (int w = kPairWarps; w >= 1; --w) {
      int per_sm = 0;
      if (per_warp * w > room) continue;
      SEVP_CUDA_TRY(
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, w * 32, per_warp * w));
      found.slots[w] = per_sm * found.sms;
      if (found.slots[w] * w > found.slots[found.best] * found.best) found.best = w;
    }
    if (!found.best) {
      sevp_internal_set_message("tile pass: a warp's rows do not fit the shared memory");
      return SEVP_BAD_ARG;
    }
    f = found;
  }
  fit = f;
  return SEVP_OK;
}

template <typename V, int W, int HM, bool UPDATE, bool DOTS>
int tile_pair_launch_k(const PairLaunch<V> &L) {
  auto kern = k_tile_pair<V, W, HM, UPDATE, DOTS>;
  const TileGeom &tg = L.tg;
  const size_t per_warp = pair_smem_per_warp<V, W, HM>(tg.nbmax);
  PairFit fit;
  const int s = pair_fit<V, W, HM, UPDATE, DOTS>(tg.nbmax, fit);
  if (s) return s;
  const long long ntasks = (long long)tg.ty * pair_cols(tg);
  // few tasks: fewer warps per CTA, so that they spread over the SMs, where
  // all tasks are then resident at once (a second round doubles the pass: 16 x
  // 16 tiles at 592 x 344, FP64, 220 tasks on 148 one-warp CTAs: 45 us, on 220:
  // 27 us)
  int warps = (int)std::min<long long>(fit.best, std::max<long long>(1, ntasks / fit.sms));
  if ((long long)fit.slots[warps] * warps < ntasks) warps = fit.best;
  const long long want = std::min<long long>((ntasks + warps - 1) / warps, fit.slots[warps]);
  const unsigned blocks =
      (unsigned)std::max<long long>(1, std::min<long long>(want, (long long)(L.partials_n / 2)));
  // vector copies: every lane's first column is even, its pair in one row, and
  // every array aligned to the pair (callers pass their own buffers)
  bool vec = tg.nx % 2 == 0 && tg.tm % 2 == 0 && tg.xs % 2 == 0;
  const void *const vp[3] = {L.r, L.q, L.z}, *const cp[3] = {L.c.ac, L.c.ar, L.c.at};
  for (int k = 0; k < 3; ++k)
    vec = vec && ((uintptr_t)vp[k] & (2 * sizeof(V) - 1)) == 0 && ((uintptr_t)cp[k] & 7) == 0;
  bool quad = vec && tg.nx % 4 == 0 && tg.tm == W && tg.xs == 0;
  for (int k = 0; k < 3; ++k)
    quad = quad && ((uintptr_t)vp[k] & 15) == 0 && ((uintptr_t)cp[k] & 15) == 0;
  // a solve's kernels only: the planes are read before the kernel ahead has
  // ended, and outside a solve that kernel may be the caller's, writing them
  SEVP_CUDA_TRY(launch_overlapped(kern, blocks, warps * 32, per_warp * warps, L.stream,
                                  UPDATE || DOTS, tg, L.c.ac, L.c.ar, L.c.at, L.mats, L.r, L.q,
                                  L.z, L.st, L.partials, L.ticket, quad ? 2 : (vec ? 1 : 0)));
  return SEVP_OK;
}

template <typename V, int W, int HM>
int tile_pair_launch_w(const PairLaunch<V> &L) {
  if (L.update) {
    if (L.dots) return tile_pair_launch_k<V, W, HM, true, true>(L);
    return tile_pair_launch_k<V, W, HM, true, false>(L);
  }
  if (L.dots) return tile_pair_launch_k<V, W, HM, false, true>(L);
  return tile_pair_launch_k<V, W, HM, false, false>(L);
}

// Calls f with the tiling's lane segment and row instantiation.
template <int HM, class F>
int pair_dispatch_w(const TileGeom &tg, F &&f) {
  using std::integral_constant;
  const integral_constant<int, HM> hm;
  if (tg.wseg == 8) return f(integral_constant<int, 8>(), hm);
  if (tg.wseg == 16) return f(integral_constant<int, 16>(), hm);
  return f(integral_constant<int, 32>(), hm);
}
template <class F>
int pair_dispatch(const TileGeom &tg, F &&f) {
  if (tg.hmax <= 6) return pair_dispatch_w<6>(tg, f);
  if (tg.hmax <= 8) return pair_dispatch_w<8>(tg, f);
  if (tg.hmax <= 16) return pair_dispatch_w<16>(tg, f);
  return pair_dispatch_w<32>(tg, f);
}

template <typename V>
int tile_pair_launch_any(const PairLaunch<V> &L) {
  return pair_dispatch(L.tg, [&](auto w, auto hm) {
    return tile_pair_launch_w<V, decltype(w)::value, decltype(hm)::value>(L);
  });
}

template <typename V>
int tile_pair_resident_any(const TileGeom &tg, long long &warps) {
  return pair_dispatch(tg, [&](auto w, auto hm) {
    PairFit fit;
    const int s =
        pair_fit<V, decltype(w)::value, decltype(hm)::value, true, true>(tg.nbmax, fit);
    warps = (long long)fit.slots[fit.best] * fit.best;
    return s;
  });
}

}  // namespace sevp
