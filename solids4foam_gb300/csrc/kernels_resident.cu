// PCG of one corrector in one thread-block cluster.
//
// The launches of a PCG iteration -- preconditioner, SpMV, loop condition --
// cost more than the work of an iteration on a small mesh, and the exact
// DIC's sweeps, scheduled part by part through global memory, wait some ten
// microseconds at every link of the part chain.  Here the whole PCG loop of
// a corrector (lduMatrix PCG with DIC, processor-local DIC or the diagonal
// preconditioner, as in kernels_pcg.cu and kernels_local.cu) is one launch
// of one cluster of up to 16 CTAs: the vector that rows read from one another
// -- w in the substitutions, p in the product -- stays in the CTAs' shared
// memory, where every CTA of the cluster reads it, and levels, sums and
// phases are separated by the cluster's hardware barrier (about 0.2 us)
// instead of launches and flags.
//
// Rows are kept in a PCG order of their own: the cluster's CTAs own
// contiguous chunks of it, each sorted by level of the triangular sweeps
// (ResPlan).  With the exact DIC a level is one of the whole mesh's
// lower-triangular DAG, split evenly over the CTAs, and a cluster barrier
// ends it; with the processor-local DIC a CTA owns whole parts, so its
// levels need a CTA barrier only.  The right-hand-side pass writes r at a
// row's PCG position and the post pass reads x there (MeshView::pcgPos).
//
// Every vector entry is computed by the operations of the separate kernels in
// the same order, and so are the global sums (to the last bit): see "Sums" below.
// Rows have at most kResW neighbours (hexahedra, prisms, tetrahedra); other
// meshes, and those whose shared row vector does not fit, run the separate
// kernels.  So does FP64 with the processor-local DIC or the diagonal
// preconditioner.

#include <algorithm>

#include "kernels.cuh"
#include "pcg_common.cuh"
#include "sweep.cuh"

namespace s4g {
namespace {

// Forms: exact DIC with a cluster barrier per level, processor-local DIC,
// diagonal, exact DIC with the substitutions inside one CTA.
enum { kResExact = 0, kResLocal = 1, kResDiag = 2, kResSingle = 3 };
// (processor-local, FP32) six values of each of 64 lanes over the part groups, and 15
// words of up to 32 rows
constexpr size_t kResGroupBytes = 64 * 6 * sizeof(double) + 15 * 32 * 4;

template <typename T>
struct ResSweeps {
  ResSweepTab<T> tb[2], more[2];
  ResAddr ad[2];
};
template <bool CROSS, bool RING, bool SPLIT, bool MORE, bool WIDE, typename T>
__device__ __forceinline__ void sweepPair(const ResSweeps<T>& sw, const ResView& rv, unsigned uBase,
                                          unsigned rank, unsigned lva, int walk) {
  resSweep<0, CROSS, RING, SPLIT, MORE, WIDE, ResEnt<T>>(sw.tb[0], sw.more[0], sw.ad[0], uBase, rank, lva,
                                              rv.nLev, walk, rv.ring);
  resSweep<1, CROSS, RING, SPLIT, MORE, WIDE, ResEnt<T>>(sw.tb[1], sw.more[1], sw.ad[1], uBase, rank, lva,
                                              rv.nLev, walk, rv.ring);
}
template <bool CROSS, bool RING, typename T>
__device__ __forceinline__ void sweepForm(const ResSweeps<T>& sw, const ResView& rv, unsigned uBase,
                                          unsigned rank, unsigned lva, int walk) {
  if (rv.wide) {
    sweepPair<CROSS, RING, false, true, true>(sw, rv, uBase, rank, lva, walk);
  } else if (sizeof(T) == 8 && rv.split) {
    if (rv.more) sweepPair<CROSS, RING, sizeof(T) == 8, true, false>(sw, rv, uBase, rank, lva, walk);
    else sweepPair<CROSS, RING, sizeof(T) == 8, false, false>(sw, rv, uBase, rank, lva, walk);
  } else {
    if (rv.more) sweepPair<CROSS, RING, false, true, false>(sw, rv, uBase, rank, lva, walk);
    else sweepPair<CROSS, RING, false, false, false>(sw, rv, uBase, rank, lva, walk);
  }
}
// Both substitutions; the CTA (CROSS: the cluster) is synchronised at the end.
template <int NT, bool CROSS, typename T>
__device__ __forceinline__ void sweeps(const ResSweeps<T>& sw, const ResView& rv, unsigned uBase,
                                       unsigned rank, unsigned lva) {
  const int walk = CROSS ? NT : rv.walk;
  if (rv.nLev > 1 && (int)threadIdx.x < walk) {
    if (rv.place & 2) sweepForm<CROSS, false>(sw, rv, uBase, rank, lva, walk);
    else sweepForm<CROSS, true>(sw, rv, uBase, rank, lva, walk);
  }
  if (!CROSS) __syncthreads();
}

// Barrier between phases: of the cluster, or of its only CTA.
__device__ __forceinline__ void phaseBarrier(bool cluster) {
  if (cluster) { clArrive(); clWait(); }
  else __syncthreads();
}

// ---- Sums -------------------------------------------------------------------------
// The corrector loop can amplify a last bit of w.r or p.q a thousandfold every ten
// correctors (FP64, processor-local, 17 x 14 x 14: 1e-13 after 60 correctors, 2e-6
// after 100; exact DIC, 23 x 16 x 19: 2e-7 after 35), and in FP32 a last bit of the
// FP64 sum can turn the rounding of alpha or beta.  So the sums are added up in the
// order of the separate kernels, whatever form a mesh runs:
//   exact DIC   w.r by part (kernels_pcg.cu): 64 lanes that take a row of each
//               level, last level first, then by parts; sum|r| and p.q by storage
//               row, 256 rows a block, then by blocks.
//   diagonal    all three by storage row.
//   processor-  w.r and sum|r| by part (kernels_local.cu): 64 lanes over the part's
//   local DIC   rows in storage order, parts in groups of 32; p.q by storage row.
// A lane adds up its rows as Acc<T> does there, from there on in FP64.
//
// With the exact DIC and the diagonal the CTAs own rows in another order, so the
// rows' values go through global memory (L2), a warp takes 32 lanes of a part or 32
// rows, and every CTA adds up the records: two cluster barriers a sum (FP64, cube of
// 8, exact DIC: 30 us an iteration, 26 with the CTAs' own sums).  A CTA of the
// processor-local form owns whole parts and a contiguous range of storage rows, so
// only the records cross CTAs: one cluster barrier a sum.
// The row kernels' grid: blocks of 256 storage rows, and rows this far apart are one
// thread's.
__device__ __forceinline__ int ordStride(const MeshView& mv) { return mv.rowGrid * kRowBlock; }
// records of 32 virtual rows
__device__ __forceinline__ int ordGroups(const MeshView& mv) {
  return (min(mv.nC, ordStride(mv)) + 31) / 32;
}
// w.r of the components K0 .. K0 + NK - 1 over 32 lanes of a part (w and r by PCG row):
// the lanes' rows in the order of their sums, a step at a time (ResView::ordRow), the
// rows of the next steps read while those before them are added.  FP64 contracts the
// product with the addition, as the sweep does.
__device__ __forceinline__ void ordAdd(Acc<double>& a, double w, double r) { a.s = fma(w, r, a.s); }
__device__ __forceinline__ void ordAdd(Acc<float>& a, float w, float r) { a.add(__fmul_rn(w, r)); }
template <int NK, typename T>
__device__ __forceinline__ void ordPart(const int* rowOf, int steps, const T* w, const T* r, int k0,
                                        Acc<T> (&s)[NK]) {
  constexpr int B = NK == 1 ? 8 : 4;
  const int* const at = rowOf + (threadIdx.x & 31);
  T wv[B][NK], rv[B][NK];
  auto read = [&](int n0, T (&wn)[B][NK], T (&rn)[B][NK]) {
    int q[B];
#pragma unroll
    for (int u = 0; u < B; ++u) q[u] = n0 + u < steps ? __ldg(at + 32 * (n0 + u)) : -1;
#pragma unroll
    for (int u = 0; u < B; ++u)
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        wn[u][k] = q[u] >= 0 ? __ldcg(w + 3 * (size_t)q[u] + k0 + k) : T(0);
        rn[u][k] = q[u] >= 0 ? __ldcg(r + 3 * (size_t)q[u] + k0 + k) : T(0);
      }
  };
  read(0, wv, rv);
  for (int n = 0; n < steps; n += B) {
    T wn[B][NK], rn[B][NK];
    read(n + B, wn, rn);
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (n + u < steps)  // (a lane without a row: plus zero)
#pragma unroll
        for (int k = 0; k < NK; ++k) ordAdd(s[k], wv[u][k], rv[u][k]);
#pragma unroll
    for (int u = 0; u < B; ++u)
#pragma unroll
      for (int k = 0; k < NK; ++k) { wv[u][k] = wn[u][k]; rv[u][k] = rn[u][k]; }
  }
}
// N x 32 virtual rows of the row kernels, from row0 on, `apart` rows between the groups:
// per group and component the sums of |r| (ABS) or the terms a, three values a row by
// PCG row; component k of group n in lane 8 k of s[n].
template <bool ABS, int N, typename T>
__device__ __forceinline__ void ordRows(const MeshView& mv, const int* pos, const T* a, int row0, int apart,
                                        double (&s)[N]) {
  const bool one = mv.nC <= ordStride(mv);  // a row a lane (an addition to zero is one too)
  double v[N][4];
  T x[N][3];
  const int lane = (int)threadIdx.x & 31;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const int row = row0 + n * apart + lane;
    const bool on = row < mv.nC && row < ordStride(mv);
    const size_t q = on ? 3 * (size_t)__ldg(pos + row) : 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) x[n][k] = on ? __ldcg(a + q + k) : T(0);
  }
  if constexpr (sizeof(T) == 4)
    if (one) {
#pragma unroll
      for (int n = 0; n < N; ++n)
#pragma unroll
        for (int k = 0; k < 3; ++k) x[n][k] = ABS ? fabsf(x[n][k]) : x[n][k];
      warpFloatSums<N>(x, s);
      return;
    }
#pragma unroll
  for (int n = 0; n < N; ++n) {
    v[n][3] = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) v[n][k] = toF64(ABS ? fabs(x[n][k]) : x[n][k]);
    if (!one) {
      Acc<T> c[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) c[k].s = ABS ? fabs(x[n][k]) : x[n][k];
      const int r0 = row0 + n * apart + lane;
      for (int row = r0 + ordStride(mv); r0 < ordStride(mv) && row < mv.nC; row += ordStride(mv)) {
        const size_t q = 3 * (size_t)__ldg(pos + row);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const T y = __ldcg(a + q + k);
          c[k].add(ABS ? fabs(y) : y);
        }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) v[n][k] = accValue(c[k]);
    }
  }
  warpSpreadSums<4, N>(v, s);
}
// w.r and |r| of the diagonal form (FP32) over 32 virtual rows (a row a lane: the form has
// at most kResMaxDiagRows rows): w.r of component k in lane 8 k, sum|r| in lane 8 k + 1
__device__ __forceinline__ double ordRowsDiag(const MeshView& mv, const int* pos, const float* w, const float* r,
                                              int g) {
  const int lane = (int)threadIdx.x & 31, row = 32 * g + lane;
  float x[2][3] = {{0, 0, 0}, {0, 0, 0}};
  if (row < mv.nC) {
    const size_t q = 3 * (size_t)__ldg(pos + row);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float v = __ldcg(r + q + k);
      x[0][k] = mulT(__ldcg(w + q + k), v);
      x[1][k] = fabsf(v);
    }
  }
  double s[2];
  warpFloatSums<2>(x, s);
  return (lane & 1) ? s[1] : s[0];
}
// The sum over the row records (stride values each), of value k, blocks 32 h ... (and
// every 256th after them)
__device__ __forceinline__ double ordBlocks(const MeshView& mv, const double* rec, int stride, int k, int h) {
  const int nB = mv.rowGrid, nG = ordGroups(mv), b0 = 32 * h + (int)(threadIdx.x & 31);
  double v = 0;
  for (int b = b0; b < nB; b += kRowBlock) {
    double x[kRowBlock / 32];
#pragma unroll
    for (int j = 0; j < kRowBlock / 32; ++j) {
      const int g = b * (kRowBlock / 32) + j;
      x[j] = g < nG ? __ldcg(rec + stride * (size_t)g + k) : 0.0;
    }
    double t = x[0];
#pragma unroll
    for (int j = 1; j < kRowBlock / 32; ++j) t += x[j];
    v = b == b0 ? t : v + t;
  }
  return warpTree(v, nB - 32 * h);
}
// Row sums of NV values from their records into out[0..NV): the end of a sum, by the
// whole CTA; complete for the threads 0 .. NV - 1.
template <int NT, int NV>
__device__ __forceinline__ void ordRowTotal(const MeshView& mv, const double* rec, double* blk, double* out) {
  constexpr int W = NT / 32;
  const int lane = (int)threadIdx.x & 31, wid = (int)threadIdx.x >> 5;
  const int nH = mv.rowGrid < kRowBlock ? (mv.rowGrid + 31) / 32 : W;
  for (int q = wid; q < NV * nH; q += W) {
    const double s = ordBlocks(mv, rec, NV, q % NV, q / NV);
    if (lane == 0) blk[q] = s;
  }
  __syncthreads();
  if ((int)threadIdx.x < NV) {
    double s = blk[threadIdx.x];
    for (int h = 1; h < nH; ++h) s += blk[NV * h + (int)threadIdx.x];
    out[threadIdx.x] = s;
  }
}
// The sum over the part records of component k (reduceRecords)
__device__ __forceinline__ double ordParts(const double* rec, int nParts, int k) {
  const int lane = (int)(threadIdx.x & 31);
  double b = 0;
  for (int j = 0; 32 * j < nParts && j < 8; ++j) {
    double a = 0;
    for (int p = lane + 32 * j; p < nParts; p += 256) {
      const double x = __ldcg(rec + 6 * (size_t)p + k), y = __ldcg(rec + 6 * (size_t)p + 3 + k);
      a = p < 256 ? x + y : a + (x + y);
    }
    b = j == 0 ? a : b + a;
  }
  return warpTree(b, nParts);
}
// Exact DIC and diagonal.  DOTS: w.r and sum|r| (w, r by PCG row) into out[0..5];
// else the terms w into out[0..2].  The rows' values are written; out is complete for
// the lanes 0 .. 2 of warp 0.  (blk: 3 + 48 values.)
template <int NT, bool DOTS, bool DIAG, typename T>
__device__ __forceinline__ void orderedSum(const MeshView& mv, const ResView& rv, const T* w, const T* r,
                                           double* rec, double* blk, double* out, int C, unsigned rank,
                                           bool cluster) {
  // FP64: a component of a half part a warp (a multiply-add of a warp takes 64 cycles);
  // FP32: the three together (9 FP64 additions for 18)
  constexpr int W = NT / 32, NK = sizeof(T) == 8 ? 1 : 3, N = 4;
  const int lane = (int)threadIdx.x & 31, wid = (int)threadIdx.x >> 5;
  const int nG = ordGroups(mv), nP = DOTS && !DIAG ? 6 / NK * mv.nParts : 0;
  double* const rows = rec + 6 * (size_t)mv.nParts + (DOTS ? 0 : 6 * (size_t)nG);
  phaseBarrier(cluster);
  int q = (int)rank + C * wid;
  for (; q < nP; q += C * W) {
    const int task = q / (3 / NK), n0 = rv.ordStep[task];
    Acc<T> a[NK];
    ordPart(rv.ordRow + 32 * (size_t)n0, rv.ordStep[task + 1] - n0, w, r, q % (3 / NK), a);
    if (NK == 1) {
      const double s = warpTree(accValue(a[0]));
      if (lane == 0) rec[q] = s;
    }
    if constexpr (NK == 3) {
      const float x[1][3] = {{a[0].s, a[1].s, a[2].s}}, c[1][3] = {{a[0].c, a[1].c, a[2].c}};
      double s[1];
      warpFloatSums<1, true>(x, c, s);
      if ((lane & 7) == 0 && lane < 24) rec[3 * (size_t)q + (lane >> 3)] = s[0];
    }
  }
  q -= nP;
  if constexpr (DOTS && DIAG) {
    for (; q < nG; q += C * W) {
      const double s = ordRowsDiag(mv, rv.pos, w, r, q);
      if ((lane & 7) < 2 && lane < 24) rows[6 * (size_t)q + 3 * (lane & 1) + (lane >> 3)] = s;
    }
  } else {
    auto put = [&](int g, double s) {
      if ((lane & 7) == 0 && lane < 24 && g < nG) rows[3 * (size_t)g + (lane >> 3)] = s;
    };
    for (; q + (N - 1) * C * W < nG; q += N * C * W) {
      double s[N];
      ordRows<DOTS, N>(mv, rv.pos, DOTS ? r : w, 32 * q, 32 * C * W, s);
#pragma unroll
      for (int n = 0; n < N; ++n) put(q + n * C * W, s[n]);
    }
    for (; q < nG; q += 2 * C * W) {
      double s[2];
      ordRows<DOTS, 2>(mv, rv.pos, DOTS ? r : w, 32 * q, 32 * C * W, s);
      put(q, s[0]);
      put(q + C * W, s[1]);
    }
  }
  phaseBarrier(cluster);
  if (DOTS && DIAG) {
    ordRowTotal<NT, 6>(mv, rows, blk, out);
    __syncwarp();  // (threads 0 .. 5 to threads 0 .. 2)
    return;
  }
  if (DOTS && wid >= W - 3) {
    const double s = ordParts(rec, mv.nParts, wid - (W - 3));
    if (lane == 0) blk[48 + wid - (W - 3)] = s;
  }
  ordRowTotal<NT, 3>(mv, rows, blk, out + (DOTS ? 3 : 0));
  if (DOTS && threadIdx.x < 3) out[lane] = blk[48 + lane];
}
// Processor-local: w.r and sum|r| by part into out[0..5], from w of the CTA's rows in
// the shared vector and r by row of the CTA.  A warp takes half of a part's lanes and one
// of the two sums.  rec: 12 values a part ([half][w.r, sum|r|][component]); grp: 6 values
// of each of 64 lanes over the groups.
template <int NT, typename T>
__device__ __forceinline__ void localDots(const MeshView& mv, const ResView& rv, unsigned uBase, const T* r,
                                          int base, const unsigned short* pos, double* rec, double* grp, double* out, unsigned rank,
                                          bool cluster) {
  constexpr int W = NT / 32, B = 8;
  const int lane = (int)threadIdx.x & 31, wid = (int)threadIdx.x >> 5;
  const int p0 = rv.part0[rank], p1 = rv.part0[rank + 1];
  for (int q = 4 * p0 + wid; q < 4 * p1; q += W) {
    const int part = q >> 2, lo = mv.partStart[part], hi = mv.partStart[part + 1];
    const bool dots = (q & 1) == 0;
    Acc<T> a[3];
    for (int s0 = lo + 16 * (q & 2) + lane; s0 < hi; s0 += 64 * B) {
      int at[B];
#pragma unroll
      for (int u = 0; u < B; ++u) at[u] = s0 + 64 * u < hi ? pos[s0 + 64 * u - base] : -1;
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (at[u] >= 0) {
          T w[3];
          if (dots) URow<T>::load(uBase + URow<T>::kBytes * (unsigned)at[u], w);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const T x = r[3 * (size_t)at[u] + k];
            a[k].add(dots ? mulT(w[k], x) : fabs(x));
          }
        }
    }
    const float x[1][3] = {{a[0].s, a[1].s, a[2].s}}, c[1][3] = {{a[0].c, a[1].c, a[2].c}};
    double s[1];
    warpFloatSums<1, true>(x, c, s);
    if ((lane & 7) == 0 && lane < 24) rec[3 * (size_t)q + (lane >> 3)] = s[0];
  }
  phaseBarrier(cluster);
  // groups of 32 parts; lane v of 64 adds up the groups v, v + 64, ... in that order
  const int nGrp = (mv.nParts + 31) / 32;
  for (int j = wid; j < 6 * min(nGrp, 64); j += W) {
    const int k = j % 6;
    double s = 0;
    for (int g = j / 6; g < nGrp; g += 64) {
      const int part = 32 * g + lane;
      const double* const x = rec + 12 * (size_t)part + k;
      const double v = warpTree(part < mv.nParts ? __ldcg(x) + __ldcg(x + 6) : 0.0, mv.nParts - 32 * g);
      s = g < 64 ? v : s + v;
    }
    if (lane == 0) grp[6 * (j / 6) + k] = s;
  }
  __syncthreads();
  groupTotal<W>(grp, nGrp, out);
  __syncthreads();
}
// Processor-local: the terms y v by storage row into out[0..2], from y by row of the
// CTA and v in the shared vector.  A 32-row record is the CTA's that owns its first row;
// other(s, t): the terms t of a row s of another CTA.
template <int NT, typename T, typename F>
__device__ __forceinline__ void localRowSum(const MeshView& mv, unsigned uBase, const T* y, int base, int R,
                                            const unsigned short* pos, double* rec, double* blk, double* out,
                                            bool cluster, F other) {
  constexpr int W = NT / 32, N = 2;
  const int lane = (int)threadIdx.x & 31, wid = (int)threadIdx.x >> 5;
  const int gEnd = (base + R + 31) / 32;
  __syncthreads();
  for (int g0 = (base + 31) / 32 + wid; g0 < gEnd; g0 += N * W) {
    T t[N][3];
    double s[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const int row = 32 * (g0 + n * W) + lane;
      t[n][0] = t[n][1] = t[n][2] = T(0);
      if (row < base + R) {
        const int i = pos[row - base];
        T u[3];
        URow<T>::load(uBase + URow<T>::kBytes * (unsigned)i, u);
#pragma unroll
        for (int k = 0; k < 3; ++k) t[n][k] = mulT(y[3 * (size_t)i + k], u[k]);
      } else if (g0 + n * W < gEnd && row < mv.nC) {
        other(row, t[n]);
      }
    }
    warpFloatSums<N>(t, s);
#pragma unroll
    for (int n = 0; n < N; ++n)
      if ((lane & 7) == 0 && lane < 24 && g0 + n * W < gEnd) rec[3 * (size_t)(g0 + n * W) + (lane >> 3)] = s[n];
  }
  phaseBarrier(cluster);
  ordRowTotal<NT, 3>(mv, rec, blk, out);
}

// Scalars of the iteration, in shared memory, decided by warp 0.
template <typename T>
struct ResScalars {
  double sum[8];
  double blk[51];  // (the sums' records over blocks)
  double norm[3], lim[3], last[3], wArA[3], wApA[3], alpha[3], beta[3];
  T alphaT[3], betaT[3];  // in the value type (a conversion is an FP64 operation)
  int active[3], pend[3], nIter[3];
  int any, iters;
  unsigned status;
};

// OCC: CTAs per SM the registers are limited to: 1 for a single solve, 2 where
// several meshes or load cases run at once (a tenth slower alone, and twice the
// clusters on the device).  Both compute the same bits.
template <typename T, int NT, int MODE, int OCC>
__global__ void __launch_bounds__(NT, OCC)
kResPcg(MeshView mv, Controls c, ResView rv, ResPtrs<T> rp, PcgPtrs<T> p, DevState* st,
        double* partials) {
  constexpr bool LOCAL = MODE == kResLocal, DIAG = MODE == kResDiag;
  p = casePcg(p, blockIdx.y, mv.nC);
  st += blockIdx.y;
  double* const ordRec = partials + (size_t)blockIdx.y * mv.caseRec + mv.ordOff;
  if (!st->pcgContinue) return;  // the same in every CTA: rank 0 writes it at the end
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ ResScalars<T> sc;
  constexpr int kRows = 2;  // rows of a thread in flight
  constexpr unsigned kU = URow<T>::kBytes;
  const int C = (int)gridDim.x, t = (int)threadIdx.x;
  const bool cluster = C > 1;
  const unsigned rank = cluster ? clRank() : 0u;
  const int base = rv.chunk[rank], R = rv.chunk[rank + 1] - base;
  const int mr = rv.maxRows;
  // ---- shared memory: u and its zero row | group sums | level starts | vectors |
  //      tables
  unsigned char* sp = smraw;
  const unsigned uBase = (unsigned)__cvta_generic_to_shared(sp);
  sp += (size_t)kU * rv.uRows;
  // (processor-local) sums of part groups; columns, coefficients, position, diagonal and
  // entry count of the up to 31 rows after the CTA's own that share a 32-row record with
  // its last ones
  double* const grp = (double*)sp;
  uint32_t* const ext = (uint32_t*)(grp + 64 * 6);
  float* const extT = (float*)ext;
  unsigned short* const posS = (unsigned short*)(sp + kResGroupBytes);  // row of each storage row
  if (rv.local) sp += kResGroupBytes + 2 * (size_t)((mr + 7) / 8 * 8);
  // (first, end) of the levels, with two empty levels before and after them
  int2* lv = (int2*)sp;
  const unsigned lva = (unsigned)__cvta_generic_to_shared(lv + 2);
  sp += sizeof(int2) * ((rv.nLev + 5) / 2 * 2);
  T *rg = p.r + 3 * (size_t)base, *qg = p.q + 3 * (size_t)base, *pg = p.p + 3 * (size_t)base,
    *xg = p.x + 3 * (size_t)base;
  T* const rGlob = rg;
  T* const wGlob = p.w + 3 * (size_t)base;
  T* const xGlob = xg;
  if (rv.place & 1) {
    const size_t b = sizeof(T) * 3 * (size_t)mr;
    rg = (T*)sp; qg = (T*)(sp + b); pg = (T*)(sp + 2 * b); xg = (T*)(sp + 3 * b);
    sp += 4 * b;
  }
  // sweep tables by row of the sweeping CTA (kResSingle: of the whole mesh)
  const int sBase = MODE == kResSingle ? 0 : base, sRows = MODE == kResSingle ? mv.nC : R;
  ResSweeps<T> sw{{rp.sweep[0], rp.sweep[1]}, {rp.more[0], rp.more[1]}, {}};
  if (MODE != kResDiag) {
    using Q = typename ResSweepTab<T>::Q;
    using Rw = typename ResSweepTab<T>::R;
    const bool ringed = !(rv.place & 2);
    const int cap = ringed ? kResAhead * rv.ring : MODE == kResSingle ? rv.uRows : mr;
    // a table's place in shared memory, filled unless it is the ring
    auto place = [&](ResSweepTab<T>& tb, unsigned& q, unsigned& r) {
      tb.q += sBase; tb.r += sBase;
      Q* const a = (Q*)sp;
      Rw* const b = (Rw*)(a + cap);
      sp = (unsigned char*)(b + cap);
      if (!ringed)
        for (int i = t; i < sRows; i += NT) { a[i] = tb.q[i]; b[i] = tb.r[i]; }
      q = (unsigned)__cvta_generic_to_shared(a);
      r = (unsigned)__cvta_generic_to_shared(b);
    };
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      unsigned char* const sp0 = sp;
      place(sw.tb[d], sw.ad[d].q, sw.ad[d].r);
      if (rv.more) place(sw.more[d], sw.ad[d].mq, sw.ad[d].mr);
      if (ringed && d == 0) sp = sp0;  // both sweeps use the same ring
    }
  }
  const uint32_t* cnt = rv.cnt + base;
  const uint32_t* col = rv.col + base;
  const T* val = rp.val + base;
  const T* diag = rp.diag + base;
  const T* rD = rp.rD + base;
  int ldP = mv.nC;
  if (rv.place & 4) {
    T* a = (T*)sp;
    T* dg = a + kResW * (size_t)mr;
    T* rd = dg + mr;
    uint32_t* cl = (uint32_t*)(rd + mr);
    uint32_t* cn = cl + kResW * (size_t)mr;
    for (int i = t; i < R; i += NT) {
      dg[i] = diag[i];
      rd[i] = rD[i];
      cn[i] = cnt[i];
#pragma unroll
      for (int k = 0; k < kResW; ++k) {
        cl[k * mr + i] = col[(size_t)k * mv.nC + i];
        a[k * mr + i] = val[(size_t)k * mv.nC + i];
      }
    }
    col = cl; val = a; diag = dg; rD = rd; cnt = cn; ldP = mr;
  }
  if (MODE != kResDiag)
    for (int l = t; l < rv.nLev + 4; l += NT) {
      const int* g = rv.lvl + (size_t)(MODE == kResSingle ? 0u : rank) * (rv.nLev + 1) + (l - 2);
      lv[l] = l < 2 || l >= rv.nLev + 2 ? make_int2(0, 0) : make_int2(g[0], g[1]);
    }
  if (t < 3) {
    const double nf = st->normFactor[t], ir = st->initRes[t];
    sc.norm[t] = nf;
    sc.lim[t] = pcgLimit(c, ir);
    sc.last[t] = ir * nf;
    sc.wArA[t] = st->wArA[t]; sc.wApA[t] = st->wApA[t]; sc.alpha[t] = 0; sc.beta[t] = 0; sc.alphaT[t] = T(0); sc.betaT[t] = T(0);
    sc.active[t] = st->active[t]; sc.pend[t] = 0; sc.nIter[t] = 0;
    const T z[3] = {T(0), T(0), T(0)};
    if (t == 0) URow<T>::store(uBase + kU * (rv.uRows - 1), z);
  }
  if (t == 0) { sc.any = 1; sc.iters = 0; sc.status = 0; }
  if (LOCAL)
    for (int i = t; i < R; i += NT) posS[i] = (unsigned short)(rv.pos[base + i] - base);
  if (LOCAL && t < 32) {
    const int row = (base + R) / 32 * 32 + t;  // (a storage row: the chunks are storage ranges)
    if (row >= base + R && row < mv.nC) {
      const int g = rv.pos[row];
      unsigned owner = rank;
      while (rv.chunk[owner + 1] <= g) ++owner;
      ext[32 * 2 * kResW + t] = owner << 24 | (unsigned)(g - rv.chunk[owner]);
      ext[32 * (2 * kResW + 2) + t] = rv.cnt[g];
      extT[32 * (2 * kResW + 1) + t] = (float)rp.diag[g];
      for (int e = 0; e < kResW; ++e) {
        ext[32 * e + t] = rv.col[(size_t)e * mv.nC + g];
        extT[32 * (kResW + e) + t] = (float)rp.val[(size_t)e * mv.nC + g];
      }
    }
  }
  if (rv.place & 1)  // (in global memory the right-hand-side pass has set both)
    for (int i = t; i < R; i += NT)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        rg[3 * i + k] = rGlob[3 * (size_t)i + k];
        xg[3 * i + k] = T(0);
      }
  // where w of the own rows is written and, after the sweeps, read
  const unsigned wBase = MODE == kResSingle && cluster ? mapa(uBase + kU * (unsigned)base, 0)
                                                       : uBase + (MODE == kResSingle ? kU * (unsigned)base : 0u);
  phaseBarrier(cluster);  // every CTA has started: its shared memory may be written
  for (;;) {
    // pending r -= alpha q, sum|r|, w = rD r
    bool pend[3];
    T al[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) { pend[k] = sc.pend[k] != 0; al[k] = sc.alphaT[k]; }
    for (int i0 = t; i0 < R; i0 += kRows * NT) {
      T rd[kRows], rr[kRows][3], qv[kRows][3];
#pragma unroll
      for (int h = 0; h < kRows; ++h) {
        const int i = i0 + h * NT;
        if (i < R) {
          rd[h] = rD[i];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            rr[h][k] = rg[3 * i + k];
            if (pend[k]) qv[h][k] = qg[3 * i + k];
          }
        }
      }
#pragma unroll
      for (int h = 0; h < kRows; ++h) {
        const int i = i0 + h * NT;
        if (i < R) {
          T w[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            if (pend[k]) {
              rr[h][k] = fmaT(-al[k], qv[h][k], rr[h][k]);
              rg[3 * i + k] = rr[h][k];
            }
            w[k] = mulT(rd[h], rr[h][k]);
            if (DIAG) {
              wGlob[3 * (size_t)i + k] = w[k];
              if (rv.place & 1) rGlob[3 * (size_t)i + k] = rr[h][k];
            }
          }
          if (MODE == kResSingle && cluster) URow<T>::storeCluster(wBase + kU * i, w);
          else URow<T>::store(wBase + kU * i, w);
        }
      }
    }
    if (MODE == kResExact) {
      phaseBarrier(true);
      sweeps<NT, true>(sw, rv, uBase, rank, lva);
    } else if (MODE == kResLocal) {
      __syncthreads();
      sweeps<NT, false>(sw, rv, uBase, rank, lva);
    } else if (MODE == kResSingle) {
      phaseBarrier(cluster);
      if (rank == 0) sweeps<NT, false>(sw, rv, uBase, rank, lva);
      if (cluster) phaseBarrier(true);
    }
    if (!DIAG && !LOCAL)
      for (int i = t; i < R; i += NT) {
        T w[3];
        if (MODE == kResSingle && cluster) {
          URow<T>::loadCluster(wBase + kU * i, w);
          if (rank != 0) URow<T>::store(uBase + kU * i, w);  // rank 0's rows are in place
        } else {
          URow<T>::load(uBase + kU * i, w);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          wGlob[3 * (size_t)i + k] = w[k];
          if (rv.place & 1) rGlob[3 * (size_t)i + k] = rg[3 * i + k];
        }
      }
    if constexpr (LOCAL) localDots<NT>(mv, rv, uBase, rg, base, posS, ordRec, grp, sc.sum, rank, cluster);
    else orderedSum<NT, true, DIAG>(mv, rv, p.w, p.r, ordRec, sc.blk, sc.sum, C, rank, cluster);
    // the residual test of the pending iteration, beta (a lane per component)
    if (t < 32) {
      int act = 0;
      unsigned bad = 0;
      const bool anyPend = sc.pend[0] || sc.pend[1] || sc.pend[2];
      __syncwarp();
      if (t < 3) {
        act = sc.active[t];
        int it = sc.nIter[t];
        if (sc.pend[t]) {
          const double s = sc.sum[3 + t];
          sc.last[t] = s;
          sc.nIter[t] = ++it;
          if (!isfinite(s)) bad = kErrNaN;
          act = (!pcgConverged(s, sc.norm[t], sc.lim[t]) && it < c.maxIter && isfinite(s)) ? 1 : 0;
          sc.active[t] = act;
        }
        if (act) {
          const double beta = it == 0 ? 0.0 : sc.sum[t] / sc.wArA[t];
          sc.beta[t] = beta;
          sc.betaT[t] = (T)beta;
          sc.wArA[t] = sc.sum[t];
        }
      }
      const unsigned any = __ballot_sync(0xffffffffu, act != 0);
      const unsigned nan = __ballot_sync(0xffffffffu, bad != 0);
      if (t == 0) {
        if (nan) sc.status |= kErrNaN;
        sc.any = any != 0 && !nan;
        if (anyPend) sc.iters += 1;
      }
    }
    __syncthreads();
    const bool go = sc.any != 0;
    // pending x += alpha p_old; p = w + beta p_old into p and the shared vector
    bool act[3], first[3];
    T b[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      act[k] = sc.active[k] != 0; first[k] = sc.nIter[k] == 0; b[k] = sc.betaT[k];
    }
    for (int i0 = t; i0 < R; i0 += kRows * NT) {
      T u[kRows][3], po[kRows][3], xo[kRows][3];
#pragma unroll
      for (int h = 0; h < kRows; ++h) {
        const int i = i0 + h * NT;
        if (i < R) {
          if (go) URow<T>::load(uBase + kU * i, u[h]);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            po[h][k] = first[k] ? T(0) : pg[3 * i + k];
            if (pend[k]) xo[h][k] = xg[3 * i + k];
          }
        }
      }
#pragma unroll
      for (int h = 0; h < kRows; ++h) {
        const int i = i0 + h * NT;
        if (i < R) {
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            if (pend[k]) xg[3 * i + k] = fmaT(al[k], po[h][k], xo[h][k]);
            if (go && act[k]) {
              if (!first[k]) u[h][k] = fmaT(b[k], po[h][k], u[h][k]);
              pg[3 * i + k] = u[h][k];
            }
          }
          if (go) URow<T>::store(uBase + kU * i, u[h]);
        }
      }
    }
    if (!go) break;
    phaseBarrier(cluster);
    // q = A p, p.q
    for (int i0 = t; i0 < R; i0 += kRows * NT) {
      int n[kRows];
      T dg[kRows], a[kRows][kResW];
      uint32_t cl[kRows][kResW];
#pragma unroll
      for (int h = 0; h < kRows; ++h) {
        const int i = i0 + h * NT;
        n[h] = 0;
        if (i < R) {
          n[h] = (int)cnt[i];
          dg[h] = diag[i];
#pragma unroll
          for (int e = 0; e < kResW; ++e) { cl[h][e] = col[e * ldP + i]; a[h][e] = val[e * ldP + i]; }
        }
      }
#pragma unroll
      for (int h = 0; h < kRows; ++h) {
        const int i = i0 + h * NT;
        if (i < R) {
          T v[3], y[3], x[kResW][3];
          URow<T>::load(uBase + kU * i, v);
#pragma unroll
          for (int e = 0; e < kResW; ++e) {
            const unsigned at = uBase + kU * (cl[h][e] & 0xffffffu);
            if ((cl[h][e] >> 24) == rank) URow<T>::load(at, x[e]);
            else URow<T>::loadCluster(mapa(at, cl[h][e] >> 24), x[e]);
          }
#pragma unroll
          for (int k = 0; k < 3; ++k) y[k] = mulT(dg[h], v[k]);
#pragma unroll
          for (int e = 0; e < kResW; ++e)
            if (e < n[h])
#pragma unroll
              for (int k = 0; k < 3; ++k) y[k] = fmaT(a[h][e], x[e][k], y[k]);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            if (act[k]) qg[3 * i + k] = y[k];
            if (!LOCAL) wGlob[3 * (size_t)i + k] = mulT(y[k], v[k]);
          }
        }
      }
    }
    if constexpr (LOCAL) {
      // a row of another CTA: its product, as there
      auto other = [&](int, T (&term)[3]) {
        const int e0 = t & 31;
        T v[3], y[3], x[kResW][3];
        const uint32_t own = ext[32 * 2 * kResW + e0];
        URow<T>::loadCluster(mapa(uBase + kU * (own & 0xffffffu), own >> 24), v);
        const int n = (int)ext[32 * (2 * kResW + 2) + e0];
#pragma unroll
        for (int e = 0; e < kResW; ++e) {
          const uint32_t cl = ext[32 * e + e0];
          URow<T>::loadCluster(mapa(uBase + kU * (cl & 0xffffffu), cl >> 24), x[e]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) y[k] = mulT(extT[32 * (2 * kResW + 1) + e0], v[k]);
#pragma unroll
        for (int e = 0; e < kResW; ++e)
          if (e < n)
#pragma unroll
            for (int k = 0; k < 3; ++k) y[k] = fmaT(extT[32 * (kResW + e) + e0], x[e][k], y[k]);
#pragma unroll
        for (int k = 0; k < 3; ++k) term[k] = mulT(y[k], v[k]);
      };
      localRowSum<NT>(mv, uBase, qg, base, R, posS, ordRec + 12 * (size_t)mv.nParts, sc.blk, sc.sum, cluster, other);
    } else orderedSum<NT, false, DIAG>(mv, rv, p.w, p.r, ordRec, sc.blk, sc.sum, C, rank, cluster);
    if (t < 32) {
      int on = 0;
      unsigned bad = 0;
      if (t < 3) {
        sc.pend[t] = 0;
        if (sc.active[t]) {
          const double s = sc.sum[t];
          sc.wApA[t] = s;
          if (fabs(s) < 1e-300 * sc.norm[t]) {  // checkSingularity: stop this component
            sc.active[t] = 0;
          } else {
            if (s <= 0) bad = kErrIndefinite;
            const double alpha = sc.wArA[t] / s;
            sc.alpha[t] = alpha;
            sc.alphaT[t] = (T)alpha;
            sc.pend[t] = 1;
            on = 1;
          }
        }
      }
      const unsigned any = __ballot_sync(0xffffffffu, on != 0);
      const unsigned ind = __ballot_sync(0xffffffffu, bad != 0);
      if (t == 0) {
        if (ind) sc.status |= kErrIndefinite;
        sc.any = any != 0;
      }
    }
    __syncthreads();
    if (!sc.any) break;
  }
  if (rv.place & 1)  // each thread its own rows
    for (int i = t; i < R; i += NT)
#pragma unroll
      for (int k = 0; k < 3; ++k) xGlob[3 * (size_t)i + k] = xg[3 * i + k];
  // no CTA leaves while another may still read its shared memory
  if (cluster) phaseBarrier(true);
  if (rank == 0 && t == 0) {
    for (int k = 0; k < 3; ++k) {
      st->nIter[k] = sc.nIter[k]; st->finalRes[k] = sc.last[k] / sc.norm[k]; st->active[k] = 0;
      st->wArA[k] = sc.wArA[k]; st->wApA[k] = sc.wApA[k]; st->alpha[k] = sc.alpha[k]; st->beta[k] = sc.beta[k];
    }
    if (sc.status) atomicOr(&st->status, sc.status);
    st->pcgIter += sc.iters;
    st->pcgContinue = 0;
  }
}

// The tables of the plan, from the storage-order CSR: entry lists of the
// product (CSR order) and of the substitutions (lower entries in CSR order,
// then upper ones in reverse; only in-part entries with the processor-local
// DIC), values in T.
template <typename T>
__global__ void kResTables(MeshView mv, ResView rv, const int* pos, const double* val,
                           const double* diag, const double* rD, const double* rDa, int diagOnly,
                           uint32_t* col, uint32_t* cnt, ResPtrs<T> out) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= mv.nC) return;
  const int i = pos[s];
  int lo = 0, hi = mv.nC;
  if (rv.local) {  // the part of row s
    int a = 0, b = mv.nParts;
    while (b - a > 1) {
      const int m = (a + b) / 2;
      if (mv.partStart[m] <= s) a = m; else b = m;
    }
    lo = mv.partStart[a];
    hi = mv.partStart[a + 1];
  }
  auto rankOf = [&](int q) {
    int r = 0;
    while (r + 1 < rv.C && rv.chunk[r + 1] <= q) ++r;
    return r;
  };
  auto code = [&](int row) {  // product column
    const int q = pos[row], r = rankOf(q);
    return ((uint32_t)r << 24) | (uint32_t)(q - rv.chunk[r]);
  };
  auto sweepCode = [&](int row) {
    const int q = pos[row];
    if (rv.single) return (uint32_t)q;
    const int r = rankOf(q);
    const uint32_t w = (uint32_t)(q - rv.chunk[r]);
    return rv.local ? w : ((uint32_t)r << 14) | w;
  };
  T* oval = const_cast<T*>(out.val);
  const int e0 = mv.rowptr[s], n = mv.rowptr[s + 1] - e0;
  const uint32_t own = code(s);
  const uint32_t zero = (rv.single || rv.local) ? (uint32_t)(rv.uRows - 1)
                                                : (own >> 24 << 14) | (uint32_t)(rv.uRows - 1);
  for (int k = 0; k < kResW; ++k) {
    col[(size_t)k * mv.nC + i] = k < n ? code(mv.col[e0 + k]) : own;
    oval[(size_t)k * mv.nC + i] = k < n ? (T)val[e0 + k] : T(0);
  }
  int num[2] = {0, 0};
  if (!diagOnly)
    for (int dir = 0; dir < 2; ++dir) {
      T a[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
      uint32_t w[6] = {zero, zero, zero, zero, zero, zero};
      for (int j = 0; j < n; ++j) {
        const int k = dir == 0 ? j : n - 1 - j;
        const int cl = mv.col[e0 + k];
        if (dir == 0 ? !(cl < s && cl >= lo) : !(cl > s && cl < hi)) continue;
        const int u = num[dir]++;
        a[u] = (T)rDa[e0 + k];
        w[u] = sweepCode(cl);
      }
      for (int h = 0; h < 2; ++h) {
        if (h == 1 && !out.more[dir].q) break;
        const T a3[3] = {a[3 * h], a[3 * h + 1], a[3 * h + 2]};
        const unsigned long long pack =
            (unsigned long long)w[3 * h] | ((unsigned long long)w[3 * h + 1] << 18) |
            ((unsigned long long)w[3 * h + 2] << 36) |
            ((unsigned long long)(h == 0 && num[dir] > 3 ? 1 : 0) << 54);
        (h == 0 ? out.sweep[dir] : out.more[dir]).put(i, a3, pack);
      }
    }
  cnt[i] = (uint32_t)n;
  const_cast<T*>(out.diag)[i] = (T)diag[s];
  const_cast<T*>(out.rD)[i] = (T)rD[s];
}

template <typename T, int OCC>
const void* resKernel(int mode) {
  constexpr int NT = kResThreads;
  if constexpr (sizeof(T) == 4) {  // (FP64 has the exact DIC only)
    if (mode == kResLocal) return (const void*)kResPcg<T, NT, kResLocal, OCC>;
    if (mode == kResDiag) return (const void*)kResPcg<T, NT, kResDiag, OCC>;
  }
  return mode == kResExact ? (const void*)kResPcg<T, NT, kResExact, OCC>
                           : (const void*)kResPcg<T, NT, kResSingle, OCC>;
}
template <typename T>
const void* resKernelOf(int mode, int occ) {
  return occ == 2 ? resKernel<T, 2>(mode) : resKernel<T, 1>(mode);
}

int resMode(bool diag, const ResView& rv) {
  return diag ? kResDiag : rv.local ? kResLocal : rv.single ? kResSingle : kResExact;
}

}  // namespace

template <typename T>
size_t resSmemBytes(const ResView& rv, int place) {
  const size_t mr = rv.maxRows;
  size_t b = (size_t)URow<T>::kBytes * rv.uRows + (rv.local ? kResGroupBytes + 2 * ((mr + 7) / 8 * 8) : 0) +
             sizeof(int2) * (size_t)((rv.nLev + 5) / 2 * 2);
  if (place & 1) b += sizeof(T) * 12 * mr;
  b += (rv.more ? 2 : 1) * (sizeof(typename ResSweepTab<T>::Q) + sizeof(typename ResSweepTab<T>::R)) *
       (size_t)((place & 2) ? 2 * (rv.single ? rv.uRows : mr) : kResAhead * rv.ring);
  if (place & 4) b += (kResW * (sizeof(T) + 4) + 2 * sizeof(T) + 4) * mr;
  return b;
}

// The largest set of {vectors, sweep tables, product tables} that fits beside the
// row vector in `limit` bytes; -1 if not even the row vector does.
template <typename T>
int resPlacement(const ResView& rv, size_t limit) {
  for (int place : {7, 3, 2, 5, 1, 0})
    if (resSmemBytes<T>(rv, place) <= limit) return place;
  return -1;
}

namespace {
template <typename T>
cudaLaunchConfig_t resConfig(const ResView& rv, int nCases, cudaStream_t s, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cf{};
  cf.gridDim = dim3(rv.C, nCases);
  cf.blockDim = dim3(kResThreads);
  cf.dynamicSmemBytes = resSmemBytes<T>(rv, rv.place);
  cf.stream = s;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = rv.C; at->val.clusterDim.y = 1; at->val.clusterDim.z = 1;
  cf.attrs = at;
  cf.numAttrs = 1;
  return cf;
}
}  // namespace

template <typename T>
cudaError_t resPrepare(const ResView& rv, int* clusters) {
  *clusters = 1 << 30;
  for (int occ = 1; occ <= 2; ++occ)
    for (int diag = 0; diag < (sizeof(T) == 4 ? 2 : 1); ++diag) {
      const void* k = resKernelOf<T>(resMode(diag != 0, rv), occ);
      int dev = 0, optin = 0;
      cudaError_t e = cudaGetDevice(&dev);
      if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
      cudaFuncAttributes fa;
      if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 optin - (int)fa.sharedSizeBytes);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e != cudaSuccess) return e;
      cudaLaunchAttribute at[1];
      const cudaLaunchConfig_t cf = resConfig<T>(rv, 1, nullptr, at);
      int n = 0;
      e = cudaOccupancyMaxActiveClusters(&n, k, &cf);
      if (e != cudaSuccess) return e;
      *clusters = std::min(*clusters, n);
    }
  return cudaSuccess;
}

template <typename T>
cudaError_t launchResPcg(const MeshView& mv, const Controls& c, const ResView& rv,
                         const ResPtrs<T>& rp, const PcgPtrs<T>& p, DevState* st, double* partials,
                         cudaStream_t s, int nCases, bool many) {
  cudaLaunchAttribute at[1];
  const cudaLaunchConfig_t cf = resConfig<T>(rv, nCases, s, at);
  void* args[] = {(void*)&mv, (void*)&c, (void*)&rv, (void*)&rp, (void*)&p, (void*)&st,
                  (void*)&partials};
  return cudaLaunchKernelExC(&cf, resKernelOf<T>(resMode(c.precond != 0, rv), many ? 2 : 1), args);
}

template <typename T>
void launchResTables(const MeshView& mv, const ResView& rv, const int* pos, const double* val,
                     const double* diag, const double* rD, const double* rDa, bool diagOnly,
                     const ResPtrs<T>& out, cudaStream_t s) {
  kResTables<T><<<(mv.nC + 255) / 256, 256, 0, s>>>(mv, rv, pos, val, diag, rD, rDa,
                                                    diagOnly ? 1 : 0, const_cast<uint32_t*>(rv.col),
                                                    const_cast<uint32_t*>(rv.cnt), out);
}

#define S4G_INSTANTIATE(T)                                                                     \
  template size_t resSmemBytes<T>(const ResView&, int);                                        \
  template int resPlacement<T>(const ResView&, size_t);                                        \
  template cudaError_t resPrepare<T>(const ResView&, int*);                                    \
  template cudaError_t launchResPcg<T>(const MeshView&, const Controls&, const ResView&,       \
                                       const ResPtrs<T>&, const PcgPtrs<T>&, DevState*,        \
                                       double*, cudaStream_t, int, bool);                      \
  template void launchResTables<T>(const MeshView&, const ResView&, const int*, const double*, \
                                   const double*, const double*, const double*, bool,          \
                                   const ResPtrs<T>&, cudaStream_t);
S4G_INSTANTIATE(double)
S4G_INSTANTIATE(float)
#undef S4G_INSTANTIATE

}  // namespace s4g
