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
// Every vector entry is computed by the operations of the separate kernels
// in the same order (to the last bit).  The global sums are, in FP32, the same
// compensated sums per thread, added up in FP64, in an order that depends on
// the mesh and the value type only; in FP64 they are those of kernels_pcg.cu
// bit for bit (orderedSum below).  Rows have at most kResW neighbours
// (hexahedra, prisms, tetrahedra); other meshes, and those whose shared row
// vector does not fit, run the separate kernels.  So does FP64 with the
// processor-local DIC or the diagonal preconditioner.

#include <algorithm>

#include "kernels.cuh"
#include "pcg_common.cuh"
#include "sweep.cuh"

namespace s4g {
namespace {

// Forms: exact DIC with a cluster barrier per level, processor-local DIC,
// diagonal, exact DIC with the substitutions inside one CTA.
enum { kResExact = 0, kResLocal = 1, kResDiag = 2, kResSingle = 3 };

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

// Cluster-wide sum of N <= M values of every thread: warp sums, the CTA's sum
// by warp 0, which stores it in a slot of every CTA's `rec` (rank order), and
// after the cluster barrier warp 0 of each CTA adds the slots in that order:
// all CTAs get the same bits.  The sums are left in out[0..N) for warp 0; the
// caller synchronises the CTA before other warps read what it derives.
template <typename T, int NT, int N, int M>
__device__ __forceinline__ void clusterSum(typename Part<T>::V (&v)[M], typename Part<T>::V* wrec,
                                           typename Part<T>::V* rec, double* out, int C,
                                           unsigned rank, bool cluster) {
  constexpr int W = NT / 32, G = 32 / M;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int k = lane / G, g = lane % G;  // the value a lane holds, its copy
  const typename Part<T>::V s = warpSpreadSum<T, M>(v);
  if (k < N && g == 0) wrec[wid * N + k] = s;
  __syncthreads();
  if (wid == 0) {
    const typename Part<T>::V a = warpRecords<T, N, M>(wrec, W);
    if (!cluster) {
      if (k < N && g == 0) out[k] = Part<T>::value(a);
    } else if (k < N) {
      const unsigned at = (unsigned)__cvta_generic_to_shared(rec + (int)rank * N + k);
      for (int j = g; j < C; j += G) stRemote(mapa(at, (unsigned)j), a);
    }
    __syncwarp();
  }
  if (cluster) {
    clArrive();
    clWait();
    if (wid == 0) {
      const typename Part<T>::V a = warpRecords<T, N, M>(rec, C);
      if (k < N && g == 0) out[k] = Part<T>::value(a);
      __syncwarp();
    }
  }
}

// Barrier between phases: of the cluster, or of its only CTA.
__device__ __forceinline__ void phaseBarrier(bool cluster) {
  if (cluster) { clArrive(); clWait(); }
  else __syncthreads();
}

// The FP64 form's sums.  The corrector loop can amplify a last bit of w.r or p.q
// a thousandfold every ten correctors (a processor-local 17 x 14 x 14 run: 1e-13
// after 60 correctors, 2e-6 after 100; exact DIC, 23 x 16 x 19: 2e-7 after 35), so
// they are added up in the order of kernels_pcg.cu: w.r by part, 64 lanes that
// take a row of each level, last level first, then by parts; sum|r| and p.q by
// storage row, 256 rows a block, then by blocks.  The CTAs own rows in another
// order, so rows go through global memory (L2), a warp takes 32 lanes of a part or
// 32 rows, and every CTA adds up the records.  Two cluster barriers a sum instead
// of one: cube of 8, exact DIC, 26 -> 30 us an iteration.
__device__ __forceinline__ double warpTree(double v) {  // in lane 0
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
// w.r of component k over 32 lanes of a part (w and r by PCG row): the lanes' rows
// in the order of their sums, a step at a time (ResView::ordRow), the rows of
// kOrdAhead steps read while those before them are added.
constexpr int kOrdAhead = 8;
__device__ __forceinline__ double ordPart(const int* rowOf, int steps, const double* w, const double* r,
                                          int k) {
  constexpr int B = kOrdAhead;
  const int* const at = rowOf + (threadIdx.x & 31);
  double s = 0, wv[B], rv[B];
  auto read = [&](int n0, double (&wn)[B], double (&rn)[B]) {
    int q[B];
#pragma unroll
    for (int u = 0; u < B; ++u) q[u] = n0 + u < steps ? __ldg(at + 32 * (n0 + u)) : -1;
#pragma unroll
    for (int u = 0; u < B; ++u) {
      wn[u] = q[u] >= 0 ? __ldcg(w + 3 * (size_t)q[u] + k) : 0.0;
      rn[u] = q[u] >= 0 ? __ldcg(r + 3 * (size_t)q[u] + k) : 0.0;
    }
  };
  read(0, wv, rv);
  for (int n = 0; n < steps; n += B) {
    double wn[B], rn[B];
    read(n + B, wn, rn);
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (n + u < steps) s = fma(wv[u], rv[u], s);
#pragma unroll
    for (int u = 0; u < B; ++u) { wv[u] = wn[u]; rv[u] = rn[u]; }
  }
  return warpTree(s);
}
// The sums over 32 storage rows of three values a row: value k in lane 8 k
template <bool ABS>
__device__ __forceinline__ double ordRows(const int* pos, const double* a, int nC, int g) {
  const int s = 32 * g + (int)(threadIdx.x & 31);
  const size_t q = 3 * (size_t)(s < nC ? __ldg(pos + s) : 0);
  double v[4] = {0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double x = s < nC ? __ldcg(a + q + k) : 0.0;
    v[k] = ABS ? fabs(x) : x;
  }
  return warpSpreadSum<double, 4>(v);
}
// The sum over the row records, of component k, blocks 32 h ... (and every 256th
// after them)
__device__ __forceinline__ double ordBlocks(const double* rec, int nC, int k, int h) {
  const int nB = (nC + kRowBlock - 1) / kRowBlock, nG = (nC + 31) / 32;
  double v = 0;
  for (int b = 32 * h + (int)(threadIdx.x & 31); b < nB; b += kRowBlock) {
    double x[kRowBlock / 32], t = 0;
#pragma unroll
    for (int j = 0; j < kRowBlock / 32; ++j) {
      const int g = b * (kRowBlock / 32) + j;
      x[j] = g < nG ? __ldcg(rec + 3 * (size_t)g + k) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kRowBlock / 32; ++j) t += x[j];
    v += t;
  }
  return warpTree(v);
}
// The sum over the part records of component k
__device__ __forceinline__ double ordParts(const double* rec, int nParts, int k) {
  const int lane = (int)(threadIdx.x & 31);
  double b = 0;
  for (int j = 0; 32 * j < nParts && j < 8; ++j) {
    double a = 0;
    for (int p = lane + 32 * j; p < nParts; p += 256) {
      const double x = __ldcg(rec + 6 * (size_t)p + k), y = __ldcg(rec + 6 * (size_t)p + 3 + k);
      a += x + y;
    }
    b += a;
  }
  return warpTree(b);
}
// DOTS: w.r by part and sum|r| (w, r by PCG row) into out[0..5]; else the terms w by
// storage row into out[0..2].  The rows' values are written; out is complete for the
// lanes 0 .. 2 of warp 0.
template <int NT, bool DOTS>
__device__ __forceinline__ void orderedSum(const MeshView& mv, const ResView& rv, const double* w,
                                           const double* r, double* rec, double* blk, double* out,
                                           int C, unsigned rank, bool cluster) {
  constexpr int W = NT / 32;
  const int lane = (int)threadIdx.x & 31, wid = (int)threadIdx.x >> 5;
  const int nG = (mv.nC + 31) / 32, nP = DOTS ? 6 * mv.nParts : 0;
  double* const rows = rec + 6 * (size_t)mv.nParts + (DOTS ? 0 : 3 * (size_t)nG);
  phaseBarrier(cluster);
  for (int q = (int)rank + C * wid; q < nP + nG; q += C * W) {
    if (q < nP) {
      const int task = q / 3, n0 = rv.ordStep[task];
      const double s = ordPart(rv.ordRow + 32 * (size_t)n0, rv.ordStep[task + 1] - n0, w, r, q % 3);
      if (lane == 0) rec[q] = s;
    } else {
      const double s = ordRows<DOTS>(rv.pos, DOTS ? r : w, mv.nC, q - nP);
      if ((lane & 7) == 0 && lane < 24) rows[3 * (size_t)(q - nP) + (lane >> 3)] = s;
    }
  }
  phaseBarrier(cluster);
  const int nB = (mv.nC + kRowBlock - 1) / kRowBlock, nH = nB < kRowBlock ? (nB + 31) / 32 : W;
  for (int q = wid; q < (DOTS ? 3 : 0) + 3 * nH; q += W) {
    if (DOTS && q < 3) {
      const double s = ordParts(rec, mv.nParts, q);
      if (lane == 0) blk[24 + q] = s;
    } else {
      const int k = (q - (DOTS ? 3 : 0)) % 3, h = (q - (DOTS ? 3 : 0)) / 3;
      const double s = ordBlocks(rows, mv.nC, k, h);
      if (lane == 0) blk[3 * h + k] = s;
    }
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double s = 0;
    for (int h = 0; h < nH; ++h) s += blk[3 * h + lane];
    out[(DOTS ? 3 : 0) + lane] = s;
    if (DOTS) out[lane] = blk[24 + lane];
  }
}

// Scalars of the iteration, in shared memory, decided by warp 0.
template <typename T>
struct ResScalars {
  double sum[8];
  double blk[27];  // (ordered sums)
  double norm[3], lim[3], last[3], wArA[3], alpha[3], beta[3];
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
  constexpr bool ORD = sizeof(T) == 8;
  using P = Part<T>;
  using V = typename P::V;
  p = casePcg(p, blockIdx.y, mv.nC);
  st += blockIdx.y;
  double* const ordRec = partials + (size_t)blockIdx.y * mv.caseRec + mv.ordOff;
  if (!st->pcgContinue) return;  // the same in every CTA: rank 0 writes it at the end
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ ResScalars<T> sc;
  constexpr int W = NT / 32;
  constexpr int kRows = 2;  // rows of a thread in flight
  constexpr unsigned kU = URow<T>::kBytes;
  const int C = (int)gridDim.x, t = (int)threadIdx.x;
  const bool cluster = C > 1;
  const unsigned rank = cluster ? clRank() : 0u;
  const int base = rv.chunk[rank], R = rv.chunk[rank + 1] - base;
  const int mr = rv.maxRows;
  // ---- shared memory: u and its zero row | sum records | level starts |
  //      vectors | tables
  unsigned char* sp = smraw;
  const unsigned uBase = (unsigned)__cvta_generic_to_shared(sp);
  sp += (size_t)kU * rv.uRows;
  V* wrec = (V*)sp;  // warp records, then the CTAs' records of the two sums
  sp += sizeof(V) * 6 * W;
  V* rec0 = (V*)sp;
  sp += sizeof(V) * 6 * kResMaxCtas;
  V* rec1 = (V*)sp;
  sp += sizeof(V) * 3 * kResMaxCtas;
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
    sc.wArA[t] = st->wArA[t]; sc.alpha[t] = 0; sc.beta[t] = 0; sc.alphaT[t] = T(0); sc.betaT[t] = T(0);
    sc.active[t] = st->active[t]; sc.pend[t] = 0; sc.nIter[t] = 0;
    const T z[3] = {T(0), T(0), T(0)};
    if (t == 0) URow<T>::store(uBase + kU * (rv.uRows - 1), z);
  }
  if (t == 0) { sc.any = 1; sc.iters = 0; sc.status = 0; }
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
    Acc<T> ar[3], wr[3];
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
            if (!ORD) ar[k].add(fabs(rr[h][k]));
            w[k] = mulT(rd[h], rr[h][k]);
            if (MODE == kResDiag) wr[k].add(mulT(w[k], rr[h][k]));
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
    if (MODE != kResDiag)
      for (int i = t; i < R; i += NT) {
        T w[3];
        if (MODE == kResSingle && cluster) {
          URow<T>::loadCluster(wBase + kU * i, w);
          if (rank != 0) URow<T>::store(uBase + kU * i, w);  // rank 0's rows are in place
        } else {
          URow<T>::load(uBase + kU * i, w);
        }
        if (ORD) {
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            wGlob[3 * (size_t)i + k] = w[k];
            if (rv.place & 1) rGlob[3 * (size_t)i + k] = rg[3 * i + k];
          }
        } else {
#pragma unroll
          for (int k = 0; k < 3; ++k) wr[k].add(mulT(w[k], rg[3 * i + k]));
        }
      }
    if constexpr (ORD) {
      orderedSum<NT, true>(mv, rv, p.w, p.r, ordRec, sc.blk, sc.sum, C, rank, cluster);
    } else {
      V v[8] = {P::of(wr[0]), P::of(wr[1]), P::of(wr[2]), P::of(ar[0]),
                P::of(ar[1]), P::of(ar[2]), P::zero(), P::zero()};
      clusterSum<T, NT, 6>(v, wrec, rec0, sc.sum, C, rank, cluster);
    }
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
    Acc<T> pq[3];
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
            if (ORD) wGlob[3 * (size_t)i + k] = mulT(y[k], v[k]);
            else pq[k].add(mulT(y[k], v[k]));
          }
        }
      }
    }
    if constexpr (ORD) {
      orderedSum<NT, false>(mv, rv, p.w, nullptr, ordRec, sc.blk, sc.sum, C, rank, cluster);
    } else {
      V v[4] = {P::of(pq[0]), P::of(pq[1]), P::of(pq[2]), P::zero()};
      clusterSum<T, NT, 3>(v, wrec, rec1, sc.sum, C, rank, cluster);
    }
    if (t < 32) {
      int on = 0;
      unsigned bad = 0;
      if (t < 3) {
        sc.pend[t] = 0;
        if (sc.active[t]) {
          const double s = sc.sum[t];
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
      st->wArA[k] = sc.wArA[k]; st->alpha[k] = sc.alpha[k]; st->beta[k] = sc.beta[k];
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
  const size_t W = kResThreads / 32, mr = rv.maxRows;
  size_t b = (size_t)URow<T>::kBytes * rv.uRows +
             sizeof(typename Part<T>::V) * (6 * W + 9 * kResMaxCtas) +
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
