// PCG with the processor-local DIC on the whole device, a CTA per part, for meshes
// beyond the cluster-resident PCG; in FP32 three kernels per iteration:
//
//   kPartPrecond  r -= alpha q of the pending iteration, sum|r|, w = M^-1 r of
//                 each part and w.r; the last CTA runs the residual test and
//                 decides beta.
//   kPartSpmv     the pending x += alpha p, p_new = w + beta p_old, q = A p_new.
//   kPartDot      p.q; the last CTA decides alpha.
//
// The first two hold a part's rows in shared memory while they work on it: w during
// the substitutions, p_new -- of the part's rows and of the rows around it that
// they touch -- during the product, so that a row's six neighbours are shared-
// memory reads instead of gathers of w and p_old through L1.  In FP64 the product
// stays with kernels_local.cu.
//
// The arithmetic of every vector entry is that of the separate kernels
// (kernels_local.cu), and so is that of the global sums, to the bit: w.r and sum|r| by
// 64 lanes over a part's rows, parts in groups of 32 (part_sums.cuh); p.q by storage
// row, the rows of a thread of the row kernels' grid together, blocks of 256 threads.
// The corrector loop of some runs amplifies a last bit of a sum a thousandfold every
// ten correctors (FP64: 1e-13 after 60, 2e-6 after 100), and in FP32 a last bit of the
// FP64 sum can turn the rounding of alpha or beta.
//
// Parts of rows with at most six neighbours that fit shared memory (in FP32
// at most 1016 rows: 10-bit columns); others run kernels_local.cu.

#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "pcg_common.cuh"
#include "part_sums.cuh"
#include "sweep.cuh"

namespace s4g {
namespace {

// Threads of a part's preconditioner: FP32 a thread per row of the widest
// levels (48 rows of an 8^3-cell part), FP64 one per row and component.
template <typename T> struct PartCfg;
template <> struct PartCfg<float> {
  using Ent = PartEnt;
  // (8 resident CTAs at 119 registers; with 6 at 139 a launch at 128^3 took 61.4 us for
  // 60.1, 16 cases of 40^3 39.4 for 35.5; with fewer rows a thread keeps 65 and 70 us.
  // The sums' order came after these: 128^3 68.1 us)
  static constexpr int kNT = 64, kKeep = 8, kOcc = 7;
  static constexpr bool kSplit = false;
};
template <> struct PartCfg<double> {
  using Ent = ResEnt<double>;
  static constexpr int kNT = 192, kKeep = 3, kOcc = 4;
  static constexpr bool kSplit = true;
};
constexpr int kPartSpmvThreads = 128;

template <typename T>
__device__ __forceinline__ void ldRow(const T* v, size_t i, T (&o)[3]) {
  o[0] = v[3 * i]; o[1] = v[3 * i + 1]; o[2] = v[3 * i + 2];
}
template <typename T>
__device__ __forceinline__ void stRow(T* v, size_t i, const T (&o)[3]) {
  v[3 * i] = o[0]; v[3 * i + 1] = o[1]; v[3 * i + 2] = o[2];
}

template <typename T, bool MORE, bool WIDE>
__global__ void __launch_bounds__(PartCfg<T>::kNT, PartCfg<T>::kOcc)
kPartPrecond(MeshView mv, Controls c, PartView pv, PartPtrs<T> pt, PcgPtrs<T> p, DevState* st,
             double* partials) {
  using C = PartCfg<T>;
  using E = typename C::Ent;
  constexpr int NT = C::kNT, KR = C::kKeep;
  // the sums' 64 lanes: lane l the rows l, l + 64, ... of a part.  With 64 threads they
  // are the thread's own rows.
  constexpr bool OWN = NT == 64;
  constexpr unsigned kU = URow<T>::kBytes, kB = E::kB;
  p = casePcg(p, blockIdx.y, mv.nC);
  st += blockIdx.y;
  partials += (size_t)blockIdx.y * mv.caseRec;
  if (!st->pcgContinue) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ __align__(16) int4 sDesc[2][2];
  __shared__ double sum[12];
  __shared__ int sGroup;
  const int t = (int)threadIdx.x, cap = pv.capRows;
  // w and its zero row | tables forward, backward | level bounds
  const unsigned uBase = (unsigned)__cvta_generic_to_shared(smraw);
  ResAddr ad[2];
  unsigned at = uBase + kU * (unsigned)(cap + 4);
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    ad[d].q = at; at += 16u * cap;
    ad[d].r = at; at += kB * cap;
    if (MORE) {
      ad[d].mq = at; at += 16u * cap;
      ad[d].mr = at; at += kB * cap;
    }
  }
  const unsigned lva = at + 16;  // two empty levels before the first
  // (not OWN) the part's residual, in the tables' place after the sweeps
  T* const sr = (T*)(smraw + (ad[0].q - uBase));
  double* grec = partials + mv.locGrpOff;
  unsigned* gcnt = reinterpret_cast<unsigned*>(grec + 8 * (size_t)mv.locGroups);
  const T* __restrict__ qg = p.q;
  const T* __restrict__ rDg = p.rD;
  T* __restrict__ rg = p.r;
  bool pend[3];
  T al[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) { pend[k] = st->pending[k] != 0; al[k] = (T)st->alpha[k]; }
  const bool anyPend = pend[0] || pend[1] || pend[2];
  const int nParts = mv.nParts;
  if (t == 0) {
    const T z[3] = {T(0), T(0), T(0)};
    URow<T>::store(uBase + kU * (unsigned)pv.zeroRow, z);
  }
  int part = (int)blockIdx.x;
  if (t == 0 && part < nParts) {
    cpAsync16(&sDesc[0][0], mv.locDesc + 2 * part);
    cpAsync16(&sDesc[0][1], mv.locDesc + 2 * part + 1);
  }
  cpAsyncWaitAll();
  __syncthreads();
  for (int buf = 0; part < nParts; part += (int)gridDim.x, buf ^= 1) {
    const int4 dA = sDesc[buf][0], dB = sDesc[buf][1];
    const int pLo = dA.x, nR = dA.y, l0 = dB.z, nL = dB.w;
    const int next = part + (int)gridDim.x;
    if (t == 0 && next < nParts) {
      cpAsync16(&sDesc[buf ^ 1][0], mv.locDesc + 2 * next);
      cpAsync16(&sDesc[buf ^ 1][1], mv.locDesc + 2 * next + 1);
    }
    // the part's tables in flight while the vectors stream
    for (int i = t; i < nR; i += NT)
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        E::fetch(ad[d].q + 16u * i, ad[d].r + kB * i, pt.sweep[d], pLo + i);
        if (MORE) E::fetch(ad[d].mq + 16u * i, ad[d].mr + kB * i, pt.more[d], pLo + i);
      }
    for (int l = t; l < nL + 4; l += NT) {
      int2 b = make_int2(0, 0);
      if (l >= 2 && l < nL + 2)
        b = make_int2(mv.lvlStart[l0 + l - 2] - pLo, mv.lvlStart[l0 + l - 1] - pLo);
      asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(lva - 16 + 8u * l), "r"(b.x), "r"(b.y) : "memory");
    }
    // pending r -= alpha q and w = rD r, every load of the thread's first KR
    // rows before any store; their residual stays in registers
    T rK[KR][3];
    {
      T qv[KR][3], rd[KR];
#pragma unroll
      for (int j = 0; j < KR; ++j) {
        const int i = t + j * NT;
        if (i < nR) {
          const size_t g = 3 * (size_t)(pLo + i);
          rd[j] = rDg[pLo + i];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            rK[j][k] = rg[g + k];
            if (pend[k]) qv[j][k] = qg[g + k];
          }
        }
      }
#pragma unroll
      for (int j = 0; j < KR; ++j) {
        const int i = t + j * NT;
        if (i < nR) {
          const size_t g = 3 * (size_t)(pLo + i);
          T w[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            if (pend[k]) {
              rK[j][k] = fmaT(-al[k], qv[j][k], rK[j][k]);
              rg[g + k] = rK[j][k];
            }
            w[k] = mulT(rd[j], rK[j][k]);
          }
          URow<T>::store(uBase + kU * (unsigned)i, w);
        }
      }
    }
    for (int i = t + KR * NT; i < nR; i += NT) {  // parts of more rows
      const size_t g = 3 * (size_t)(pLo + i);
      const T rd = rDg[pLo + i];
      T w[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        T rv = rg[g + k];
        if (pend[k]) {
          rv = fmaT(-al[k], qg[g + k], rv);
          rg[g + k] = rv;
        }
        w[k] = mulT(rd, rv);
      }
      URow<T>::store(uBase + kU * (unsigned)i, w);
    }
    cpAsyncWaitAll();
    __syncthreads();
    if (nL > 1) {
      resSweepBody<0, false, false, C::kSplit, MORE, WIDE, E>(pt.sweep[0], pt.more[0], ad[0], uBase, 0u,
                                                              lva, nL, NT, 0);
      resSweepBody<1, false, false, C::kSplit, MORE, WIDE, E>(pt.sweep[1], pt.more[1], ad[1], uBase, 0u,
                                                              lva, nL, NT, 0);
    }
    // w out, w.r and sum|r| of the lane's rows in row order
    Acc<T> wr[3], ar[3];
#pragma unroll
    for (int j = 0; j < KR; ++j) {
      const int i = t + j * NT;
      if (i < nR) {
        T w[3];
        URow<T>::load(uBase + kU * (unsigned)i, w);
        stRow(p.w, (size_t)(pLo + i), w);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (OWN) {
            wr[k].add(mulT(w[k], rK[j][k]));
            ar[k].add(fabs(rK[j][k]));
          } else {
            sr[3 * i + k] = rK[j][k];
          }
        }
      }
    }
    for (int i = t + KR * NT; i < nR; i += NT) {
      T w[3];
      URow<T>::load(uBase + kU * (unsigned)i, w);
      stRow(p.w, (size_t)(pLo + i), w);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const T r = rg[3 * (size_t)(pLo + i) + k];  // written by this thread
        if (OWN) {
          wr[k].add(mulT(w[k], r));
          ar[k].add(fabs(r));
        } else {
          sr[3 * i + k] = r;
        }
      }
    }
    if (!OWN) __syncthreads();
    // then a fixed tree: sum64's
    // w.r of component k in lane 8 k, sum|r| in lane 8 k + 1
    const int l8 = t & 7, k3 = (t & 31) >> 3;
    double s6 = 0;
    if (t < 64) {
      double d[2];
      if constexpr (OWN) {
        const T x[2][3] = {{wr[0].s, wr[1].s, wr[2].s}, {ar[0].s, ar[1].s, ar[2].s}};
        const T e[2][3] = {{wr[0].c, wr[1].c, wr[2].c}, {ar[0].c, ar[1].c, ar[2].c}};
        warpFloatSums<2, true>(x, e, d);
      } else {
        double v[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
        for (int i = t; i < nR; i += 64) {
          T w[3];
          URow<T>::load(uBase + kU * (unsigned)i, w);
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const T r = sr[3 * i + m];
            v[0][m] = fma((double)w[m], (double)r, v[0][m]);
            v[1][m] += fabs((double)r);
          }
        }
        warpSpreadSums<4, 2>(v, d);
      }
      s6 = l8 == 0 ? d[0] : d[1];
      if (t >= 32 && l8 < 2 && k3 < 3) sum[3 * l8 + k3] = s6;
    }
    __syncthreads();  // the next part reuses the vector and the tables
    if (t < 32 && l8 < 2 && k3 < 3) partials[8 * (size_t)part + 3 * l8 + k3] = s6 + sum[3 * l8 + k3];
  }
  // the records are reported on their groups' counters at the end (a fence for every part
  // would wait for the part's w to drain, some 1.5 us each)
  if (t < 32) {
    __syncwarp();
    const int step = (int)gridDim.x;
    for (int p0 = (int)blockIdx.x; p0 < nParts; p0 += 32 * step) {
      const long mine = p0 + (long)t * step;
      unsigned full = __ballot_sync(0xffffffffu, mine < nParts && locArrive(gcnt, (int)mine, nParts));
      for (; full; full &= full - 1)
        locGroupSum(partials, grec, gcnt, (p0 + (__ffs((int)full) - 1) * step) / kLocGroup, nParts);
    }
  }
  __syncthreads();
  locFinish(mv, c, st, partials, -1, anyPend, sum, &sGroup);
}

__global__ void __launch_bounds__(kPartSpmvThreads, 8)
kPartSpmv(MeshView mv, PartView pv, PartPtrs<float> pt, PcgPtrs<float> p, const DevState* st) {
  using T = float;
  constexpr int NT = kPartSpmvThreads, RP = 1, KH = 4;
  constexpr unsigned kU = URow<T>::kBytes;
  p = casePcg(p, blockIdx.y, mv.nC);
  st += blockIdx.y;
  if (!st->pcgContinue) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  const unsigned uBase = (unsigned)__cvta_generic_to_shared(smraw);
  const int t = (int)threadIdx.x;
  const int pb = st->pbuf;
  const T* __restrict__ po = pb ? p.p2 : p.p;
  T* __restrict__ pn = pb ? p.p : p.p2;
  const T* __restrict__ wv = p.w;
  T* __restrict__ qo = p.q;
  T* __restrict__ xg = p.x;
  bool act[3], first[3], xp[3];
  T b[3], al[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    act[k] = st->active[k] != 0; first[k] = st->nIter[k] == 0; b[k] = (T)st->beta[k];
    xp[k] = st->xPend[k] != 0; al[k] = (T)st->alpha[k];
  }
  // the part's first row, rows and halo, read a part ahead
  int part = (int)blockIdx.x, pLo = 0, nR = 0, nH = 0;
  if (part < mv.nParts) {
    pLo = mv.partStart[part];
    nR = mv.partStart[part + 1] - pLo;
    nH = pv.haloCnt[part];
  }
  for (; part < mv.nParts;) {
    const int next = part + (int)gridDim.x;
    int pLo1 = 0, nR1 = 0, nH1 = 0;
    if (next < mv.nParts) {
      pLo1 = mv.partStart[next];
      nR1 = mv.partStart[next + 1];
      nH1 = pv.haloCnt[next];
    }
    const int* __restrict__ hi = pv.halo + (size_t)part * pv.haloCap;
    int hx[KH];  // the rows of the thread's first halo places
#pragma unroll
    for (int j = 0; j < KH; ++j) hx[j] = t + j * NT < nH ? hi[t + j * NT] : -1;
    // a row's coefficients are read a row ahead, the first one's while p_new is
    // formed
    T aN[kResW], dgN = T(0);
    unsigned short clN[kResW];
    auto coefs = [&](int i) {
      if (i >= nR) return;
      dgN = p.diag[pLo + i];
#pragma unroll
      for (int e = 0; e < kResW; ++e) {
        clN[e] = pv.slot[(size_t)e * mv.nC + pLo + i];
        aN[e] = pt.val[(size_t)e * mv.nC + pLo + i];
      }
    };
    coefs(t);
    // p_new of the part's rows and of the rows around it
    for (int i0 = t; i0 < nR; i0 += RP * NT) {
      T w[RP][3], o[RP][3], x[RP][3];
#pragma unroll
      for (int h = 0; h < RP; ++h) {
        const int i = i0 + h * NT;
        const size_t g = 3 * (size_t)(pLo + i);
        if (i < nR) {
          ldRow(wv, (size_t)(pLo + i), w[h]);
          ldRow(po, (size_t)(pLo + i), o[h]);
#pragma unroll
          for (int k = 0; k < 3; ++k)
            if (xp[k]) x[h][k] = xg[g + k];
        }
      }
#pragma unroll
      for (int h = 0; h < RP; ++h) {
        const int i = i0 + h * NT;
        const size_t g = 3 * (size_t)(pLo + i);
        if (i < nR) {
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            if (xp[k]) xg[g + k] = fmaT(al[k], o[h][k], x[h][k]);
            if (!first[k]) w[h][k] = fmaT(b[k], o[h][k], w[h][k]);
          }
          // (a stopped component's p is not read again: its x is complete
          // with this pass)
          stRow(pn, (size_t)(pLo + i), w[h]);
          URow<T>::store(uBase + kU * (unsigned)i, w[h]);
        }
      }
    }
#pragma unroll
    for (int j0 = 0; j0 < KH; j0 += RP) {
      T w[RP][3], o[RP][3];
#pragma unroll
      for (int h = 0; h < RP; ++h)
        if (hx[j0 + h] >= 0) {
          ldRow(wv, (size_t)hx[j0 + h], w[h]);
          ldRow(po, (size_t)hx[j0 + h], o[h]);
        }
#pragma unroll
      for (int h = 0; h < RP; ++h)
        if (hx[j0 + h] >= 0) {
#pragma unroll
          for (int k = 0; k < 3; ++k)
            if (!first[k]) w[h][k] = fmaT(b[k], o[h][k], w[h][k]);
          URow<T>::store(uBase + kU * (unsigned)(nR + t + (j0 + h) * NT), w[h]);
        }
    }
    for (int h = t + KH * NT; h < nH; h += NT) {
      T v[3], o[3];
      ldRow(wv, (size_t)hi[h], v);
      ldRow(po, (size_t)hi[h], o);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (!first[k]) v[k] = fmaT(b[k], o[k], v[k]);
      URow<T>::store(uBase + kU * (unsigned)(nR + h), v);
    }
    __syncthreads();
    for (int i = t; i < nR; i += NT) {
      T a[kResW], v[3], y[3], x[kResW][3];
      const T dg = dgN;
      unsigned short cl[kResW];
#pragma unroll
      for (int e = 0; e < kResW; ++e) { a[e] = aN[e]; cl[e] = clN[e]; }
      coefs(i + NT);
      URow<T>::load(uBase + kU * (unsigned)i, v);
#pragma unroll
      for (int e = 0; e < kResW; ++e) URow<T>::load(uBase + kU * (unsigned)cl[e], x[e]);
#pragma unroll
      for (int k = 0; k < 3; ++k) y[k] = mulT(dg, v[k]);
#pragma unroll
      for (int e = 0; e < kResW; ++e)  // (padded: the row itself times zero)
#pragma unroll
        for (int k = 0; k < 3; ++k) y[k] = fmaT(a[e], x[e][k], y[k]);
      const size_t g = 3 * (size_t)(pLo + i);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (act[k]) qo[g + k] = y[k];
    }
    __syncthreads();
    part = next; pLo = pLo1; nR = nR1 - pLo1; nH = nH1;
  }
}

// p.q of the product, in the order of kLocSpmv: a thread the storage rows of the row
// kernels' grid, blocks of 256 threads, then the blocks.  (In the product itself the
// rows are by part.)  Reads q and p_new.  128^3: 20 us, 50 MB from DRAM; 64^3: 11 us,
// the latency of its chain (state, rows, block sums, the last block's total, alpha).
__global__ void __launch_bounds__(kRowBlock)
kPartDot(MeshView mv, PcgPtrs<float> p, DevState* st, double* partials) {
  p = casePcg(p, blockIdx.y, mv.nC);
  st += blockIdx.y;
  partials += (size_t)blockIdx.y * mv.caseRec;
  if (!st->pcgContinue) return;
  constexpr int W = kRowBlock / 32, B = 7;
  __shared__ double red[3 * W];
  const int t = (int)threadIdx.x, lane = t & 31, wid = t >> 5;
  const int pb = st->pbuf;
  const float* __restrict__ pn = pb ? p.p : p.p2;
  const float* __restrict__ q = p.q;
  const int step = (int)(gridDim.x * kRowBlock);
  Acc<float> a[3];
  for (int s0 = (int)blockIdx.x * kRowBlock + t; s0 < mv.nC; s0 += B * step) {
    float y[B][3], v[B][3];
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (s0 + u * step < mv.nC) {
        ldRow(q, (size_t)(s0 + u * step), y[u]);
        ldRow(pn, (size_t)(s0 + u * step), v[u]);
      }
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (s0 + u * step < mv.nC)
#pragma unroll
        for (int k = 0; k < 3; ++k) a[k].add(mulT(y[u][k], v[u][k]));
  }
  // blockSum's order, by the spread sum
  auto blockTotal = [&](double s) {  // value k in thread k, from the warps' sums in lanes 8 k
    if ((lane & 7) == 0 && lane < 24) red[3 * wid + (lane >> 3)] = s;
    __syncthreads();
    double o = 0;
    if (t < 3) {
      o = red[t];
#pragma unroll
      for (int w = 1; w < W; ++w) o += red[3 * w + t];
    }
    return o;
  };
  const float x[1][3] = {{a[0].s, a[1].s, a[2].s}}, cmp[1][3] = {{a[0].c, a[1].c, a[2].c}};
  double own[1];
  warpFloatSums<1, true>(x, cmp, own);
  const double mine = blockTotal(own[0]);
  if (t < 3) {
    partials[8 * (size_t)blockIdx.x + t] = mine;
    __threadfence();
  }
  if (!lastBlockDone(&st->counter[6], gridDim.x)) return;
  double v[4] = {0, 0, 0, 0};
  for (int j = t; j < (int)gridDim.x; j += kRowBlock)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double x = __ldcg(partials + 8 * (size_t)j + k);
      v[k] = j == t ? x : v[k] + x;
    }
  const double total = blockTotal(warpSpreadSum<4>(v));
  if (t >= 32) return;
  if (t == 0) st->counter[6] = 0;
  pcgDecideAlpha(st, total, pb);
}

// ---- the whole loop of a corrector in one launch ---------------------------------
// Meshes whose parts are all resident at once (a CTA per part; FP32): the
// launches of the part kernels, their reading of the state and their ends take longer
// than a part's work, so one cooperative launch runs the PCG loop of a corrector.
// r, x, p and q stay in registers, the tables in shared memory; the part's halo keeps
// its p in shared memory and needs only w from other parts once per iteration.
//
// What CTAs tell one another goes through 16-byte packets that carry their own
// tag (the count of sums so far): a reader polls the packet itself, so neither a
// counter nor a fence stands between a value and its use.  Rows publish w; a CTA
// publishes its records of a sum, CTA 0 adds the records up, decides and publishes the
// result in kLoopCopies lines.  A packet is written again only after its readers have
// taken part in a later sum.
//
// The sums have the order of kernels_local.cu (the comment at the top):
//   w.r, sum|r|  64 lanes over the part's rows, lane l the rows l, l + 64, ...: the
//                first half of them in thread l, the rest in thread l + 64, which goes
//                on with that thread's sum (sum|r|'s second half runs beside the walk).
//                A record of six values per part; CTA 0 adds up groups of 32 parts.
//   p.q          blocks of 256 storage rows, in each lane the rows a row kernels' grid
//                apart.  A block is added up by the CTA that owns its first row; the rows
//                of it that other CTAs own come as packets.
constexpr int kLoopThreads = 128, kLoopRows = 4, kLoopWalk = 64;
constexpr int kLoopMaxRows = kLoopThreads * kLoopRows;
constexpr int kLoopAhead = 2;  // part groups whose packets a warp of CTA 0 has in flight
constexpr int kLoopCopies = 32, kLoopLine = 8;  // result packets, 128 bytes apart

__device__ __forceinline__ uint4 ldPacket(const uint4* p) {
  unsigned long long a, b;
  asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
               : "=l"(a), "=l"(b) : "l"(p) : "memory");
  return make_uint4((unsigned)a, (unsigned)(a >> 32), (unsigned)b, (unsigned)(b >> 32));
}
__device__ __forceinline__ void stPacket(uint4* p, unsigned x, unsigned y, unsigned z, unsigned w) {
  const unsigned long long a = x | (unsigned long long)y << 32, b = z | (unsigned long long)w << 32;
  asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }"
               ::"l"(p), "l"(a), "l"(b) : "memory");
}
// The packet with this tag, after at most limit polls; false if it did not come.
// shift: bits of the last word below the tag.
__device__ __forceinline__ bool waitPacket(const uint4* p, unsigned tag, int shift, int limit, uint4& v) {
  v = ldPacket(p);
  for (int it = 0; (v.w ^ tag) >> shift; v = ldPacket(p))
    if (++it > limit) return false;
  return true;
}
// N packets with this tag (addr(n) null: none), polled together: one after the other,
// each would cost a round trip to L2 of its own once its first load came too early.
template <int N, typename F>
__device__ __forceinline__ bool waitPackets(F addr, unsigned tag, int limit, uint4 (&v)[N]) {
#pragma unroll
  for (int n = 0; n < N; ++n) v[n] = addr(n) ? ldPacket(addr(n)) : make_uint4(0, 0, 0, tag);
  for (int it = 0;;) {
    bool all = true;
#pragma unroll
    for (int n = 0; n < N; ++n) all = all && v[n].w == tag;
    if (all) return true;
    if (++it > limit) return false;
#pragma unroll
    for (int n = 0; n < N; ++n)
      if (v[n].w != tag) v[n] = ldPacket(addr(n));
  }
}
// FP64 values in packets: value k in the words 2 k, 2 k + 1; three words a packet.
__device__ __forceinline__ unsigned valueWord(double v, int w) {
  return (unsigned)((w & 1) ? __double2hiint(v) : __double2loint(v));
}
__device__ __forceinline__ double wordsValue(unsigned lo, unsigned hi) {
  return __hiloint2double((int)hi, (int)lo);
}
// CTA 0: the sum over the parts' records (value k in lane k of warp 0); false if some did
// not come.  grp: 6 values of each of 64 lanes over the groups; out: 6 values.
__device__ __forceinline__ bool loopPartTotal(const uint4* rec, int n, double* grp, double* out, unsigned tag,
                                              int limit, double& mine) {
  constexpr int W = kLoopThreads / 32, A = kLoopAhead;
  const int lane = (int)threadIdx.x & 31, wid = (int)threadIdx.x >> 5, nGrp = (n + 31) / 32;
  bool ok = true;
  for (int g0 = wid; g0 < nGrp; g0 += A * W) {
    uint4 x[4 * A];
    ok = waitPackets(
             [&](int i) {
               const int part = 32 * (g0 + i / 4 * W) + lane;
               return part < n ? rec + (size_t)(i % 4) * n + part : (const uint4*)nullptr;
             },
             tag, limit, x) && ok;
    double v[A][8], s[A];
#pragma unroll
    for (int u = 0; u < A; ++u) {
      const uint4 *const y = x + 4 * u;
      const double d[6] = {wordsValue(y[0].x, y[0].y), wordsValue(y[0].z, y[1].x), wordsValue(y[1].y, y[1].z),
                           wordsValue(y[2].x, y[2].y), wordsValue(y[2].z, y[3].x), wordsValue(y[3].y, y[3].z)};
#pragma unroll
      for (int k = 0; k < 8; ++k) v[u][k] = k < 6 ? d[k < 6 ? k : 0] : 0.0;
    }
    warpSpreadSums<8, A>(v, s);
#pragma unroll
    for (int u = 0; u < A; ++u) {
      const int g = g0 + u * W;
      if ((lane & 3) == 0 && lane < 24 && g < nGrp) {
        double* const o = grp + 6 * (g & 63) + (lane >> 2);
        *o = g < 64 ? s[u] : *o + s[u];
      }
    }
  }
  ok = __syncthreads_and(ok) != 0;
  groupTotal<W>(grp, nGrp, out);
  __syncthreads();
  if (lane < 6) mine = out[lane];
  return ok;
}
// CTA 0: the sum over the n row blocks' records (reducePartials with 256 threads), value k
// in lane k of warp 0.  red: 24 values.
__device__ __forceinline__ bool loopBlockTotal(const uint4* rec, int n, double* red, unsigned tag, int limit,
                                               double& mine) {
  constexpr int NT = kLoopThreads;
  const int t = (int)threadIdx.x, lane = t & 31, wid = t >> 5;
  bool ok = true;
  double v[2][4], s[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) v[h][0] = v[h][1] = v[h][2] = v[h][3] = 0;
  for (int j0 = t; j0 < n; j0 += kRowBlock) {
    uint4 x[4];
    ok = waitPackets(
             [&](int i) {
               const int j = j0 + NT * (i / 2);
               return j < n ? rec + (size_t)(i % 2) * n + j : (const uint4*)nullptr;
             },
             tag, limit, x) && ok;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 &y0 = x[2 * h], &y1 = x[2 * h + 1];
      const double d[3] = {wordsValue(y0.x, y0.y), wordsValue(y0.z, y1.x), wordsValue(y1.y, y1.z)};
#pragma unroll
      for (int k = 0; k < 3; ++k) v[h][k] = j0 == t ? d[k] : v[h][k] + d[k];
    }
  }
  warpSpreadSums<4, 2>(v, s);
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if ((lane & 7) == 0 && lane < 24) red[3 * (wid + 4 * h) + (lane >> 3)] = s[h];
  ok = __syncthreads_and(ok) != 0;
  if (t < 3) {
    double a = red[t];
#pragma unroll
    for (int w = 1; w < kRowBlock / 32; ++w) a += red[3 * w + t];
    mine = a;
  }
  return ok;
}
// The result of a sum: three values and flag bits beside the tag.  CTA 0 (the
// values in lanes 0 .. 2 of warp 0) writes the copies, the others poll theirs.
__device__ __forceinline__ void resultPut(uint4* out, unsigned tag, float v, unsigned flags) {
  const int lane = threadIdx.x & 31;
  const unsigned x = __float_as_uint(__shfl_sync(0xffffffffu, v, 0));
  const unsigned y = __float_as_uint(__shfl_sync(0xffffffffu, v, 1));
  const unsigned z = __float_as_uint(__shfl_sync(0xffffffffu, v, 2));
  stPacket(out + kLoopLine * lane, x, y, z, tag << 8 | flags);
}

template <bool MORE, bool WIDE>
__global__ void __launch_bounds__(kLoopThreads, 4)
kPartLoop(MeshView mv, Controls c, PartView pv, PartPtrs<float> pt, LoopPtrs lp, PcgPtrs<float> p,
          DevState* st) {
  using T = float;
  using E = PartEnt;
  constexpr int NT = kLoopThreads, KR = kLoopRows, KH = 4;
  constexpr unsigned kU = URow<T>::kBytes;
  if (!st->pcgContinue) return;  // the same in every CTA: CTA 0 writes the state at its end
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double grp[64 * 6];  // (CTA 0: sums over part groups); before that, in sums of
  float2* const hand = reinterpret_cast<float2*>(grp);  // lanes: the first halves' sums [3][64]
  __shared__ double red[6], blk[2][24];
  __shared__ T sVal[3];
  __shared__ unsigned sFlags;
  __shared__ DevState sst;  // CTA 0: the state while the loop runs
  const int t = (int)threadIdx.x, cap = pv.capRows, part = (int)blockIdx.x, nP = (int)gridDim.x;
  const int lane = t & 31, wid = t >> 5;
  const int pLo = mv.partStart[part], nR = mv.partStart[part + 1] - pLo, nH = pv.haloCnt[part];
  const int l0 = mv.lvlOff[part], nL = mv.lvlOff[part + 1] - l0;
  const bool lead = part == 0;
  const int limit = mv.packetLimit;
  // the thread's rows: i0, i0 + 64, ..., nMine of them
  const int half = (nR + 127) / 128, i0 = (t & 63) + (t >> 6) * 64 * half;
  const int nMine = i0 < nR ? min(half, (nR - i0 + 63) / 64) : 0;
  // the row blocks that the CTA adds up, the distance of a lane's rows
  const int nB = mv.rowGrid, stride = nB * kRowBlock, b0 = (pLo + kRowBlock - 1) / kRowBlock;
  const int nMyB = min((pLo + nR + kRowBlock - 1) / kRowBlock, nB) - b0;  // at most 2
  uint4* const rec2 = lp.rec + 4 * (size_t)nP;
  uint4* const out = rec2 + 2 * (size_t)nB;
  unsigned* const count = reinterpret_cast<unsigned*>(out + kLoopLine * kLoopCopies);
  unsigned tag = ldRelaxed(count);  // of the last sum; CTA 0 writes it at its end
  const uint4* const mine = out + kLoopLine * (part % kLoopCopies);
  // ---- shared memory: w, p or p.q's terms of the rows, the zero row, p of the halo |
  //      sweep tables | level bounds | product coefficients | product columns
  const unsigned uBase = (unsigned)__cvta_generic_to_shared(smraw);
  const int halo0 = cap + 4;
  ResAddr ad[2];
  unsigned at = uBase + kU * (unsigned)(halo0 + pv.haloCap);
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    ad[d].q = at; at += 16u * cap;
    ad[d].r = at;
    if (MORE) { ad[d].mq = at; at += 16u * cap; ad[d].mr = at; }
  }
  const unsigned lva = at + 16;
  T* const sval = (T*)(smraw + (at - uBase) + 8 * (mv.maxLevels + 5));
  unsigned short* const sslot = (unsigned short*)(sval + kResW * cap);
  for (int i = t; i < nR; i += NT) {
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      E::fetch(ad[d].q + 16u * i, 0u, pt.sweep[d], pLo + i);
      if (MORE) E::fetch(ad[d].mq + 16u * i, 0u, pt.more[d], pLo + i);
    }
#pragma unroll
    for (int e = 0; e < kResW; ++e) {
      sval[e * cap + i] = pt.val[(size_t)e * mv.nC + pLo + i];
      const int w = pv.slot[(size_t)e * mv.nC + pLo + i];
      sslot[e * cap + i] = (unsigned short)(w < nR ? w : w - nR + halo0);
    }
  }
  for (int l = t; l < nL + 4; l += NT) {
    int2 b = make_int2(0, 0);
    if (l >= 2 && l < nL + 2)
      b = make_int2(mv.lvlStart[l0 + l - 2] - pLo, mv.lvlStart[l0 + l - 1] - pLo);
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(lva - 16 + 8u * l), "r"(b.x), "r"(b.y) : "memory");
  }
  if (t == 0) {
    const T z[3] = {0, 0, 0};
    URow<T>::store(uBase + kU * (unsigned)pv.zeroRow, z);
    if (lead) sst = *st;
  }
  int hx[KH];
  const int* __restrict__ hi = pv.halo + (size_t)part * pv.haloCap;
#pragma unroll
  for (int j = 0; j < KH; ++j) hx[j] = t + j * NT < nH ? hi[t + j * NT] : -1;
  T r[KR][3], x[KR][3], pp[KR][3], q[KR][3], rd[KR], dg[KR];
#pragma unroll
  for (int j = 0; j < KR; ++j) {
    const int i = i0 + 64 * j;
    rd[j] = j < nMine ? p.rD[pLo + i] : T(0);
    dg[j] = j < nMine ? p.diag[pLo + i] : T(0);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      r[j][k] = j < nMine ? p.r[3 * (size_t)(pLo + i) + k] : T(0);
      x[j][k] = 0; pp[j][k] = 0; q[j][k] = 0;
    }
  }
  cpAsyncWaitAll();
  __syncthreads();
  bool ok = true;
  unsigned pend = 0;  // components with a pending update (bits)
  T al[3] = {0, 0, 0};
  // result of a sum: in sVal and sFlags after the next barrier
  auto result = [&]() {
    if (t == 0 && !lead) {
      uint4 v;
      ok = waitPacket(mine, tag << 8, 8, limit, v) && ok;
      sVal[0] = __uint_as_float(v.x); sVal[1] = __uint_as_float(v.y); sVal[2] = __uint_as_float(v.z);
      sFlags = v.w & 0xffu;
    }
    ok = __syncthreads_and(ok) != 0;
  };
  // a lane's sums between its two threads
  auto handOver = [&](const Acc<T> (&a)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) hand[64 * k + t] = make_float2(a[k].s, a[k].c);
  };
  auto takeOver = [&](Acc<T> (&a)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float2 h = hand[64 * k + t - 64];
      a[k].s = h.x; a[k].c = h.y;
    }
  };
  auto laneSums = [](const Acc<T> (&a)[3]) {  // component k in lane 8 k
    const T x[1][3] = {{a[0].s, a[1].s, a[2].s}}, e[1][3] = {{a[0].c, a[1].c, a[2].c}};
    double s[1];
    warpFloatSums<1, true>(x, e, s);
    return s[0];
  };
  // p.q of the CTA's NB row blocks: the warps' sums in blk.  The terms of the CTA's own rows
  // are in the shared vector.
  auto blockSums = [&](auto nb) {
    constexpr int NB = decltype(nb)::value;
    bool came = true;
    Acc<T> a[2 * NB][3];
    const bool two = mv.nC > stride;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (e == 1 && !two) break;
      auto rowOf = [&](int n) { return b0 * kRowBlock + NT * n + t + stride * e; };
      uint4 pk[2 * NB];
      came = waitPackets(
                 [&](int n) {
                   const int row = rowOf(n);
                   return row < mv.nC && (row < pLo || row >= pLo + nR) ? lp.t + row : (const uint4*)nullptr;
                 },
                 tag, limit, pk) && came;
#pragma unroll
      for (int n = 0; n < 2 * NB; ++n) {
        const int row = rowOf(n);
        if (row >= mv.nC) continue;
        T u[3];
        if (row < pLo || row >= pLo + nR) {
          u[0] = __uint_as_float(pk[n].x); u[1] = __uint_as_float(pk[n].y); u[2] = __uint_as_float(pk[n].z);
        } else {
          URow<T>::load(uBase + kU * (unsigned)(row - pLo), u);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (e == 0) a[n][k].s = u[k];
          else a[n][k].add(u[k]);
      }
    }
    T x[2 * NB][3], cmp[2 * NB][3];
    double s[2 * NB];
#pragma unroll
    for (int n = 0; n < 2 * NB; ++n)
#pragma unroll
      for (int k = 0; k < 3; ++k) { x[n][k] = a[n][k].s; cmp[n][k] = a[n][k].c; }
    if (two) warpFloatSums<2 * NB, true>(x, cmp, s);
    else warpFloatSums<2 * NB>(x, s);
#pragma unroll
    for (int n = 0; n < 2 * NB; ++n)
      if ((lane & 7) == 0 && lane < 24) blk[n >> 1][3 * (wid + 4 * (n & 1)) + (lane >> 3)] = s[n];
    return came;
  };
  for (;;) {
    ++tag;
    // pending r -= alpha q, w = rD r; sum|r| of the lanes' first halves
#pragma unroll
    for (int j = 0; j < KR; ++j)
      if (j < nMine) {
        T w[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (pend >> k & 1) r[j][k] = fmaT(-al[k], q[j][k], r[j][k]);
          w[k] = mulT(rd[j], r[j][k]);
        }
        URow<T>::store(uBase + kU * (unsigned)(i0 + 64 * j), w);
      }
    Acc<T> ar[3], wr[3];
    auto addAbs = [&]() {
#pragma unroll
      for (int j = 0; j < KR; ++j)
        if (j < nMine)
#pragma unroll
          for (int k = 0; k < 3; ++k) ar[k].add(fabs(r[j][k]));
    };
    if (t < 64) {
      addAbs();
      handOver(ar);
    }
    __syncthreads();
    double absHalf = 0;  // (warps 2, 3) sum|r| over half of the lanes: value k in lane 8 k
    if (t < kLoopWalk) {
      if (nL > 1) {
        resSweepBody<0, false, false, false, MORE, WIDE, E>(pt.sweep[0], pt.more[0], ad[0], uBase, 0u, lva,
                                                            nL, kLoopWalk, 0);
        resSweepBody<1, false, false, false, MORE, WIDE, E>(pt.sweep[1], pt.more[1], ad[1], uBase, 0u, lva,
                                                            nL, kLoopWalk, 0);
      }
    } else {
      takeOver(ar);
      addAbs();
      absHalf = laneSums(ar);
    }
    __syncthreads();
    auto addDots = [&]() {
#pragma unroll
      for (int j = 0; j < KR; ++j)
        if (j < nMine) {
          T w[3];
          URow<T>::load(uBase + kU * (unsigned)(i0 + 64 * j), w);
#pragma unroll
          for (int k = 0; k < 3; ++k) wr[k].add(mulT(w[k], r[j][k]));
        }
    };
#pragma unroll
    for (int j = 0; j < KR; ++j)
      if (j < nMine) {
        const int i = i0 + 64 * j;
        T w[3];
        URow<T>::load(uBase + kU * (unsigned)i, w);
        stPacket(lp.w + pLo + i, __float_as_uint(w[0]), __float_as_uint(w[1]), __float_as_uint(w[2]), tag);
      }
    if (t < 64) {
      addDots();
      handOver(wr);
    }
    __syncthreads();
    double dotHalf = 0;
    if (t >= 64) {
      takeOver(wr);
      addDots();
      dotHalf = laneSums(wr);
      if (wid == 3 && (lane & 7) == 0 && lane < 24) {
        red[lane >> 3] = dotHalf;
        red[3 + (lane >> 3)] = absHalf;
      }
    }
    __syncthreads();
    if (wid == 2) {
      const int k = (lane >> 3) % 3;
      const double d = dotHalf + red[k], a = absHalf + red[3 + k];
      unsigned b[3];
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const int m = 3 * (lane & 3) + e, from = 8 * ((m >> 1) % 3);
        const double vd = __shfl_sync(0xffffffffu, d, from), va = __shfl_sync(0xffffffffu, a, from);
        b[e] = valueWord(m < 6 ? vd : va, m);
      }
      if (lane < 4) stPacket(lp.rec + (size_t)lane * nP + part, b[0], b[1], b[2], tag);
    }
    if (lead) {
      double sum = 0;
      ok = loopPartTotal(lp.rec, nP, grp, blk[0], tag, limit, sum) && ok;
      if (t < 32) {
        pcgDecideBeta(c, &sst, sum, pend != 0);
        __syncwarp();
        const bool act = t < 3 && sst.active[t < 3 ? t : 0], first = t < 3 && sst.nIter[t < 3 ? t : 0] == 0;
        const unsigned f = __ballot_sync(0xffffffffu, act) | __ballot_sync(0xffffffffu, first) << 3 |
                           (sst.pcgContinue ? 64u : 0u);
        const T b = t < 3 ? (T)sst.beta[t] : T(0);
        resultPut(out, tag, b, f);
        if (t < 3) sVal[t] = b;
        if (t == 0) sFlags = f;
      }
    }
    // (the halo's w while CTA 0 decides)
    uint4 wh[KH];
    ok = waitPackets([&](int j) { return hx[j] >= 0 ? lp.w + hx[j] : (const uint4*)nullptr; }, tag, limit, wh) && ok;
    result();
    if (!ok) break;
    const unsigned fl = sFlags;
    const bool go = (fl & 64u) != 0;
    // pending x += alpha p_old; p = w + beta p_old
    T b[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) b[k] = sVal[k];
#pragma unroll
    for (int j = 0; j < KR; ++j)
      if (j < nMine) {
        const int i = i0 + 64 * j;
        T u[3];
        URow<T>::load(uBase + kU * (unsigned)i, u);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (pend >> k & 1) x[j][k] = fmaT(al[k], pp[j][k], x[j][k]);
          if (!(fl >> (3 + k) & 1)) u[k] = fmaT(b[k], pp[j][k], u[k]);
          if (fl >> k & 1) pp[j][k] = u[k];
        }
        URow<T>::store(uBase + kU * (unsigned)i, u);
      }
    if (!go) break;
#pragma unroll
    for (int j = 0; j < KH; ++j)
      if (hx[j] >= 0) {
        const unsigned a = uBase + kU * (unsigned)(halo0 + t + j * NT);
        T o[3], w[3] = {__uint_as_float(wh[j].x), __uint_as_float(wh[j].y), __uint_as_float(wh[j].z)};
        URow<T>::load(a, o);
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (!(fl >> (3 + k) & 1)) w[k] = fmaT(b[k], o[k], w[k]);
        URow<T>::store(a, w);
      }
    __syncthreads();
    ++tag;
    // q = A p
#pragma unroll
    for (int j = 0; j < KR; ++j)
      if (j < nMine) {
        const int i = i0 + 64 * j;
        T v[3], y[3], xv[kResW][3];
        URow<T>::load(uBase + kU * (unsigned)i, v);
#pragma unroll
        for (int e = 0; e < kResW; ++e) URow<T>::load(uBase + kU * (unsigned)sslot[e * cap + i], xv[e]);
#pragma unroll
        for (int k = 0; k < 3; ++k) y[k] = mulT(dg[j], v[k]);
#pragma unroll
        for (int e = 0; e < kResW; ++e) {
          const T a = sval[e * cap + i];
#pragma unroll
          for (int k = 0; k < 3; ++k) y[k] = fmaT(a, xv[e][k], y[k]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (fl >> k & 1) q[j][k] = y[k];
      }
    __syncthreads();  // (p of the rows has been read)
    // the terms of p.q in its place; those that another CTA adds up as packets (a stopped
    // component's are not used)
#pragma unroll
    for (int j = 0; j < KR; ++j)
      if (j < nMine) {
        const int i = i0 + 64 * j, row = pLo + i;
        const int first = (row < stride ? row : row - stride) / kRowBlock * kRowBlock;
        T u[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) u[k] = mulT(q[j][k], pp[j][k]);
        if (first < pLo || first >= pLo + nR)
          stPacket(lp.t + row, __float_as_uint(u[0]), __float_as_uint(u[1]), __float_as_uint(u[2]), tag);
        URow<T>::store(uBase + kU * (unsigned)i, u);
      }
    __syncthreads();
    if (nMyB == 2) ok = blockSums(std::integral_constant<int, 2>()) && ok;
    else if (nMyB == 1) ok = blockSums(std::integral_constant<int, 1>()) && ok;
    __syncthreads();
    if (wid == 0 && nMyB > 0) {  // the blocks' sums in lanes 0 .. 3 nMyB - 1, then two packets each
      double s = 0;
      if (lane < 3 * nMyB) {
        s = blk[lane / 3][lane % 3];
#pragma unroll
        for (int w = 1; w < kRowBlock / 32; ++w) s += blk[lane / 3][3 * w + lane % 3];
      }
      unsigned b3[3];
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const int m = 3 * (lane & 1) + e;
        const double v = __shfl_sync(0xffffffffu, s, 3 * (lane >> 1 & 1) + (m >> 1));
        b3[e] = valueWord(v, m);
      }
      if (lane < 2 * nMyB) stPacket(rec2 + (size_t)(lane & 1) * nB + b0 + (lane >> 1), b3[0], b3[1], b3[2], tag);
    }
    if (lead) {
      __syncthreads();  // (the blocks' records have been read)
      double sum = 0;
      ok = loopBlockTotal(rec2, nB, blk[0], tag, limit, sum) && ok;
      if (t < 32) {
        pcgDecideAlpha(&sst, sum, 0);
        __syncwarp();
        const bool on = t < 3 && sst.pending[t < 3 ? t : 0];
        const unsigned f = __ballot_sync(0xffffffffu, on) | (sst.pcgContinue ? 64u : 0u);
        const T a = t < 3 ? (T)sst.alpha[t] : T(0);
        resultPut(out, tag, a, f);
        if (t < 3) sVal[t] = a;
        if (t == 0) sFlags = f;
      }
    }
    result();
    if (!ok) break;
    pend = sFlags & 7u;
#pragma unroll
    for (int k = 0; k < 3; ++k) al[k] = sVal[k];
    if (!(sFlags & 64u)) break;
  }
#pragma unroll
  for (int j = 0; j < KR; ++j)
    if (j < nMine) stRow(p.x, (size_t)(pLo + i0 + 64 * j), x[j]);
  if (t == 0 && !ok) atomicOr(&st->status, kErrTimeout);
  if (lead) {
    // the state back; x is complete
    __syncthreads();
    if (t < 3) {
      st->active[t] = sst.active[t]; st->nIter[t] = sst.nIter[t]; st->finalRes[t] = sst.finalRes[t];
      st->wArA[t] = sst.wArA[t]; st->wApA[t] = sst.wApA[t];
      st->alpha[t] = sst.alpha[t]; st->beta[t] = sst.beta[t];
      st->pending[t] = sst.pending[t];
      st->xPend[t] = 0;
    }
    if (t == 0) {
      st->pcgIter = sst.pcgIter;
      st->pcgContinue = sst.pcgContinue;
      if (sst.status) atomicOr(&st->status, sst.status);
      *count = tag;
    }
  }
}

// ---- tables --------------------------------------------------------------------
// Entries of a part's rows that lead out of it (the largest count in *most).
__global__ void kPartCount(MeshView mv, int* cnt, int* most) {
  const int part = blockIdx.x;
  const int lo = mv.partStart[part], hi = mv.partStart[part + 1];
  __shared__ int n;
  if (threadIdx.x == 0) n = 0;
  __syncthreads();
  int m = 0;
  for (int e = mv.rowptr[lo] + threadIdx.x; e < mv.rowptr[hi]; e += blockDim.x) {
    const int cl = mv.col[e];
    if (cl < lo || cl >= hi) ++m;
  }
  atomicAdd(&n, m);
  __syncthreads();
  if (threadIdx.x == 0) {
    cnt[part] = n;
    atomicMax(most, n);
  }
}
// Their rows (a place each, in any order: the places do not enter the results),
// and every row's product columns as places in the part's shared memory.
__global__ void kPartSlots(MeshView mv, PartView pv, int* halo, unsigned short* slot) {
  const int part = blockIdx.x;
  const int lo = mv.partStart[part], hi = mv.partStart[part + 1];
  __shared__ int n;
  if (threadIdx.x == 0) n = 0;
  __syncthreads();
  for (int s = lo + threadIdx.x; s < hi; s += blockDim.x) {
    const int e0 = mv.rowptr[s], m = mv.rowptr[s + 1] - e0;
    for (int k = 0; k < kResW; ++k) {
      int w = s - lo;
      if (k < m) {
        const int cl = mv.col[e0 + k];
        if (cl >= lo && cl < hi) {
          w = cl - lo;
        } else {
          const int at = atomicAdd(&n, 1);
          halo[(size_t)part * pv.haloCap + at] = cl;
          w = hi - lo + at;
        }
      }
      slot[(size_t)k * mv.nC + s] = (unsigned short)w;
    }
  }
}

__device__ __forceinline__ void putPart(const PartTab<float>& tb, int i, const float* a, const unsigned* w, bool more) {
  const unsigned pack = w[0] | (w[1] << 10) | (w[2] << 20) | (more ? 1u << 30 : 0u);
  const_cast<float4*>(tb.q)[i] = make_float4(a[0], a[1], a[2], __uint_as_float(pack));
}
__device__ __forceinline__ void putPart(const ResSweepTab<double>& tb, int i, const double* a, const unsigned* w, bool more) {
  const double a3[3] = {a[0], a[1], a[2]};
  tb.put(i, a3, (unsigned long long)w[0] | ((unsigned long long)w[1] << 18) |
                    ((unsigned long long)w[2] << 36) | ((unsigned long long)(more ? 1 : 0) << 54));
}
// Coefficients of the product and of the substitutions (in-part entries: lower
// ones in CSR order, upper ones in reverse) in T, padded with zeros.
template <typename T>
__global__ void kPartTables(MeshView mv, PartView pv, const double* val, const double* rDa, PartPtrs<T> out) {
  const int part = blockIdx.x;
  const int lo = mv.partStart[part], hi = mv.partStart[part + 1];
  for (int s = lo + threadIdx.x; s < hi; s += blockDim.x) {
    const int e0 = mv.rowptr[s], n = mv.rowptr[s + 1] - e0;
    if (out.val)
      for (int k = 0; k < kResW; ++k)
        const_cast<T*>(out.val)[(size_t)k * mv.nC + s] = k < n ? (T)val[e0 + k] : T(0);
    for (int dir = 0; dir < 2; ++dir) {
      T a[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
      const unsigned z = (unsigned)pv.zeroRow;
      unsigned w[6] = {z, z, z, z, z, z};
      int num = 0;
      for (int j = 0; j < n; ++j) {
        const int k = dir == 0 ? j : n - 1 - j, cl = mv.col[e0 + k];
        if (dir == 0 ? !(cl < s && cl >= lo) : !(cl > s && cl < hi)) continue;
        a[num] = (T)rDa[e0 + k];
        w[num++] = (unsigned)(cl - lo);
      }
      putPart(out.sweep[dir], s, a, w, num > 3);
      if (pv.more) putPart(out.more[dir], s, a + 3, w + 3, false);
    }
  }
}

template <typename T>
const void* precondKernel(const PartView& pv) {
  if (pv.wide) return (const void*)kPartPrecond<T, true, true>;
  return pv.more ? (const void*)kPartPrecond<T, true, false> : (const void*)kPartPrecond<T, false, false>;
}
template <typename T>
size_t precondSmem(const MeshView& mv, const PartView& pv) {
  const size_t ent = 16 + PartCfg<T>::Ent::kB;
  return URow<T>::kBytes * (size_t)(pv.capRows + 4) + 2 * (pv.more ? 2 : 1) * ent * pv.capRows +
         8 * (size_t)(mv.maxLevels + 5);
}
size_t spmvSmem(const PartView& pv) {
  return URow<float>::kBytes * (size_t)(pv.capRows + pv.haloCap);
}

}  // namespace

// Largest part in rows: the columns' 10 bits in FP32.
template <typename T>
int partMaxRows() { return sizeof(T) == 4 ? 1016 : 1 << 16; }
// Threads that walk a part's levels at once.
template <typename T>
int partWalkRows() { return PartCfg<T>::kSplit ? PartCfg<T>::kNT / 3 : PartCfg<T>::kNT; }

template <typename T>
cudaError_t partPrepare(const MeshView& mv, const PartView& pv, int* blocks) {
  const void* k[2] = {precondKernel<T>(pv), (const void*)kPartSpmv};
  const size_t sm[2] = {precondSmem<T>(mv, pv), spmvSmem(pv)};
  const int nt[2] = {PartCfg<T>::kNT, kPartSpmvThreads};
  blocks[1] = 1;
  for (int j = 0; j < (sizeof(T) == 8 ? 1 : 2); ++j) {
    cudaError_t e = setMaxDynamicSmem(k[j]);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks[j], k[j], nt[j], sm[j]);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

namespace {
const void* loopKernel(const PartView& pv) {
  if (pv.wide) return (const void*)kPartLoop<true, true>;
  return pv.more ? (const void*)kPartLoop<true, false> : (const void*)kPartLoop<false, false>;
}
size_t loopSmem(const MeshView& mv, const PartView& pv) {
  const size_t cap = pv.capRows;
  return URow<float>::kBytes * (cap + 4 + pv.haloCap) + 16 * (pv.more ? 4 : 2) * cap +
         8 * (size_t)(mv.maxLevels + 5) + kResW * 6 * cap;
}
}  // namespace

size_t partLoopPackets(const MeshView& mv) {
  return 4 * (size_t)mv.nParts + 2 * (size_t)mv.rowGrid + kLoopLine * kLoopCopies + 1;
}

cudaError_t partLoopPrepare(const MeshView& mv, const PartView& pv, int* blocks) {
  *blocks = 0;
  if (pv.capRows > kLoopMaxRows || pv.haloCap > 4 * kLoopThreads) return cudaSuccess;
  if (mv.nC > 2 * mv.rowGrid * kRowBlock) return cudaSuccess;  // (two rows a lane of p.q)
  const void* k = loopKernel(pv);
  const cudaError_t e = setMaxDynamicSmem(k);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k, kLoopThreads, loopSmem(mv, pv));
}
cudaError_t launchPartLoop(const MeshView& mv, const Controls& c, const PartView& pv,
                           const PartPtrs<float>& pt, const LoopPtrs& lp, const PcgPtrs<float>& p,
                           DevState* st, cudaStream_t s) {
  cudaLaunchConfig_t cf{};
  cf.gridDim = dim3(mv.nParts);
  cf.blockDim = dim3(kLoopThreads);
  cf.dynamicSmemBytes = loopSmem(mv, pv);
  cf.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cf.attrs = at;
  cf.numAttrs = 1;
  void* args[] = {(void*)&mv, (void*)&c, (void*)&pv, (void*)&pt, (void*)&lp, (void*)&p, (void*)&st};
  return cudaLaunchKernelExC(&cf, loopKernel(pv), args);
}

cudaError_t launchPartCount(const MeshView& mv, int* cnt, int* most, cudaStream_t s) {
  kPartCount<<<mv.nParts, 128, 0, s>>>(mv, cnt, most);
  return cudaGetLastError();
}
cudaError_t launchPartSlots(const MeshView& mv, const PartView& pv, cudaStream_t s) {
  kPartSlots<<<mv.nParts, 128, 0, s>>>(mv, pv, const_cast<int*>(pv.halo), const_cast<unsigned short*>(pv.slot));
  return cudaGetLastError();
}
template <typename T>
cudaError_t launchPartTables(const MeshView& mv, const PartView& pv, const double* val, const double* rDa,
                             const PartPtrs<T>& out, cudaStream_t s) {
  kPartTables<T><<<mv.nParts, 128, 0, s>>>(mv, pv, val, rDa, out);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launchPartIteration(const MeshView& mv, const Controls& c, const PartView& pv,
                                const PartPtrs<T>& pt, const PcgPtrs<T>& p, DevState* st,
                                double* partials, const LocalTuning& t, cudaStream_t s,
                                LaunchTimer* tm, int nCases) {
  {
    TimeScope ts(tm, S4G_K_LOC_PRECOND, s);
    void* args[] = {(void*)&mv, (void*)&c, (void*)&pv, (void*)&pt, (void*)&p, (void*)&st, (void*)&partials};
    const cudaError_t e = cudaLaunchKernel(precondKernel<T>(pv), dim3(pv.grid[0], nCases),
                                           dim3(PartCfg<T>::kNT), args, precondSmem<T>(mv, pv), s);
    if (e != cudaSuccess) return e;
  }
  {
    TimeScope ts(tm, S4G_K_LOC_SPMV, s);
    if constexpr (sizeof(T) == 8) {
      launchLocalSpmv<T>(mv, p, st, partials, t, s, nCases);
    } else {
      kPartSpmv<<<dim3(pv.grid[1], nCases), kPartSpmvThreads, spmvSmem(pv), s>>>(mv, pv, pt, p, st);
      kPartDot<<<dim3(mv.rowGrid, nCases), kRowBlock, 0, s>>>(mv, p, st, partials);
    }
  }
  return cudaGetLastError();
}

#define S4G_INSTANTIATE(T)                                                                       \
  template int partMaxRows<T>();                                                                 \
  template int partWalkRows<T>();                                                                \
  template cudaError_t partPrepare<T>(const MeshView&, const PartView&, int*);                   \
  template cudaError_t launchPartTables<T>(const MeshView&, const PartView&, const double*,      \
                                           const double*, const PartPtrs<T>&, cudaStream_t);     \
  template cudaError_t launchPartIteration<T>(const MeshView&, const Controls&, const PartView&, \
                                              const PartPtrs<T>&, const PcgPtrs<T>&, DevState*,  \
                                              double*, const LocalTuning&, cudaStream_t,         \
                                              LaunchTimer*, int);
S4G_INSTANTIATE(double)
S4G_INSTANTIATE(float)
#undef S4G_INSTANTIATE

}  // namespace s4g
