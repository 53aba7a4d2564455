// PCG with the processor-local DIC on the whole device, a CTA per part: two
// kernels per iteration, for meshes beyond the cluster-resident PCG.
//
//   kPartPrecond  r -= alpha q of the pending iteration, sum|r|, w = M^-1 r of
//                 each part and w.r; the last CTA runs the residual test and
//                 decides beta.
//   kPartSpmv     the pending x += alpha p, p_new = w + beta p_old, q = A p_new
//                 and p.q; the last CTA decides alpha.
//
// Both hold a part's rows in shared memory while they work on it: w during the
// substitutions, p_new -- of the part's rows and of the rows around it that
// they touch -- during the product, so that a row's six neighbours are shared-
// memory reads instead of gathers of w and p_old through L1.  The arithmetic of
// every vector entry is that of the separate kernels (kernels_local.cu), to the
// bit in FP32; a CTA takes parts b, b + G, ... and adds up its threads' sums
// once, at the end, and the last CTA adds the CTAs' records in order: the order
// of the sums depends on the mesh, the value type and the device only.
//
// In FP64 the corrector loop of some processor-local runs amplifies a last bit of
// a sum a thousandfold every ten correctors (measured: 1e-13 after 60, 2e-6
// after 100).  There the preconditioner keeps the sums of kernels_local.cu in
// their order -- 64 lanes over a part's rows, parts in groups of 32
// (part_sums.cuh) -- and the product and its sums stay with kernels_local.cu.
//
// Parts of rows with at most six neighbours that fit shared memory (in FP32
// at most 1022 rows: 10-bit columns); others run kernels_local.cu.

#include <algorithm>

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
  // (8 resident CTAs at 123 registers; 6 at 139 before: 128^3 61.4 -> 60.1 us a
  // launch, 16 cases of 40^3 39.4 -> 35.5; fewer rows a thread keeps: 65 and 70 us)
  static constexpr int kNT = 64, kKeep = 8, kOcc = 7;
  static constexpr bool kSplit = false, kOrdered = false;
};
template <> struct PartCfg<double> {
  using Ent = ResEnt<double>;
  static constexpr int kNT = 192, kKeep = 3, kOcc = 4;
  static constexpr bool kSplit = true, kOrdered = true;
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

// Sums of N values of every thread of the CTA into its record (rec[value][CTA]),
// and by the last CTA of the launch over all records: thread t sums CTAs t,
// t + NT, ..., four records' loads in flight, then a fixed tree.  True in every
// thread of the last CTA; its threads 0 .. 31 find the sums in out[0..N).
template <typename T, int NT, int N, int M>
__device__ __forceinline__ bool gridSum(typename Part<T>::V (&v)[M], typename Part<T>::V* rec,
                                        typename Part<T>::V* wrec, double* out, unsigned* counter) {
  using P = Part<T>;
  using V = typename P::V;
  constexpr int W = NT / 32, G = 32 / M;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, k = lane / G, g = lane % G;
  const V s = warpSpreadSum<T, M>(v);
  if (k < N && g == 0) wrec[wid * N + k] = s;
  __syncthreads();
  if (wid == 0) {
    const V a = warpRecords<T, N, M>(wrec, W);
    if (k < N && g == 0) rec[(size_t)k * gridDim.x + blockIdx.x] = a;
    __syncwarp();
    if (lane < N) __threadfence();
  }
  if (!lastBlockDone(counter, gridDim.x)) return false;
  const int n = (int)gridDim.x;
#pragma unroll
  for (int m = 0; m < M; ++m) v[m] = P::zero();
  for (int j0 = (int)threadIdx.x; j0 < n; j0 += 4 * NT) {
    V x[4][N];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int m = 0; m < N; ++m)
        x[u][m] = j0 + u * NT < n ? P::ldcg(rec + (size_t)m * n + j0 + u * NT) : P::zero();
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int m = 0; m < N; ++m) v[m] = P::add(v[m], x[u][m]);
  }
  const V a = warpSpreadSum<T, M>(v);
  if (k < N && g == 0) wrec[wid * N + k] = a;
  __syncthreads();
  if (wid == 0) {
    const V b = warpRecords<T, N, M>(wrec, W);
    if (k < N && g == 0) out[k] = P::value(b);
    __syncwarp();
  }
  return true;
}

template <typename T, bool MORE, bool WIDE>
__global__ void __launch_bounds__(PartCfg<T>::kNT, PartCfg<T>::kOcc)
kPartPrecond(MeshView mv, Controls c, PartView pv, PartPtrs<T> pt, PcgPtrs<T> p, DevState* st,
             double* partials) {
  using C = PartCfg<T>;
  using E = typename C::Ent;
  using P = Part<T>;
  using V = typename P::V;
  constexpr int NT = C::kNT, KR = C::kKeep;
  constexpr unsigned kU = URow<T>::kBytes, kB = E::kB;
  p = casePcg(p, blockIdx.y, mv.nC);
  st += blockIdx.y;
  partials += (size_t)blockIdx.y * mv.caseRec;
  if (!st->pcgContinue) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ __align__(16) int4 sDesc[2][2];
  __shared__ V wrec[6 * (NT / 32)];
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
  // (ordered sums) the part's residual, in the tables' place after the sweeps
  T* const sr = (T*)(smraw + (ad[0].q - uBase));
  double* grec = partials + mv.locGrpOff;
  unsigned* gcnt = reinterpret_cast<unsigned*>(grec + 8 * (size_t)mv.locGroups);
  int prev = -1;
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
  Acc<T> wr[3], ar[3];
  for (int buf = 0; part < nParts; part += (int)gridDim.x, buf ^= 1) {
    const int4 dA = sDesc[buf][0], dB = sDesc[buf][1];
    const int pLo = dA.x, nR = dA.y, l0 = dB.z, nL = dB.w;
    const int next = part + (int)gridDim.x;
    if (t == 0 && next < nParts) {
      cpAsync16(&sDesc[buf ^ 1][0], mv.locDesc + 2 * next);
      cpAsync16(&sDesc[buf ^ 1][1], mv.locDesc + 2 * next + 1);
    }
    // the previous part's record is reported on its group's counter
    bool done = false;
    if (C::kOrdered && t == 0 && prev >= 0) done = locArrive(gcnt, prev, nParts);
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
    // w out, w.r and sum|r| over the thread's rows in row order
#pragma unroll
    for (int j = 0; j < KR; ++j) {
      const int i = t + j * NT;
      if (i < nR) {
        T w[3];
        URow<T>::load(uBase + kU * (unsigned)i, w);
        stRow(p.w, (size_t)(pLo + i), w);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (C::kOrdered) {
            sr[3 * i + k] = rK[j][k];
            continue;
          }
          wr[k].add(mulT(w[k], rK[j][k]));
          ar[k].add(fabs(rK[j][k]));
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
        if (C::kOrdered) {
          sr[3 * i + k] = r;
          continue;
        }
        wr[k].add(mulT(w[k], r));
        ar[k].add(fabs(r));
      }
    }
    if (C::kOrdered) {
      // lane l of 64 sums rows l, l + 64, ..., then a fixed tree: sum64's, by the
      // spread sum (9 additions a warp for 30)
      __syncthreads();
      const int k = (t & 31) / 4;
      double s6 = 0;
      if (t < 64) {
        double d[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int i = t; i < nR; i += 64) {
          T w[3];
          URow<T>::load(uBase + kU * (unsigned)i, w);
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const T r = sr[3 * i + m];
            d[m] = fma((double)w[m], (double)r, d[m]);
            d[3 + m] += fabs((double)r);
          }
        }
        s6 = warpSpreadSum<double, 8>(d);
        if (t >= 32 && t % 4 == 0 && k < 6) sum[k] = s6;
      }
      if (t == 0) sGroup = done ? prev / kLocGroup : -1;
      __syncthreads();
      if (t < 32 && t % 4 == 0 && k < 6) partials[8 * (size_t)part + k] = s6 + sum[k];
      if (sGroup >= 0 && t < 32) locGroupSum(partials, grec, gcnt, sGroup, nParts);
      prev = part;
    }
    __syncthreads();  // the next part reuses the shared memory
  }
  if (C::kOrdered) {
    locFinish(mv, c, st, partials, prev, anyPend, sum, &sGroup);
    return;
  }
  V v[8] = {P::of(wr[0]), P::of(wr[1]), P::of(wr[2]), P::of(ar[0]),
            P::of(ar[1]), P::of(ar[2]), P::zero(), P::zero()};
  if (!gridSum<T, NT, 6>(v, (V*)partials, wrec, sum, &st->counter[5])) return;
  if (t >= 32) return;
  if (t == 0) st->counter[5] = 0;
  pcgDecideBeta(c, st, t < 6 ? sum[t] : 0.0, anyPend);
}

__global__ void __launch_bounds__(kPartSpmvThreads, 8)
kPartSpmv(MeshView mv, PartView pv, PartPtrs<float> pt, PcgPtrs<float> p, DevState* st, double* partials) {
  using T = float;
  using P = Part<T>;
  using V = typename P::V;
  constexpr int NT = kPartSpmvThreads, RP = 1, KH = 4;
  constexpr unsigned kU = URow<T>::kBytes;
  p = casePcg(p, blockIdx.y, mv.nC);
  st += blockIdx.y;
  partials += (size_t)blockIdx.y * mv.caseRec;
  if (!st->pcgContinue) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ V wrec[3 * (NT / 32)];
  __shared__ double sum[4];
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
  Acc<T> pq[3];
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
      for (int k = 0; k < 3; ++k) {
        if (act[k]) qo[g + k] = y[k];
        pq[k].add(mulT(y[k], v[k]));
      }
    }
    __syncthreads();
    part = next; pLo = pLo1; nR = nR1 - pLo1; nH = nH1;
  }
  V v[4] = {P::of(pq[0]), P::of(pq[1]), P::of(pq[2]), P::zero()};
  if (!gridSum<T, NT, 3>(v, (V*)partials, wrec, sum, &st->counter[6])) return;
  if (t >= 32) return;
  if (t == 0) st->counter[6] = 0;
  pcgDecideAlpha(st, t < 3 ? sum[t] : 0.0, pb);
}

// ---- the whole loop of a corrector in one launch ---------------------------------
// Meshes whose parts are all resident at once (a CTA per part; FP32): the
// launches of kPartPrecond and kPartSpmv, their reading of the state and their
// ends take longer than a part's work, so one cooperative launch runs the PCG
// loop of a corrector.  r, x, p and q stay in registers, the tables in shared
// memory; the part's halo keeps its p in shared memory and needs only w from
// other parts once per iteration.
//
// What CTAs tell one another goes through 16-byte packets that carry their own
// tag (the count of sums so far): a reader polls the packet itself, so neither a
// counter nor a fence stands between a value and its use.  Rows publish w; a CTA
// publishes its part of a sum, CTA 0 adds the parts up, decides and publishes the
// result in kLoopCopies lines.  (With a counter, fences and the last CTA deciding
// on the state in memory a sum took 7 us of a 27 us iteration of 512 parts.)  A
// packet is written again only after its readers have taken part in a later sum.
constexpr int kLoopThreads = 128, kLoopRows = 4, kLoopWalk = 64;
constexpr int kLoopMaxRows = kLoopThreads * kLoopRows;
constexpr int kLoopAhead = 2;  // CTAs whose packets a thread of CTA 0 has in flight
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

// All CTAs' sums of N values.  A CTA's packets: the first parts of three values'
// compensated sums, their second parts, the same of the next three.  CTA 0 leaves
// the sums in its warp 0 (value k in lane k) and returns whether all came.
template <int N, int M>
__device__ __forceinline__ bool gridPut(float2 (&v)[M], uint4* rec, float2* wrec, unsigned tag, int limit,
                                        double& mine) {
  using P = Part<float>;
  constexpr int NT = kLoopThreads, W = NT / 32, G = 32 / M, Q = 2 * N / 3;
  const int t = (int)threadIdx.x, lane = t & 31, wid = t >> 5, k = lane / G, g = lane % G;
  const int n = (int)gridDim.x;
  const float2 s = warpSpreadSum<float, M>(v);
  if (k < N && g == 0) wrec[wid * N + k] = s;
  __syncthreads();
  if (wid == 0) {
    const float2 a = warpRecords<float, N, M>(wrec, W);
    unsigned b[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const int from = (3 * ((lane % Q) >> 1) + m) * G;
      const float x = __shfl_sync(0xffffffffu, a.x, from), y = __shfl_sync(0xffffffffu, a.y, from);
      b[m] = __float_as_uint((lane & 1) ? y : x);
    }
    if (lane < Q) stPacket(rec + (size_t)lane * n + blockIdx.x, b[0], b[1], b[2], tag);
  }
  if (blockIdx.x != 0) return true;
  // thread t adds up the CTAs t, t + NT, ..., kLoopAhead at a time
  bool ok = true;
#pragma unroll
  for (int m = 0; m < M; ++m) v[m] = P::zero();
  for (int j0 = t; j0 < n; j0 += kLoopAhead * NT) {
    uint4 x[kLoopAhead][Q];
#pragma unroll
    for (int u = 0; u < kLoopAhead; ++u)
#pragma unroll
      for (int q = 0; q < Q; ++q)
        x[u][q] = j0 + u * NT < n ? ldPacket(rec + (size_t)q * n + j0 + u * NT) : make_uint4(0, 0, 0, tag);
#pragma unroll
    for (int u = 0; u < kLoopAhead; ++u)
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (x[u][q].w != tag)
          ok = waitPacket(rec + (size_t)q * n + j0 + u * NT, tag, 0, limit, x[u][q]) && ok;
#pragma unroll
    for (int u = 0; u < kLoopAhead; ++u)
#pragma unroll
      for (int q = 0; q < Q; q += 2) {
        const uint4 h = x[u][q], l = x[u][q + 1];
        const int m = 3 * (q / 2);
        v[m] = P::add(v[m], make_float2(__uint_as_float(h.x), __uint_as_float(l.x)));
        v[m + 1] = P::add(v[m + 1], make_float2(__uint_as_float(h.y), __uint_as_float(l.y)));
        v[m + 2] = P::add(v[m + 2], make_float2(__uint_as_float(h.z), __uint_as_float(l.z)));
      }
  }
  const float2 a = warpSpreadSum<float, M>(v);
  __syncthreads();  // (warp 0 has read the records of its CTA)
  if (k < N && g == 0) wrec[wid * N + k] = a;
  ok = __syncthreads_and(ok) != 0;
  if (wid == 0) {
    const float2 b = warpRecords<float, N, M>(wrec, W);
    mine = __shfl_sync(0xffffffffu, P::value(b), lane < N ? lane * G : 0);
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
  using P = Part<T>;
  constexpr int NT = kLoopThreads, KR = kLoopRows, KH = 4;
  constexpr unsigned kU = URow<T>::kBytes;
  if (!st->pcgContinue) return;  // the same in every CTA: CTA 0 writes the state at its end
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ float2 wrec[6 * (NT / 32)];
  __shared__ T sVal[3];
  __shared__ unsigned sFlags;
  __shared__ DevState sst;  // CTA 0: the state while the loop runs
  const int t = (int)threadIdx.x, cap = pv.capRows, part = (int)blockIdx.x, nP = (int)gridDim.x;
  const int pLo = mv.partStart[part], nR = mv.partStart[part + 1] - pLo, nH = pv.haloCnt[part];
  const int l0 = mv.lvlOff[part], nL = mv.lvlOff[part + 1] - l0;
  const bool lead = part == 0;
  // (a shorter limit is for the waits between parts of the exact DIC's sweeps)
  const int limit = mv.spinLimit > kSpinLimit ? mv.spinLimit : kSpinLimit;
  uint4* const rec2 = lp.rec + 4 * (size_t)nP;
  uint4* const out = rec2 + 2 * (size_t)nP;
  unsigned* const count = reinterpret_cast<unsigned*>(out + kLoopLine * kLoopCopies);
  unsigned tag = ldRelaxed(count);  // of the last sum; CTA 0 writes it at its end
  const uint4* const mine = out + kLoopLine * (part % kLoopCopies);
  // ---- shared memory: w or p of the rows, the zero row, p of the halo | sweep
  //      tables | level bounds | product coefficients | product columns
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
    const int i = t + j * NT;
    rd[j] = i < nR ? p.rD[pLo + i] : T(0);
    dg[j] = i < nR ? p.diag[pLo + i] : T(0);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      r[j][k] = i < nR ? p.r[3 * (size_t)(pLo + i) + k] : T(0);
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
  for (;;) {
    ++tag;
    // pending r -= alpha q, sum|r|, w = rD r
    Acc<T> ar[3], wr[3];
#pragma unroll
    for (int j = 0; j < KR; ++j) {
      const int i = t + j * NT;
      if (i < nR) {
        T w[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (pend >> k & 1) r[j][k] = fmaT(-al[k], q[j][k], r[j][k]);
          ar[k].add(fabs(r[j][k]));
          w[k] = mulT(rd[j], r[j][k]);
        }
        URow<T>::store(uBase + kU * (unsigned)i, w);
      }
    }
    __syncthreads();
    if (nL > 1 && t < kLoopWalk) {
      resSweepBody<0, false, false, false, MORE, WIDE, E>(pt.sweep[0], pt.more[0], ad[0], uBase, 0u, lva,
                                                          nL, kLoopWalk, 0);
      resSweepBody<1, false, false, false, MORE, WIDE, E>(pt.sweep[1], pt.more[1], ad[1], uBase, 0u, lva,
                                                          nL, kLoopWalk, 0);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < KR; ++j) {
      const int i = t + j * NT;
      if (i < nR) {
        T w[3];
        URow<T>::load(uBase + kU * (unsigned)i, w);
        stPacket(lp.w + pLo + i, __float_as_uint(w[0]), __float_as_uint(w[1]), __float_as_uint(w[2]), tag);
#pragma unroll
        for (int k = 0; k < 3; ++k) wr[k].add(mulT(w[k], r[j][k]));
      }
    }
    {
      float2 v[8] = {P::of(wr[0]), P::of(wr[1]), P::of(wr[2]), P::of(ar[0]),
                     P::of(ar[1]), P::of(ar[2]), P::zero(), P::zero()};
      double sum = 0;
      ok = gridPut<6>(v, lp.rec, wrec, tag, limit, sum) && ok;
      if (lead && t < 32) {
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
#pragma unroll
    for (int j = 0; j < KH; ++j)
      if (hx[j] >= 0) wh[j] = ldPacket(lp.w + hx[j]);
#pragma unroll
    for (int j = 0; j < KH; ++j)
      if (hx[j] >= 0 && wh[j].w != tag) ok = waitPacket(lp.w + hx[j], tag, 0, limit, wh[j]) && ok;
    result();
    if (!ok) break;
    const unsigned fl = sFlags;
    const bool go = (fl & 64u) != 0;
    // pending x += alpha p_old; p = w + beta p_old
    T b[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) b[k] = sVal[k];
#pragma unroll
    for (int j = 0; j < KR; ++j) {
      const int i = t + j * NT;
      if (i < nR) {
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
    // q = A p, p.q
    Acc<T> pq[3];
#pragma unroll
    for (int j = 0; j < KR; ++j) {
      const int i = t + j * NT;
      if (i < nR) {
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
        for (int k = 0; k < 3; ++k) {
          if (fl >> k & 1) q[j][k] = y[k];
          pq[k].add(mulT(y[k], v[k]));
        }
      }
    }
    {
      float2 v[4] = {P::of(pq[0]), P::of(pq[1]), P::of(pq[2]), P::zero()};
      double sum = 0;
      ok = gridPut<3>(v, rec2, wrec, tag, limit, sum) && ok;
      if (lead && t < 32) {
        pcgDecideAlpha(&sst, sum, 0);
        __syncwarp();
        const bool on = t < 3 && sst.pending[t < 3 ? t : 0];
        const unsigned f = __ballot_sync(0xffffffffu, on) | (sst.pcgContinue ? 64u : 0u);
        const T b = t < 3 ? (T)sst.alpha[t] : T(0);
        resultPut(out, tag, b, f);
        if (t < 3) sVal[t] = b;
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
  for (int j = 0; j < KR; ++j) {
    const int i = t + j * NT;
    if (i < nR) stRow(p.x, (size_t)(pLo + i), x[j]);
  }
  if (t == 0 && !ok) atomicOr(&st->status, kErrTimeout);
  if (lead) {
    // the state back; x is complete.  (No tag of a wait that gave up comes again.)
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
      *count = tag + 4;
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
  for (int j = 0; j < (PartCfg<T>::kOrdered ? 1 : 2); ++j) {
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

size_t partLoopPackets(int nParts) { return 6 * (size_t)nParts + kLoopLine * kLoopCopies + 1; }

cudaError_t partLoopPrepare(const MeshView& mv, const PartView& pv, int* blocks) {
  *blocks = 0;
  if (pv.capRows > kLoopMaxRows || pv.haloCap > 4 * kLoopThreads) return cudaSuccess;
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
    if constexpr (PartCfg<T>::kOrdered) launchLocalSpmv<T>(mv, p, st, partials, t, s, nCases);
    else
      kPartSpmv<<<dim3(pv.grid[1], nCases), kPartSpmvThreads, spmvSmem(pv), s>>>(mv, pv, pt, p, st, partials);
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
