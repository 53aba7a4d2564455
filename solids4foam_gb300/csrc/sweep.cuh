// Device helpers of the PCG kernels that keep a part's or a cluster's rows in shared
// memory (kernels_resident.cu, kernels_part.cu): cluster primitives, rows of the
// shared vector, the triangular substitutions over levels, sums.
#pragma once

#include "kernels.cuh"
#include "pcg_common.cuh"

namespace s4g {

// ---- cluster primitives ------------------------------------------------------
__device__ __forceinline__ void clArrive() {
  __syncwarp();  // .aligned: the warp arrives as one
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void clWait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned clRank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared-memory address of the same variable in CTA `rank` of the cluster
__device__ __forceinline__ unsigned mapa(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

__device__ __forceinline__ float fmaT(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmaT(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mulT(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mulT(double a, double b) { return __dmul_rn(a, b); }

// One row of the shared vector: 16 bytes in FP32 (one load), 24 in FP64.
template <typename T> struct URow;
template <> struct URow<float> {
  static constexpr unsigned kBytes = 16;
  static __device__ __forceinline__ void load(unsigned a, float (&v)[3]) {
    float pad;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(pad) : "r"(a) : "memory");
  }
  static __device__ __forceinline__ void loadCluster(unsigned a, float (&v)[3]) {
    float pad;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(pad) : "r"(a) : "memory");
  }
  static __device__ __forceinline__ void store(unsigned a, const float (&v)[3]) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};"
                 ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(0.0f) : "memory");
  }
  static __device__ __forceinline__ void storeCluster(unsigned a, const float (&v)[3]) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};"
                 ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(0.0f) : "memory");
  }
};
template <> struct URow<double> {
  static constexpr unsigned kBytes = 24;
  static __device__ __forceinline__ void load(unsigned a, double (&v)[3]) {
    asm volatile("ld.shared.f64 %0, [%3];\nld.shared.f64 %1, [%3+8];\nld.shared.f64 %2, [%3+16];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]) : "r"(a) : "memory");
  }
  static __device__ __forceinline__ void loadCluster(unsigned a, double (&v)[3]) {
    asm volatile("ld.shared::cluster.f64 %0, [%3];\nld.shared::cluster.f64 %1, [%3+8];\n"
                 "ld.shared::cluster.f64 %2, [%3+16];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]) : "r"(a) : "memory");
  }
  static __device__ __forceinline__ void store(unsigned a, const double (&v)[3]) {
    asm volatile("st.shared.f64 [%0], %1;\nst.shared.f64 [%0+8], %2;\nst.shared.f64 [%0+16], %3;"
                 ::"r"(a), "d"(v[0]), "d"(v[1]), "d"(v[2]) : "memory");
  }
  static __device__ __forceinline__ void storeCluster(unsigned a, const double (&v)[3]) {
    asm volatile("st.shared::cluster.f64 [%0], %1;\nst.shared::cluster.f64 [%0+8], %2;\n"
                 "st.shared::cluster.f64 [%0+16], %3;"
                 ::"r"(a), "d"(v[0]), "d"(v[1]), "d"(v[2]) : "memory");
  }
};

// ---- substitutions -------------------------------------------------------------
// A row's data of one sweep: its first three coefficients and their columns (18
// bits each: row in the CTA, with the CTA's rank << 14 where columns cross
// CTAs), padded with a zero coefficient on the CTA's zero row.  Bit 54: up to
// three more entries, in the second table.  An entry lies in two arrays (16 + 4
// bytes in FP32, 16 + 16 in FP64), at shared addresses qa and ra.
template <typename T> struct ResEnt;
template <> struct ResEnt<float> {
  using T = float;
  using Tab = ResSweepTab<float>;
  static constexpr unsigned kB = 4;  // bytes in the second array
  float a0, a1, a2; unsigned lo, hi;
  __device__ __forceinline__ void load(unsigned qa, unsigned ra) {
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(a0), "=f"(a1), "=f"(a2), "=r"(lo) : "r"(qa) : "memory");
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(hi) : "r"(ra) : "memory");
  }
  __device__ __forceinline__ void loadGlobal(const ResSweepTab<float>& tb, int i) {
    const float4 q = tb.q[i];
    a0 = q.x; a1 = q.y; a2 = q.z; lo = __float_as_uint(q.w); hi = tb.r[i];
  }
  __device__ __forceinline__ unsigned i0() const { return lo & 0x3ffffu; }
  __device__ __forceinline__ unsigned i1() const { return __funnelshift_r(lo, hi, 18) & 0x3ffffu; }
  __device__ __forceinline__ unsigned i2() const { return (hi >> 4) & 0x3ffffu; }
  __device__ __forceinline__ bool more() const { return (hi >> 22) != 0; }
  static __device__ __forceinline__ void fetch(unsigned qa, unsigned ra, const ResSweepTab<float>& tb, int i) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(qa), "l"(tb.q + i) : "memory");
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(ra), "l"(tb.r + i) : "memory");
  }
};
template <> struct ResEnt<double> {
  using T = double;
  using Tab = ResSweepTab<double>;
  static constexpr unsigned kB = 16;
  double a0, a1, a2; unsigned lo, hi;
  __device__ __forceinline__ void load(unsigned qa, unsigned ra) {
    double p;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a0), "=d"(a1) : "r"(qa) : "memory");
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a2), "=d"(p) : "r"(ra) : "memory");
    lo = (unsigned)__double2loint(p);
    hi = (unsigned)__double2hiint(p);
  }
  __device__ __forceinline__ void loadGlobal(const ResSweepTab<double>& tb, int i) {
    const double2 q = tb.q[i], r = tb.r[i];
    a0 = q.x; a1 = q.y; a2 = r.x;
    lo = (unsigned)__double2loint(r.y);
    hi = (unsigned)__double2hiint(r.y);
  }
  __device__ __forceinline__ unsigned i0() const { return lo & 0x3ffffu; }
  __device__ __forceinline__ unsigned i1() const { return __funnelshift_r(lo, hi, 18) & 0x3ffffu; }
  __device__ __forceinline__ unsigned i2() const { return (hi >> 4) & 0x3ffffu; }
  __device__ __forceinline__ bool more() const { return (hi >> 22) != 0; }
  static __device__ __forceinline__ void fetch(unsigned qa, unsigned ra, const ResSweepTab<double>& tb, int i) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(qa), "l"(tb.q + i) : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ra), "l"(tb.r + i) : "memory");
  }
};

// The entry of a part of at most 1022 rows in FP32 (kernels_part.cu): 16 bytes,
// columns of 10 bits, bit 30: more entries.
struct PartEnt {
  using T = float;
  using Tab = PartTab<float>;
  static constexpr unsigned kB = 0;
  float a0, a1, a2; unsigned w;
  __device__ __forceinline__ void load(unsigned qa, unsigned) {
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(a0), "=f"(a1), "=f"(a2), "=r"(w) : "r"(qa) : "memory");
  }
  __device__ __forceinline__ void loadGlobal(const Tab& tb, int i) {
    const float4 q = tb.q[i];
    a0 = q.x; a1 = q.y; a2 = q.z; w = __float_as_uint(q.w);
  }
  __device__ __forceinline__ unsigned i0() const { return w & 0x3ffu; }
  __device__ __forceinline__ unsigned i1() const { return (w >> 10) & 0x3ffu; }
  __device__ __forceinline__ unsigned i2() const { return (w >> 20) & 0x3ffu; }
  __device__ __forceinline__ bool more() const { return (w >> 30) != 0; }
  static __device__ __forceinline__ void fetch(unsigned qa, unsigned, const Tab& tb, int i) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(qa), "l"(tb.q + i) : "memory");
  }
};

// first row and end of a level
__device__ __forceinline__ void ldBounds(unsigned a, int& lo, int& hi) {
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(lo), "=r"(hi) : "r"(a) : "memory");
}

// Components of the shared vector that a thread works on: all three of a row, or
// (SPLIT) one.  `uc`: the vector's shared address, plus the component's offset.
template <typename T, bool SPLIT> struct ResVec;
template <typename T> struct ResVec<T, false> {
  T v[3];
  __device__ __forceinline__ void load(unsigned at) { URow<T>::load(at, v); }
  __device__ __forceinline__ void loadCluster(unsigned at) { URow<T>::loadCluster(at, v); }
  __device__ __forceinline__ void store(unsigned at) const { URow<T>::store(at, v); }
  __device__ __forceinline__ void sub(T a, const ResVec& x) {
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = fmaT(-a, x.v[k], v[k]);
  }
};
template <> struct ResVec<float, true> {
  float v;
  __device__ __forceinline__ void load(unsigned at) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  }
  __device__ __forceinline__ void loadCluster(unsigned at) {
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  }
  __device__ __forceinline__ void store(unsigned at) const {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
  }
  __device__ __forceinline__ void sub(float a, const ResVec& x) { v = fmaT(-a, x.v, v); }
};
template <> struct ResVec<double, true> {
  double v;
  __device__ __forceinline__ void load(unsigned at) {
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
  }
  __device__ __forceinline__ void loadCluster(unsigned at) {
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
  }
  __device__ __forceinline__ void store(unsigned at) const {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
  }
  __device__ __forceinline__ void sub(double a, const ResVec& x) { v = fmaT(-a, x.v, v); }
};

template <bool CROSS, typename T, bool SPLIT>
__device__ __forceinline__ void resGather(unsigned uc, unsigned rank, unsigned idx,
                                          ResVec<T, SPLIT>& x) {
  const unsigned at = uc + URow<T>::kBytes * (CROSS ? idx & 0x3fffu : idx);
  if (CROSS && (idx >> 14) != rank) x.loadCluster(mapa(at, idx >> 14));
  else x.load(at);
}
// v -= a_u x_u for the entry's three columns in order
template <bool CROSS, typename E, typename T, bool SPLIT>
__device__ __forceinline__ void resSub(unsigned uc, unsigned rank, const E& en, ResVec<T, SPLIT>& v) {
  ResVec<T, SPLIT> x0, x1, x2;
  resGather<CROSS>(uc, rank, en.i0(), x0);
  resGather<CROSS>(uc, rank, en.i1(), x1);
  resGather<CROSS>(uc, rank, en.i2(), x2);
  v.sub(en.a0, x0);
  v.sub(en.a1, x1);
  v.sub(en.a2, x2);
}
// One substitution over the levels (DIR 0 forward, 1 backward): a level's rows in
// parallel, a barrier after each level.  The first level of a sweep has no
// entries.  Ends with a barrier.  A level is a chain -- the gathers, three
// dependent multiply-adds, a store, the barrier -- run by a warp or two, so
// what does not belong to the chain is read before the barrier that opens the
// level (its rows' entries, its bounds one level earlier), and branches and
// unrolling are kept out of the loop.  Cycles per level of an 8^3-cell part in
// FP32, 64 threads at work: 421 unrolled over the levels with the entries in
// registers, 305 as a loop that reads bounds and entries after the barrier,
// 253 with both read ahead, 178 without the branch for rows of more than three
// entries and the loop for rows beyond the walking threads (WIDE).
//   RING: the tables are in global memory; a level's entries are copied to
//   shared memory kResAhead levels before (tables that fit are there whole).
//   MORE: some rows have more than three entries; every row then applies a
//   second entry, padded like the first.
//   SPLIT: a thread per component of a row, for FP64: a warp issues an FP64
//   multiply-add every 64 cycles, so the nine of a thread per row made a
//   level 890 cycles long, the three of a component 400.
//   walk: the threads that take part, a multiple of 32 (all of them if CROSS:
//   the cluster's barrier counts every thread); rs: entries of a ring slot.
constexpr int kResAhead = 8;
// shared addresses of a sweep's tables, or of its ring (m: the second entries)
struct ResAddr { unsigned q, r, mq, mr; };
template <int DIR, bool CROSS, bool RING, bool SPLIT, bool MORE, bool WIDE, typename E>
__device__ __forceinline__ void resSweepBody(const typename E::Tab tb, const typename E::Tab more,
                                      const ResAddr ad, unsigned uBase, unsigned rank,
                                      unsigned lva, int nL, int walk, int rs) {
  using T = typename E::T;
  constexpr unsigned kB = E::kB;
  constexpr unsigned kU = URow<T>::kBytes;
  const int t = (int)threadIdx.x;
  const int nR = SPLIT ? walk / 3 : walk;  // rows at once
  const int off = SPLIT ? (t < 3 * nR ? t / 3 : 1 << 28) : t;
  const unsigned uc = SPLIT ? uBase + (unsigned)sizeof(T) * (t % 3) : uBase;
  constexpr int step = DIR == 0 ? 8 : -8;
  unsigned lp = lva + 8u * (DIR == 0 ? 1 : nL - 2);  // bounds of level q
  auto barrier = [&]() {
    if (CROSS) clWait();
    else asm volatile("bar.sync 1, %0;" ::"r"(walk) : "memory");
  };
  auto fetch = [&](int slot, int i) {
    const unsigned k = (unsigned)(slot * rs + t);
    E::fetch(ad.q + 16 * k, ad.r + kB * k, tb, i);
    if (MORE) E::fetch(ad.mq + 16 * k, ad.mr + kB * k, more, i);
  };
  if (RING) {
    for (int j = 0; j < kResAhead; ++j) {
      if (1 + j < nL && t < nR) {
        int a, b;
        ldBounds(lp + j * step, a, b);
        if (a + t < b) fetch(j, a + t);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(SPLIT ? kResAhead - 2 : kResAhead - 1) : "memory");
    if (SPLIT) {  // an entry is read by other threads than its copier
      if (CROSS) clArrive();
      barrier();
    }
  }
  int slot = 0;
  int lo, hi, lo1 = 0, hi1 = 0;
  ldBounds(lp, lo, hi);
  if (nL > 2) ldBounds(lp + step, lo1, hi1);
  E en{}, e2{};
  if (lo + off < hi) {
    const unsigned at = RING ? (unsigned)off : (unsigned)(lo + off);
    en.load(ad.q + 16 * at, ad.r + kB * at);
    if (MORE) e2.load(ad.mq + 16 * at, ad.mr + kB * at);
  }
  for (int q = 1; q < nL; ++q, lp += step) {
    int i = lo + off;
    if (i < hi) {
      const unsigned at = uc + kU * (unsigned)i;
      ResVec<T, SPLIT> v;
      v.load(at);
      resSub<CROSS>(uc, rank, en, v);
      if (MORE) resSub<CROSS>(uc, rank, e2, v);
      v.store(at);
      if (WIDE)
        for (i += nR; i < hi; i += nR) {
          const unsigned at2 = uc + kU * (unsigned)i;
          if (RING) en.loadGlobal(tb, i);
          else en.load(ad.q + 16 * (unsigned)i, ad.r + kB * (unsigned)i);
          v.load(at2);
          resSub<CROSS>(uc, rank, en, v);
          if (MORE && en.more()) {
            if (RING) e2.loadGlobal(more, i);
            else e2.load(ad.mq + 16 * (unsigned)i, ad.mr + kB * (unsigned)i);
            resSub<CROSS>(uc, rank, e2, v);
          }
          v.store(at2);
        }
    }
    if (CROSS) clArrive();
    if (RING) {
      // the slot of level q (SPLIT: of level q - 1, which every thread has
      // read) takes the entries of the level kResAhead after it
      constexpr int back = SPLIT ? 1 : 0;
      if (!SPLIT || q > 1) {
        if (q - back + kResAhead < nL && t < nR) {
          int a, b;
          ldBounds(lp + (kResAhead - back) * step, a, b);
          if (a + t < b) fetch(back ? (slot == 0 ? kResAhead - 1 : slot - 1) : slot, a + t);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      asm volatile("cp.async.wait_group %0;" ::"n"(SPLIT ? kResAhead - 3 : kResAhead - 1) : "memory");
      slot = slot + 1 == kResAhead ? 0 : slot + 1;
    }
    lo = lo1; hi = hi1;
    if (lo + off < hi) {
      const unsigned at = RING ? (unsigned)(slot * rs + off) : (unsigned)(lo + off);
      en.load(ad.q + 16 * at, ad.r + kB * at);
      if (MORE) e2.load(ad.mq + 16 * at, ad.mr + kB * at);
    }
    ldBounds(lp + 2 * step, lo1, hi1);  // (the levels have two empty ones at either end)
    barrier();
  }
}

// The same as a function of its own (the resident kernel's many forms).
template <int DIR, bool CROSS, bool RING, bool SPLIT, bool MORE, bool WIDE, typename E>
__device__ __noinline__ void resSweep(const typename E::Tab tb, const typename E::Tab more,
                                      const ResAddr ad, unsigned uBase, unsigned rank,
                                      unsigned lva, int nL, int walk, int rs) {
  resSweepBody<DIR, CROSS, RING, SPLIT, MORE, WIDE, E>(tb, more, ad, uBase, rank, lva, nL, walk, rs);
}

// ---- sums ------------------------------------------------------------------------
// Sum of M values (a power of two) over a warp.  A lane adds M/2, M/4, ..., 1
// values while the values are spread over the lanes, then one value per
// remaining step: 9 (M = 8) or 6 (M = 4) additions per lane instead of 5 M --
// an FP64 addition of a warp takes ~19 cycles of the SM's FP64 unit.  Value k
// ends in the lanes k * 32 / M + (0 .. 32 / M - 1).  The pairs of lanes that are
// added, and their order, are blockSum's and sum64's (16, 8, 4, 2, 1 apart).
// N such sums side by side: their chains (some 130 cycles a step) overlap.
template <int M, int N>
__device__ __forceinline__ void warpSpreadSums(double (&v)[N][M], double (&s)[N]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = M / 2, o = 16; h >= 1; h /= 2, o /= 2) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
      for (int k = 0; k < h; ++k) {
        const double give = up ? v[n][k] : v[n][k + h];
        const double keep = up ? v[n][k + h] : v[n][k];
        v[n][k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
  }
#pragma unroll
  for (int n = 0; n < N; ++n) s[n] = v[n][0];
#pragma unroll
  for (int o = 32 / M / 2; o >= 1; o /= 2)
#pragma unroll
    for (int n = 0; n < N; ++n) s[n] += __shfl_xor_sync(0xffffffffu, s[n], o);
}
template <int M>
__device__ __forceinline__ double warpSpreadSum(double (&v)[M]) {
  double w[1][M], s[1];
#pragma unroll
  for (int k = 0; k < M; ++k) w[0][k] = v[k];
  warpSpreadSums<M, 1>(w, s);
  return s[0];
}
// warpSpreadSums<4, N> of N x 3 floats x (and their compensations c, added to them first:
// PAIR), component k in the lanes 8 k ...; the same bits.  Where every float is a multiple
// of 2^-46 of the largest one's power of two, the FP64 additions of that sum are exact,
// whatever their order, and integer sums of the warp give it: some 70 instructions and 9
// warp reductions instead of 6 FP64 additions, which take 114 cycles of the SM's FP64 unit
// and 660 one after the other.  Else the additions are done.
template <int N, bool PAIR>
__device__ __forceinline__ void warpFloatSums(const float (&x)[N][3], const float (&c)[N][3], double (&s)[N]) {
  constexpr int L = 23;  // bits below those of the largest: 24 + 23 + 5 < 53
  const int comp = (int)(threadIdx.x & 31) >> 3;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    int top[3], hi[3], lo[3];
    bool exact = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      unsigned a = __float_as_uint(x[n][k]) & 0x7fffffffu;
      if (PAIR) a = max(a, __float_as_uint(c[n][k]) & 0x7fffffffu);
      top[k] = max(1, (int)(__reduce_max_sync(0xffffffffu, a) >> 23));
      exact = exact && top[k] < 255;
      hi[k] = lo[k] = 0;
      auto add = [&](float f) {
        const unsigned b = __float_as_uint(f), q = b & 0x7fffffffu;
        const int e = max(1, (int)(q >> 23)), sh = top[k] - e;
        const unsigned m = (q & 0x7fffffu) | (q >= 0x00800000u ? 0x800000u : 0u);
        // m 2^L >> sh in two parts of L bits and the rest
        const unsigned h = sh < 32 ? m >> sh : 0u;
        unsigned l;
        if (sh <= L) {
          l = (m << (L - sh)) & ((1u << L) - 1);
        } else {
          const int d = sh - L;
          l = d < 32 ? m >> d : 0u;
          exact = exact && (d < 32 ? l << d : 0u) == m;
        }
        hi[k] += (b >> 31) ? -(int)h : (int)h;
        lo[k] += (b >> 31) ? -(int)l : (int)l;
      };
      add(x[n][k]);
      if (PAIR) add(c[n][k]);
    }
    if (__all_sync(0xffffffffu, exact)) {
      long long sum = 0;
      int e = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const long long t = ((long long)__reduce_add_sync(0xffffffffu, hi[k]) << L) +
                            (long long)__reduce_add_sync(0xffffffffu, lo[k]);
        if (comp == k) { sum = t; e = top[k]; }
      }
      // sum 2^(e - 150 - L)
      const unsigned long long u = (unsigned long long)(sum < 0 ? -sum : sum);
      const int z = __clzll((long long)u);
      const unsigned long long m = (u << (z & 63)) >> 11 & 0xfffffffffffffull;
      const unsigned long long ex = (unsigned long long)(1023 + 63 - z + e - 150 - L);
      const unsigned long long r = u ? ex << 52 | m | (sum < 0 ? 1ull << 63 : 0ull) : 0ull;
      s[n] = __longlong_as_double((long long)r);
    } else {
      double v[4] = {0, 0, 0, 0};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        v[k] = toF64(x[n][k]);
        if (PAIR) v[k] += toF64(c[n][k]);
      }
      s[n] = warpSpreadSum<4>(v);
    }
  }
}
template <int N>
__device__ __forceinline__ void warpFloatSums(const float (&x)[N][3], double (&s)[N]) {
  warpFloatSums<N, false>(x, x, s);
}

// Sum over the lanes below n (the others hold zero), in lane 0: blockSum's tree without
// its steps that add zeros (a loop: unrolled, they would be added and dropped).
__device__ __forceinline__ double warpTree(double v, int n = 32) {
#pragma unroll 1
  for (int o = n > 32 ? 16 : n > 1 ? 1 << (31 - __clz(n - 1)) : 0; o > 0; o >>= 1)
    v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// locGroupsTotal's sums of six values over the part groups into out[0..5], by W warps:
// grp holds them for 64 lanes (lane v: groups v, v + 64, ...).  The caller synchronises
// the CTA before and after it.
template <int W>
__device__ __forceinline__ void groupTotal(const double* grp, int nGrp, double* out) {
  const int lane = (int)threadIdx.x & 31, wid = (int)threadIdx.x >> 5;
  for (int k = wid; k < 6; k += W) {
    double s = warpTree(lane < nGrp ? grp[6 * lane + k] : 0.0, nGrp);
    if (nGrp > 32) s += warpTree(32 + lane < nGrp ? grp[6 * (32 + lane) + k] : 0.0, nGrp - 32);
    if (lane == 0) out[k] = s;
  }
}

}  // namespace s4g
