// Helpers shared by the PCG kernels.
#pragma once

#include "device_common.cuh"
#include "kernels.cuh"

namespace s4g {

// Asynchronous global->shared copies (LDGSTS): a part's static data is put in
// flight at once and waited for with one hardware wait.
template <int BYTES>
__device__ __forceinline__ void cpAsync(void* sm, const void* gm) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(sm);
  if (BYTES == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(gm) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gm) : "memory");
}
template <typename T>
__device__ __forceinline__ void cpAsyncT(T* sm, const T* gm) { cpAsync<sizeof(T)>(sm, gm); }
__device__ __forceinline__ void cpAsyncWaitAll() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_all;" ::: "memory");
}

// Sum of T values: plain for double; Neumaier-compensated for float.
template <typename T> struct Acc;
template <> struct Acc<double> {
  double s = 0;
  __device__ __forceinline__ void add(double x) { s += x; }
  __device__ __forceinline__ double value() const { return s; }
};
template <> struct Acc<float> {
  float s = 0, c = 0;
  __device__ __forceinline__ void add(float x) {
    const float t = s + x;
    c += (fabsf(s) >= fabsf(x)) ? (s - t) + x : (x - t) + s;
    s = t;
  }
  __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

// (double)x of a float by integer instructions: a conversion is an operation of the
// FP64 unit, one warp instruction per 19 cycles of an SM.
__device__ __forceinline__ double toF64(float x) {
  const unsigned b = __float_as_uint(x), a = b & 0x7fffffffu;
  unsigned e = (a >> 23) + 896u, m = a & 0x7fffffu;
  if (a < 0x00800000u) {  // zero, subnormal
    const int z = __clz((int)a) - 8;
    m = a ? (a << z) & 0x7fffffu : 0u;
    e = a ? 897u - (unsigned)z : 0u;
  }
  if (a >= 0x7f800000u) e = 2047u;  // infinite, NaN
  return __hiloint2double((int)((b & 0x80000000u) | e << 20 | m >> 3), (int)(m << 29));
}
__device__ __forceinline__ double toF64(double x) { return x; }
// Acc::value(), converted so
__device__ __forceinline__ double accValue(const Acc<double>& a) { return a.s; }
__device__ __forceinline__ double accValue(const Acc<float>& a) { return toF64(a.s) + toF64(a.c); }

// sum|r| / normFactor < the limit (tolerance, or relTol * the initial residual),
// as that quotient compares, but divided only where rounding could decide (an FP64
// division takes 564 cycles of the chain).
__device__ __forceinline__ double pcgLimit(const Controls& c, double initRes) {
  return fmax(c.tol, c.relTol > 1e-20 ? c.relTol * initRes : 0.0);
}
__device__ __forceinline__ bool pcgConverged(double s, double norm, double lim) {
  const double b = lim * norm;
  if (b > 1e-290) {
    if (s < b * (1 - 4e-15)) return true;
    if (s > b * (1 + 4e-15)) return false;
  }
  return s / norm < lim;
}

// A wait that gave up or a value that is not finite ends the loop with its iteration (the
// loop's own condition looks only once in kPcgUnroll of them).
__device__ __forceinline__ bool pcgFailed(const DevState* st) {
  return (*(const volatile unsigned*)&st->status & (kErrTimeout | kErrNaN)) != 0;
}

// End of a processor-local preconditioner launch, by warp 0 of its last CTA:
// S = w.r of the components, then sum|r| (S[k] in lane k and k + 3 for lanes
// 0 .. 5 of `mine`).  Per component the residual test of the pending iteration,
// beta and wArA, and whether the loop goes on.  A lane per component with its
// state read at once: one thread going through the three with their dependent
// loads and divisions (564 cycles each) took about 6 us of every iteration.
__device__ __forceinline__ void pcgDecideBeta(const Controls& c, DevState* st, double mine, bool anyPend) {
  const int l = threadIdx.x & 31;
  const double rs = __shfl_down_sync(0xffffffffu, mine, 3);
  int act = 0;
  if (l < 3) {
    const int pend = st->pending[l], it0 = st->nIter[l], a0 = st->active[l];
    const double nf = st->normFactor[l], ir = st->initRes[l], wa = st->wArA[l];
    act = a0;
    int it = it0;
    if (pend) {
      st->pending[l] = 0;
      st->nIter[l] = ++it;
      const bool conv = pcgConverged(rs, nf, pcgLimit(c, ir));
      const bool fin = isfinite(rs);
      if (!fin) atomicOr(&st->status, kErrNaN);
      act = (!conv && it < c.maxIter && fin) ? 1 : 0;
      st->active[l] = act;
      if (!act) st->finalRes[l] = rs / nf;
    }
    if (act) {
      st->beta[l] = it == 0 ? 0.0 : mine / wa;
      st->wArA[l] = mine;
    }
  }
  const unsigned any = __ballot_sync(0xffffffffu, act != 0);
  if (l == 0) {
    if (anyPend) st->pcgIter += 1;
    st->pcgContinue = any != 0 && !pcgFailed(st);
  }
}

// End of the product's launch, by warp 0 of its last CTA: mine = p.q of the
// component in lanes 0 .. 2.  alpha, and which components have an iteration
// pending; pb: the p buffer the launch read.
__device__ __forceinline__ void pcgDecideAlpha(DevState* st, double mine, int pb) {
  const int l = threadIdx.x & 31;
  int on = 0;
  if (l < 3) {
    const int act = st->active[l];
    const double nf = st->normFactor[l], wa = st->wArA[l];
    st->xPend[l] = 0;  // applied by this pass
    if (act) {
      st->wApA[l] = mine;
      if (fabs(mine) < 1e-300 * nf) {  // checkSingularity: stop this component
        st->active[l] = 0;
      } else {
        if (mine <= 0) atomicOr(&st->status, kErrIndefinite);
        st->alpha[l] = wa / mine;
        st->pending[l] = 1;
        st->xPend[l] = 1;
        on = 1;
      }
    }
  }
  const unsigned any = __ballot_sync(0xffffffffu, on != 0);
  if (l == 0) {
    st->pbuf = pb ^ 1;
    st->pcgContinue = any != 0;
  }
}

// 16-byte asynchronous global->shared copy that bypasses L1 (data read once).
__device__ __forceinline__ void cpAsync16(void* sm, const void* gm) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(sm);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gm) : "memory");
}

}  // namespace s4g
