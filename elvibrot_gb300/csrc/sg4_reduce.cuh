// sg4_reduce.cuh -- the weighted accumulation of the Smolyak terms
// (tabR_AT_iG_TO_tabPackedBasis, sub_module_basis_BtoG_GtoB_SG4.f90:1255):
// the sum of a packed function's term contributions.
//
// The Smolyak weights alternate in sign and cancel, so plain sums lose digits,
// and compensated ones run seven dependent FP64 additions a value on a unit
// that does two a clock and SM.  Here the values of a function and column are
// added as 128-bit integers on the scale of their largest exponent: integer
// instructions only, and an associative sum, so that a block's threads share
// it freely and the result does not depend on how.  A value is cut below
// 2^-116 of the largest one's leading bit (2^(k-116) for a list of up to
// 2^(9+k) values), so n values are summed to n 2^-116 of it, against some
// n 2^-106 for the compensated sums, and rounded once.  Bound by the latency of
// an index and a value load.  Against two kernels of compensated chunk sums and
// joins: 4-D L=7, one complex vector, an order-30 Chebyshev step 1.53 -> 1.01 ms
// and an RK4 stage's two kernels 33 -> 10 us; one vector of a 3-D L=6 operator
// 34.5 -> 24.3 us.
#pragma once
#include <cuda_runtime.h>

namespace evr {

#define EVR_SUM_THREADS 128
#define EVR_SUM_KEEP 4  // values a thread keeps between the two passes

// the largest value's 53-bit mantissa has its top at bit 116 - k: above are the
// sign and room for 2^(9+k) values
__device__ __forceinline__ int sum_shift(long long n) { return n > 512 ? 55 - __clzll(n - 1) : 0; }

__device__ __forceinline__ __int128 sum_term(double x, int emax, int k) {
  const long long b = __double_as_longlong(x);
  const int e = (int)(b >> 52) & 0x7ff;
  const unsigned long long m = ((unsigned long long)b & 0xFFFFFFFFFFFFFull) | (e ? 0x10000000000000ull : 0ull);
  const int d = min(emax - max(e, 1) + k, 127);
  const __int128 v = (__int128)(((unsigned __int128)m << 64) >> d);
  return b < 0 ? -v : v;
}

__device__ __forceinline__ double sum_value(__int128 v, int emax, int k) {
  const bool neg = v < 0;
  unsigned __int128 a = neg ? (unsigned __int128)(-v) : (unsigned __int128)v;
  if (a == 0) return 0.0;
  const unsigned long long hi = (unsigned long long)(a >> 64);
  const int lz = hi ? __clzll((long long)hi) : 64 + __clzll((long long)(unsigned long long)a);
  a <<= lz;
  const unsigned long long top = (unsigned long long)(a >> 64) | ((unsigned long long)a != 0);  // sticky
  const double r = scalbn(__ull2double_rn(top), k - lz + emax - 1075);
  return neg ? -r : r;
}

__device__ __forceinline__ __int128 shfl_xor128(__int128 v, int off) {
  const unsigned long long lo = __shfl_xor_sync(0xffffffffu, (unsigned long long)v, off);
  const unsigned long long hi = __shfl_xor_sync(0xffffffffu, (unsigned long long)(v >> 64), off);
  return (__int128)(((unsigned __int128)hi << 64) | lo);
}

// The sums of a function over its contributions contrib[idx[q] * nv + v], q in
// [q0, q1), for the columns v in [v0, v0 + cw), into out[v]; one block of
// EVR_SUM_THREADS.  The cw columns (a power of two up to 32) lie side by side
// in a warp, the rest of the threads share the list.  A sum over a value that
// is not finite is NaN (the compensated sums gave NaN as well).
__device__ __forceinline__ void sum_function(const double* __restrict__ contrib, const long long* __restrict__ idx,
                                             long long q0, long long q1, int nv, int v0, int cw,
                                             double* __restrict__ out) {
  __shared__ int se[EVR_SUM_THREADS];
  __shared__ __int128 ss[EVR_SUM_THREADS];
  const int tid = threadIdx.x, col = tid & (cw - 1), lane = tid & 31, warp = tid >> 5;
  const int step = EVR_SUM_THREADS / cw;
  const int v = v0 + col;
  const bool on = v < nv;
  const int k2 = sum_shift(q1 - q0);
  double keep[EVR_SUM_KEEP];
  int em = 1;
  const long long qs = q0 + tid / cw;
  if (on) {
#pragma unroll
    for (int k = 0; k < EVR_SUM_KEEP; ++k) {
      const long long q = qs + (long long)k * step;
      keep[k] = q < q1 ? contrib[idx[q] * nv + v] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < EVR_SUM_KEEP; ++k) em = max(em, (__double2hiint(keep[k]) >> 20) & 0x7ff);
#pragma unroll 4
    for (long long q = qs + (long long)EVR_SUM_KEEP * step; q < q1; q += step)
      em = max(em, (__double2hiint(contrib[idx[q] * nv + v]) >> 20) & 0x7ff);
  }
  for (int off = 16; off >= cw; off >>= 1) em = max(em, __shfl_xor_sync(0xffffffffu, em, off));
  if (lane < cw) se[warp * cw + lane] = em;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < EVR_SUM_THREADS / 32; ++w) em = max(em, se[w * cw + col]);
  __int128 s = 0;
  if (on) {
#pragma unroll
    for (int k = 0; k < EVR_SUM_KEEP; ++k) s += sum_term(keep[k], em, k2);
#pragma unroll 4
    for (long long q = qs + (long long)EVR_SUM_KEEP * step; q < q1; q += step)
      s += sum_term(contrib[idx[q] * nv + v], em, k2);
  }
  for (int off = 16; off >= cw; off >>= 1) s += shfl_xor128(s, off);
  if (lane < cw) ss[warp * cw + lane] = s;
  __syncthreads();
  if (tid < cw && on) {
    s = 0;
#pragma unroll
    for (int w = 0; w < EVR_SUM_THREADS / 32; ++w) s += ss[w * cw + col];
    out[v] = em == 0x7ff ? __longlong_as_double(0x7FF8000000000000LL) : sum_value(s, em, k2);
  }
}

}  // namespace evr
