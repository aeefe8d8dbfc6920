// Warp sums and scalar tests of the solvers' kernels, kept off GB300's FP64 pipe:
// it starts one warp's instruction per 64 cycles and SM quarter, whatever the
// number of useful lanes.
#pragma once

#include <cuda_runtime.h>

namespace bmfp
{
namespace reduce
{
// Sum over a warp, the same on every lane: each value's mantissa shifted to
// the largest exponent of the warp (five guard bits: more than the FP64 adds
// of a butterfly keep), the integers added exactly in three limbs by redux,
// one rounding (to nearest, halves away from zero) where the result is put
// together. A butterfly's five dependent warp-wide FP64 adds take 600 cycles
// on GB300, whose FP64 pipe starts one warp's instruction per 64 cycles and SM
// quarter, and keep that pipe busy throughout; this runs on the integer pipes.
// Zeros, subnormals, infinities and NaN go to the butterfly.
// NK values at a time: their chains of redux run side by side.
template <int NK> __device__ __forceinline__ void warp_sums (const double (&v)[NK], double (&out)[NK])
{
  constexpr unsigned kAll = 0xffffffffu;
  int top[NK];
#pragma unroll
  for (int k = 0; k < NK; k++)
    top[k] = (int) __reduce_max_sync (kAll, (unsigned) ((__double2hiint (v[k]) >> 20) & 0x7ff));
#pragma unroll
  for (int k = 0; k < NK; k++)
    {
      const long long bits = __double_as_longlong (v[k]);
      const int ex = (int) ((bits >> 52) & 0x7ff);
      const int d = top[k] - ex;
      long long m = ex ? ((bits & 0xfffffffffffffll) | 0x10000000000000ll) << 5 : 0;
      m = d < 58 ? (m + ((1ll << d) >> 1)) >> d : 0;
      if (bits < 0)
        m = -m;
      const unsigned lo = __reduce_add_sync (kAll, (unsigned) (m & 0xfffff));
      const unsigned mid = __reduce_add_sync (kAll, (unsigned) ((m >> 20) & 0xfffff));
      const int hi = __reduce_add_sync (kAll, (int) (m >> 40));
      const long long sum = ((long long) hi << 40) + ((long long) mid << 20) + lo;
      unsigned long long u = (unsigned long long) (sum < 0 ? -sum : sum);
      const int lz = __clzll ((long long) u);
      u <<= lz & 63;
      const unsigned long long man = (u >> 11) + ((u >> 10) & 1); // 2^52 .. 2^53
      const unsigned long long r = ((unsigned long long) (top[k] + 5 - lz) << 52) + man;
      out[k] = __longlong_as_double (sum ? (long long) (r | (sum < 0 ? 1ull << 63 : 0)) : 0);
    }
#pragma unroll
  for (int k = 0; k < NK; k++)
    if (top[k] < 64 || top[k] > 2047 - 64)
      {
        double a = v[k];
        if (__any_sync (kAll, (__double_as_longlong (a) << 1) != 0))
#pragma unroll
          for (int off = 16; off > 0; off >>= 1)
            a += __shfl_xor_sync (kAll, a, off);
        out[k] = a;
      }
}

__device__ __forceinline__ double warp_sum (double v)
{
  const double in[1] = { v };
  double out[1];
  warp_sums<1> (in, out);
  return out[0];
}

// Sum over a warp and the M values of each of its lanes (M <= 32), as
// warp_sums does it: 1024 terms of 58 bits take 68.
template <int M> __device__ __forceinline__ double warp_sum_of (const double (&v)[M])
{
  constexpr unsigned kAll = 0xffffffffu;
  static_assert (M <= 32, "a lane's terms fit 63 bits");
  int ex[M], top = 0;
#pragma unroll
  for (int j = 0; j < M; j++)
    {
      ex[j] = (__double2hiint (v[j]) >> 20) & 0x7ff;
      top = max (top, ex[j]);
    }
  top = (int) __reduce_max_sync (kAll, (unsigned) top);
  if (top < 64 || top > 2047 - 64)
    {
      double a = v[0];
#pragma unroll
      for (int j = 1; j < M; j++)
        a += v[j];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        a += __shfl_xor_sync (kAll, a, off);
      return a;
    }
  long long m = 0;
#pragma unroll
  for (int j = 0; j < M; j++)
    {
      const long long bits = __double_as_longlong (v[j]);
      const int d = top - ex[j];
      long long a = ex[j] ? ((bits & 0xfffffffffffffll) | 0x10000000000000ll) << 5 : 0;
      a = d < 58 ? (a + ((1ll << d) >> 1)) >> d : 0;
      m += bits < 0 ? -a : a;
    }
  const unsigned lo = __reduce_add_sync (kAll, (unsigned) (m & 0xfffff));
  const unsigned mid = __reduce_add_sync (kAll, (unsigned) ((m >> 20) & 0xfffff));
  const int hi = __reduce_add_sync (kAll, (int) (m >> 40));
  // in units of 2^20, and the rest
  long long a = ((long long) hi << 20) + mid + (lo >> 20);
  unsigned b = lo & 0xfffff;
  const bool minus = a < 0;
  if (minus)
    {
      a = -a - (b != 0);
      b = (0x100000u - b) & 0xfffff;
    }
  if (a == 0 && b == 0)
    return 0.0;
  // normalised: bit 63 set, bits below the last place of 68 dropped
  const int la = __clzll (a);
  int lz; // zeros above the value's first bit in 84 bits
  unsigned long long u;
  if (la < 64)
    {
      lz = la;
      u = la >= 20 ? ((unsigned long long) a << la) | ((unsigned long long) b << (la - 20))
                   : ((unsigned long long) a << la) | (b >> (20 - la));
    }
  else
    {
      lz = 64 + __clz ((int) b) - 12;
      u = (unsigned long long) b << (32 + __clz ((int) b));
    }
  const unsigned long long man = (u >> 11) + ((u >> 10) & 1); // 2^52 .. 2^53
  const unsigned long long r = ((unsigned long long) (top + 5 + 20 - lz) << 52) + man;
  return __longlong_as_double ((long long) (r | (minus ? 1ull << 63 : 0)));
}

// Tests of doubles on the integer pipes (a DSETP costs what a DFMA does).
__device__ __forceinline__ bool is_zero (double v) { return (__double_as_longlong (v) << 1) == 0; }
__device__ __forceinline__ bool is_finite (double v) { return ((__double2hiint (v) >> 20) & 0x7ff) != 0x7ff; }
// a < b for a and b non-negative, infinite or NaN (false then).
__device__ __forceinline__ bool less_abs (double a, double b)
{
  const unsigned long long ua = (unsigned long long) __double_as_longlong (a),
                           ub = (unsigned long long) __double_as_longlong (b);
  return ua < ub && ub <= 0x7ff0000000000000ull;
}

// (double) x by integer operations, for every x: a conversion costs what a DFMA
// does. Subnormals are scaled into the normal range first.
__device__ __forceinline__ double widen (float x)
{
  const bool tiny = (__float_as_uint (x) & 0x7fffffffu) < 0x00800000u;
  const unsigned u = __float_as_uint (tiny ? x * 4294967296.0f : x), m = u & 0x7fffffffu;
  // exponent bias 127 -> 1023 (less the 32 of the scaling); infinities and NaN
  // keep the largest exponent
  const unsigned bias = m >= 0x7f800000u ? 0x70000000u : tiny ? 0x36000000u : 0x38000000u;
  const unsigned hi = (u & 0x80000000u) | (m ? (m >> 3) + bias : 0u);
  return __hiloint2double ((int) hi, (int) (u << 29));
}
__device__ __forceinline__ double widen (double x) { return x; }
} // namespace reduce
} // namespace bmfp
