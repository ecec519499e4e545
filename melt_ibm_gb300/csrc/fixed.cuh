// fixed.cuh -- FP64 values as 64-bit fixed point with a shared exponent, for
// kernels that do their arithmetic on the integer pipe (fft_int.cuh, the
// explicit terms of stencil.cu): an FP64 instruction costs as much issue as
// some 32 integer ones on this part.
//
// The products of halves also build for the host (without CUDA), so that a
// CPU test can check them against exact arithmetic.
#pragma once

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#define FIXED_FN __host__ __device__ __forceinline__
#else
#define FIXED_FN inline
#endif

namespace mibm {
namespace fixed {

// signed halves of x: x = hi 2^32 + lo, lo in [-2^31, 2^31).  -lo does not
// always fit a half: products are subtracted, halves never negated.
FIXED_FN void halves(long long x, int& hi, int& lo) {
  lo = (int)x;
  hi = (int)(x >> 32) + (int)((unsigned)lo >> 31);
}
FIXED_FN long long wide(int a, int b) { return (long long)a * b; }

struct I2 { long long x, y; };
// (cos, -sin) 2^62 of the forward twiddle as signed halves
struct Tw { int ch, cl, sh, sl; };

// v w / 2^S (w, or its conjugate for INV), S = 1 or 2; a component is
// within half a unit plus the two products of low halves left out, 2^-S each
template <int S, bool INV>
FIXED_FN I2 twiddle(I2 v, Tw w) {
  int xh, xl, yh, yl;
  halves(v.x, xh, xl);
  halves(v.y, yh, yl);
  constexpr long long half = 1ll << (29 + S);
  // forward: (x c - y s, y c + x s); inverse: (x c + y s, y c - x s)
  const long long pr = wide(yh, w.sh), pi = wide(xh, w.sh);
  const long long qr = wide(yh, w.sl) + wide(yl, w.sh), qi = wide(xh, w.sl) + wide(xl, w.sh);
  const long long mr = INV ? wide(xh, w.ch) + pr : wide(xh, w.ch) - pr;
  const long long mi = INV ? wide(yh, w.ch) - pi : wide(yh, w.ch) + pi;
  const long long lr = half + wide(xh, w.cl) + wide(xl, w.ch) + (INV ? qr : -qr);
  const long long li = half + wide(yh, w.cl) + wide(yl, w.ch) + (INV ? -qi : qi);
  return I2{mr * (1ll << (2 - S)) + (lr >> (30 + S)), mi * (1ll << (2 - S)) + (li >> (30 + S))};
}

#if defined(__CUDACC__)

// biased exponent field (zero and subnormal values: 0)
__device__ __forceinline__ int expo(double d) { return (int)((__double_as_longlong(d) >> 52) & 0x7ff); }

// d at the exponent E >= 1 (at least its own): d 2^(1075 - E + UP), cut to an
// integer (UP guard bits below the last bit of the largest value keep what
// the cut loses out of the result's rounding); below 2^(53 + UP) in magnitude
template <int UP>
__device__ __forceinline__ long long from_double(double d, int E) {
  const long long b = __double_as_longlong(d);
  const int e = (int)((b >> 52) & 0x7ff);
  const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffull) | (e ? 1ull << 52 : 0);
  const long long a = (long long)((m << UP) >> min(E - max(e, 1), 63));
  const long long s = b >> 63;
  return (a ^ s) - s;
}

// to_double below the normal range or above it: integer operations only (an
// integer to FP64 conversion issues at the FP64 rate, and would be taken on
// every call if it were inlined)
static __device__ __noinline__ double to_double_edge(unsigned long long s, unsigned long long a, int e) {
  if (e > 2046) return __longlong_as_double((long long)(s | 0x7ff0000000000000ull));
  const int sh = 12 - e;                                // a's leading bit at 63; subnormals end at bit 0
  const unsigned long long m = sh > 63 ? 0 : ((a >> (sh - 1)) + 1) >> 1;
  return __longlong_as_double((long long)(s | m));
}

// f 2^(X - 1075) as a double, rounded to nearest (halves away from zero)
__device__ __forceinline__ double to_double(long long f, int X) {
  const unsigned long long s = (unsigned long long)f & 0x8000000000000000ull;
  const long long n = f >> 63;
  unsigned long long a = (unsigned long long)((f ^ n) - n);
  const int lz = __clzll((long long)a);
  a <<= lz & 63;                                         // 2^63 <= a < 2^64, or 0
  const int e = 63 - lz + X - 52;                        // biased exponent of the leading bit: 63 - lz + (X - 1075) + 1023
  if (a != 0 && (unsigned)(e - 1) >= 2045u) return to_double_edge(s, a, e);
  const unsigned long long m = (a >> 11) + ((a >> 10) & 1);
  const unsigned long long r = ((unsigned long long)(unsigned)(e - 1) << 52) + m;
  return a == 0 ? 0.0 : __longlong_as_double((long long)(s | r));
}

__device__ __forceinline__ double quiet_nan() { return __longlong_as_double(0x7ff8000000000000ll); }

// a b / 2^64 without lo*lo, rounded down: within one unit (|a|, |b| < 2^62)
__device__ __forceinline__ long long mul_high(long long a, long long b) {
  int ah, al, bh, bl;
  halves(a, ah, al);
  halves(b, bh, bl);
  return wide(ah, bh) + ((wide(ah, bl) + wide(al, bh)) >> 32);
}
__device__ __forceinline__ long long square_high(long long a) {
  int ah, al;
  halves(a, ah, al);
  return wide(ah, ah) + (wide(ah, al) >> 31);
}
#endif

}  // namespace fixed
}  // namespace mibm
