// Host build of the products of halves of melt_ibm_gb300/csrc/fixed.cuh and of
// fpconv.cuh's guarded sum for the CPU tests: the same source the kernels use,
// over a C ABI in batches.
#include <stdint.h>

#include "fixed.cuh"
#include "fpconv.cuh"

extern "C" {

// n complex products v w / 2^shift (v: pairs; w: quadruples of halves)
void fixed_twiddle(int shift, int inverse, long long n, const long long* v, const int* w, long long* out) {
  using namespace mibm::fixed;
  for (long long t = 0; t < n; ++t) {
    const I2 a{v[2 * t], v[2 * t + 1]};
    const Tw b{w[4 * t], w[4 * t + 1], w[4 * t + 2], w[4 * t + 3]};
    const I2 r = shift == 1 ? (inverse ? twiddle<1, true>(a, b) : twiddle<1, false>(a, b))
                            : (inverse ? twiddle<2, true>(a, b) : twiddle<2, false>(a, b));
    out[2 * t] = r.x;
    out[2 * t + 1] = r.y;
  }
}

// n sextuples; ok: whether the sum was taken
void guarded_sum6(long long n, const double* x, double* out, int* ok) {
  for (long long t = 0; t < n; ++t, x += 6) {
    out[t] = 0.0;
    ok[t] = mibm::sum6_guarded(x[0], x[1], x[2], x[3], x[4], x[5], out[t]);
  }
}
}
