// fft_int.cuh -- the FP64 Poisson solve's x and y transforms (phcalc.f90:11-97,
// same chain and conventions as fft.cu) on the integer pipe.
//
// An FP64 instruction occupies a quarter of an SM for 64 clocks on this part;
// a 64-bit integer addition takes two instructions and a 64-bit product's
// upper half three wide multiply-adds, each a few clocks.  The FP64 passes
// (fft_fast.cuh) are bound by 25 FP64 operations per complex value, so here a
// line is transformed in 64-bit fixed point with one exponent per line (block
// floating point):
//   load    the line's largest exponent is found, every value becomes
//           mantissa << 6 (x inverse: << 5) at that exponent;
//   stages  radix-4/2/3 Stockham stages as in fft_fast.cuh; before each stage
//           but the first, values are halved (rounded) as often as the stage
//           may grow them: ceil(log2(points combined)) in all, so that
//           |z| <= 2^61.5 always holds;
//   store   back to FP64, rounded once.
// A twiddle factor is held to 2^-62 in two 32-bit halves; a product is hi*hi +
// (hi*lo + lo*hi + 2^31 >> 32), which leaves out lo*lo: below a unit of the
// last place kept.  The unit at the end is n 2^-61 of the line's largest
// input, against outputs of about sqrt(n) times its rms: below 2^-55 of them
// for inputs up to 16 times their rms, less than the rounding of the result.
// One line against extended precision, before that rounding, relative 2-norm (FP64
// stages): noise 1e-17 .. 6e-17 (2e-16); a spike, the worst input for one
// scale per line, 5e-17 at 128, 1.4e-16 at 192, 2.2e-16 at 512 (6e-17 .. 1.2e-16).
// The whole solve against one in extended precision, relative 2-norm of phi /
// of its gradient, with the z lines of fft_int_z.cu (the FP64 passes): 32^3 noise
// 2.9e-16 / 3.4e-16 (1.1e-15 / 7.8e-16), 64^3 noise 2.5e-16 / 4.4e-16 (3.4e-15 /
// 1.2e-15), one spike 2.3e-16 / 4.1e-16 (3.7e-15 / 1.2e-15), values over nine
// decades 2.7e-16 / 4.4e-16 (4.1e-15 / 1.2e-15).  A line that holds an infinity
// or a NaN comes out as NaN.
// Per pass, FP64 -> integer: 128^3 x forward 61 -> 20, y 60 -> 20, x inverse 60
// -> 20 us; 192^3 212 -> 58, 192 -> 57, 208 -> 56 us; 108 x 108 x 72 (no
// compile-time FP64 instance) 45 -> 15, 47 -> 15, 44 -> 15 us.
#pragma once

#include "fft_common.cuh"
#include "fixed.cuh"

namespace mibm {
namespace intfft {

using namespace fixed;

__host__ __device__ constexpr int nstages(int n) {
  int s = 0;
  while (n % 4 == 0) { n /= 4; ++s; }
  while (n % 2 == 0) { n /= 2; ++s; }
  while (n % 3 == 0) { n /= 3; ++s; }
  return s;
}
__host__ __device__ constexpr int radix_at(int n, int st) {
  int s = 0;
  while (n % 4 == 0) { if (s == st) return 4; n /= 4; ++s; }
  while (n % 2 == 0) { if (s == st) return 2; n /= 2; ++s; }
  while (n % 3 == 0) { if (s == st) return 3; n /= 3; ++s; }
  return 1;
}
__host__ __device__ constexpr int clog2(int n) { int l = 0; while ((1 << l) < n) ++l; return l; }
// halvings over all stages
__host__ __device__ constexpr int total_shift(int n) { return clog2(n) - clog2(radix_at(n, 0)); }

// Lines per block: 8 at least (128 contiguous bytes per spectrum row), more
// for short lines so that a block has about 1024 values
template <int N>
struct Shape {
  static constexpr int T = 256;
  static constexpr int L = N >= 128 ? 8 : (N >= 64 ? 16 : 32);
  static constexpr int ES = L + 1;
  static constexpr int kWarps = T / 32, kLinesPerWarp = L / kWarps;
  static constexpr size_t smem = sizeof(Tw) * N + sizeof(I2) * (size_t)N * ES;
};

// x / 2^S, rounded
template <int S>
__device__ __forceinline__ long long down(long long x) { return (x + (1ll << (S - 1))) >> S; }
template <int S>
__device__ __forceinline__ I2 down(I2 v) { return I2{down<S>(v.x), down<S>(v.y)}; }

__device__ __forceinline__ I2 add(I2 a, I2 b) { return I2{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ I2 sub(I2 a, I2 b) { return I2{a.x - b.x, a.y - b.y}; }

// x sqrt(3)/2
__device__ __forceinline__ long long times_s3(long long x) {
  constexpr long long c = 3993837246235628775ll;        // sqrt(3)/2 2^62
  constexpr int cl = (int)(unsigned)(c & 0xffffffffll), ch = (int)((c - cl) >> 32);
  int h, l;
  halves(x, h, l);
  return (wide(h, ch) << 2) + ((wide(h, cl) + wide(l, ch) + (1ll << 29)) >> 30);
}

template <int R, bool INV>
__device__ __forceinline__ void butterfly(I2 (&v)[R]) {
  if constexpr (R == 4) {
    const I2 a02p = add(v[0], v[2]), a02m = sub(v[0], v[2]);
    const I2 a13p = add(v[1], v[3]), a13m = sub(v[1], v[3]);
    v[0] = add(a02p, a13p);
    v[2] = sub(a02p, a13p);
    // -i (a1 - a3) for the forward sign, +i (a1 - a3) for the inverse
    const I2 p{a02m.x + a13m.y, a02m.y - a13m.x}, q{a02m.x - a13m.y, a02m.y + a13m.x};
    v[1] = INV ? q : p;
    v[3] = INV ? p : q;
  } else if constexpr (R == 2) {
    const I2 a = v[0], b = v[1];
    v[0] = add(a, b);
    v[1] = sub(a, b);
  } else {
    const I2 t1 = add(v[1], v[2]), t2 = sub(v[1], v[2]);
    const I2 m = sub(v[0], down<1>(t1));
    const long long sx = times_s3(t2.y), sy = times_s3(t2.x);
    v[0] = add(v[0], t1);
    // forward: -i s3 t2 added to v[1]; inverse: +i s3 t2
    const I2 p{m.x + sx, m.y - sy}, q{m.x - sx, m.y + sy};
    v[1] = INV ? q : p;
    v[2] = INV ? p : q;
  }
}

// one Stockham stage of radix R after NS points have been combined
template <int N, int L, int T, int R, int NS, bool INV>
__device__ __forceinline__ void stage(I2* buf, const Tw* tw) {
  constexpr int ES = L + 1, NB = N / R, TOT = NB * L, PER = (TOT + T - 1) / T, TS = N / (NS * R);
  constexpr int S = clog2(NS * R) - clog2(NS);           // halvings before this stage (none before the first)
  I2 v[PER][R];
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int b = threadIdx.x + p * T;
    if (TOT % T == 0 || b < TOT) {
      const int l = b % L, j = b / L;
#pragma unroll
      for (int r = 0; r < R; ++r) v[p][r] = buf[(j + r * NB) * ES + l];
    }
  }
  __syncthreads();
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int b = threadIdx.x + p * T;
    if (TOT % T == 0 || b < TOT) {
      const int l = b % L, j = b / L, kk = j % NS;
      if constexpr (NS > 1) {
        v[p][0] = down<S>(v[p][0]);
#pragma unroll
        for (int r = 1; r < R; ++r) v[p][r] = twiddle<S, INV>(v[p][r], tw[kk * r * TS]);
      }
      butterfly<R, INV>(v[p]);
      const int o = (j / NS) * NS * R + kk;
#pragma unroll
      for (int r = 0; r < R; ++r) buf[(o + r * NS) * ES + l] = v[p][r];
    }
  }
  __syncthreads();
}

template <int N, int L, int T, bool INV, int S = 0, int NS = 1>
__device__ __forceinline__ void run(I2* buf, const Tw* tw) {
  if constexpr (S < nstages(N)) {
    constexpr int R = radix_at(N, S);
    stage<N, L, T, R, NS, INV>(buf, tw);
    run<N, L, T, INV, S + 1, NS * R>(buf, tw);
  }
}

// to_double, or NaN where the line (exponent E) held a non-finite value
__device__ __forceinline__ double real(long long f, int X, int E) { return E == 0x7ff ? quiet_nan() : to_double(f, X); }

template <int N, int T>
__device__ __forceinline__ void stage_twiddles(Tw* s, const Tw* __restrict__ tw) {
  for (int m = threadIdx.x; m < N; m += T) s[m] = tw[m];
}

// X forward: rows (j, j+1) of plane k packed as one complex line, r2c split.
// A warp loads and stores whole lines, so a line's exponent is a warp maximum.
template <int N>
__global__ void __launch_bounds__(Shape<N>::T, 3) x_fwd(Grid g, const Tw* __restrict__ twg,
                                                        const double* __restrict__ src, double2* __restrict__ spec) {
  typedef Shape<N> Sh;
  constexpr int L = Sh::L, T = Sh::T, ES = Sh::ES, PER = (N + 31) / 32, LW = Sh::kLinesPerWarp;
  extern __shared__ __align__(16) unsigned char shraw[];
  Tw* tw = (Tw*)shraw;
  I2* buf = (I2*)(tw + N);
  stage_twiddles<N, T>(tw, twg);
  const int k = blockIdx.y, jp0 = blockIdx.x * L, npairs = min(L, g.n2m / 2 - jp0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int E[LW];
#pragma unroll
  for (int q = 0; q < LW; ++q) {
    const int l = warp * LW + q;
    double a[PER], b[PER];
    const double* __restrict__ ra = src + cidx(g, 0, l < npairs ? 2 * (jp0 + l) : 0, k);
    const double* __restrict__ rb = ra + g.P;
    int e = 1;
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int i = lane + 32 * p;
      const bool ok = l < npairs && (N % 32 == 0 || i < N);
      a[p] = ok ? ra[i] : 0.0;
      b[p] = ok ? rb[i] : 0.0;
      e = max(e, max(expo(a[p]), expo(b[p])));
    }
    E[q] = __reduce_max_sync(0xffffffffu, e);
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int i = lane + 32 * p;
      if (N % 32 == 0 || i < N) buf[i * ES + l] = I2{from_double<6>(a[p], E[q]), from_double<6>(b[p], E[q])};
    }
  }
  __syncthreads();
  run<N, L, T, false>(buf, tw);
#pragma unroll
  for (int q = 0; q < LW; ++q) {
    const int l = warp * LW + q;
    if (l >= npairs) continue;
    const int X = E[q] - 6 + total_shift(N) - 1;          // the halves below
    double2* __restrict__ sa = spec + (size_t)g.HP * ((size_t)(2 * (jp0 + l)) + (size_t)g.n2m * k);
    double2* __restrict__ sb = sa + g.HP;
    for (int kx = lane; kx <= N / 2; kx += 32) {
      const I2 z = buf[kx * ES + l], c = buf[((N - kx) % N) * ES + l];
      // X_a = (Z + conj Z_-)/2 ; X_b = (Z - conj Z_-)/(2i)
      sa[kx] = make_double2(real(z.x + c.x, X, E[q]), real(z.y - c.y, X, E[q]));
      sb[kx] = make_double2(real(z.y + c.y, X, E[q]), real(c.x - z.x, X, E[q]));
    }
  }
}

// X inverse (c2r): half spectra of rows (j, j+1) -> real rows; the imaginary
// parts of the kx = 0 and kx = n1m/2 bins are dropped
template <int N>
__global__ void __launch_bounds__(Shape<N>::T, 3) x_inv(Grid g, const Tw* __restrict__ twg,
                                                        const double2* __restrict__ spec, double* __restrict__ dst) {
  typedef Shape<N> Sh;
  constexpr int L = Sh::L, T = Sh::T, ES = Sh::ES, H = N / 2 + 1, PER = (H + 31) / 32, LW = Sh::kLinesPerWarp;
  extern __shared__ __align__(16) unsigned char shraw[];
  Tw* tw = (Tw*)shraw;
  I2* buf = (I2*)(tw + N);
  stage_twiddles<N, T>(tw, twg);
  const int k = blockIdx.y, jp0 = blockIdx.x * L, npairs = min(L, g.n2m / 2 - jp0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int E[LW];
#pragma unroll
  for (int q = 0; q < LW; ++q) {
    const int l = warp * LW + q;
    double2 a[PER], b[PER];
    const double2* __restrict__ sa =
        spec + (size_t)g.HP * ((size_t)(l < npairs ? 2 * (jp0 + l) : 0) + (size_t)g.n2m * k);
    const double2* __restrict__ sb = sa + g.HP;
    int e = 1;
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int kx = lane + 32 * p;
      const bool ok = l < npairs && kx < H;
      a[p] = ok ? sa[kx] : make_double2(0.0, 0.0);
      b[p] = ok ? sb[kx] : make_double2(0.0, 0.0);
      if (kx == 0 || 2 * kx == N) { a[p].y = 0.0; b[p].y = 0.0; }
      e = max(e, max(max(expo(a[p].x), expo(a[p].y)), max(expo(b[p].x), expo(b[p].y))));
    }
    E[q] = __reduce_max_sync(0xffffffffu, e);
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int kx = lane + 32 * p;
      if (kx >= H) continue;
      const long long ax = from_double<5>(a[p].x, E[q]), ay = from_double<5>(a[p].y, E[q]);
      const long long bx = from_double<5>(b[p].x, E[q]), by = from_double<5>(b[p].y, E[q]);
      buf[kx * ES + l] = I2{ax - by, ay + bx};            // Z = Xa + i Xb
      if (kx > 0 && 2 * kx < N) buf[(N - kx) * ES + l] = I2{ax + by, bx - ay};
    }
  }
  __syncthreads();
  run<N, L, T, true>(buf, tw);
#pragma unroll
  for (int q = 0; q < LW; ++q) {
    const int l = warp * LW + q;
    if (l >= npairs) continue;
    const int X = E[q] - 5 + total_shift(N);
    double* __restrict__ ra = dst + cidx(g, 0, 2 * (jp0 + l), k);
    double* __restrict__ rb = ra + g.P;
    for (int i = lane; i < N; i += 32) {
      const I2 z = buf[i * ES + l];
      ra[i] = real(z.x, X, E[q]);
      rb[i] = real(z.y, X, E[q]);
    }
  }
}

// Y pass (forward or inverse) on L kx columns of plane k: a thread keeps the
// line threadIdx.x % L throughout
template <int N, bool INV>
__global__ void __launch_bounds__(Shape<N>::T, 3) y_pass(Grid g, const Tw* __restrict__ twg,
                                                         double2* __restrict__ spec) {
  typedef Shape<N> Sh;
  constexpr int L = Sh::L, T = Sh::T, ES = Sh::ES, PER = (N * L + T - 1) / T;
  __shared__ int sE[L];
  extern __shared__ __align__(16) unsigned char shraw[];
  Tw* tw = (Tw*)shraw;
  I2* buf = (I2*)(tw + N);
  stage_twiddles<N, T>(tw, twg);
  const int kx0 = blockIdx.x * L, k = blockIdx.y, l = threadIdx.x % L, e0 = threadIdx.x / L;
  if (threadIdx.x < L) sE[threadIdx.x] = 1;
  double2* __restrict__ col = spec + (size_t)kx0 + l + (size_t)g.HP * g.n2m * k;
  const bool act = kx0 + l < g.H;
  double2 v[PER];
  int m = 1;
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int e = e0 + p * (T / L);
    const bool ok = act && (N * L % T == 0 || e < N);
    v[p] = ok ? col[(size_t)g.HP * e] : make_double2(0.0, 0.0);
    m = max(m, max(expo(v[p].x), expo(v[p].y)));
  }
#pragma unroll
  for (int off = L; off < 32; off <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
  __syncthreads();
  if ((threadIdx.x & 31) < L) atomicMax(&sE[l], m);
  __syncthreads();
  const int E = sE[l];
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int e = e0 + p * (T / L);
    if (N * L % T == 0 || e < N) buf[e * ES + l] = I2{from_double<6>(v[p].x, E), from_double<6>(v[p].y, E)};
  }
  __syncthreads();
  run<N, L, T, INV>(buf, tw);
  const int X = E - 6 + total_shift(N);
  if (!act) return;
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int e = e0 + p * (T / L);
    if (N * L % T == 0 || e < N) {
      const I2 z = buf[e * ES + l];
      col[(size_t)g.HP * e] = make_double2(real(z.x, X, E), real(z.y, X, E));
    }
  }
}

template <typename K>
inline bool smem_attr(Ctx* c, K kern, size_t bytes) {
  if (bytes <= 48 * 1024) return true;
  return cuda_ok(c, cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes),
                 "fft smem");
}

template <int N>
void launch_x_fwd(Ctx* c, const Tw* tw, const double* src, double2* spec) {
  typedef Shape<N> Sh;
  if (!smem_attr(c, x_fwd<N>, Sh::smem)) return;
  x_fwd<N><<<dim3(div_up(c->g.n2m / 2, Sh::L), c->g.n3m), Sh::T, Sh::smem, c->stream>>>(c->g, tw, src, spec);
}
template <int N>
void launch_x_inv(Ctx* c, const Tw* tw, const double2* spec, double* dst) {
  typedef Shape<N> Sh;
  if (!smem_attr(c, x_inv<N>, Sh::smem)) return;
  x_inv<N><<<dim3(div_up(c->g.n2m / 2, Sh::L), c->g.n3m), Sh::T, Sh::smem, c->stream>>>(c->g, tw, spec, dst);
}
template <int N>
void launch_y(Ctx* c, const Tw* tw, double2* spec, int sign) {
  typedef Shape<N> Sh;
  if (!smem_attr(c, y_pass<N, false>, Sh::smem) || !smem_attr(c, y_pass<N, true>, Sh::smem)) return;
  const dim3 grid(div_up(c->g.H, Sh::L), c->g.n3m);
  if (sign < 0) y_pass<N, false><<<grid, Sh::T, Sh::smem, c->stream>>>(c->g, tw, spec);
  else y_pass<N, true><<<grid, Sh::T, Sh::smem, c->stream>>>(c->g, tw, spec);
}

}  // namespace intfft

// line lengths with an instance: every 2^a 3^b the library takes
#define MIBM_INTFFT_SIZES(X)                                                                              \
  X(8) X(12) X(16) X(18) X(24) X(32) X(36) X(48) X(54) X(64) X(72) X(96) X(108) X(128) X(144) X(162) X(192) \
  X(216) X(256) X(288) X(324) X(384) X(432) X(486) X(512)

}  // namespace mibm
