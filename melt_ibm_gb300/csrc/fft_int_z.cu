// fft_int_z.cu -- the z lines of the FP64 Poisson solve on the integer pipe.
//
// After the x and y transforms a line (kx, ky) is the periodic system
// (D_zz - lambda) phi = r (fft.cu make_ztri), circulant like the line solves
// of tridiag.cu: with G = dx3q / lambda and e = 2 / (1 + sqrt(1 + 4 G)), rho =
// 1 - e, it factors into y_i = r_i + rho y_{i-1}, x_i = y_i + rho x_{i+1},
// phi = -e^2 / lambda x.  The recurrences run in 64-bit fixed point (fixed.cuh)
// with one exponent per real line; the factor, with the transforms' scale, is
// the only FP64 operation: 2 per complex value instead of 10, and 48 bytes of
// constants per line instead of its factor tables (7 n + 5 n/M values read per
// line and solve).  A warp's lanes are 16 lines (consecutive in kx + H ky) by
// real and imaginary part, its block's warps their n/M chunks of M cells, held
// in registers.  A chunk sweeps from a zero entry, takes its entry value from
// the end values of the K chunks before it (weights rho^{mM} / (1 - rho^n),
// 2^-60 dropped), and adds the entry's decay to its cells.  Per line the host
// gives the bits that a sweep may grow values by: they start as far up as the
// first sweep allows.  Before the second they are shifted down, rounded, from
// what the first has made of them: a line that oscillates in z has not grown and is
// left where it is.
// The zero line (lambda = 0, mean set to 0) is two running sums, exact in
// 128-bit integers, in a block of its own beside the others.
// Error (see also fft_int.cuh; phi, relative 2-norm, 8 x 8 lines of 16 to 512 cells
// times cos x, FP64 lines / these): noise, a spike or the lowest mode in z 1e-15 ..
// 1e-12 / 1e-16 .. 4e-16; modes from n/8 up, alone, on the average 0.2 to 0.6
// of the FP64 lines' in cubic and taller boxes (256 cells, n/2 - 1: 6e-14 / 7e-15),
// up to 5 times them in boxes 0.4 as tall as wide, where 1/e is 100 and more.
// The alternating mode and n/4 by themselves come out of the FP64 lines to a few
// 1e-15 at some lengths (216, 288, 432), where all their roundings cancel; here to
// 2e-14 (216) .. 1e-13 (288).  The table's wavenumbers are those of the half-angle
// formula, which alone takes 64^3 noise from 5.1e-15 to 2.5e-16.
// Per solve, FP64 -> this: 48^3 25 -> 8.8 us,
// 96^3 39 -> 14.4, 128^3 49 -> 25, 192^3 145 -> 58, 108 x 108 x 72 63 -> 15.
#include <cmath>
#include <cstring>
#include <vector>

#include "fft_common.cuh"
#include "fixed.cuh"

namespace mibm {
namespace {

using namespace fixed;

constexpr int kMaxChunks = 32, kMaxLine = 512;

// a line's constants, times 2^62 as signed halves: rho, rho^M and 1/(1 -
// rho^n) - 1; guard bits of the load (may be negative), bits that a sweep may
// grow values by, K; and the final factor
struct alignas(16) ZLine {
  int rh, rl, mh, ml;
  int wh, wl, up, grow;
  int K, pad;
  double scale;
};

// x f / 2^62, rounded
__device__ __forceinline__ long long frac(long long x, int fh, int fl) {
  int h, l;
  halves(x, h, l);
  return (wide(h, fh) << 2) + ((wide(h, fl) + wide(l, fh) + (1ll << 29)) >> 30);
}

// from_double with `up` guard bits, -16 <= up <= 8
__device__ __forceinline__ long long load_fixed(double d, int E, int up) {
  const long long b = __double_as_longlong(d);
  const int e = (int)((b >> 52) & 0x7ff);
  const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffull) | (e ? 1ull << 52 : 0);
  const long long a = (long long)((m << 8) >> min(E - max(e, 1) + 8 - up, 63));
  const long long s = b >> 63;
  return (a ^ s) - s;
}

// inclusive sums of one value per thread of the first n threads; all threads call
__device__ __forceinline__ __int128 running_sum(__int128 v, __int128* buf, int t, int n) {
  for (int d = 1; d < n; d <<= 1) {
    if (t < n) buf[t] = v;
    __syncthreads();
    if (t < n && t >= d) v += buf[t - d];
    __syncthreads();
  }
  if (t < n) buf[t] = v;
  __syncthreads();
  return v;
}

// D_zz phi = r - mean(r), mean(phi) = 0: with running sums s of r, S = n s - (k+1)
// s_{n-1} of n (r - mean) and P the sums before k of n S - sum S, phi dx3q n^3 is
// n P - sum P.  r has 59 bits, P n 107 at most.
__device__ __noinline__ void zero_line(int n, size_t st, double2* __restrict__ spec, double scale, __int128* buf,
                                       int* sE) {
  const int t = threadIdx.x + 32 * threadIdx.y;
  for (int part = 0; part < 2; ++part) {
    double* __restrict__ p = (double*)spec + part + (size_t)min(t, n - 1) * st;
    const double v = *p;
    if (t == 0) *sE = 1;
    __syncthreads();
    atomicMax(sE, expo(v));
    __syncthreads();
    const int E = *sE;
    const __int128 s = running_sum(from_double<6>(v, E), buf, t, n);
    const __int128 S = s * n - buf[n - 1] * (t + 1);
    __syncthreads();
    const __int128 q = running_sum(S, buf, t, n);
    const __int128 P = (q - S) * n - buf[n - 1] * t;
    __syncthreads();
    running_sum(P, buf, t, n);
    const __int128 F = P * n - buf[n - 1];
    __syncthreads();
    if (t >= n) continue;
    const unsigned __int128 a = F < 0 ? -(unsigned __int128)F : (unsigned __int128)F;
    const unsigned long long hi = (unsigned long long)(a >> 64);
    const int sh = hi ? 66 - __clzll((long long)hi) : ((unsigned long long)a >> 62 ? 2 : 0);   // 62 bits are left
    *p = E == 0x7ff ? quiet_nan() : to_double((long long)(F >> sh), E - 6 + sh) * scale;
  }
}

// threads: up to 32 n/M; T bounds it for the register count
template <int M, int T>
__global__ void __launch_bounds__(T, T <= 512 ? 2 : 1) z_lines(Grid g, const ZLine* __restrict__ tab, double2* __restrict__ spec) {
  __shared__ __align__(16) long long sC[kMaxChunks][32], sD[kMaxChunks][32];
  __shared__ int sE[32], sB[32];
  static_assert(sizeof(sC) >= kMaxLine * sizeof(__int128), "the zero line's sums fit");
  const size_t st = 2 * (size_t)g.HP * g.n2m;
  if (blockIdx.x == 0) {
    zero_line(g.n3m, st, spec, tab[0].scale, (__int128*)&sC[0][0], sE);
    return;
  }
  const int lane = threadIdx.x, w = threadIdx.y, G = blockDim.y, H = g.H;
  const int l = (blockIdx.x - 1) * 16 + (lane >> 1);
  const bool act = l > 0 && l < H * g.n2m;
  const int kx = act ? l % H : 1, ky = act ? l / H : 0;
  const ZLine Z = tab[kx + H * min(ky, g.n2m - ky)];
  double* __restrict__ rp = (double*)(spec + kx + (size_t)g.HP * ky) + (lane & 1) + (size_t)(w * M) * st;
  if (w == 0) {
    sE[lane] = 1;
    sB[lane] = 0;
  }
  long long r[M];
  int E = 1;
  {
    double v[M];
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] = act ? rp[(size_t)i * st] : 0.0;
#pragma unroll
    for (int i = 0; i < M; ++i) E = max(E, expo(v[i]));
    __syncthreads();
    atomicMax(&sE[lane], E);
    __syncthreads();
    E = sE[lane];
#pragma unroll
    for (int i = 0; i < M; ++i) r[i] = load_fixed(v[i], E, Z.up);
  }
  // a chunk's entry value from the end values of the chunks on one side
  const int K = __reduce_max_sync(0xffffffffu, Z.K);
  auto entry = [&](const long long (*e)[32], int dir) {
    int src = w + dir * K;
    src = src < 0 ? src + G : (src >= G ? src - G : src);
    long long s = 0;
    for (int m = 0; m < K; ++m) {
      s = e[src][lane] + frac(s, Z.mh, Z.ml);
      src -= dir;
      src = src < 0 ? G - 1 : (src == G ? 0 : src);
    }
    return s + frac(s, Z.wh, Z.wl);
  };
#pragma unroll
  for (int i = 1; i < M; ++i) r[i] += frac(r[i - 1], Z.rh, Z.rl);
  sC[w][lane] = r[M - 1];
  __syncthreads();
  long long t = entry(sC, -1);
  int top = 0;
#pragma unroll
  for (int i = 0; i < M; ++i) {
    t = frac(t, Z.rh, Z.rl);
    r[i] += t;
    top |= (int)(r[i] >> 32) ^ (int)(r[i] >> 63);
  }
  // down to where the second sweep's growth just fits
  atomicMax(&sB[lane], 64 - __clz(top));
  __syncthreads();
  const int down = max(sB[lane] + Z.grow - 61, 0);
  const long long half = (1ll << down) >> 1;
#pragma unroll
  for (int i = 0; i < M; ++i) r[i] = (r[i] + half) >> down;
#pragma unroll
  for (int i = M - 2; i >= 0; --i) r[i] += frac(r[i + 1], Z.rh, Z.rl);
  sD[w][lane] = r[0];
  __syncthreads();
  t = entry(sD, 1);
  const int X = E - Z.up + down;
#pragma unroll
  for (int i = M - 1; i >= 0; --i) {
    t = frac(t, Z.rh, Z.rl);
    if (act) rp[(size_t)i * st] = E == 0x7ff ? quiet_nan() : to_double(r[i] + t, X) * Z.scale;
  }
}

// chunk length: the shortest with at most 16 chunks (blocks of up to 512 threads
// at 64 registers, two on an SM: 192 cells, one solve, 12: 56 us, 8 with 24
// chunks: 69 us; below 16 chunks the lengths are within 5% of each other),
// else the longest
int chunk_of(int n) {
  for (int m : {8, 12, 16, 18})
    if (n % m == 0 && n / m <= 16) return m;
  for (int m : {18, 16})
    if (n % m == 0 && n / m <= kMaxChunks && n <= kMaxLine) return m;
  return 0;
}

typedef unsigned __int128 u128;
constexpr u128 kOne = (u128)1 << 62;
u128 mul62(u128 a, u128 b) { return (a * b + (kOne >> 1)) >> 62; }

void put(u128 v, int& hi, int& lo) {
  const long long x = (long long)v;
  lo = (int)(unsigned)(x & 0xffffffffll);
  hi = (int)((x - lo) >> 32);
}

template <int M, int T>
void launch(Ctx* c, const void* tab, double2* spec) {
  const Grid& g = c->g;
  z_lines<M, T><<<1 + (unsigned)div_up((size_t)g.H * g.n2m, 16), dim3(32, g.n3m / M), 0, c->stream>>>(
      g, (const ZLine*)tab, spec);
}

}  // namespace

// Constants of every line, lt = kx + H min(ky, n2m - ky); empty where the
// scheme does not cover the grid: a box so flat (rho^n) or lines so stiff
// that the solution would outgrow its bits
void intfft_z_table(const Grid& g, std::vector<char>& out) {
  out.clear();
  const int n = g.n3m, M = chunk_of(n), H = g.H;
  if (!M || H < 2) return;
  std::vector<ZLine> tab((size_t)H * (g.n2m / 2 + 1));
  const double nfac = 1.0 / ((double)g.n1m * (double)g.n2m);
  // phini.f90's ak1, ak2 by the half-angle formula: 1 - cos(a) of a small a has few digits left
  auto ak = [](int k, int m, double dq) { const double s = std::sin(M_PI * k / m); return 4.0 * s * s * dq; };
  for (int ky = 0; ky <= g.n2m / 2; ++ky)
    for (int kx = 0; kx < H; ++kx) {
      ZLine& z = tab[kx + (size_t)H * ky];
      if (kx == 0 && ky == 0) {
        z.scale = nfac / ((double)n * (double)n * (double)n * g.dx3q);
        continue;
      }
      const double lambda = ak(kx, g.n1m, g.dx1q) + ak(ky, g.n2m, g.dx2q), G = g.dx3q / lambda;
      const double e = 2.0 / (1.0 + std::sqrt(1.0 + 4.0 * G));
      if (!(e > 1.0 / 256.0 && e < 1.0)) return;
      const u128 rho = e < 0.5 ? kOne - (u128)std::ldexp(e, 62) : (u128)std::ldexp(G * e * e, 62);
      u128 rm = kOne, rn = kOne;
      for (int i = 0; i < M; ++i) rm = mul62(rm, rho);
      for (int i = 0; i < n / M; ++i) rn = mul62(rn, rm);
      if (rn > kOne / 3) return;
      const u128 w = (rn << 62) / (kOne - rn);
      put(rho, z.rh, z.rl);
      put(rm, z.mh, z.ml);
      put(w, z.wh, z.wl);
      // a sweep grows values by at most (1 + w) / e
      const int bits = (int)std::ceil(std::log2((1.0 + std::ldexp((double)w, -62)) / e) + 0.01);
      z.up = 8 - bits;                                      // below 2^61 after the first sweep
      z.grow = bits;
      const double drop = 60.0 / (-std::log2(std::max(std::ldexp((double)rm, -62), 1e-300)));
      z.K = (int)std::min((double)(n / M), std::ceil(drop));
      z.scale = -nfac / lambda * e * e;
    }
  out.resize(tab.size() * sizeof(ZLine));
  std::memcpy(out.data(), tab.data(), out.size());
}

void intfft_z(Ctx* c, const void* tab, double2* spec) {
  const int M = chunk_of(c->g.n3m);
  const bool small = c->g.n3m <= 16 * M;
  if (M == 8) launch<8, 512>(c, tab, spec);
  else if (M == 12) launch<12, 512>(c, tab, spec);
  else if (M == 16) small ? launch<16, 512>(c, tab, spec) : launch<16, 1024>(c, tab, spec);
  else small ? launch<18, 512>(c, tab, spec) : launch<18, 1024>(c, tab, spec);
}

}  // namespace mibm
