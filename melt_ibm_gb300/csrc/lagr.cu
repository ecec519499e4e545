// lagr.cu -- immersed-boundary (Lagrangian) part of the substep.
//
// Restates on the device:
//   findCentroidIndices.f90:14-50           centroid cage indices
//   mlsWeight.f90:48-412, geom.f90:24-53     MLS shape functions (FP64 4x4 LU)
//   mlsForce.f90:13-33, forc1/2/3/temp.f90  interpolation + force spreading
//   velforce.f90:13-52, tempforce.f90:13-40 mean removal and field update
//   findProbeIndices.f90:20-74              +/- normal probe cages
//   mls_heatFlux.f90:77-395                 MLS gradient of T, face->vertex
//   stefanCondition.f90:12-31               Stefan front advance
//   triaux.f90:53-323, RigidAuxRoutines.f90:653-780  geometry refresh
//   genSDF.f90:120-365, tagCells.f90:85-111 narrow-band tagging
//   pencil_rayTag.f90:37-460                initial full tagging
//
// Determinism: no floating-point atomics anywhere.  Force spreading gathers:
// the 27 cage cells of every triangle are grouped by cell once per geometry
// (the scatter plan below; integer atomics only, and its finished order
// depends only on the mesh), then each touched cell sums its contributions in
// triangle order -- the reference's summation order.  Face->vertex sums use
// a vertex->face adjacency list in ascending face order.  The narrow band
// takes the minimum distance with 64-bit integer atomicMin on the
// (non-negative) IEEE bit pattern and the earliest triangle among equal
// distances, exactly the strict "<" update rule of genSDF.f90:167.
#include <climits>
#include <string>
#include <cstddef>
#include <cmath>
#include <utility>
#include <vector>

#include "common.cuh"
#include "fpconv.cuh"
#include "mls_exp.h"

namespace mibm {

// ---------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------
struct LagArgs {
  Grid g;
  int nf, nv, coff, clen;
  const double* xc; const double* xm; const double* yc; const double* ym; const double* zc; const double* zm;
  double wcon, wscl;
  // the weights' divisors and their reciprocals: wscl/dx per direction, wcon, wcon^2
  double wr[3], iwr[3], iwcon, wc2, iwc2, dcoef;   // dcoef: -2 / wcon^2
};

static LagArgs lag_args(Ctx* c) {
  LagArgs a;
  a.g = c->g; a.nf = c->maxnf; a.nv = c->maxnv; a.coff = c->coord_off; a.clen = 3 * c->coord_off;
  a.xc = c->xc; a.xm = c->xm; a.yc = c->yc; a.ym = c->ym; a.zc = c->zc; a.zm = c->zm;
  a.wcon = c->S(MIBM_S_WCON); a.wscl = c->S(MIBM_S_WSCL);
  a.wr[0] = a.wscl / c->g.dx1; a.wr[1] = a.wscl / c->g.dx2; a.wr[2] = a.wscl / c->g.dx3;
  for (int d = 0; d < 3; ++d) a.iwr[d] = 1.0 / a.wr[d];
  a.iwcon = 1.0 / a.wcon;
  a.wc2 = a.wcon * a.wcon;
  a.iwc2 = 1.0 / a.wc2;
  a.dcoef = -2.0 / a.wc2;
  return a;
}

template <typename T> static T* M(Ctx* c, int id) { return (T*)c->dm[id]; }

__device__ __forceinline__ int ffloor(double x) { return (int)floor(x); }
__device__ __forceinline__ int fnint(double x) { return (int)round(x); }
__device__ __forceinline__ double sqd(double x) { return x * x; }

__device__ __forceinline__ double coord(const LagArgs& A, int dir, int sel, int idx) {
  // sel 0 = c (face) coordinates, 1 = m (centre).  The tables span
  // [-coff, 2*coff) grid indices, more than the reference's -n..2n; a body
  // outside that range is clamped instead of read out of bounds.
  int t = min(max(idx + A.coff, 0), A.clen - 1);
  if (dir == 0) return sel == 0 ? A.xc[t] : A.xm[t];
  if (dir == 1) return sel == 0 ? A.yc[t] : A.ym[t];
  return sel == 0 ? A.zc[t] : A.zm[t];
}

// Gaussian weight and its radial derivative (geom.f90:24-53).  exp is the
// written-out mls_exp (mls_exp.h), shared with the oracle, so that the
// plain form's MLS construction gives the oracle's bits.
// a / b, correctly rounded, for a constant b whose reciprocal y has been rounded
// once: after one correction the quotient is within an ulp, from where the
// second rounds it correctly (Markstein, Computation of elementary functions on
// the IBM RISC System/6000, 1990).  Five FP64 operations; quotient and
// remainder must not underflow (0 does not).
__device__ __forceinline__ double div_const(double a, double b, double y) {
  const double q = a * y, q1 = fma(fma(-b, q, a), y, q);
  return fma(fma(-b, q1, a), y, q1);
}
// limit < x <= infinity for x >= 0 (false for a NaN), limit >= 0: an FP64
// comparison issues at the FP64 rate, one of the bits does not
__device__ __forceinline__ bool above(double x, double limit) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x),
                           l = (unsigned long long)__double_as_longlong(limit);
  return b > l && b <= 0x7ff0000000000000ull;
}
// |pos - pc| / (wscl/dx) along axis d, or 2 where it is above 4
__device__ __forceinline__ double axis_norp(const LagArgs& A, int d, double diff) {
  const double a = fabs(diff);
  return above(a, 4.0 * A.wr[d]) ? 2.0 : div_const(a, A.wr[d], A.iwr[d]);
}
// the Gaussian weight of norp (mlsWeight.f90): 0 above 1
__device__ __forceinline__ double mls_gaussian(const LagArgs& A, double r) {
  return above(r, 1.0) ? 0.0 : mls_exp(-sqd(div_const(r, A.wcon, A.iwcon)));
}
// In-place inverse of a 4x4 column-major matrix: LU with partial pivoting
// (dgetrf semantics, first maximal pivot) and inversion from the factors
// (dgetri).  Returns false if a pivot is exactly zero.
__device__ __forceinline__ bool inv4(double* a) {
  constexpr int n = 4;
  int ipiv[4];
  double rp[4];                                   // 1 / pivot, used by both factors
#pragma unroll
  for (int j = 0; j < n; ++j) {
    int p = j;
    double amax = fabs(a[j + n * j]);
#pragma unroll
    for (int i = j + 1; i < n; ++i)
      if (above(fabs(a[i + n * j]), amax)) { amax = fabs(a[i + n * j]); p = i; }
    ipiv[j] = p;
    if (__double_as_longlong(amax) == 0) return false;
#pragma unroll
    for (int i = j + 1; i < n; ++i)
#pragma unroll
      for (int cc = 0; cc < n; ++cc) {            // rows j and p change places, in registers
        const double t = a[j + n * cc], u = a[i + n * cc];
        a[j + n * cc] = p == i ? u : t;
        a[i + n * cc] = p == i ? t : u;
      }
    const double r = 1.0 / a[j + n * j];
    rp[j] = r;
#pragma unroll
    for (int i = j + 1; i < n; ++i) a[i + n * j] *= r;
#pragma unroll
    for (int cc = j + 1; cc < n; ++cc) {
      double t = a[j + n * cc];
#pragma unroll
      for (int i = j + 1; i < n; ++i) a[i + n * cc] -= t * a[i + n * j];
    }
  }
#pragma unroll
  for (int j = 0; j < n; ++j) {
    a[j + n * j] = rp[j];
    const double ajj = -rp[j];
#pragma unroll
    for (int i = 0; i < j; ++i) {
      double s = a[i + n * i] * a[i + n * j];
#pragma unroll
      for (int k = i + 1; k < j; ++k) s += a[i + n * k] * a[k + n * j];
      a[i + n * j] = s;
    }
#pragma unroll
    for (int i = 0; i < j; ++i) a[i + n * j] *= ajj;
  }
#pragma unroll
  for (int j = n - 2; j >= 0; --j) {
    double work[4];
#pragma unroll
    for (int i = j + 1; i < n; ++i) { work[i] = a[i + n * j]; a[i + n * j] = 0.0; }
#pragma unroll
    for (int i = 0; i < n; ++i) {
      double s = a[i + n * (j + 1)] * work[j + 1];
#pragma unroll
      for (int k = j + 2; k < n; ++k) s += a[i + n * k] * work[k];
      a[i + n * j] -= s;
    }
  }
#pragma unroll
  for (int j = n - 2; j >= 0; --j)
#pragma unroll
    for (int c = j + 1; c < n; ++c)
#pragma unroll
      for (int i = 0; i < n; ++i) {               // columns j and ipiv[j] change places
        const double t = a[i + n * j], u = a[i + n * c];
        a[i + n * j] = ipiv[j] == c ? u : t;
        a[i + n * c] = ipiv[j] == c ? t : u;
      }
  return true;
}

// Blocks of one warp for the kernels over faces, probes and vertices.  Their
// warps are chains of FP64 instructions, which the warps of an SM share a
// narrow pipe for, and a body has few of them (1280 faces: 40 to 160 warps):
// blocks of four warps left most SMs idle beside some with eight warps to run.
// Blocks of 128 -> 32 threads: mls_weight_sep 69 -> 49 us (5120 faces), 166 ->
// 146 us (20480), heat_flux_sep 125 -> 104 us (20480), the others unchanged.
constexpr int kLagBlock = 32;

// ---------------------------------------------------------------------
// findCentroidIndices / findProbeIndices
// ---------------------------------------------------------------------
__device__ __forceinline__ void centroid_idx_one(const Grid& g, double px, double py, double pz, int* p) {
  int i1 = ffloor(px * g.dx1) + 1, ist = fnint(px * g.dx1) + 1;
  int j1 = ffloor(py * g.dx2) + 1, jst = fnint(py * g.dx2) + 1;
  int k1 = ffloor(pz * g.dx3) + 1, kst = fnint(pz * g.dx3) + 1;
  k1 = fmod_pos(k1 - 1, g.n3m) + 1;
  kst = fmod_pos(kst - 1, g.n3m) + 1;
  p[0] = i1; p[1] = j1; p[2] = k1; p[3] = ist; p[4] = jst; p[5] = kst;
}

__global__ void centroid_idx_kernel(LagArgs A, const double* __restrict__ tri_bar, const int* __restrict__ ghost,
                                    int* __restrict__ pind) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= A.nf || ghost[t]) return;
  centroid_idx_one(A.g, tri_bar[3 * t], tri_bar[3 * t + 1], tri_bar[3 * t + 2], pind + 6 * t);
}

__global__ void probe_idx_kernel(LagArgs A, const double* __restrict__ tri_bar, const double* __restrict__ tri_nor,
                                 const int* __restrict__ ghost, double h, int* __restrict__ pind) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= A.nf || ghost[t]) return;
  const Grid& g = A.g;
  double n0 = tri_nor[3 * t], n1 = tri_nor[3 * t + 1], n2 = tri_nor[3 * t + 2];
  double s = sqrt(n0 * n0 + n1 * n1 + n2 * n2);
  for (int side = 0; side < 2; ++side) {
    double pos[3];
    for (int d = 0; d < 3; ++d) {
      double nd = tri_nor[3 * t + d];
      pos[d] = side == 0 ? tri_bar[3 * t + d] + h * nd / s : tri_bar[3 * t + d] - h * nd / s;
    }
    int i1 = ffloor(pos[0] * g.dx1) + 1, j1 = ffloor(pos[1] * g.dx2) + 1, k1 = ffloor(pos[2] * g.dx3) + 1;
    k1 = fmod_pos(k1 - 1, g.n3m) + 1;
    pind[6 * t + 3 * side + 0] = i1; pind[6 * t + 3 * side + 1] = j1; pind[6 * t + 3 * side + 2] = k1;
  }
}

// ---------------------------------------------------------------------
// mlsWeight: one thread per (triangle, component)
// component 0 = wght1 (vx), 1 = wght2 (vy), 2 = wght3 (vz), 3 = wghttemp
// ---------------------------------------------------------------------
struct CageSpec {
  int ix, iy;      // pind slot (0-based) of the x and y cage centre
  int sx, sy, sz;  // coordinate selector per axis (0 = c, 1 = m)
  bool znint;      // z centre from nint (wght3) or floor
};
__device__ __forceinline__ CageSpec cage_spec(int comp) {
  switch (comp) {
    case 0: return CageSpec{3, 1, 0, 1, 1, false};   // xc, ym, zm ; pind(4), pind(2)
    case 1: return CageSpec{0, 4, 1, 0, 1, false};   // xm, yc, zm ; pind(1), pind(5)
    case 2: return CageSpec{0, 1, 1, 1, 0, true};    // xm, ym, zc ; pind(1), pind(2)
  }
  return CageSpec{0, 1, 1, 1, 1, false};             // xm, ym, zm ; pind(1), pind(2)
}

// One z layer of the cage added to the moment sums M = sum_n w_n p_n p_n^T in the
// reference's order (rank-one updates (w p_cc) p_r, nodes in cage order), the
// FIRST into empty sums; TWICE for the gradient's second layer, whose values the
// repeated layer of mls_heatFlux.f90:213 has again.  Row 0 of column cc sums
// what row cc of column 0 does and is left to lit_symmetric.
template <bool FIRST, bool TWICE = !FIRST>
__device__ __forceinline__ void lit_layer(const double (&w)[9], const double (&x)[3], const double (&y)[3], double z,
                                          double (&M)[16]) {
#pragma unroll
  for (int cc = 0; cc < 4; ++cc) {
    double t[9];
#pragma unroll
    for (int n = 0; n < 9; ++n) t[n] = cc == 0 ? w[n] : w[n] * (cc == 1 ? x[n % 3] : cc == 2 ? y[n / 3] : z);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (r == 0 && cc > 0) continue;
      double p[9];
#pragma unroll
      for (int n = 0; n < 9; ++n) p[n] = r == 0 ? t[n] : t[n] * (r == 1 ? x[n % 3] : r == 2 ? y[n / 3] : z);
      double s = FIRST ? p[0] : M[r + 4 * cc] + p[0];
#pragma unroll
      for (int n = 1; n < 9; ++n) s = s + p[n];
      if (TWICE) {
#pragma unroll
        for (int n = 0; n < 9; ++n) s = s + p[n];
      }
      M[r + 4 * cc] = s;
    }
  }
}
__device__ __forceinline__ void lit_symmetric(double (&M)[16]) { M[4] = M[1]; M[8] = M[2]; M[12] = M[3]; }

// The reference's MLS shape functions at pos for the 27-point cage centred on
// (i0, j0, k0) with per-axis staggering sx, sy, sz (mls_shape of wght1/2/3/
// temp, mlsWeight.f90:48-412, and of wght_press, mls_structLoads.f90:271-
// 404): basis [1, x, y, z] in absolute coordinates, A = sum W p p^T by
// rank-one updates in cage order, A^-1 by LU with partial pivoting, then
// phi = (p(x)^T A^-1) B.  IEEE operations in the oracle's order (this file is
// compiled without FMA contraction): the same bits.  Returns false on a
// singular A.
__device__ bool shape_lit(const LagArgs& A, const double pos[3], int i0, int j0, int k0, int sx, int sy, int sz,
                          double out[27]) {
  const Grid& g = A.g;
  const double ptx[4] = {1.0, pos[0], pos[1], pos[2]};
  // separable Gaussian weights (the reference evaluates the same 9 values)
  double wz[3], wy[3], wx[3], cz[3], cy[3], cx[3];
  for (int q = 0; q < 3; ++q) {
    cz[q] = coord(A, 2, sz, k0 - 1 + q);
    cy[q] = coord(A, 1, sy, j0 - 1 + q);
    cx[q] = coord(A, 0, sx, i0 - 1 + q);
    wz[q] = mls_gaussian(A, axis_norp(A, 2, cz[q] - pos[2]));
    wy[q] = mls_gaussian(A, axis_norp(A, 1, cy[q] - pos[1]));
    wx[q] = mls_gaussian(A, axis_norp(A, 0, cx[q] - pos[0]));
  }
  double Am[16], w[9];
  auto layer = [&](int kk) {
    for (int n = 0; n < 9; ++n) w[n] = wx[n % 3] * (wy[n / 3] * wz[kk]);
  };
  layer(0);
  lit_layer<true>(w, cx, cy, cz[0], Am);
  layer(1);
  lit_layer<false, false>(w, cx, cy, cz[1], Am);
  layer(2);
  lit_layer<false, false>(w, cx, cy, cz[2], Am);
  lit_symmetric(Am);
  if (!inv4(Am)) return false;
  double ptxA[4];
  for (int cc = 0; cc < 4; ++cc) {
    double s = 0;
    for (int r = 0; r < 4; ++r) s += ptx[r] * Am[r + 4 * cc];
    ptxA[cc] = s;
  }
  for (int kk = 0; kk < 3; ++kk)
    for (int jj = 0; jj < 3; ++jj) {
      double w23 = wy[jj] * wz[kk];
      for (int ii = 0; ii < 3; ++ii) {
        double wtx = wx[ii] * w23;
        // B(:,n) = wtx * [1, x, y, z]
        out[ii + 3 * jj + 9 * kk] =
            ptxA[0] * (wtx * 1.0) + ptxA[1] * (wtx * cx[ii]) + ptxA[2] * (wtx * cy[jj]) + ptxA[3] * (wtx * cz[kk]);
      }
    }
  return true;
}

// One thread per (triangle, component): the serial order of the reference,
// and the fewest FP64 operations (the part's scarce resource).
__global__ void mls_weight_kernel(LagArgs A, const double* __restrict__ tri_bar, const int* __restrict__ ghost,
                                  const int* __restrict__ pind, double* __restrict__ p1, double* __restrict__ p2,
                                  double* __restrict__ p3, double* __restrict__ pt, int* __restrict__ flag) {
  int gid = blockIdx.x * blockDim.x + threadIdx.x;
  int t = gid >> 2, comp = gid & 3;
  if (t >= A.nf || ghost[t]) return;
  const Grid& g = A.g;
  double pos[3] = {tri_bar[3 * t], tri_bar[3 * t + 1], tri_bar[3 * t + 2]};
  CageSpec cs = cage_spec(comp);
  int i0 = pind[6 * t + cs.ix], j0 = pind[6 * t + cs.iy];
  int k0 = cs.znint ? fnint(pos[2] * g.dx3) + 1 : ffloor(pos[2] * g.dx3) + 1;
  double* out = (comp == 0) ? p1 : (comp == 1) ? p2 : (comp == 2) ? p3 : pt;
  double phi[27];
  if (!shape_lit(A, pos, i0, j0, k0, cs.sx, cs.sy, cs.sz, phi)) { atomicOr(flag, 1); return; }
  out += 27 * (size_t)t;
  for (int n = 0; n < 27; ++n) out[n] = phi[n];
}

// Weight and weight derivative of one cage coordinate for the literal
// gradient, as wght_grad_field evaluates them (mls_heatFlux.f90:166-185):
// norp = |pos - pc| / (wscl/dx); W = gaussian(norp); dW = 0 at norp < eps,
// else gauss_deriv(norp) * ((pos - pc) / |pos - pc| / (wscl/dx)).  The
// Gaussian's exp is evaluated once for both (the same value either way).
__device__ __forceinline__ void lit_axis_weight(const LagArgs& A, int d, double pos, double pc, double& W, double& dW) {
  const double eps = 2.220446049250313e-16;       // EPSILON(1.0d0)
  const double diff = pos - pc;
  const double norp = axis_norp(A, d, diff);
  if (above(norp, 1.0)) {
    W = 0.0;
    dW = 0.0;
    return;
  }
  const double e = mls_exp(-sqd(div_const(norp, A.wcon, A.iwcon)));
  W = e;
  // (pos - pc) / |pos - pc| is +-1
  dW = __double_as_longlong(norp) < __double_as_longlong(eps)
           ? 0.0 : (div_const(-2.0 * norp, A.wc2, A.iwc2) * e) * copysign(A.iwr[d], diff);
}

// weights of a layer's nodes: of A (D < 0), of dA_d
__device__ __forceinline__ void lit_node_weights(int d, const double (&W0)[3], const double (&dW0)[3],
                                                 const double (&W1)[3], const double (&dW1)[3], double W2, double dW2,
                                                 double (&w)[9]) {
#pragma unroll
  for (int n = 0; n < 9; ++n) {
    const int i = n % 3, j = n / 3;
    w[n] = d < 0 ? W0[i] * (W1[j] * W2)
         : d == 0 ? (dW0[i] * W1[j]) * W2 : d == 1 ? (W0[i] * dW1[j]) * W2 : (W0[i] * W1[j]) * dW2;
  }
}

// dgam . (wt p) + gam . (dw p) of a layer's nodes
__device__ __forceinline__ void lit_node_values(const double (&wt)[9], const double (&dw)[9], const double (&dgam)[4],
                                                const double (&gam)[4], const double (&x)[3], const double (&y)[3],
                                                double z, double (&v)[9]) {
#pragma unroll
  for (int n = 0; n < 9; ++n) {
    const double px = x[n % 3], py = y[n / 3];
    const double t1 = ((dgam[0] * wt[n] + dgam[1] * (wt[n] * px)) + dgam[2] * (wt[n] * py)) + dgam[3] * (wt[n] * z);
    const double t2 = ((gam[0] * dw[n] + gam[1] * (dw[n] * px)) + gam[2] * (dw[n] * py)) + gam[3] * (dw[n] * z);
    v[n] = t1 + t2;
  }
}

// The reference's MLS gradient at a probe, literally (wght_gradT,
// mls_heatFlux.f90:161-376; wght_gradP/U/V/W, mls_structLoads.f90:406-1298):
// basis [1, x, y, z] in absolute coordinates; A, dA/dx_d, B, dB/dx_d
// accumulated point by point in cage order (z layer, y, x) as the reference's
// rank-one DGEMM updates; A^-1 by LU with partial pivoting; gamma = A^-1 p(x);
//   d phi / dx_d = (A^-1 (e_d - dA_d gamma))^T B + gamma^T dB_d,
// contracted with the field over the cage.  Cage i, j around (pi1, pi2);
// z layers [k1-1, k1, k1] (the repeated layer of mls_heatFlux.f90:213) with
// k1 = floor(z*dx3)+1, or nint for the w-velocity; coordinates per axis from
// the field's staggering (sel 0 = face, 1 = centre); field values at the
// wrapped cage, z from [k1w-1, k1w, k1w+1].  Every operation is the oracle's
// (wght_grad_field) in its order, so the two agree bit for bit.  B and dB are
// not stored: each entry is a product of per-axis weight factors and a basis
// entry, recomputed where it is used from the same factors in the same order
// (the same bits); dA_d is accumulated in its own pass per direction.  The
// repeated layer has the middle one's coordinates and weights, so its products
// are not formed again.
// Returns false on a singular A.
__device__ bool probe_grad_lit(const LagArgs& A, const double pos[3], int pi1, int pi2, int sx, int sy, int sz,
                               bool knint, const double* __restrict__ q, double grad[3]) {
  const Grid& g = A.g;
  const double ptx[4] = {1.0, pos[0], pos[1], pos[2]};
  const int k1 = knint ? fnint(pos[2] * g.dx3) + 1 : ffloor(pos[2] * g.dx3) + 1;
  const int k1w = fmod_pos(k1 - 1, g.n3m) + 1;
  const int keul[3] = {k1w - 1, k1w, k1w + 1};
  double x[3], y[3], z[2], W0[3], W1[3], W2[2], dW0[3], dW1[3], dW2[2];
  for (int r = 0; r < 3; ++r) {
    x[r] = coord(A, 0, sx, pi1 - 1 + r);
    y[r] = coord(A, 1, sy, pi2 - 1 + r);
    lit_axis_weight(A, 0, pos[0], x[r], W0[r], dW0[r]);
    lit_axis_weight(A, 1, pos[1], y[r], W1[r], dW1[r]);
    if (r < 2) {
      z[r] = coord(A, 2, sz, k1 - 1 + r);
      lit_axis_weight(A, 2, pos[2], z[r], W2[r], dW2[r]);
    }
  }
  double Am[16], wt[9], dw[9];
  lit_node_weights(-1, W0, dW0, W1, dW1, W2[0], dW2[0], wt);
  lit_layer<true>(wt, x, y, z[0], Am);
  lit_node_weights(-1, W0, dW0, W1, dW1, W2[1], dW2[1], wt);
  lit_layer<false>(wt, x, y, z[1], Am);
  lit_symmetric(Am);
  if (!inv4(Am)) return false;
  double gam[4];
  for (int r = 0; r < 4; ++r) {                   // DGEMV('N', invA, ptx)
    double t = 0;
    for (int cc = 0; cc < 4; ++cc) t += Am[r + 4 * cc] * ptx[cc];
    gam[r] = t;
  }
  const int kk_[3] = {wrap(keul[0] - 1, g.n3m), wrap(keul[1] - 1, g.n3m), wrap(keul[2] - 1, g.n3m)};
  for (int d = 0; d < 3; ++d) {
    double dA[16];
    lit_node_weights(d, W0, dW0, W1, dW1, W2[0], dW2[0], dw);
    lit_layer<true>(dw, x, y, z[0], dA);
    lit_node_weights(d, W0, dW0, W1, dW1, W2[1], dW2[1], dw);
    lit_layer<false>(dw, x, y, z[1], dA);
    lit_symmetric(dA);
    double pk_d[4] = {0.0, 0.0, 0.0, 0.0};
    pk_d[d + 1] = 1.0;
    for (int r = 0; r < 4; ++r) {                 // pk = -dA gamma + pk
      double t = 0;
      for (int cc = 0; cc < 4; ++cc) t += dA[r + 4 * cc] * gam[cc];
      pk_d[r] = pk_d[r] - t;
    }
    double dgam[4];
    for (int r = 0; r < 4; ++r) {
      double t = 0;
      for (int cc = 0; cc < 4; ++cc) t += Am[r + 4 * cc] * pk_d[cc];
      dgam[r] = t;
    }
    double gsum = 0, v[9];
    for (int nk = 0; nk < 3; ++nk) {
      if (nk < 2) {
        lit_node_weights(-1, W0, dW0, W1, dW1, W2[nk], dW2[nk], wt);
        lit_node_weights(d, W0, dW0, W1, dW1, W2[nk], dW2[nk], dw);
        lit_node_values(wt, dw, dgam, gam, x, y, z[nk], v);
      }
#pragma unroll
      for (int n = 0; n < 9; ++n)
        gsum += v[n] * q[cidx(g, fmod_pos(pi1 - 1 + n % 3 - 1, g.n1m), fmod_pos(pi2 - 1 + n / 3 - 1, g.n2m), kk_[nk])];
    }
    grad[d] = gsum;
  }
  return true;
}

// The reference's MLS value at a probe, literally (wght_press,
// mls_structLoads.f90:271-404): shape functions of the cell-centred cage
// around (i0, j0), z layers k1-1, k1, k1+1 with k1 = floor(z*dx3)+1, summed
// against the field in cage order as the oracle does.
__device__ bool probe_value_lit(const LagArgs& A, const double pos[3], int i0, int j0, const double* __restrict__ q,
                                double& val) {
  const Grid& g = A.g;
  const int k1 = ffloor(pos[2] * g.dx3) + 1;
  double phi[27];
  if (!shape_lit(A, pos, i0, j0, k1, 1, 1, 1, phi)) return false;
  const int k1w = fmod_pos(k1 - 1, g.n3m) + 1;
  double v = 0.0;
  int inw = 0;
  for (int kk = 0; kk < 3; ++kk) {
    const int kc = wrap(k1w - 1 + kk - 1, g.n3m);
    for (int j = 0; j < 3; ++j) {
      const int jj = fmod_pos(j0 - 1 + j - 1, g.n2m);
      for (int i = 0; i < 3; ++i) {
        v = v + q[cidx(g, fmod_pos(i0 - 1 + i - 1, g.n1m), jj, kc)] * phi[inw];
        ++inw;
      }
    }
  }
  val = v;
  return true;
}

// ---------------------------------------------------------------------
// mlsForce: interpolation Um per (triangle, component) and coefficient
// cfac*(target - Um); the spread goes through the sorted scatter plan.
// ---------------------------------------------------------------------
struct ForceArgs {
  const double* q[4];       // vx, vy, vz, temp (compact)
  const double* ptx[4];
  const double* vel_tri;
  const double* cfac;
  const int* pind;
  const int* ghost;
};

__device__ __forceinline__ void cage_center(int comp, const int* p, int& i0, int& j0, int& k0) {
  // forc1: pind(4), pind(2), pind(3); forc2: pind(1), pind(5), pind(3)
  // forc3: pind(1), pind(2), pind(6); forctemp: pind(1), pind(2), pind(3)
  switch (comp) {
    case 0: i0 = p[3]; j0 = p[1]; k0 = p[2]; return;
    case 1: i0 = p[0]; j0 = p[4]; k0 = p[2]; return;
    case 2: i0 = p[0]; j0 = p[1]; k0 = p[5]; return;
  }
  i0 = p[0]; j0 = p[1]; k0 = p[2];
}

__device__ __forceinline__ size_t cage_cell(const Grid& g, int i0, int j0, int k0, int slot) {
  int ii = fmod_pos(i0 - 2 + slot % 3, g.n1m);
  int jj = fmod_pos(j0 - 2 + (slot / 3) % 3, g.n2m);
  int kk = fmod_pos(k0 - 2 + slot / 9, g.n3m);
  return cidx(g, ii, jj, kk);
}

__global__ void force_coef_kernel(Grid g, int nf, ForceArgs F, double tmelt, double* __restrict__ coef) {
  int gid = blockIdx.x * blockDim.x + threadIdx.x;
  int t = gid >> 2, comp = gid & 3;
  if (t >= nf) return;
  if (F.ghost[t]) { coef[comp * (size_t)nf + t] = 0.0; return; }
  int i0, j0, k0;
  cage_center(comp, F.pind + 6 * t, i0, j0, k0);
  const double* phi = F.ptx[comp] + 27 * (size_t)t;
  const double* q = F.q[comp];
  double Um = 0.0;
  for (int s = 0; s < 27; ++s) Um = Um + q[cage_cell(g, i0, j0, k0, s)] * phi[s];
  double target = (comp == 3) ? tmelt : F.vel_tri[3 * t + comp];
  coef[comp * (size_t)nf + t] = F.cfac[t] * (target - Um);
}

// ---------------------------------------------------------------------
// Scatter plan: the entries grouped by cell, without a sort of the entries.
// ---------------------------------------------------------------------
// The four cage sets (x, y, z staggered, cell-centred) are merged into one
// plan: entry e = comp*27*nf + 27*t + slot, key = comp*cells + cage cell
// (ghost faces have no entries).  A run is the entries of one key, in triangle
// order; runs are numbered in key order.  The keys touched are marked in a
// bitmap of 4*cells bits; a scan of its population counts numbers the runs in
// key order; entries then take slots of their runs with atomics, runs take
// storage from a cursor, and half a warp per run puts its few tens of entries
// into triangle order by rank (a block where there are more).  The slots and the storage depend on the order
// of the atomics, the finished runs do not.  Eight launches, each a few
// microseconds: this chain is on the step's critical path at small and
// moderate grids.  A radix sort of all entries by key in its place took 3 or 4
// passes of five launches and five more for the run heads (serial kernel time
// of the plan, 5120 faces on 128^3: 170 -> 95 us per substep; 20480 faces, radius
// 0.3 on 16^3 / 0.4 on 64^3: 166 -> 155 / 216 -> 114 us).
// The plan depends only on the cage centres (pind) and the ghost flags;
// `plan_check` compares them with the values the plan was built from and
// every kernel of the rebuild returns at once when nothing changed, so a
// rebuild costs nothing on a stationary cage.
__global__ void plan_check_kernel(int nf, const int* __restrict__ pind, const int* __restrict__ ghost,
                                  const int* __restrict__ saved, int* __restrict__ dirty,
                                  const StepParams* __restrict__ pp) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0 && pp && pp->force_plan) atomicOr(dirty, 1);   // rebuild requested by the host
  if (t >= nf) return;
  const int* sv = saved + 7 * (size_t)t;
  bool diff = (sv[6] != ghost[t]);
  if (!ghost[t])
    for (int q = 0; q < 6; ++q) diff = diff || (sv[q] != pind[6 * t + q]);
  if (diff) atomicOr(dirty, 1);
}

// The kernels over entries take them slot by slot: thread p has the entry of
// triangle p % nf, so that a warp's entries are those of neighbouring triangles at one
// cage slot and many of them share a cell (plan_slot).
// key and number of entry p, key -1 for a ghost face
__device__ __forceinline__ int plan_key(const Grid& g, int nf, const int* __restrict__ pind,
                                        const int* __restrict__ ghost, int p, int& e) {
  const int q = p / nf, t = p - q * nf, comp = q / 27, sl = q - 27 * comp;
  e = 27 * (comp * nf + t) + sl;
  if (ghost[t]) return -1;
  int i0, j0, k0;
  cage_center(comp, pind + 6 * t, i0, j0, k0);
  return (int)((size_t)comp * g.cells + cage_cell(g, i0, j0, k0, sl));
}

__global__ void __launch_bounds__(256) plan_mark_kernel(Grid g, int nf, const int* __restrict__ pind,
                                                        const int* __restrict__ ghost, const int* __restrict__ dirty,
                                                        unsigned* __restrict__ bitmap) {
  if (!*dirty) return;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  int e, key = -1;
  if (p < 108 * nf) key = plan_key(g, nf, pind, ghost, p, e);
  const unsigned same = __match_any_sync(0xffffffffu, key);
  if (key < 0 || (threadIdx.x & 31) != __ffs(same) - 1) return;
  const unsigned bit = 1u << (key & 31);
  if (!(bitmap[key >> 5] & bit)) atomicOr(bitmap + (key >> 5), bit);   // a stale 0 only repeats the atomic
}

// Bitmap scan in tiles of 4096 words (256 threads x 16 words): the tiles'
// population counts, then (plan_runs_kernel) each tile's base from those of
// the tiles before it, the run number at the start of every marked word, and
// the runs' keys with their counts reset.
constexpr int kPlanTile = 4096;
__device__ __forceinline__ int plan_words(const unsigned* __restrict__ bitmap, int words, int w0, unsigned (&v)[16]) {
  int n = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint4 u = make_uint4(0, 0, 0, 0);
    if (w0 + 4 * q < words) u = reinterpret_cast<const uint4*>(bitmap + w0)[q];   // padded to a multiple of 4
    v[4 * q] = u.x; v[4 * q + 1] = u.y; v[4 * q + 2] = u.z; v[4 * q + 3] = u.w;
    n += __popc(u.x) + __popc(u.y) + __popc(u.z) + __popc(u.w);
  }
  return n;
}

// exclusive scan of one value per thread of a 256-thread block, and the total
__device__ __forceinline__ int block_scan(int v, int* wsum, int& total) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
  for (int off = 1; off < 32; off <<= 1) {
    const int u = __shfl_up_sync(FULL, x, off);
    if (lane >= off) x += u;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  int base = 0;
  total = 0;
  for (int q = 0; q < 8; ++q) {
    if (q < w) base += wsum[q];
    total += wsum[q];
  }
  __syncthreads();
  return base + x - v;
}

__global__ void __launch_bounds__(256) plan_count_kernel(const unsigned* __restrict__ bitmap, int words,
                                                         const int* __restrict__ dirty, int* __restrict__ tsum) {
  if (!*dirty) return;
  __shared__ int wsum[8];
  unsigned v[16];
  int total;
  block_scan(plan_words(bitmap, words, blockIdx.x * kPlanTile + 16 * threadIdx.x, v), wsum, total);
  if (threadIdx.x == 0) tsum[blockIdx.x] = total;
}

__global__ void __launch_bounds__(256) plan_runs_kernel(const unsigned* __restrict__ bitmap, int words,
                                                        const int* __restrict__ dirty, const int* __restrict__ tsum,
                                                        int* __restrict__ wpre, int* __restrict__ run_key,
                                                        int* __restrict__ run_cnt, int* __restrict__ nruns) {
  if (!*dirty) return;
  __shared__ int wsum[8];
  int before = 0, base;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += 256) before += tsum[b];
  block_scan(before, wsum, base);
  unsigned v[16];
  const int w0 = blockIdx.x * kPlanTile + 16 * threadIdx.x;
  int total, at = block_scan(plan_words(bitmap, words, w0, v), wsum, total) + base;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    unsigned m = v[q];
    if (!m) continue;
    wpre[w0 + q] = at;
    for (; m; m &= m - 1) {
      run_key[at] = 32 * (w0 + q) + __ffs(m) - 1;
      run_cnt[at] = 0;
      ++at;
    }
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    nruns[0] = base + total;
    nruns[1] = 0;                        // the storage cursor
    nruns[2] = 0;                        // long runs
  }
}

// a slot of its run for every entry: one atomic for the entries of a warp that
// share a run (a body of 20480 faces within a few cells has runs of as many entries: 240 -> 35 us)
__global__ void __launch_bounds__(256) plan_slot_kernel(Grid g, int nf, const int* __restrict__ pind,
                                                        const int* __restrict__ ghost, const int* __restrict__ dirty,
                                                        const unsigned* __restrict__ bitmap,
                                                        const int* __restrict__ wpre, int* __restrict__ run_cnt,
                                                        int2* __restrict__ slot) {
  if (!*dirty) return;
  const unsigned FULL = 0xffffffffu;
  const int p = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  int e, run = -1;
  if (p < 108 * nf) {
    const int key = plan_key(g, nf, pind, ghost, p, e);
    if (key >= 0) run = wpre[key >> 5] + __popc(bitmap[key >> 5] & ((1u << (key & 31)) - 1u));
  }
  const unsigned same = __match_any_sync(FULL, run);
  const int first = __ffs(same) - 1;
  int at = 0;
  if (run >= 0 && lane == first) at = atomicAdd(run_cnt + run, __popc(same));
  at = __shfl_sync(FULL, at, first) + __popc(same & ((1u << lane) - 1u));
  if (p < 108 * nf) slot[p] = make_int2(run, at);
}

// storage for every run: a warp of runs takes its total from the cursor; runs
// of more than kLongRun entries are listed
constexpr int kLongRun = 128;
__global__ void __launch_bounds__(256) plan_store_kernel(const int* __restrict__ dirty, const int* __restrict__ run_cnt,
                                                         int* __restrict__ run_off, int* __restrict__ nruns,
                                                         int* __restrict__ long_run) {
  if (!*dirty) return;
  const unsigned FULL = 0xffffffffu;
  const int n = nruns[0], lane = threadIdx.x & 31;
  for (int h0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); h0 < n; h0 += gridDim.x * blockDim.x) {
    const int h = h0 + lane, v = h < n ? run_cnt[h] : 0;
    int x = v;
    for (int off = 1; off < 32; off <<= 1) {
      const int u = __shfl_up_sync(FULL, x, off);
      if (lane >= off) x += u;
    }
    int base = 0;
    if (lane == 31) base = atomicAdd(nruns + 1, x);
    base = __shfl_sync(FULL, base, 31);
    if (h < n) run_off[h] = base + x - v;
    if (h < n && v > kLongRun) long_run[atomicAdd(nruns + 2, 1)] = h;
  }
}

// entries into their slots; the cage centres the plan was built from
__global__ void __launch_bounds__(256) plan_place_kernel(int nf, const int* __restrict__ pind,
                                                         const int* __restrict__ ghost, const int* __restrict__ dirty,
                                                         const int2* __restrict__ slot, const int* __restrict__ run_off,
                                                         int* __restrict__ entry, int* __restrict__ saved) {
  if (!*dirty) return;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= 108 * nf) return;
  const int2 s = slot[p];
  const int q = p / nf, t = p - q * nf;                   // plan_key's order
  if (s.x >= 0) entry[run_off[s.x] + s.y] = 27 * (q / 27 * nf + t) + q % 27;
  if (p < nf) {
    for (int d = 0; d < 6; ++d) saved[7 * (size_t)p + d] = pind[6 * p + d];
    saved[7 * (size_t)p + 6] = ghost[p];
  }
}

// A long run into triangle order, by a block: a triangle has one entry of a run
// (its 27 cage cells differ), so a bitmap of the triangles, by tiles, gives every entry its
// rank.  All threads of the block call.  Tiles of 8192 triangles: with 32768 the
// kernel's 8 KB of shared memory cost the 48^3 step 1%.
constexpr int kSortWords = 256;
__device__ void plan_sort_long(int nf, int len, const int* __restrict__ entry, int* __restrict__ src) {
  __shared__ unsigned bits[kSortWords];
  __shared__ int before[kSortWords], wsum[8];
  constexpr int kPer = kSortWords / 256, kTile = 32 * kSortWords;
  const int t = threadIdx.x, per = 27 * nf, base = entry[0] / per * per;          // of the run's component
  int done = 0;
  for (int t0 = 0; t0 < nf; t0 += kTile) {
    for (int w = t; w < kSortWords; w += 256) bits[w] = 0u;
    __syncthreads();
    for (int i = t; i < len; i += 256) {
      const unsigned f = (unsigned)((entry[i] - base) / 27 - t0);
      if (f < (unsigned)kTile) atomicOr(bits + f / 32, 1u << (f & 31));
    }
    __syncthreads();
    int n = 0, total;
#pragma unroll
    for (int q = 0; q < kPer; ++q) n += __popc(bits[kPer * t + q]);
    int at = block_scan(n, wsum, total) + done;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      before[kPer * t + q] = at;
      at += __popc(bits[kPer * t + q]);
    }
    __syncthreads();
    for (int i = t; i < len; i += 256) {
      const int e = entry[i];
      const unsigned f = (unsigned)((e - base) / 27 - t0);
      if (f < (unsigned)kTile) src[before[f / 32] + __popc(bits[f / 32] & ((1u << (f & 31)) - 1u))] = e;
    }
    done += total;
    __syncthreads();
  }
}

// half a warp per run: the run's entries into triangle order (the rank of an
// entry is the number of smaller ones), and its word of the bitmap back to zero
// for the next build.  A run has about ten entries, so half of a whole warp would idle:
// 20480 faces 58 -> 50 us (32 runs loaded at once by a warp: 118, too few warps).
// Ranks cost the square of the length: the long runs of a fine mesh on a coarse grid, or
// of a body that has melted to a few cells, go to whole blocks (20480 faces, radius 0.3 on
// 16^3: 271 ms -> 51 us, 0.4 on 64^3 1003 -> 35 us, 0.5 on 128^3 94 -> 78 us).
__global__ void __launch_bounds__(256) plan_order_kernel(int nf, const int* __restrict__ dirty, const int* __restrict__ nruns,
                                                         const int* __restrict__ run_key,
                                                         const int* __restrict__ run_off,
                                                         const int* __restrict__ run_cnt,
                                                         const int* __restrict__ long_run,
                                                         const int* __restrict__ entry, int* __restrict__ src,
                                                         unsigned* __restrict__ bitmap) {
  if (!*dirty) return;
  constexpr int W = 16;
  const unsigned FULL = 0xffffffffu;
  const int n = nruns[0], lane = threadIdx.x % W, step = gridDim.x * (256 / W);
  // h0: the first run of the warp, the loop is uniform over it
  for (int h0 = (blockIdx.x * 256 + (threadIdx.x & ~31)) / W; h0 < n; h0 += step) {
    const int h = h0 + ((threadIdx.x & 31) / W);
    const bool act = h < n;
    const int o = act ? run_off[h] : 0, all = act ? run_cnt[h] : 0, len = all > kLongRun ? 0 : all;
    const int longest = max(len, __shfl_xor_sync(FULL, len, W));
    if (act && lane == 0) bitmap[run_key[h] >> 5] = 0u;
    for (int i0 = 0; i0 < longest; i0 += W) {
      const int v = i0 + lane < len ? entry[o + i0 + lane] : 0;
      int rank = 0;
      for (int j0 = 0; j0 < longest; j0 += W) {
        const int u = j0 + lane < len ? entry[o + j0 + lane] : 0x7fffffff;
#pragma unroll
        for (int q = 0; q < W; ++q) rank += __shfl_sync(FULL, u, q, W) < v;
      }
      if (i0 + lane < len) src[o + rank] = v;
    }
  }
  for (int q = blockIdx.x; q < nruns[2]; q += gridDim.x) {
    const int h = long_run[q], o = run_off[h];
    plan_sort_long(nf, run_cnt[h], entry + o, src + o);
  }
}

// Heads of the runs of equal keys (one cell of one component) sum their run
// in triangle order and add the sum to that component's target field; with
// `segval` the head also records the sum (for the mean force).
struct ScatterOut {
  double* f[4];
  const double* phi[4];
  float* m32[4];   // FP32 mirrors of f (precision form), null where none
};

__device__ __forceinline__ int key_comp(int k, size_t cells) {
  size_t u = (size_t)k;
  return (u >= cells) + (u >= 2 * cells) + (u >= 3 * cells);
}

// One warp per run (a cell of one component): the lanes take every 32nd
// entry of the run (face order), a fixed shuffle tree adds the 32 partial
// sums, lane 0 adds the total to the target field.  A warp instruction costs
// the same with 1 or 32 active lanes, and FP64 ones issue at a small fraction
// of the FP32 rate, so the runs (tens of entries each) are not summed by one
// thread.  With `segval` the run sum is also recorded at the run's index
// (for the mean force).
constexpr int kScatterBlocks = 1216;     // 8 blocks of 8 warps per SM on 152 SMs; the warps loop over runs
struct PlanRuns {
  const int* n;       // number of runs
  const int* key;     // per run, ascending: key, first entry in src, entries
  const int* off;
  const int* cnt;
  const int* src;     // entries in triangle order within a run
};
__global__ void __launch_bounds__(256) scatter_apply_kernel(int nf, size_t cells, PlanRuns P,
                                     const double* __restrict__ coef, ScatterOut O, int comp_lo, int comp_hi,
                                     double* __restrict__ segval) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * (blockDim.x >> 5);
  const int nh = *P.n;
  const int per = 27 * nf;
  for (int h = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); h < nh; h += nw) {
    const int k = P.key[h];
    const int comp = key_comp(k, cells);
    if (comp < comp_lo || comp >= comp_hi) continue;            // uniform over the warp
    const int e0 = P.off[h], e1 = e0 + P.cnt[h];
    const double* __restrict__ phi = O.phi[comp];
    const double* __restrict__ cf = coef + (size_t)comp * nf;
    double sum = 0.0;
    for (int q = e0 + lane; q < e1; q += 32) {
      const int sr = P.src[q] - comp * per;
      if (!MIBM_IDX_OK(sr, per)) continue;
      sum = fma(cf[sr / 27], phi[sr], sum);
    }
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(FULL, sum, off);
    if (lane == 0 && MIBM_IDX_OK((size_t)k - (size_t)comp * cells, cells)) {
      const size_t cell = (size_t)k - (size_t)comp * cells;
      const double v = O.f[comp][cell] + sum;
      O.f[comp][cell] = v;
      if (O.m32[comp]) O.m32[comp][cell] = (float)v;
      if (segval) segval[h] = sum;
    }
  }
}

// fixed-order sum of the recorded run sums per velocity component: 256
// blocks over contiguous ranges of runs (shuffle trees, then the 8 warps in
// order); the last block to finish (a ticket in mean3's slot 7, reset by that
// block) adds the 256 block sums, one component per warp: lane l sums blocks
// l, l+32, l+64, ... in that order, then a fixed shuffle tree adds the 32
// lane sums (a fixed order, so the result is deterministic); it writes the
// means divided by the cell count (FP64 at mean3[0..2], an FP32
// copy for the precision form at float offset 8)
constexpr int kMeanBlocks = 256;
__global__ void __launch_bounds__(256) seg_mean_kernel(PlanRuns P, size_t cells,
                                                      const double* __restrict__ segval, double* __restrict__ part,
                                                      double ncell, double* __restrict__ mean3) {
  const unsigned FULL = 0xffffffffu;
  __shared__ double ws[8][3];
  __shared__ bool last;
  const int n = *P.n;
  int per = (n + gridDim.x - 1) / gridDim.x;
  int lo = blockIdx.x * per, hi = min(n, lo + per);
  double s[3] = {0, 0, 0};
  for (int h = lo + threadIdx.x; h < hi; h += blockDim.x) {
    int comp = key_comp(P.key[h], cells);
    if (comp < 3) s[comp] += segval[h];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q = 0; q < 3; ++q) {
    double v = s[q];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(FULL, v, off);
    if (lane == 0) ws[warp][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double v = ws[0][threadIdx.x];
    for (int w = 1; w < 8; ++w) v += ws[w][threadIdx.x];
    part[3 * (size_t)blockIdx.x + threadIdx.x] = v;
  }
  unsigned* ticket = reinterpret_cast<unsigned*>(mean3 + 7);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (warp < 3) {
    double v = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32) v += __ldcg(part + 3 * (size_t)b + warp);
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(FULL, v, off);
    if (lane == 0) {
      double m = v / ncell;
      mean3[warp] = m;
      reinterpret_cast<float*>(mean3 + 4)[warp] = (float)m;   // FP32 copy for the precision form
    }
  }
  if (threadIdx.x == 0) *ticket = 0u;
}

// ---------------------------------------------------------------------
// deterministic sums
// ---------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Mean of the three force fields over the owned cells -> mean3[0..2], in a fixed
// order: kFieldMeanBlocks blocks over strided rows, block sums as in seg_mean_kernel,
// added by the last block to finish (the ticket in mean3's slot 7).  A force is
// zero off the markers' cages, so a warp whose pieces are all zero adds nothing
// (an FP64 addition costs it 16 clocks).
// Bound by the reads (128^3, 50 MB): 119 -> 25 us against one block and three
// shuffle trees per row and a second launch.
constexpr int kFieldMeanBlocks = 152 * 4;
__global__ void __launch_bounds__(256) field_mean_kernel(Grid g, const double* __restrict__ a,
                                                         const double* __restrict__ b, const double* __restrict__ cc,
                                                         double* __restrict__ part, double ncell,
                                                         double* __restrict__ mean3) {
  constexpr int kU = 4;
  const unsigned FULL = 0xffffffffu;
  __shared__ double ws[8][3];
  __shared__ bool last;
  const double* f[3] = {a, b, cc};
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = gridDim.x * 8, rows = g.n2m * g.n3m, per = (g.n1m + 31) / 32;
  double s[3] = {0, 0, 0};
  // a warp's pieces of 32 cells, kU of each field in flight
  for (int p0 = blockIdx.x * 8 + warp; p0 < rows * per; p0 += kU * warps) {
    double v[3][kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int p = p0 + u * warps, row = p / per, i = (p - row * per) * 32 + lane;
      const bool ok = p < rows * per && i < g.n1m;
      const size_t c0 = ok ? cidx(g, i, row % g.n2m, row / g.n2m) : 0;
#pragma unroll
      for (int q = 0; q < 3; ++q) v[q][u] = ok ? f[q][c0] : 0.0;
    }
    long long bits = 0;
#pragma unroll
    for (int u = 0; u < kU; ++u)
#pragma unroll
      for (int q = 0; q < 3; ++q) bits |= __double_as_longlong(v[q][u]);
    if (!__any_sync(FULL, bits << 1 != 0)) continue;
#pragma unroll
    for (int u = 0; u < kU; ++u)
#pragma unroll
      for (int q = 0; q < 3; ++q) s[q] += v[q][u];
  }
  for (int q = 0; q < 3; ++q) {
    const double v = warp_sum(s[q]);
    if (lane == 0) ws[warp][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double v = ws[0][threadIdx.x];
    for (int w = 1; w < 8; ++w) v += ws[w][threadIdx.x];
    part[3 * (size_t)blockIdx.x + threadIdx.x] = v;
  }
  unsigned* ticket = reinterpret_cast<unsigned*>(mean3 + 7);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (warp < 3) {
    double v = 0.0;
    for (int q = lane; q < (int)gridDim.x; q += 32) v += __ldcg(part + 3 * (size_t)q + warp);
    v = warp_sum(v);
    if (lane == 0) mean3[warp] = v / ncell;
  }
  if (threadIdx.x == 0) *ticket = 0u;
}

__device__ __forceinline__ void cross3(double r[3], const double x[3], const double y[3]) {
  r[0] = x[1] * y[2] - y[1] * x[2];
  r[1] = x[2] * y[0] - y[2] * x[0];
  r[2] = x[0] * y[1] - y[0] * x[1];
}

// Per-face loads in the reference's order (mls_structLoads.f90:52-202):
// c[0..3) pressure force, [3..6) viscous force, [6..9) pressure torque,
// [9..12) viscous torque.
__device__ void face_loads(const double* __restrict__ e, const double nrm[3], const double rad[3], double sur,
                           double h, double ren, double c[12]) {
  double press_tri = e[0] - h * (e[1] * nrm[0] + e[2] * nrm[1] + e[3] * nrm[2]);
  double pn[3], buf[3];
  for (int d = 0; d < 3; ++d) { c[d] = press_tri * sur * nrm[d]; pn[d] = press_tri * nrm[d]; }
  cross3(buf, rad, pn);
  for (int d = 0; d < 3; ++d) c[6 + d] = buf[d] * sur;
  double S11 = e[4], S12 = e[5], S13 = e[6], S21 = e[7], S22 = e[8], S23 = e[9];
  double S31 = e[10], S32 = e[11], S33 = e[12];
  double sr = sur / ren;
  double tv[3];
  tv[0] = sr * (2.0 * S11 * nrm[0] + (S12 + S21) * nrm[1] + S13 * nrm[2]);
  tv[1] = sr * ((S21 + S12) * nrm[0] + 2.0 * S22 * nrm[1] + S23 * nrm[2]);
  tv[2] = sr * (S13 * nrm[0] + S23 * nrm[1]);
  double tn[3], rt[3];
  for (int d = 0; d < 3; ++d) tn[d] = 0.0 + tv[d];
  cross3(buf, rad, tv);
  for (int d = 0; d < 3; ++d) rt[d] = 0.0 + buf[d];
  tv[0] = sr * (S31 * nrm[2]);
  tv[1] = sr * (S32 * nrm[2]);
  tv[2] = sr * (S31 * nrm[0] + S32 * nrm[1] + 2.0 * S33 * nrm[2]);
  for (int d = 0; d < 3; ++d) tn[d] = tn[d] + tv[d];
  cross3(buf, rad, tv);
  for (int d = 0; d < 3; ++d) rt[d] = rt[d] + buf[d];
  for (int d = 0; d < 3; ++d) { c[3 + d] = tn[d]; c[9 + d] = rt[d]; }
}

// ---------------------------------------------------------------------
// Precision form of mlsWeight and mls_heatFlux.  MLS with the complete
// linear basis is invariant under an affine change of basis, so the shape
// functions (and their gradients) can be built from the basis
// p = (1, x - x0, y - y0, z - z0) shifted to the interpolation point x0,
// where p(x0) = e0.  With separable Gaussian weights w_n = wx_i wy_j wz_k
// every moment sum factorises into 1-D moments S_m = sum_q w_q d_q^m
// (m = 0, 1, 2) and the derivative weights likewise (D_m), so the 4x4
// moment matrix and its three derivatives take a few dozen FP64 operations
// instead of 27 rank-one updates each, and are far better conditioned than
// with absolute coordinates.  The 4x4 inversion is the FP64 LU of the plain
// form.  The values agree with the reference construction to its round-off
// (amplified by its conditioning), not bit for bit.
// ---------------------------------------------------------------------
__device__ __forceinline__ void moments3(const double w[3], const double d[3], double S[3]) {
  S[0] = w[0] + w[1] + w[2];
  S[1] = fma(w[0], d[0], fma(w[1], d[1], w[2] * d[2]));
  S[2] = fma(w[0] * d[0], d[0], fma(w[1] * d[1], d[1], (w[2] * d[2]) * d[2]));
}

// symmetric moment matrix (column-major) of the shifted linear basis from
// 1-D moments X, Y, Z (each S0, S1, S2)
__device__ __forceinline__ void moment_matrix(const double X[3], const double Y[3], const double Z[3], double M[16]) {
  double a00 = X[0] * Y[0] * Z[0];
  double a01 = X[1] * Y[0] * Z[0], a02 = X[0] * Y[1] * Z[0], a03 = X[0] * Y[0] * Z[1];
  double a11 = X[2] * Y[0] * Z[0], a22 = X[0] * Y[2] * Z[0], a33 = X[0] * Y[0] * Z[2];
  double a12 = X[1] * Y[1] * Z[0], a13 = X[1] * Y[0] * Z[1], a23 = X[0] * Y[1] * Z[1];
  M[0] = a00; M[1] = a01; M[2] = a02; M[3] = a03;
  M[4] = a01; M[5] = a11; M[6] = a12; M[7] = a13;
  M[8] = a02; M[9] = a12; M[10] = a22; M[11] = a23;
  M[12] = a03; M[13] = a13; M[14] = a23; M[15] = a33;
}

__global__ void mls_weight_sep_kernel(LagArgs A, const double* __restrict__ tri_bar, const int* __restrict__ ghost,
                                      const int* __restrict__ pind, double* __restrict__ p1, double* __restrict__ p2,
                                      double* __restrict__ p3, double* __restrict__ pt, int* __restrict__ flag) {
  int gid = blockIdx.x * blockDim.x + threadIdx.x;
  int t = gid >> 2, comp = gid & 3;
  if (t >= A.nf || ghost[t]) return;
  const Grid& g = A.g;
  double pos[3] = {tri_bar[3 * t], tri_bar[3 * t + 1], tri_bar[3 * t + 2]};
  CageSpec cs = cage_spec(comp);
  int i0 = pind[6 * t + cs.ix], j0 = pind[6 * t + cs.iy];
  int k0 = cs.znint ? fnint(pos[2] * g.dx3) + 1 : ffloor(pos[2] * g.dx3) + 1;
  double wx[3], wy[3], wz[3], dx[3], dy[3], dz[3];
  for (int q = 0; q < 3; ++q) {
    double cz = coord(A, 2, cs.sz, k0 - 1 + q), cy = coord(A, 1, cs.sy, j0 - 1 + q), cx = coord(A, 0, cs.sx, i0 - 1 + q);
    wz[q] = mls_gaussian(A, axis_norp(A, 2, cz - pos[2]));
    wy[q] = mls_gaussian(A, axis_norp(A, 1, cy - pos[1]));
    wx[q] = mls_gaussian(A, axis_norp(A, 0, cx - pos[0]));
    dx[q] = cx - pos[0]; dy[q] = cy - pos[1]; dz[q] = cz - pos[2];
  }
  double X[3], Y[3], Z[3], M[16];
  moments3(wx, dx, X); moments3(wy, dy, Y); moments3(wz, dz, Z);
  moment_matrix(X, Y, Z, M);
  if (!inv4(M)) { atomicOr(flag, 1); return; }
  const double c0 = M[0], c1 = M[1], c2 = M[2], c3 = M[3];   // A^{-1} e0
  double* out = (comp == 0) ? p1 : (comp == 1) ? p2 : (comp == 2) ? p3 : pt;
  out += 27 * (size_t)t;
  for (int kk = 0; kk < 3; ++kk)
    for (int jj = 0; jj < 3; ++jj) {
      double wyz = wy[jj] * wz[kk], base = fma(c2, dy[jj], fma(c3, dz[kk], c0));
      for (int ii = 0; ii < 3; ++ii) out[ii + 3 * jj + 9 * kk] = (wx[ii] * wyz) * fma(c1, dx[ii], base);
    }
}

// Gaussian weight of one cage coordinate and its derivative along the axis
// (geom.f90:24-53 with the chain-rule factor of mls_heatFlux.f90:176-180).
// The cut-off decision r > 1 uses r = |x - x_c| / (wscl/dx) rounded as the
// reference rounds it; the rest uses precomputed reciprocals (the separable
// construction is insensitive to last-ulp changes of the weights).
__device__ __forceinline__ void axis_weight(const LagArgs& A, int d, double pos, double pc, double& w, double& dw) {
  const double eps = 2.220446049250313e-16;
  const double rr = pos - pc;
  const double np = axis_norp(A, d, rr);
  if (above(np, 1.0)) { w = 0.0; dw = 0.0; return; }
  double e = exp(-sqd(np * A.iwcon));
  w = e;
  dw = __double_as_longlong(np) < __double_as_longlong(eps) ? 0.0 : (A.dcoef * np) * e * copysign(A.iwr[d], rr);
}

// Separable MLS gradient at a probe: the gradient of wght_gradT (mls_heatFlux
// .f90:161-376) and wght_gradP/U/V/W (mls_structLoads.f90:406-1298).  Cage
// i, j centred on (pi1, pi2); z layers [k1-1, k1, k1] (the repeated layer of
// the reference) with k1 = floor(z*dx3)+1, or nint for the w-velocity;
// coordinates per axis from the field's staggering (sel 0 = face, 1 =
// centre); field values at the wrapped cage, z from [k1w-1, k1w, k1w+1].
// Returns false on a singular moment matrix.
__device__ bool probe_grad_sep(const LagArgs& A, const double pos[3], int pi1, int pi2, int sx, int sy, int sz,
                               bool knint, const double* __restrict__ q, double grad[3]) {
  const Grid& g = A.g;
  int k1 = knint ? fnint(pos[2] * g.dx3) + 1 : ffloor(pos[2] * g.dx3) + 1;
  int kin[3] = {k1 - 1, k1, k1};                  // mls_heatFlux.f90:213 (third layer repeats k1)
  int k1w = fmod_pos(k1 - 1, g.n3m) + 1;
  int keul[3] = {k1w - 1, k1w, k1w + 1};
  const int sel[3] = {sx, sy, sz};
  double w[3][3], dw[3][3], dd[3][3];             // [axis][point]
  for (int r = 0; r < 3; ++r) {
    double pc[3] = {coord(A, 0, sel[0], pi1 - 1 + r), coord(A, 1, sel[1], pi2 - 1 + r), coord(A, 2, sel[2], kin[r])};
    for (int a = 0; a < 3; ++a) {
      if (a == 2 && r == 2) {                     // the repeated layer
        w[2][2] = w[2][1]; dw[2][2] = dw[2][1]; dd[2][2] = dd[2][1];
        break;
      }
      axis_weight(A, a, pos[a], pc[a], w[a][r], dw[a][r]);
      dd[a][r] = pc[a] - pos[a];
    }
  }
  double S[3][3], D[3][3];
  for (int a = 0; a < 3; ++a) { moments3(w[a], dd[a], S[a]); moments3(dw[a], dd[a], D[a]); }
  double Ai[16];
  moment_matrix(S[0], S[1], S[2], Ai);
  if (!inv4(Ai)) return false;
  const double gam[4] = {Ai[0], Ai[1], Ai[2], Ai[3]};     // A^{-1} p(x0), p(x0) = e0
  // sums over the cage of the field times the weighted basis p = (1, d0, d1,
  // d2): MT (weights), MD[d] (derivative of the weights along d).  Weights
  // and basis factor by axis, so the sums are contracted one axis at a time
  // (x, then y, then z): about 250 FP64 operations instead of 675.
  double wd[3][3], dwd[3][3];
  for (int a = 0; a < 3; ++a)
    for (int r = 0; r < 3; ++r) { wd[a][r] = w[a][r] * dd[a][r]; dwd[a][r] = dw[a][r] * dd[a][r]; }
  double MT[4] = {0, 0, 0, 0}, MD[3][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0}};
  for (int kk = 0; kk < 3; ++kk) {
    const int kk_ = wrap(keul[kk] - 1, g.n3m);
    // y sums of the x sums A = sum w0 q, B = sum w0 d0 q, C = sum dw0 q, D = sum dw0 d0 q
    double SA = 0, SAd = 0, SAw = 0, SAwd = 0, SB = 0, SBw = 0, SC = 0, SCd = 0, SD = 0;
    for (int jj = 0; jj < 3; ++jj) {
      const int jj_ = fmod_pos(pi2 - 1 + jj - 1, g.n2m);
      double qa = 0, qb = 0, qc = 0, qd = 0;
      for (int ii = 0; ii < 3; ++ii) {
        const double T = q[cidx(g, fmod_pos(pi1 - 1 + ii - 1, g.n1m), jj_, kk_)];
        qa = fma(w[0][ii], T, qa); qb = fma(wd[0][ii], T, qb);
        qc = fma(dw[0][ii], T, qc); qd = fma(dwd[0][ii], T, qd);
      }
      SA = fma(w[1][jj], qa, SA); SAd = fma(wd[1][jj], qa, SAd);
      SAw = fma(dw[1][jj], qa, SAw); SAwd = fma(dwd[1][jj], qa, SAwd);
      SB = fma(w[1][jj], qb, SB); SBw = fma(dw[1][jj], qb, SBw);
      SC = fma(w[1][jj], qc, SC); SCd = fma(wd[1][jj], qc, SCd);
      SD = fma(w[1][jj], qd, SD);
    }
    const double z = w[2][kk], zd = wd[2][kk], dz = dw[2][kk], dzd = dwd[2][kk];
    MT[0] = fma(z, SA, MT[0]); MT[1] = fma(z, SB, MT[1]); MT[2] = fma(z, SAd, MT[2]); MT[3] = fma(zd, SA, MT[3]);
    MD[0][0] = fma(z, SC, MD[0][0]); MD[0][1] = fma(z, SD, MD[0][1]);
    MD[0][2] = fma(z, SCd, MD[0][2]); MD[0][3] = fma(zd, SC, MD[0][3]);
    MD[1][0] = fma(z, SAw, MD[1][0]); MD[1][1] = fma(z, SBw, MD[1][1]);
    MD[1][2] = fma(z, SAwd, MD[1][2]); MD[1][3] = fma(zd, SAw, MD[1][3]);
    MD[2][0] = fma(dz, SA, MD[2][0]); MD[2][1] = fma(dz, SB, MD[2][1]);
    MD[2][2] = fma(dz, SAd, MD[2][2]); MD[2][3] = fma(dzd, SA, MD[2][3]);
  }
  for (int d = 0; d < 3; ++d) {
    double dA[16];
    double X[3], Y[3], Z[3];
    for (int m = 0; m < 3; ++m) {
      X[m] = d == 0 ? D[0][m] : S[0][m];
      Y[m] = d == 1 ? D[1][m] : S[1][m];
      Z[m] = d == 2 ? D[2][m] : S[2][m];
    }
    moment_matrix(X, Y, Z, dA);
    double pk[4];
    for (int r = 0; r < 4; ++r) {
      double a = 0;
      for (int cc = 0; cc < 4; ++cc) a = fma(dA[r + 4 * cc], gam[cc], a);
      pk[r] = (r == d + 1 ? 1.0 : 0.0) - a;
    }
    double acc = 0;
    for (int r = 0; r < 4; ++r) {
      double dg = 0;
      for (int cc = 0; cc < 4; ++cc) dg = fma(Ai[r + 4 * cc], pk[cc], dg);
      acc = fma(dg, MT[r], fma(gam[r], MD[d][r], acc));
    }
    grad[d] = acc;
  }
  return true;
}

// Separable MLS value at a probe (wght_press, mls_structLoads.f90:271-404):
// cell-centred cage around (i0, j0), z layers k1-1, k1, k1+1 (no repeated
// layer).  value = A^{-1} e0 . sum_n w_n p_n q_n in the shifted basis.
__device__ bool probe_value_sep(const LagArgs& A, const double pos[3], int i0, int j0, const double* __restrict__ q,
                                double& val) {
  const Grid& g = A.g;
  int k1 = ffloor(pos[2] * g.dx3) + 1;
  int k1w = fmod_pos(k1 - 1, g.n3m) + 1;
  double w[3][3], dd[3][3];
  for (int r = 0; r < 3; ++r) {
    double pc[3] = {coord(A, 0, 1, i0 - 1 + r), coord(A, 1, 1, j0 - 1 + r), coord(A, 2, 1, k1 - 1 + r)};
    for (int a = 0; a < 3; ++a) {
      double dwu;
      axis_weight(A, a, pos[a], pc[a], w[a][r], dwu);
      dd[a][r] = pc[a] - pos[a];
    }
  }
  double S[3][3];
  for (int a = 0; a < 3; ++a) moments3(w[a], dd[a], S[a]);
  double Ai[16];
  moment_matrix(S[0], S[1], S[2], Ai);
  if (!inv4(Ai)) return false;
  // sum over the cage of q w p, contracted one axis at a time (as in
  // probe_grad_sep)
  double MT[4] = {0, 0, 0, 0};
  for (int kk = 0; kk < 3; ++kk) {
    const int kk_ = wrap(k1w - 1 + kk - 1, g.n3m);
    double SA = 0, SAd = 0, SB = 0;
    for (int jj = 0; jj < 3; ++jj) {
      const int jj_ = fmod_pos(j0 - 1 + jj - 1, g.n2m);
      double qa = 0, qb = 0;
      for (int ii = 0; ii < 3; ++ii) {
        const double T = q[cidx(g, fmod_pos(i0 - 1 + ii - 1, g.n1m), jj_, kk_)];
        qa = fma(w[0][ii], T, qa); qb = fma(w[0][ii] * dd[0][ii], T, qb);
      }
      SA = fma(w[1][jj], qa, SA); SAd = fma(w[1][jj] * dd[1][jj], qa, SAd); SB = fma(w[1][jj], qb, SB);
    }
    MT[0] = fma(w[2][kk], SA, MT[0]); MT[1] = fma(w[2][kk], SB, MT[1]);
    MT[2] = fma(w[2][kk], SAd, MT[2]); MT[3] = fma(w[2][kk] * dd[2][kk], SA, MT[3]);
  }
  double v = 0;
  for (int r = 0; r < 4; ++r) v = fma(Ai[r], MT[r], v);
  val = v;
  return true;
}

// mls_heatFlux.f90:77-158 at both probes of every face with the separable
// construction (precision form, moving body): one thread per (face, side).
__global__ void heat_flux_sep_kernel(LagArgs A, const double* __restrict__ temp, const double* __restrict__ tri_bar,
                                 const double* __restrict__ tri_nor, const int* __restrict__ ghost,
                                 const int* __restrict__ pind, double h, double pec, double* __restrict__ qw_o,
                                 double* __restrict__ qw_i, int* __restrict__ flag) {
  int gid = blockIdx.x * blockDim.x + threadIdx.x;
  int t = gid >> 1, side = gid & 1;
  if (t >= A.nf) return;
  double* qout = side == 0 ? qw_o : qw_i;
  if (ghost[t]) { qout[t] = 0.0; return; }
  double n0 = tri_nor[3 * t], n1 = tri_nor[3 * t + 1], n2 = tri_nor[3 * t + 2];
  double s = sqrt(n0 * n0 + n1 * n1 + n2 * n2);
  double pos[3];
  for (int d = 0; d < 3; ++d) {
    double nd = tri_nor[3 * t + d];
    pos[d] = side == 0 ? tri_bar[3 * t + d] + h * nd / s : tri_bar[3 * t + d] - h * nd / s;
  }
  // pind null (fused step): the probe's cage as probe_idx_kernel finds it
  const int pi1 = pind ? pind[6 * t + 3 * side + 0] : ffloor(pos[0] * A.g.dx1) + 1;
  const int pi2 = pind ? pind[6 * t + 3 * side + 1] : ffloor(pos[1] * A.g.dx2) + 1;
  double grad[3];
  if (!probe_grad_sep(A, pos, pi1, pi2, 1, 1, 1, false, temp, grad)) { atomicOr(flag, 1); qout[t] = 0.0; return; }
  double qv = n0 * grad[0] + n1 * grad[1] + n2 * grad[2];
  qout[t] = qv / pec;
}

// The literal heat flux of the plain form (mls_heatFlux.f90:77-158 with
// wght_gradT), spread over a block of 4 warps for 32 probes (lane = probe,
// probe q = face q/2, side q%2): warp 0 forms the probe's per-axis weights
// (shared), then the moment matrix A by the reference's rank-one updates, its
// inverse and gamma; warp w = 1..3 forms dA_d (d = w - 1) meanwhile and, once
// A^-1 and gamma are published, the direction-d gradient.  Every value comes
// from exactly the operations of probe_grad_lit in its order (the oracle's
// bits); the split only gives the device four times the independent work per
// probe that one thread would have.  Bound by the FP64 pipe (no contraction, so
// a product and its sum are two instructions): the repeated layer's and the
// symmetric sums once, divisions by constants as five operations (div_const),
// comparisons on the bits and the probe's position formed by one warp took 20480
// faces from 612 to 418 us, 5120 from 219 to 152; the MLS weights (mls_weight_kernel)
// of 20480 faces went from 313 to 279 us, the precision form's from 146 to 119.
constexpr int kHfProbes = 32;
__global__ void __launch_bounds__(4 * kHfProbes)
heat_flux_lit_kernel(LagArgs A, const double* __restrict__ temp, const double* __restrict__ tri_bar,
                     const double* __restrict__ tri_nor, const int* __restrict__ ghost,
                     const int* __restrict__ pind, double h, double pec, double* __restrict__ qw_o,
                     double* __restrict__ qw_i, int* __restrict__ flag) {
  __shared__ double sW[3][3][kHfProbes], sdW[3][3][kHfProbes], spc[3][3][kHfProbes];
  __shared__ double sAi[16][kHfProbes], sgam[4][kHfProbes], sgrad[3][kHfProbes];
  __shared__ int sok[kHfProbes], scell[3][kHfProbes];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int gid = blockIdx.x * kHfProbes + lane;
  const int t = gid >> 1, side = gid & 1;
  const bool valid = t < A.nf;
  const bool live = valid && !ghost[t];
  const Grid& g = A.g;
  double pos[3] = {0.0, 0.0, 0.0};
  if (w == 0 && live) {
    const double n0 = tri_nor[3 * t], n1 = tri_nor[3 * t + 1], n2 = tri_nor[3 * t + 2];
    const double s = sqrt(n0 * n0 + n1 * n1 + n2 * n2);
    for (int d = 0; d < 3; ++d) {
      const double nd = tri_nor[3 * t + d];
      pos[d] = side == 0 ? tri_bar[3 * t + d] + h * nd / s : tri_bar[3 * t + d] - h * nd / s;
    }
    // pind null (fused step): the probe's cage as probe_idx_kernel finds it
    const int pi1 = pind ? pind[6 * t + 3 * side + 0] : ffloor(pos[0] * g.dx1) + 1;
    const int pi2 = pind ? pind[6 * t + 3 * side + 1] : ffloor(pos[1] * g.dx2) + 1;
    const int k1 = ffloor(pos[2] * g.dx3) + 1;
    scell[0][lane] = pi1;
    scell[1][lane] = pi2;
    scell[2][lane] = k1;
    for (int r = 0; r < 3; ++r) {
      const double pc[3] = {coord(A, 0, 1, pi1 - 1 + r), coord(A, 1, 1, pi2 - 1 + r), coord(A, 2, 1, k1 - 1 + r)};
      for (int a = 0; a < 3; ++a) {
        if (a == 2 && r == 2) break;              // z layers k1 - 1, k1 and k1 again
        double W, dW;
        lit_axis_weight(A, a, pos[a], pc[a], W, dW);
        spc[a][r][lane] = pc[a];
        sW[a][r][lane] = W;
        sdW[a][r][lane] = dW;
      }
    }
  }
  __syncthreads();
  const int d = w - 1;
  double x[3], y[3];
  for (int r = 0; r < 3; ++r) {
    x[r] = spc[0][r][lane];
    y[r] = spc[1][r][lane];
  }
  // node weights of layer nk: of A (e < 0) or dA_e
  auto nodes = [&](int e, int nk, double (&out)[9]) {
    const double W0[3] = {sW[0][0][lane], sW[0][1][lane], sW[0][2][lane]};
    const double W1[3] = {sW[1][0][lane], sW[1][1][lane], sW[1][2][lane]};
    const double dW0[3] = {sdW[0][0][lane], sdW[0][1][lane], sdW[0][2][lane]};
    const double dW1[3] = {sdW[1][0][lane], sdW[1][1][lane], sdW[1][2][lane]};
    lit_node_weights(e, W0, dW0, W1, dW1, sW[2][nk][lane], sdW[2][nk][lane], out);
  };
  double Mx[16];
  if (live) {
    double wn[9];
    nodes(d, 0, wn);
    lit_layer<true>(wn, x, y, spc[2][0][lane], Mx);
    nodes(d, 1, wn);
    lit_layer<false>(wn, x, y, spc[2][1][lane], Mx);
    lit_symmetric(Mx);
  }
  if (w == 0) {
    int ok = 0;
    if (live && inv4(Mx)) {
      ok = 1;
      const double ptx[4] = {1.0, pos[0], pos[1], pos[2]};
      for (int r = 0; r < 4; ++r) {               // DGEMV('N', invA, ptx)
        double tt = 0;
        for (int cc = 0; cc < 4; ++cc) tt += Mx[r + 4 * cc] * ptx[cc];
        sgam[r][lane] = tt;
      }
      for (int e = 0; e < 16; ++e) sAi[e][lane] = Mx[e];
    }
    sok[lane] = ok;
  }
  __syncthreads();
  if (w > 0 && live && sok[lane]) {
    double gam[4];
    for (int r = 0; r < 4; ++r) gam[r] = sgam[r][lane];
    double pk_d[4] = {0.0, 0.0, 0.0, 0.0};
    pk_d[d + 1] = 1.0;
    for (int r = 0; r < 4; ++r) {                   // pk = -dA gamma + pk
      double tt = 0;
      for (int cc = 0; cc < 4; ++cc) tt += Mx[r + 4 * cc] * gam[cc];
      pk_d[r] = pk_d[r] - tt;
    }
    double dgam[4];
    for (int r = 0; r < 4; ++r) {
      double tt = 0;
      for (int cc = 0; cc < 4; ++cc) tt += sAi[r + 4 * cc][lane] * pk_d[cc];
      dgam[r] = tt;
    }
    const int pi1 = scell[0][lane], pi2 = scell[1][lane], k1w = fmod_pos(scell[2][lane] - 1, g.n3m) + 1;
    double gsum = 0, v[9];
    for (int nk = 0; nk < 3; ++nk) {
      if (nk < 2) {
        double wt[9], dw[9];
        nodes(-1, nk, wt);
        nodes(d, nk, dw);
        lit_node_values(wt, dw, dgam, gam, x, y, spc[2][nk][lane], v);
      }
      const int kk = wrap(k1w - 2 + nk, g.n3m);
#pragma unroll
      for (int n = 0; n < 9; ++n)
        gsum += v[n] * temp[cidx(g, fmod_pos(pi1 - 1 + n % 3 - 1, g.n1m), fmod_pos(pi2 - 1 + n / 3 - 1, g.n2m), kk)];
    }
    sgrad[d][lane] = gsum;
  }
  __syncthreads();
  if (w == 0 && valid) {
    double* qout = side == 0 ? qw_o : qw_i;
    if (!live) {
      qout[t] = 0.0;
    } else if (!sok[lane]) {
      atomicOr(flag, 1);
      qout[t] = 0.0;
    } else {
      const double qv = tri_nor[3 * t] * sgrad[0][lane] + tri_nor[3 * t + 1] * sgrad[1][lane] +
                        tri_nor[3 * t + 2] * sgrad[2][lane];
      qout[t] = qv / pec;
    }
  }
}

// The same construction, every value by the same operations in the same order
// (the same bits), with a probe on four lanes of each of the four warps: a
// block takes 8 probes.  A lane evaluates one of the nine axis weights,
// accumulates one column of A (warp 0) or dA_d (warps 1-3) and every fourth of
// the 27 terms of the gradient, which are then added in cage order; only the
// inversion is done by all four lanes alike.  The chain of FP64 instructions
// of a block is a third of the other kernel's and there are four times the
// blocks, at a quarter more FP64 instructions in all: faster until the SMs are
// full (1280 faces 72 -> 60 us, 5120 faces 152 -> 163, 20480 faces 418 -> 582).
constexpr int kHf4Probes = 8;
constexpr int kHf4Faces = 4096;
__global__ void __launch_bounds__(128)
heat_flux_lit4_kernel(LagArgs A, const double* __restrict__ temp, const double* __restrict__ tri_bar,
                      const double* __restrict__ tri_nor, const int* __restrict__ ghost,
                      const int* __restrict__ pind, double h, double pec, double* __restrict__ qw_o,
                      double* __restrict__ qw_i, int* __restrict__ flag) {
  constexpr int NP = kHf4Probes;
  const unsigned FULL = 0xffffffffu;
  __shared__ double sW[3][3][NP], sdW[3][3][NP], spc[3][3][NP], spos[3][NP];
  __shared__ double sAi[16][NP], sdA[3][16][NP], sgam[4][NP], sgrad[3][NP];
  __shared__ int sok[NP];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, pr = lane >> 2, c = lane & 3;
  const int gid = blockIdx.x * NP + pr;
  const int t = gid >> 1, side = gid & 1;
  const bool valid = t < A.nf;
  const bool live = valid && !ghost[t];
  const Grid& g = A.g;
  const double eps = 2.220446049250313e-16;       // EPSILON(1.0d0)
  if (w == 0) {
    double x = 0.0;
    if (live && c < 3) {
      const double n0 = tri_nor[3 * t], n1 = tri_nor[3 * t + 1], n2 = tri_nor[3 * t + 2];
      const double s = sqrt(n0 * n0 + n1 * n1 + n2 * n2);
      const double nd = c == 0 ? n0 : (c == 1 ? n1 : n2);
      x = side == 0 ? tri_bar[3 * t + c] + h * nd / s : tri_bar[3 * t + c] - h * nd / s;
    }
    if (c < 3) spos[c][pr] = x;
  }
  __syncthreads();
  const double pos[3] = {spos[0][pr], spos[1][pr], spos[2][pr]};
  int pi1 = 0, pi2 = 0, k1 = 0;
  if (live) {
    // pind null (fused step): the probe's cage as probe_idx_kernel finds it
    pi1 = pind ? pind[6 * t + 3 * side + 0] : ffloor(pos[0] * g.dx1) + 1;
    pi2 = pind ? pind[6 * t + 3 * side + 1] : ffloor(pos[1] * g.dx2) + 1;
    k1 = ffloor(pos[2] * g.dx3) + 1;
  }
  if (live && 4 * w + c < 8) {                    // one axis weight per lane
    const int a = (4 * w + c) % 3, r = (4 * w + c) / 3;
    const double pc = a == 0 ? coord(A, 0, 1, pi1 - 1 + r)
                             : (a == 1 ? coord(A, 1, 1, pi2 - 1 + r) : coord(A, 2, 1, k1 - 1 + r));
    double W, dW;
    lit_axis_weight(A, a, pos[a], pc, W, dW);
    spc[a][r][pr] = pc;
    sW[a][r][pr] = W;
    sdW[a][r][pr] = dW;
  }
  __syncthreads();
  const int d = w - 1;
  // weight of node (i, j, nk): of A, and of dA_d
  auto wt_of = [&](int i, int j, int nk) { return sW[0][i][pr] * (sW[1][j][pr] * sW[2][nk][pr]); };
  auto dw_of = [&](int i, int j, int nk) {
    return d == 0 ? (sdW[0][i][pr] * sW[1][j][pr]) * sW[2][nk][pr]
         : d == 1 ? (sW[0][i][pr] * sdW[1][j][pr]) * sW[2][nk][pr]
                  : (sW[0][i][pr] * sW[1][j][pr]) * sdW[2][nk][pr];
  };
  double col[4] = {0.0, 0.0, 0.0, 0.0};           // column c; layer 1 counts twice (lit_layer)
  if (live) {
#pragma unroll
    for (int nk = 0; nk < 2; ++nk) {
      const double pz = spc[2][nk][pr];
      double p[4][9];
#pragma unroll
      for (int n = 0; n < 9; ++n) {
        const int i = n % 3, j = n / 3;
        const double wn = w == 0 ? wt_of(i, j, nk) : dw_of(i, j, nk);
        const double px = spc[0][i][pr], py = spc[1][j][pr];
        const double tt = wn * (c == 0 ? 1.0 : (c == 1 ? px : (c == 2 ? py : pz)));
        p[0][n] = tt;
        p[1][n] = tt * px;
        p[2][n] = tt * py;
        p[3][n] = tt * pz;
      }
#pragma unroll
      for (int rep = 0; rep <= nk; ++rep)
#pragma unroll
        for (int n = 0; n < 9; ++n)
#pragma unroll
          for (int r = 0; r < 4; ++r) col[r] = col[r] + p[r][n];
    }
  }
  if (w == 0) {
    double Am[16];
    for (int cc = 0; cc < 4; ++cc)
      for (int r = 0; r < 4; ++r) Am[r + 4 * cc] = __shfl_sync(FULL, col[r], (lane & ~3) + cc);
    int ok = 0;
    if (live && inv4(Am)) {
      ok = 1;
      const double ptx[4] = {1.0, pos[0], pos[1], pos[2]};
      for (int r = 0; r < 4; ++r) {               // DGEMV('N', invA, ptx)
        double tt = 0;
        for (int cc = 0; cc < 4; ++cc) tt += Am[r + 4 * cc] * ptx[cc];
        if (r == c) sgam[r][pr] = tt;
      }
      for (int e = 0; e < 16; ++e)
        if ((e >> 2) == c) sAi[e][pr] = Am[e];
    }
    if (c == 0) sok[pr] = ok;
  } else {
    for (int r = 0; r < 4; ++r) sdA[d][r + 4 * c][pr] = col[r];
  }
  __syncthreads();
  if (w > 0) {
    const bool go = live && sok[pr];
    double gam[4] = {0.0, 0.0, 0.0, 0.0};
    double mine = 0.0;
    if (go) {
      for (int r = 0; r < 4; ++r) gam[r] = sgam[r][pr];
      double tt = 0;                               // row c of pk = -dA gamma + pk
      for (int cc = 0; cc < 4; ++cc) tt += sdA[d][c + 4 * cc][pr] * gam[cc];
      mine = (c == d + 1 ? 1.0 : 0.0) - tt;
    }
    double pk_d[4], dgam[4];
    for (int r = 0; r < 4; ++r) pk_d[r] = __shfl_sync(FULL, mine, (lane & ~3) + r);
    double dg = 0;
    if (go)
      for (int cc = 0; cc < 4; ++cc) dg += sAi[c + 4 * cc][pr] * pk_d[cc];
    for (int r = 0; r < 4; ++r) dgam[r] = __shfl_sync(FULL, dg, (lane & ~3) + r);
    const int k1w = fmod_pos(k1 - 1, g.n3m) + 1;
    double gsum = 0;
    double nv[5];                                  // nodes 4m .. 4m+3 of layers 0 and 1, one per lane
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const int nd = 4 * m + c;
      nv[m] = 0.0;
      if (go && nd < 18) {
        const int i = nd % 3, j = (nd / 3) % 3, nk = nd / 9;
        const double wtx = wt_of(i, j, nk), dwd = dw_of(i, j, nk);
        const double px = spc[0][i][pr], py = spc[1][j][pr], pz = spc[2][nk][pr];
        const double t1 = ((dgam[0] * wtx + dgam[1] * (wtx * px)) + dgam[2] * (wtx * py)) + dgam[3] * (wtx * pz);
        const double t2 = ((gam[0] * dwd + gam[1] * (dwd * px)) + gam[2] * (dwd * py)) + gam[3] * (dwd * pz);
        nv[m] = t1 + t2;
      }
    }
#pragma unroll
    for (int m = 0; m < 7; ++m) {                  // all 27 in cage order
      const int nd = 4 * m + c;
      double val = m < 5 ? nv[m] : 0.0;
      if (m >= 4) {                                // node nd - 9: lane c - 1 of group m - 2, lane 3 of m - 3 for c = 0
        const double a = __shfl_sync(FULL, nv[m - 2], (lane & ~3) + ((c + 3) & 3));
        const double b = __shfl_sync(FULL, nv[m - 3], (lane & ~3) + 3);
        if (nd >= 18) val = c == 0 ? b : a;
      }
      if (go && nd < 27)
        val *= temp[cidx(g, fmod_pos(pi1 - 1 + nd % 3 - 1, g.n1m), fmod_pos(pi2 - 1 + (nd / 3) % 3 - 1, g.n2m),
                         wrap(k1w - 2 + nd / 9, g.n3m))];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double v = __shfl_sync(FULL, val, (lane & ~3) + q);
        if (4 * m + q < 27) gsum += v;
      }
    }
    if (go && c == 0) sgrad[d][pr] = gsum;
  }
  __syncthreads();
  if (w == 0 && valid && c == 0) {
    double* qout = side == 0 ? qw_o : qw_i;
    if (!live) {
      qout[t] = 0.0;
    } else if (!sok[pr]) {
      atomicOr(flag, 1);
      qout[t] = 0.0;
    } else {
      const double qv = tri_nor[3 * t] * sgrad[0][pr] + tri_nor[3 * t + 1] * sgrad[1][pr] +
                        tri_nor[3 * t + 2] * sgrad[2][pr];
      qout[t] = qv / pec;
    }
  }
}

// ---------------------------------------------------------------------
// Structural loads (mls_structLoads.f90:1-269).  Faces go in groups of 32
// (lane = face); each group is five one-warp blocks, and warp e evaluates, at
// each face's positive probe x_p = X + h n/|n|,
//   e = 0  the pressure (wght_press: cell-centred cage, z layers k1-1..k1+1
//          without the repeated layer, mls_structLoads.f90:271-404)
//   e = 1  grad p   (wght_gradP, cage (icent, jcent))
//   e = 2  grad u   (wght_gradU, x at faces, cage (istag, jcent))
//   e = 3  grad v   (wght_gradV, y at faces, cage (icent, jstag))
//   e = 4  grad w   (wght_gradW, z at faces with nint, cage (icent, jcent))
// so every warp runs one kind of evaluation, and stores it in the group's
// slots.  One-warp blocks spread over the SMs evenly (five-warp blocks of 32
// faces left a few SMs with two blocks of the FP64-bound evaluations).  The
// last of the five warps to finish (a group ticket) forms each face's
// pressure force, viscous normal stress and their moments about pos_CM in
// the reference's operation order (face_loads) and sums the 32 faces' 12
// values with fixed shuffle trees; the last group to finish (the global
// ticket) adds the group sums (lane l takes groups l, l+32, ... in order, then
// a fixed shuffle tree) and updates the loads.  Tickets are reset by the
// warps that close them.
// Lit (the plain form): the reference's MLS construction (probe_value_lit,
// probe_grad_lit), the oracle's bits per face.  Otherwise (the precision
// form) the separable construction, which agrees with the reference's
// rank-one accumulation in absolute coordinates to that construction's
// round-off (amplified by its ~1e8 conditioning) at a fifth of the cost.
// scratch: [groups][13][32] evaluations, then [groups][12] group sums;
// tickets: [0] groups done, [1 + g] warps of group g done.
// ---------------------------------------------------------------------
constexpr int kLoadFaces = 32;

__device__ __forceinline__ void struct_probe(const double* __restrict__ tri_bar, const double* __restrict__ tri_nor,
                                             int t, double h, double pos[3], double nrm[3]) {
  for (int d = 0; d < 3; ++d) nrm[d] = tri_nor[3 * t + d];
  double s = sqrt(nrm[0] * nrm[0] + nrm[1] * nrm[1] + nrm[2] * nrm[2]);
  for (int d = 0; d < 3; ++d) pos[d] = tri_bar[3 * t + d] + h * nrm[d] / s;
}

template <bool Lit>
__global__ void __launch_bounds__(kLoadFaces)
loads_face_kernel(LagArgs A, const double* __restrict__ pr, const double* __restrict__ vx,
                  const double* __restrict__ vy, const double* __restrict__ vz, const double* __restrict__ tri_bar,
                  const double* __restrict__ tri_nor, const double* __restrict__ sur, const int* __restrict__ ghost,
                  const StepParams* __restrict__ pp, double h, double ren, double* __restrict__ scratch,
                  int* __restrict__ flag, unsigned* __restrict__ tickets, RigidDev* __restrict__ r) {
  const unsigned FULL = 0xffffffffu;
  const int lf = threadIdx.x;
  const int grp = blockIdx.x / 5, e = blockIdx.x % 5, ngrp = gridDim.x / 5;
  double* evg = scratch + (size_t)grp * 13 * kLoadFaces;
  double* part = scratch + (size_t)ngrp * 13 * kLoadFaces;
  const int t = grp * kLoadFaces + lf;
  const bool live = t < A.nf && !ghost[t];
  const Grid& g = A.g;
  double pos[3], nrm[3];
  if (live) {
    struct_probe(tri_bar, tri_nor, t, h, pos, nrm);
    int icent = ffloor(pos[0] * g.dx1) + 1, istag = fnint(pos[0] * g.dx1) + 1;
    int jcent = ffloor(pos[1] * g.dx2) + 1, jstag = fnint(pos[1] * g.dx2) + 1;
    bool ok;
    if (e == 0) {
      double v = 0.0;
      ok = Lit ? probe_value_lit(A, pos, icent, jcent, pr, v) : probe_value_sep(A, pos, icent, jcent, pr, v);
      evg[lf] = ok ? v : 0.0;
    } else {
      double gr[3] = {0, 0, 0};
      const double* q = e == 1 ? pr : e == 2 ? vx : e == 3 ? vy : vz;
      const int pi1 = e == 2 ? istag : icent, pi2 = e == 3 ? jstag : jcent;
      const int sx = e == 2 ? 0 : 1, sy = e == 3 ? 0 : 1, sz = e == 4 ? 0 : 1;
      ok = Lit ? probe_grad_lit(A, pos, pi1, pi2, sx, sy, sz, e == 4, q, gr)
               : probe_grad_sep(A, pos, pi1, pi2, sx, sy, sz, e == 4, q, gr);
      for (int d = 0; d < 3; ++d) evg[(1 + 3 * (e - 1) + d) * kLoadFaces + lf] = ok ? gr[d] : 0.0;
    }
    if (!ok) atomicOr(flag, 1);
  }
  // the last of the group's five warps forms the loads of its 32 faces
  __threadfence();
  __syncwarp();
  unsigned done = 0;
  if (lf == 0) done = atomicAdd(&tickets[1 + grp], 1u);
  if (__shfl_sync(FULL, done, 0) != 4u) return;
  __threadfence();
  double cf[12];
  for (int q = 0; q < 12; ++q) cf[q] = 0.0;
  if (live) {
    double e13[13], rad[3];
    for (int q = 0; q < 13; ++q) e13[q] = __ldcg(evg + q * kLoadFaces + lf);
    for (int d = 0; d < 3; ++d) rad[d] = tri_bar[3 * t + d] - pp->pos[d];
    face_loads(e13, nrm, rad, sur[t], h, ren, cf);
  }
  // group sums (a shuffle tree over the group's faces per quantity)
  for (int q = 0; q < 12; ++q) {
    double v = cf[q];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(FULL, v, off);
    if (lf == 0) part[12 * (size_t)grp + q] = v;
  }
  if (lf == 0) tickets[1 + grp] = 0u;
  __threadfence();
  __syncwarp();
  unsigned gdone = 0;
  if (lf == 0) gdone = atomicAdd(&tickets[0], 1u);
  if (__shfl_sync(FULL, gdone, 0) != (unsigned)ngrp - 1u) return;
  __threadfence();
  // the last group: the loads (lane l takes groups l, l+32, ... in order, then
  // a fixed shuffle tree), the previous loads to the _m1 slots, the new ones
  // stored and added to the running sums (mls_structLoads.f90:21-24, 207-262)
  double tot[12];
  for (int q = 0; q < 12; ++q) {
    double v = 0.0;
    for (int b = lf; b < ngrp; b += 32) v += __ldcg(part + 12 * (size_t)b + q);
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(FULL, v, off);
    tot[q] = v;
  }
  if (lf == 0) {
    for (int q = 0; q < 12; ++q) {        // packed [prn, tau, rprn, rtau]
      r->load1[q] = r->load[q];
      r->load[q] = tot[q];
      r->acc[q] = r->acc[q] + tot[q];
    }
    tickets[0] = 0u;
  }
}

// face -> vertex: qw_v(v) = sum over adjacent faces (ascending) of q_f*(A_f/3/A_v)
__device__ __forceinline__ void vert_flux(int v, const int* __restrict__ adj_off, const int* __restrict__ adj_face,
                                          const double* __restrict__ sur, const double* __restrict__ avert,
                                          const double* __restrict__ qf_o, const double* __restrict__ qf_i,
                                          double& so, double& si) {
  const double av = avert[v];
  so = si = 0.0;
  for (int q = adj_off[v]; q < adj_off[v + 1]; ++q) {
    int f = adj_face[q];
    double w = sur[f] / 3.0 / av;
    so = so + qf_o[f] * w;
    si = si + qf_i[f] * w;
  }
}

__global__ void face_to_vert_kernel(int nv, const int* __restrict__ adj_off, const int* __restrict__ adj_face,
                                    const double* __restrict__ sur, const double* __restrict__ avert,
                                    const double* __restrict__ qf_o, const double* __restrict__ qf_i,
                                    double* __restrict__ qv_o, double* __restrict__ qv_i) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  double so, si;
  vert_flux(v, adj_off, adj_face, sur, avert, qf_o, qf_i, so, si);
  qv_o[v] = so;
  qv_i[v] = si;
}

__device__ __forceinline__ void vert_melt(int v, const int* __restrict__ ghostv, const double* __restrict__ vert_nor,
                                          double qo, double qi, double cp_over_L, const StepParams* __restrict__ pp,
                                          double* __restrict__ vmelt, double* __restrict__ vmelt_m1,
                                          double* __restrict__ xyzv) {
  double dt = pp->dt, ga = pp->ga, ro = pp->ro;
  for (int d = 0; d < 3; ++d) vmelt_m1[3 * v + d] = vmelt[3 * v + d];
  if (ghostv[v]) return;
  double dq = qi - qo;
  for (int d = 0; d < 3; ++d) {
    double vm = cp_over_L * dq * vert_nor[3 * v + d];
    vmelt[3 * v + d] = vm;
    xyzv[3 * v + d] = xyzv[3 * v + d] + dt * (ga * vm + ro * vmelt_m1[3 * v + d]);
  }
}

__global__ void stefan_kernel(int nv, const int* __restrict__ ghostv, const double* __restrict__ vert_nor,
                              const double* __restrict__ qv_o, const double* __restrict__ qv_i, double cp_over_L,
                              const StepParams* __restrict__ pp, double* __restrict__ vmelt,
                              double* __restrict__ vmelt_m1, double* __restrict__ xyzv) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  vert_melt(v, ghostv, vert_nor, qv_o[v], qv_i[v], cp_over_L, pp, vmelt, vmelt_m1, xyzv);
}

// face_to_vert_kernel and stefan_kernel for one vertex in one launch (fused step)
__global__ void melt_vert_kernel(int nv, const int* __restrict__ adj_off, const int* __restrict__ adj_face,
                                 const double* __restrict__ sur, const double* __restrict__ avert,
                                 const double* __restrict__ qf_o, const double* __restrict__ qf_i,
                                 double* __restrict__ qv_o, double* __restrict__ qv_i, const int* __restrict__ ghostv,
                                 const double* __restrict__ vert_nor, double cp_over_L,
                                 const StepParams* __restrict__ pp, double* __restrict__ vmelt,
                                 double* __restrict__ vmelt_m1, double* __restrict__ xyzv) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  double so, si;
  vert_flux(v, adj_off, adj_face, sur, avert, qf_o, qf_i, so, si);
  qv_o[v] = so;
  qv_i[v] = si;
  vert_melt(v, ghostv, vert_nor, so, si, cp_over_L, pp, vmelt, vmelt_m1, xyzv);
}

// ---------------------------------------------------------------------
// geometry refresh (particle.f90:165-193)
// ---------------------------------------------------------------------
// calculate_area, update_tri_normal, calc_centroids_from_vert of face t and
// its summands of calculate_volume and calc_rigidBody_params
__device__ __forceinline__ void face_geom_one(int t, const int* __restrict__ vof, const double* __restrict__ x,
                                              double* __restrict__ sur, double* __restrict__ nor,
                                              double* __restrict__ bar, double pp[12]) {
  int a = vof[3 * t] - 1, b = vof[3 * t + 1] - 1, d = vof[3 * t + 2] - 1;
  double x1 = x[3 * a], y1 = x[3 * a + 1], z1 = x[3 * a + 2];
  double x2 = x[3 * b], y2 = x[3 * b + 1], z2 = x[3 * b + 2];
  double x3 = x[3 * d], y3 = x[3 * d + 1], z3 = x[3 * d + 2];
  // calculate_area (triaux.f90:82-119)
  double d12 = sqrt(sqd(x1 - x2) + sqd(y1 - y2) + sqd(z1 - z2));
  double d23 = sqrt(sqd(x2 - x3) + sqd(y2 - y3) + sqd(z2 - z3));
  double d31 = sqrt(sqd(x3 - x1) + sqd(y3 - y1) + sqd(z3 - z1));
  double sp = (d12 + d23 + d31) / 2.0;
  double ar = sqrt(sp * (sp - d12) * (sp - d23) * (sp - d31));
  sur[t] = ar;
  // update_tri_normal (triaux.f90:183-232)
  double e1x = x2 - x1, e1y = y2 - y1, e1z = z2 - z1, e2x = x3 - x1, e2y = y3 - y1, e2z = z3 - z1;
  double n0 = e1y * e2z - e1z * e2y, n1 = e1z * e2x - e1x * e2z, n2 = e1x * e2y - e1y * e2x;
  double m = sqrt(n0 * n0 + n1 * n1 + n2 * n2);
  nor[3 * t] = n0 / m; nor[3 * t + 1] = n1 / m; nor[3 * t + 2] = n2 / m;
  // calc_centroids_from_vert (triaux.f90:308-323)
  bar[3 * t] = (x1 + x2 + x3) / 3.0; bar[3 * t + 1] = (y1 + y2 + y3) / 3.0; bar[3 * t + 2] = (z1 + z2 + z3) / 3.0;
  // calculate_volume summand (triaux.f90:53-80)
  double vol = x1 * (y2 * z3 - z2 * y3) + x2 * (y3 * z1 - z3 * y1) + x3 * (y1 * z2 - z1 * y2);
  // calc_rigidBody_params summands (RigidAuxRoutines.f90:704-733)
  double v = x1 * y2 * z3 + y1 * z2 * x3 + x2 * y3 * z1 - (x3 * y2 * z1 + x2 * y1 * z3 + y3 * z2 * x1);
  double x4 = x1 + x2 + x3, y4 = y1 + y2 + y3, z4 = z1 + z2 + z3;
  pp[0] = ar; pp[1] = vol; pp[2] = v; pp[3] = v * x4; pp[4] = v * y4; pp[5] = v * z4;
  pp[6] = v * (x1 * x1 + x2 * x2 + x3 * x3 + x4 * x4);
  pp[7] = v * (y1 * y1 + y2 * y2 + y3 * y3 + y4 * y4);
  pp[8] = v * (z1 * z1 + z2 * z2 + z3 * z3 + z4 * z4);
  pp[9] = v * (y1 * x1 + y2 * x2 + y3 * x3 + y4 * x4);
  pp[10] = v * (z1 * x1 + z2 * x2 + z3 * x3 + z4 * x4);
  pp[11] = v * (z1 * y1 + z2 * y2 + z3 * y3 + z4 * y4);
}

// What the narrow band's bounds need of a face (band_bounds), in FP32 from FP64
// differences: the centroid c and R (every vertex lies within R of it), the unit normal
// and the radius about c of a disc inside the face; and the base cell of its
// 5^3 band.  Where the computed normal is not normal to the face (a sliver: some
// vertex is off its plane by more than 1e-6, or it is no number) normal and
// disc are zero; where c is not the centroid (one that the caller has set) the
// disc's radius is -R, from which band_bound makes |P - c| + R.
struct BandFace { float4 c, n; };
__device__ __forceinline__ void band_prep_one(int f, int nv, const int* __restrict__ vof, const double* __restrict__ x,
                                              const double pos[3], const Grid& g, BandFace* __restrict__ band_face,
                                              int4* __restrict__ face_cell) {
  int vid[3] = {vof[3 * f] - 1, vof[3 * f + 1] - 1, vof[3 * f + 2] - 1};
  if (!(MIBM_IDX_OK(vid[0], nv) & MIBM_IDX_OK(vid[1], nv) & MIBM_IDX_OK(vid[2], nv))) vid[0] = vid[1] = vid[2] = 0;
  float p[3][3], r2 = 0.f, l2 = 0.f;
  for (int v = 0; v < 3; ++v) {
    for (int d = 0; d < 3; ++d) p[v][d] = d2f_bits(x[3 * vid[v] + d] - pos[d]);
    r2 = fmaxf(r2, p[v][0] * p[v][0] + p[v][1] * p[v][1] + p[v][2] * p[v][2]);
  }
  float e[2][3];
  for (int d = 0; d < 3; ++d) { e[0][d] = p[1][d] - p[0][d]; e[1][d] = p[2][d] - p[0][d]; }
  for (int v = 0; v < 3; ++v) {
    const float a = p[(v + 1) % 3][0] - p[v][0], b = p[(v + 1) % 3][1] - p[v][1], c = p[(v + 1) % 3][2] - p[v][2];
    l2 = fmaxf(l2, a * a + b * b + c * c);
  }
  float n0 = e[0][1] * e[1][2] - e[0][2] * e[1][1], n1 = e[0][2] * e[1][0] - e[0][0] * e[1][2],
        n2 = e[0][0] * e[1][1] - e[0][1] * e[1][0];
  const float area2 = sqrtf(n0 * n0 + n1 * n1 + n2 * n2);
  n0 /= area2; n1 /= area2; n2 /= area2;
  float off = 0.f;
  for (int v = 0; v < 3; ++v) off = fmaxf(off, fabsf(n0 * p[v][0] + n1 * p[v][1] + n2 * p[v][2]));
  const bool flat = off <= 1e-6f && fabsf(n0) <= 1.f && fabsf(n1) <= 1.f && fabsf(n2) <= 1.f;
  BandFace b;
  bool mid = true;
  for (int d = 0; d < 3; ++d) mid = mid && fabsf(p[0][d] + p[1][d] + p[2][d]) <= 2e-6f;
  const float R = sqrtf(r2) * 1.00001f + 1e-30f;                          // rounded up
  b.c = make_float4((float)pos[0], (float)pos[1], (float)pos[2], R);
  b.n = !mid ? make_float4(0.f, 0.f, 0.f, -R)
      : flat ? make_float4(n0, n1, n2, area2 / (3.f * sqrtf(l2)) * 0.9999f) : make_float4(0.f, 0.f, 0.f, 0.f);
  band_face[f] = b;
  // base cell of the band, as band_kernel derives it (genSDF.f90:151-153)
  face_cell[f] = make_int4(ffloor(pos[0] * g.dx1) + 1, ffloor(pos[1] * g.dx2) + 1, ffloor(pos[2] * g.dx3) + 1, 0);
}

// the post-processing of calc_rigidBody_params (RigidAuxRoutines.f90:736-775)
// from the 12 body sums: [Surface, Volume1, Volume, pos_CM(3), InertTensor(9)]
__device__ void geom_finish(const double* sm, double dens_ratio, double* __restrict__ out) {
  double Surface = sm[0], Volume1 = sm[1] / 6.0;
  double Vol = sm[2], Cx = sm[3], Cy = sm[4], Cz = sm[5];
  double r = 1.0 / (4.0 * Vol);
  Cx = Cx * r; Cy = Cy * r; Cz = Cz * r;
  Vol = Vol / 6.0;
  out[0] = Surface; out[1] = Volume1; out[2] = Vol;
  out[3] = Cx; out[4] = Cy; out[5] = Cz;
  r = 1.0 / 120.0;
  double Ixy = sm[9] * r - Vol * Cy * Cx;
  double Ixz = sm[10] * r - Vol * Cz * Cx;
  double Iyz = sm[11] * r - Vol * Cz * Cy;
  double xx = sm[6] * r - Vol * Cx * Cx, yy = sm[7] * r - Vol * Cy * Cy, zz = sm[8] * r - Vol * Cz * Cz;
  double Ixx = yy + zz, Iyy = zz + xx, Izz = xx + yy;
  double I[9] = {Ixx, -Ixy, -Ixz, -Ixy, Iyy, -Iyz, -Ixz, -Iyz, Izz};
  for (int q = 0; q < 9; ++q) out[6 + q] = I[q] * dens_ratio;
}

// What the next substep derives from the faces alone, formed with them (fused
// step; null pointers: not wanted): the narrow band's bounds (band_prep_one), the cage
// indices (findCentroidIndices) and whether they differ from the ones the
// scatter plan was built from, and cfac (initmls.f90:25).  Separate kernels
// for these were three more launches on the chain between two substeps.
struct FaceNext {
  Grid g;
  int nv;
  BandFace* band_face;
  int4* face_cell;
  int* pind;
  const int* saved;      // plan_check's
  int* dirty;
  double* cfac;
  double h, celvol;
};

// One thread per face.  The 12 per-face sums are added over the block (one
// quantity per warp: four values per lane in thread order, then a shuffle
// tree) into part[12 * block + q]; the last block to finish (a ticket
// counter, reset by that block) adds the block sums the same way (lane l
// takes blocks l, l+32, ... in order, then a fixed shuffle tree over the
// lanes) and writes the body's scalars to out.  Each warp's dependent FP64
// chain is a few additions per quantity: on this part an FP64 warp
// instruction holds the pipe for about 64 cycles however few lanes run.
// SUM = false leaves the last block's part to geom_sum_kernel, off the chain
// to the next substep's tagging, which reads the faces only.
constexpr int kGeomBlock = 128;
static_assert(kGeomBlock == 128, "four values per lane in the block sums");
__device__ void geom_total(const double* __restrict__ part, int blocks, double* tot, double dens_ratio,
                           double* __restrict__ out) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q = warp; q < 12; q += kGeomBlock / 32) {
    double v = 0.0;
    for (int b = lane; b < blocks; b += 32) v += __ldcg(part + 12 * (size_t)b + q);
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(FULL, v, off);
    if (lane == 0) tot[q] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) geom_finish(tot, dens_ratio, out);
}

__global__ void __launch_bounds__(kGeomBlock) geom_sum_kernel(const double* __restrict__ part, int blocks,
                                                             double dens_ratio, double* __restrict__ out) {
  __shared__ double tot[12];
  geom_total(part, blocks, tot, dens_ratio, out);
}

template <bool SUM>
__global__ void __launch_bounds__(kGeomBlock)
face_geom_kernel(int nf, const int* __restrict__ vof, const int* __restrict__ ghost, const double* __restrict__ x,
                 double* __restrict__ sur, double* __restrict__ nor, double* __restrict__ bar,
                 double* __restrict__ part /* 12 per block */, unsigned* __restrict__ ticket, double dens_ratio,
                 double* __restrict__ out, FaceNext N) {
  const unsigned FULL = 0xffffffffu;
  __shared__ double ws[12][kGeomBlock];
  __shared__ double tot[12];
  __shared__ bool last;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  double pp[12];
  for (int q = 0; q < 12; ++q) pp[q] = 0.0;
  const bool live = t < nf && !ghost[t];
  if (live) face_geom_one(t, vof, x, sur, nor, bar, pp);
  if (t < nf) {
    const double b[3] = {bar[3 * t], bar[3 * t + 1], bar[3 * t + 2]};
    if (N.band_face) band_prep_one(t, N.nv, vof, x, b, N.g, N.band_face, N.face_cell);
    if (N.pind) {
      const int* sv = N.saved + 7 * (size_t)t;
      bool diff = sv[6] != ghost[t];
      if (live) {
        int p[6];
        centroid_idx_one(N.g, b[0], b[1], b[2], p);
        for (int q = 0; q < 6; ++q) {
          N.pind[6 * t + q] = p[q];
          diff = diff || sv[q] != p[q];
        }
      }
      if (diff) atomicOr(N.dirty, 1);
    }
    if (N.cfac) N.cfac[t] = (sur[t] * N.h) / N.celvol;
  }
  for (int q = 0; q < 12; ++q) ws[q][threadIdx.x] = pp[q];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q = warp; q < 12; q += kGeomBlock / 32) {
    double v = ws[q][lane] + ws[q][lane + 32] + ws[q][lane + 64] + ws[q][lane + 96];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(FULL, v, off);
    if (lane == 0) part[12 * (size_t)blockIdx.x + q] = v;
  }
  if constexpr (SUM) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    geom_total(part, (int)gridDim.x, tot, dens_ratio, out);
    if (threadIdx.x == 0) *ticket = 0u;
  }
}


__global__ void vert_geom_kernel(int nv, const int* __restrict__ adj_off, const int* __restrict__ adj_face,
                                 const int* __restrict__ ghostv, const double* __restrict__ sur,
                                 const double* __restrict__ nor, double* __restrict__ avert,
                                 double* __restrict__ vnor) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  double av = 0, a0 = 0, a1 = 0, a2 = 0;
  for (int q = adj_off[v]; q < adj_off[v + 1]; ++q) {
    int f = adj_face[q];
    double s = sur[f];
    av = av + s / 3.0;
    a0 = a0 + s * nor[3 * f]; a1 = a1 + s * nor[3 * f + 1]; a2 = a2 + s * nor[3 * f + 2];
  }
  avert[v] = av;
  if (ghostv[v]) { vnor[3 * v] = a0; vnor[3 * v + 1] = a1; vnor[3 * v + 2] = a2; return; }
  double m = sqrt(a0 * a0 + a1 * a1 + a2 * a2);
  vnor[3 * v] = a0 / m; vnor[3 * v + 1] = a1 / m; vnor[3 * v + 2] = a2 / m;
}

// calculate_eLengths (triaux.f90:277-306); flag bit 0 set when a live edge
// is shorter than thresh (the remesh trigger rm_flag)
__global__ void elength_kernel(int ne, const int* __restrict__ voe, const int* __restrict__ ghoste,
                               const double* __restrict__ x, double thresh, double* __restrict__ el,
                               int* __restrict__ flag) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne || ghoste[e]) return;
  int v1 = voe[2 * e] - 1, v2 = voe[2 * e + 1] - 1;
  double len = sqrt(sqd(x[3 * v1] - x[3 * v2]) + sqd(x[3 * v1 + 1] - x[3 * v2 + 1]) + sqd(x[3 * v1 + 2] - x[3 * v2 + 2]));
  el[e] = len;
  if (flag && len < thresh) atomicOr(flag, 1);
}

// calculate_skewness (triaux.f90:325-358)
__global__ void skewness_kernel(int nf, const int* __restrict__ eof, const int* __restrict__ ghost,
                                const double* __restrict__ el, const double* __restrict__ sur,
                                double* __restrict__ skew) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nf || ghost[t]) return;
  double perim = el[eof[3 * t] - 1] + el[eof[3 * t + 1] - 1] + el[eof[3 * t + 2] - 1];
  double sur_opt = sqrt(3.0) / 4.0 * sqd(perim / 3.0);
  skew[t] = (sur_opt - sur[t]) / sur_opt;
}

// update_tri_velocity (RigidAuxRoutines.f90:902-928) after a remesh:
// vel_tri = vel_CM + omega x (tri_bar - pos_CM), pos_CM of the refreshed
// geometry (geom + 3)
__global__ void tri_velocity_kernel(int nf, const int* __restrict__ ghost, const double* __restrict__ bar,
                                    const double* __restrict__ geom, const double* __restrict__ vel,
                                    const double* __restrict__ om, double* __restrict__ vel_tri) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nf || ghost[t]) return;
  double r[3];
  for (int d = 0; d < 3; ++d) r[d] = bar[3 * t + d] - geom[3 + d];
  double c0 = om[1] * r[2] - r[1] * om[2];
  double c1 = om[2] * r[0] - r[2] * om[0];
  double c2 = om[0] * r[1] - r[0] * om[1];
  vel_tri[3 * t] = vel[0] + c0;
  vel_tri[3 * t + 1] = vel[1] + c1;
  vel_tri[3 * t + 2] = vel[2] + c2;
}

// ---------------------------------------------------------------------
// narrow-band tagging (genSDF.f90:120-192)
// ---------------------------------------------------------------------
__device__ double point_tri_dist(const double P[3], const double V0[3], const double V1[3], const double V2[3]) {
  double E0[3], E1[3], DE[3];
  for (int d = 0; d < 3; ++d) { E0[d] = V1[d] - V0[d]; E1[d] = V2[d] - V0[d]; DE[d] = V0[d] - P[d]; }
  double a = E0[0] * E0[0] + E0[1] * E0[1] + E0[2] * E0[2];
  double b = E0[0] * E1[0] + E0[1] * E1[1] + E0[2] * E1[2];
  double cc = E1[0] * E1[0] + E1[1] * E1[1] + E1[2] * E1[2];
  double d = E0[0] * DE[0] + E0[1] * DE[1] + E0[2] * DE[2];
  double e = E1[0] * DE[0] + E1[1] * DE[1] + E1[2] * DE[2];
  double det = a * cc - b * b, s = b * e - cc * d, t = b * d - a * e;
  if (s + t <= det) {
    if (s < 0.0) {
      if (t < 0.0) {
        if (d < 0.0) { t = 0.0; s = (-d >= a) ? 1.0 : -d / a; }
        else { s = 0.0; if (e >= 0.0) t = 0.0; else if (-e >= cc) t = 1.0; else t = -e / cc; }
      } else {
        s = 0.0; if (e >= 0.0) t = 0.0; else if (-e >= cc) t = 1.0; else t = -e / cc;
      }
    } else if (t < 0.0) {
      t = 0.0; if (d >= 0.0) s = 0.0; else if (-d >= a) s = 1.0; else s = -d / a;
    } else {
      double invDet = 1.0 / det; s = s * invDet; t = t * invDet;
    }
  } else {
    if (s < 0.0) {
      double tmp0 = b + d, tmp1 = cc + e;
      if (tmp1 > tmp0) {
        double numer = tmp1 - tmp0, denom = a - 2.0 * b + cc;
        if (numer >= denom) { s = 1.0; t = 0.0; } else { s = numer / denom; t = 1.0 - s; }
      } else {
        s = 0.0; if (tmp1 <= 0.0) t = 1.0; else if (e >= 0.0) t = 0.0; else t = -e / cc;
      }
    } else if (t < 0.0) {
      double tmp0 = b + e, tmp1 = a + d;
      if (tmp1 > tmp0) {
        double numer = tmp1 - tmp0, denom = a - 2.0 * b + cc;
        if (numer >= denom) { t = 1.0; s = 0.0; } else { t = numer / denom; s = 1.0 - t; }
      } else {
        t = 0.0; if (tmp1 <= 0.0) s = 1.0; else if (d >= 0.0) s = 0.0; else s = -d / a;
      }
    } else {
      double numer = cc + e - b - d, denom = a - 2.0 * b + cc;
      if (numer <= 0.0) s = 0.0; else if (numer >= denom) s = 1.0; else s = numer / denom;
      t = 1.0 - s;
    }
  }
  double D0 = (V0[0] + s * E0[0] + t * E1[0]) - P[0];
  double D1 = (V0[1] + s * E0[1] + t * E1[1]) - P[1];
  double D2 = (V0[2] + s * E0[2] + t * E1[2]) - P[2];
  return sqrt(D0 * D0 + D1 * D1 + D2 * D2);
}

struct TagArgs {
  LagArgs L;
  const double* x; const int* vof; const int* ghost; const double* bar; const double* nor;
};

__device__ __forceinline__ void tri_verts(const TagArgs& T, int f, double V0[3], double V1[3], double V2[3]) {
  int a = T.vof[3 * f] - 1, b = T.vof[3 * f + 1] - 1, c = T.vof[3 * f + 2] - 1;
  if (!(MIBM_IDX_OK(a, T.L.nv) & MIBM_IDX_OK(b, T.L.nv) & MIBM_IDX_OK(c, T.L.nv))) a = b = c = 0;
  for (int d = 0; d < 3; ++d) { V0[d] = T.x[3 * a + d]; V1[d] = T.x[3 * b + d]; V2[d] = T.x[3 * c + d]; }
}

// winner (initial tagging) and band_ub (narrow band): null where not wanted; the
// narrow band's pass 0 sets the winners that its pass 1 uses
__global__ void sdf_reset_kernel(Grid g, unsigned long long* __restrict__ sdf_bits, int* __restrict__ winner,
                                 unsigned* __restrict__ band_ub) {
  size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.cells) return;
  sdf_bits[t] = (unsigned long long)__double_as_longlong(999.0);   // genSDF.f90:138
  if (winner) winner[t] = INT_MAX;
  if (band_ub) band_ub[t] = 0x7f800000u;                           // +inf
}

// Culling of the narrow-band distance pass.  A face lies in its plane, within R
// of its centroid c, and holds a disc of radius r about c, so for a cell centre
// P at height h over the plane whose projection is at rho from c
//   sqrt(h^2 + max(0, rho - R)^2)  <=  dist(P, face)  <=  sqrt(h^2 + max(0, rho - r)^2).
// Pass U takes the minimum of the upper bounds over the candidate faces of a
// cell; the exact pass skips a face whose lower bound exceeds that minimum:
// such a face is strictly farther than the nearest one, so the minimum, the
// set of faces tied at it and hence the earliest-face winner are unchanged.
// The bounds are evaluated in FP32 from FP32 copies of the coordinates, whose
// rounding grows with the coordinate: with X the largest one of the pair, both
// copies together put P - c off by 2 sqrt(3) 2^-24 X, the arithmetic by some 8
// 2^-24 |P - c| more, and a vertex may be 1e-6 off the plane.  The margin of
// either side is kBandMargin, which covers that up to X = 13 (a box of 2 pi),
// or kBandRel X if that is more.
// Without a plane (BandFace) h = r = 0 and rho = |P - c|; that bound alone let
// the exact pass evaluate so many pairs that its three passes took 64 us each
// with 20480 faces at 256^3 (now 22) and 20 us with 5120 at 128^3 (now 11).
constexpr float kBandMargin = 8e-6f, kBandRel = 6.2e-7f;

__global__ void cm32_kernel(LagArgs A, float* __restrict__ cm32) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= A.clen) return;
  cm32[t] = (float)A.xm[t];
  cm32[A.clen + t] = (float)A.ym[t];
  cm32[2 * A.clen + t] = (float)A.zm[t];
}

__global__ void band_prep_kernel(TagArgs T, BandFace* __restrict__ band_face, int4* __restrict__ face_cell) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= T.L.nf) return;
  const double pos[3] = {T.bar[3 * f], T.bar[3 * f + 1], T.bar[3 * f + 2]};
  band_prep_one(f, T.L.nv, T.vof, T.x, pos, T.L.g, band_face, face_cell);
}

// the bound of cell (ii, jj, kk) from face F with in-plane radius rad, and its margin
__device__ __forceinline__ float band_bound(const float* __restrict__ cm32, int clen, int coff, int ii, int jj, int kk,
                                            const BandFace& F, float rad, float& margin) {
  const float gx = cm32[min(max(ii + coff, 0), clen - 1)];
  const float gy = cm32[clen + min(max(jj + coff, 0), clen - 1)];
  const float gz = cm32[2 * clen + min(max(kk + coff, 0), clen - 1)];
  const float vx = gx - F.c.x, vy = gy - F.c.y, vz = gz - F.c.z;
  const float h = F.n.x * vx + F.n.y * vy + F.n.z * vz;
  const float px = vx - h * F.n.x, py = vy - h * F.n.y, pz = vz - h * F.n.z;
  const float a = fmaxf(sqrtf(px * px + py * py + pz * pz) - rad, 0.f);
  const float X = fmaxf(fmaxf(fmaxf(fabsf(gx), fabsf(gy)), fmaxf(fabsf(gz), fabsf(F.c.x))), fmaxf(fabsf(F.c.y), fabsf(F.c.z)));
  margin = fmaxf(kBandMargin, kBandRel * X);
  return sqrtf(h * h + a * a);
}

// after pass U: pairs whose lower bound does not exceed the cell's bound go
// to a compact list (warp-aggregated append)
__global__ void band_select_kernel(TagArgs T, const BandFace* __restrict__ band_face,
                                   const int4* __restrict__ face_cell, const float* __restrict__ cm32,
                                   const unsigned* __restrict__ band_ub, int* __restrict__ list,
                                   int* __restrict__ count) {
  long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int f = (int)(gid / 125), q = (int)(gid % 125);
  const LagArgs& A = T.L;
  bool keep = false;
  if (f < A.nf && !T.ghost[f]) {
    const Grid& g = A.g;
    int4 b = face_cell[f];
    int ii = b.x - 2 + q % 5, jj = b.y - 2 + (q / 5) % 5, kk = b.z - 2 + q / 25;
    int im = fmod_pos(ii - 1, g.n1m), jm = fmod_pos(jj - 1, g.n1m), km = fmod_pos(kk - 1, g.n3m);
    const BandFace F = band_face[f];
    float margin;
    const float lb = band_bound(cm32, A.clen, A.coff, ii, jj, kk, F, F.c.w, margin);
    keep = !(lb - margin > __uint_as_float(band_ub[cidx(g, im, jm, km)]));
  }
  unsigned m = __ballot_sync(0xffffffffu, keep);
  if (!m) return;
  int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(count, __popc(m));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (keep) list[base + __popc(m & ((1u << lane) - 1u))] = (int)gid;
}

// pass U: per (face, band cell) the upper bound plus the margin, min per cell
__global__ void band_ub_kernel(TagArgs T, const BandFace* __restrict__ band_face, const int4* __restrict__ face_cell,
                               const float* __restrict__ cm32, unsigned* __restrict__ band_ub) {
  long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int f = (int)(gid / 125), q = (int)(gid % 125);
  const LagArgs& A = T.L;
  if (f >= A.nf || T.ghost[f]) return;
  const Grid& g = A.g;
  int4 b = face_cell[f];
  int ii = b.x - 2 + q % 5, jj = b.y - 2 + (q / 5) % 5, kk = b.z - 2 + q / 25;
  int im = fmod_pos(ii - 1, g.n1m), jm = fmod_pos(jj - 1, g.n1m), km = fmod_pos(kk - 1, g.n3m);
  const BandFace F = band_face[f];
  float margin;
  const float ub = band_bound(cm32, A.clen, A.coff, ii, jj, kk, F, F.n.w, margin);
  atomicMin(&band_ub[cidx(g, im, jm, km)], __float_as_uint(ub + margin));
}

// one thread per (triangle, band cell) of the compact list of
// band_select_kernel (entry t < *count; the pairs it culls can neither hold
// a cell's minimum nor win it); pass 0: distance (stored) and the minimum
// per cell, pass 1: the earliest triangle at that distance, pass 2: the
// winner writes the signed distance and the VOF
__device__ __forceinline__ void band_pair(const TagArgs& T, int pass, unsigned long long* __restrict__ sdf_bits,
                                          int* __restrict__ winner, double* __restrict__ vofp,
                                          double* __restrict__ dist_buf, const int4* __restrict__ face_cell, int gid,
                                          int t) {
  int f = gid / 125, q = gid % 125;
  const LagArgs& A = T.L;
  if (f >= A.nf || T.ghost[f]) return;
  const Grid& g = A.g;
  int4 b = face_cell[f];
  int ii = b.x - 2 + q % 5, jj = b.y - 2 + (q / 5) % 5, kk = b.z - 2 + q / 25;
  int im = fmod_pos(ii - 1, g.n1m), jm = fmod_pos(jj - 1, g.n1m), km = fmod_pos(kk - 1, g.n3m);
  size_t c0 = cidx(g, im, jm, km);
  double dist;
  if (pass == 0) {
    double P[3] = {coord(A, 0, 1, ii), coord(A, 1, 1, jj), coord(A, 2, 1, kk)};
    double V0[3], V1[3], V2[3];
    tri_verts(T, f, V0, V1, V2);
    dist = point_tri_dist(P, V0, V1, V2);
    dist_buf[t] = dist;
    winner[c0] = INT_MAX;
    atomicMin(&sdf_bits[c0], (unsigned long long)__double_as_longlong(dist));
    return;
  }
  dist = dist_buf[t];
  unsigned long long bits = (unsigned long long)__double_as_longlong(dist);
  if (pass == 1) {
    if (sdf_bits[c0] == bits && dist < 999.0) atomicMin(&winner[c0], f);
    return;
  }
  if (winner[c0] != f || sdf_bits[c0] != bits) return;
  double pos[3] = {T.bar[3 * f], T.bar[3 * f + 1], T.bar[3 * f + 2]};
  double P[3] = {coord(A, 0, 1, ii), coord(A, 1, 1, jj), coord(A, 2, 1, kk)};
  double Q0 = pos[0] - P[0], Q1 = pos[1] - P[1], Q2 = pos[2] - P[2];
  double dotval = T.nor[3 * f] * Q0 + T.nor[3 * f + 1] * Q1 + T.nor[3 * f + 2] * Q2;
  double sgnd = dist * (-copysign(1.0, dotval));
  double eps = 1.0 / g.dx1, vof;
  const double pi = 3.141592653589793238462643;
  if (sgnd <= -eps) vof = 0.0;
  else if (sgnd >= eps) vof = 1.0;
  else vof = 0.5 * (1.0 + sgnd * g.dx1 + (1.0 / pi) * sin(pi * sgnd * g.dx1));
  vofp[c0] = vof;
  sdf_bits[c0] = (unsigned long long)__double_as_longlong(sgnd);
}

// interp_vof after a later tagging of the same step: only the faces around cells
// whose vofp pass 2 has written can have changed since the last one (256^3,
// 20480 faces: 103 -> 37 us beside the projection; the full pass moves 32 bytes per cell)
__global__ void band_vof_kernel(TagArgs T, const int* __restrict__ winner,
                                const double* __restrict__ vofp, double* __restrict__ vofx, double* __restrict__ vofy,
                                double* __restrict__ vofz, const int4* __restrict__ face_cell,
                                const int* __restrict__ list, const int* __restrict__ count) {
  const Grid& g = T.L.g;
  const int n = *count;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int gid = list[t], f = gid / 125, q = gid % 125;
    const int4 b = face_cell[f];
    const int i = fmod_pos(b.x - 2 + q % 5 - 1, g.n1m), j = fmod_pos(b.y - 2 + (q / 5) % 5 - 1, g.n1m),
              k = fmod_pos(b.z - 2 + q / 25 - 1, g.n3m);
    const size_t c0 = cidx(g, i, j, k);
    if (winner[c0] != f) continue;
    const double c = vofp[c0];
    const size_t ip = cidx(g, wrap(i + 1, g.n1m), j, k), jp = cidx(g, i, wrap(j + 1, g.n2m), k),
                 kp = cidx(g, i, j, wrap(k + 1, g.n3m));
    vofx[c0] = 0.5 * (vofp[cidx(g, wrap(i - 1, g.n1m), j, k)] + c);
    vofy[c0] = 0.5 * (vofp[cidx(g, i, wrap(j - 1, g.n2m), k)] + c);
    vofz[c0] = 0.5 * (vofp[cidx(g, i, j, wrap(k - 1, g.n3m))] + c);
    vofx[ip] = 0.5 * (c + vofp[ip]);
    vofy[jp] = 0.5 * (c + vofp[jp]);
    vofz[kp] = 0.5 * (c + vofp[kp]);
  }
}

constexpr int kBandBlocks = 152 * 24;
__global__ void band_kernel(TagArgs T, int pass, unsigned long long* __restrict__ sdf_bits, int* __restrict__ winner,
                            double* __restrict__ vofp, double* __restrict__ dist_buf, const int4* __restrict__ face_cell,
                            const int* __restrict__ list, const int* __restrict__ count) {
  const int n = *count;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
    band_pair(T, pass, sdf_bits, winner, vofp, dist_buf, face_cell, list[t], t);
}


// initial full tagging: one thread per cell of the bounding box
__device__ bool ray_tri(const double C[3], const double Q[3], const double V0[3], const double V1[3],
                        const double V2[3], double ip[3]) {
  const double EPS = 1e-12;
  double dir[3] = {Q[0] - C[0], Q[1] - C[1], Q[2] - C[2]};
  double e1[3], e2[3], h[3], s[3], q[3];
  for (int d = 0; d < 3; ++d) { e1[d] = V1[d] - V0[d]; e2[d] = V2[d] - V0[d]; }
  h[0] = dir[1] * e2[2] - dir[2] * e2[1]; h[1] = dir[2] * e2[0] - dir[0] * e2[2]; h[2] = dir[0] * e2[1] - dir[1] * e2[0];
  double a = e1[0] * h[0] + e1[1] * h[1] + e1[2] * h[2];
  if (fabs(a) < EPS) return false;
  double f = 1.0 / a;
  for (int d = 0; d < 3; ++d) s[d] = C[d] - V0[d];
  double u = f * (s[0] * h[0] + s[1] * h[1] + s[2] * h[2]);
  if (u < 0.0 || u > 1.0) return false;
  q[0] = s[1] * e1[2] - s[2] * e1[1]; q[1] = s[2] * e1[0] - s[0] * e1[2]; q[2] = s[0] * e1[1] - s[1] * e1[0];
  double v = f * (dir[0] * q[0] + dir[1] * q[1] + dir[2] * q[2]);
  if (v < 0.0 || u + v > 1.0) return false;
  double t = f * (e2[0] * q[0] + e2[1] * q[1] + e2[2] * q[2]);
  if (t < 0.0 || t > 1.0) return false;
  for (int d = 0; d < 3; ++d) ip[d] = C[d] + t * dir[d];
  return true;
}

// pass A: ray parity / interface rule per bounding-box cell (rayTagQ_pencil,
// pencil_rayTag.f90:381-460) -> tmp[gid]
__global__ void initial_tag_kernel(TagArgs T, int bx0, int by0, int bz0, int nbx, int nby, int nbz,
                                   double* __restrict__ tmp) {
  long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long long)nbx * nby * nbz) return;
  const LagArgs& A = T.L;
  const Grid& g = A.g;
  int i = bx0 + (int)(gid % nbx), j = by0 + (int)((gid / nbx) % nby), kk = bz0 + (int)(gid / ((long long)nbx * nby));
  double Q[3] = {coord(A, 0, 1, i), coord(A, 1, 1, j), coord(A, 2, 1, kk)};
  double C[3] = {-g.xlen * 10.0, Q[1], Q[2]};
  double ymin = Q[1] - 0.5 / g.dx2, ymax = Q[1] + 0.5 / g.dx2, zmin = Q[2] - 0.5 / g.dx3, zmax = Q[2] + 0.5 / g.dx3;
  double xmin = Q[0] - 0.5 / g.dx1, xmax = Q[0] + 0.5 / g.dx1;
  int count = 0;
  double vof = -1.0;
  for (int f = 0; f < A.nf; ++f) {
    if (T.ghost[f]) continue;
    double V0[3], V1[3], V2[3];
    tri_verts(T, f, V0, V1, V2);
    double ylo = fmin(V0[1], fmin(V1[1], V2[1])), yhi = fmax(V0[1], fmax(V1[1], V2[1]));
    double zlo = fmin(V0[2], fmin(V1[2], V2[2])), zhi = fmax(V0[2], fmax(V1[2], V2[2]));
    if (yhi < ymin || ylo > ymax || zhi < zmin || zlo > zmax) continue;
    double xlo = fmin(V0[0], fmin(V1[0], V2[0])), xhi = fmax(V0[0], fmax(V1[0], V2[0]));
    if (!(xhi < xmin || xlo > xmax)) { vof = 0.5; break; }
    double ip[3];
    if (ray_tri(C, Q, V0, V1, V2, ip)) {
      if (ip[0] >= xmin && ip[0] <= xmax && ip[1] >= ymin && ip[1] <= ymax && ip[2] >= zmin && ip[2] <= zmax) {
        vof = 0.5;
        break;
      }
      ++count;
    }
  }
  if (vof < 0) vof = (count % 2 == 0) ? 1.0 : 0.0;
  tmp[gid] = vof;
}

// reference loop order (i outermost, kk innermost) as an integer key
__device__ __forceinline__ int box_order(long long gid, int nbx, int nby, int nbz) {
  int io = (int)(gid % nbx), jo = (int)((gid / nbx) % nby), ko = (int)(gid / ((long long)nbx * nby));
  return (io * nby + jo) * nbz + ko;
}

// pass B/C: a cell reached through several periodic images keeps the first
// value below 1 in loop order (pencil_rayTag.f90:298-302)
__global__ void initial_claim_kernel(Grid g, int bx0, int by0, int bz0, int nbx, int nby, int nbz,
                                     const double* __restrict__ tmp, int* __restrict__ claim, double* __restrict__ vofp,
                                     int pass) {
  long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long long)nbx * nby * nbz) return;
  double v = tmp[gid];
  if (!(v < 1.0)) return;
  int i = bx0 + (int)(gid % nbx), j = by0 + (int)((gid / nbx) % nby), kk = bz0 + (int)(gid / ((long long)nbx * nby));
  size_t c0 = cidx(g, fmod_pos(i - 1, g.n1m), fmod_pos(j - 1, g.n2m), fmod_pos(kk - 1, g.n3m));
  int key = box_order(gid, nbx, nby, nbz);
  if (pass == 0) atomicMin(&claim[c0], key);
  else if (claim[c0] == key) vofp[c0] = v;
}

__global__ void fill_kernel(Grid g, double* __restrict__ a, double v) {
  size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < g.cells) a[t] = v;
}

// ---------------------------------------------------------------------
// per-context Lagrangian state
// ---------------------------------------------------------------------
struct LagState {
  Ctx* c = nullptr;
  int* adj_off = nullptr;
  int* adj_face = nullptr;
  int adj_nf = -1, adj_nv = -1;
  double* face_part = nullptr;
  double* geom_out = nullptr;   // device [Surface, Volume1, Vol, Cx, Cy, Cz, InertTensor(9)]
  unsigned* geom_ticket = nullptr;   // blocks of face_geom_kernel done (0 between launches)
  double* loads_ev = nullptr;   // structural loads: per 32-face group 13 x 32 evaluations, then 12 group sums
  unsigned* loads_ticket = nullptr;   // groups done, then warps done per group (0 between launches)
  int* rm_flag = nullptr;       // remesh trigger (device)
  double* mean3 = nullptr;
  int* winner = nullptr;
  double* dist_buf = nullptr;
  // narrow-band culling: per cell an FP32 upper bound of the nearest face
  // distance (float bits), per face its FP32 centroid and circumradius and
  // the base cell of its 5^3 band, FP32 cell-centre coordinates
  unsigned* band_ub = nullptr;
  int* band_list = nullptr;      // (face, cell) pairs that survive the bound, and their count
  int* band_count = nullptr;
  BandFace* band_face = nullptr;
  int4* face_cell = nullptr;
  float* cm32 = nullptr;
  // merged scatter plan
  unsigned* bitmap = nullptr;                    // one bit per key, zero between builds
  int *wpre = nullptr, *tsum = nullptr;          // run number at each marked word, marked keys per tile of words
  int plan_words = 0;
  int2* slot = nullptr;                          // per entry: its run and its slot in it
  int *run_key = nullptr, *run_cnt = nullptr, *run_off = nullptr;
  int* nruns = nullptr;                          // [0] runs, [1] storage cursor, [2] long runs
  int* long_run = nullptr;                       // the long runs, in no order
  int *entry = nullptr, *src = nullptr;          // entries by run, then in triangle order
  int* saved = nullptr;                          // 7 ints per face: pind(1:6), ghost
  int* dirty = nullptr;
  double* segval = nullptr;
  bool force_rebuild = true;
  bool weights_valid = false;                    // stationary cages: weights kept
};
static std::vector<LagState*> g_lag;

static LagState* lag_of(Ctx* c) {
  for (auto* s : g_lag)
    if (s->c == c) return s;
  LagState* s = new LagState();
  s->c = c;
  g_lag.push_back(s);
  return s;
}

// The mesh changed on the host side: the scatter plan is rebuilt from
// scratch and the MLS weights recomputed.  The step graph stays valid (the
// rebuild is requested through pinned memory read at replay) unless the
// weights of a stationary body were being reused, which changes the launch
// sequence.
void lagr_invalidate(Ctx* c) {
  ++c->geom_gen;
  LagState* s = lag_of(c);
  s->force_rebuild = true;
  if (c->I(MIBM_I_STATIONARY) && s->weights_valid) ++c->lag_gen;
  s->weights_valid = false;
}

// Per step, while its parameter blocks are filled: a pending request to
// rebuild the scatter plan from scratch goes into substep 0's block, which
// the step reads on the device (so a step graph stays valid across uploads).
int lagr_take_plan_request(Ctx* c) {
  if (c->I(MIBM_I_IMLSFOR) != 1 || c->maxnf == 0) return 0;
  LagState* s = lag_of(c);
  int r = s->force_rebuild ? 1 : 0;
  s->force_rebuild = false;
  return r;
}

// the face/vertex/edge relations changed (a remesh or a host upload of the
// connectivity): rebuild the vertex->face lists too
void lagr_topology_changed(Ctx* c) {
  lagr_invalidate(c);
  lag_of(c)->adj_nf = -1;
}

static bool ensure_adjacency(Ctx* c) {
  LagState* s = lag_of(c);
  if (s->adj_off && s->adj_nf == c->maxnf && s->adj_nv == c->maxnv) return true;
  std::vector<int> vof(3 * (size_t)c->maxnf), ghost(c->maxnf);
  cudaMemcpy(vof.data(), c->dm[MIBM_M_VERT_OF_FACE], vof.size() * 4, cudaMemcpyDeviceToHost);
  cudaMemcpy(ghost.data(), c->dm[MIBM_M_GHOST_FACE], ghost.size() * 4, cudaMemcpyDeviceToHost);
  std::vector<int> cnt(c->maxnv + 1, 0);
  for (int f = 0; f < c->maxnf; ++f) {
    if (ghost[f]) continue;
    for (int q = 0; q < 3; ++q) {
      int v = vof[3 * f + q] - 1;
      if (v < 0 || v >= c->maxnv) { fail(c, MIBM_EINVAL, "vert_of_face out of range"); return false; }
      cnt[v + 1]++;
    }
  }
  for (int v = 0; v < c->maxnv; ++v) cnt[v + 1] += cnt[v];
  std::vector<int> face(cnt[c->maxnv]), fill(cnt.begin(), cnt.end() - 1);
  for (int f = 0; f < c->maxnf; ++f) {      // ascending face order per vertex
    if (ghost[f]) continue;
    for (int q = 0; q < 3; ++q) face[fill[vof[3 * f + q] - 1]++] = f;
  }
  cudaFree(s->adj_off); cudaFree(s->adj_face);
  if (!cuda_ok(c, cudaMalloc(&s->adj_off, cnt.size() * 4), "adj")) return false;
  if (!cuda_ok(c, cudaMalloc(&s->adj_face, std::max<size_t>(1, face.size()) * 4), "adj")) return false;
  cudaMemcpy(s->adj_off, cnt.data(), cnt.size() * 4, cudaMemcpyHostToDevice);
  cudaMemcpy(s->adj_face, face.data(), face.size() * 4, cudaMemcpyHostToDevice);
  s->adj_nf = c->maxnf; s->adj_nv = c->maxnv;
  return true;
}

static bool ensure_lag_buffers(Ctx* c) {
  LagState* s = lag_of(c);
  if (!s->face_part) {
    if (!cuda_ok(c, cudaMalloc(&s->face_part, sizeof(double) * 12 * std::max(1, c->maxnf)), "lag")) return false;
    if (!cuda_ok(c, cudaMalloc(&s->geom_out, sizeof(double) * 16), "lag")) return false;
    if (!cuda_ok(c, cudaMalloc(&s->geom_ticket, sizeof(unsigned)), "lag")) return false;
    cudaMemsetAsync(s->geom_out, 0, sizeof(double) * 16, c->stream);
    cudaMemsetAsync(s->geom_ticket, 0, sizeof(unsigned), c->stream);
    // [0..3) FP64 mean force, [4..6) the same rounded to FP32 (3 floats)
    // [0..2] the means, [4..5] their FP32 copies, [7] seg_mean_kernel's ticket
    if (!cuda_ok(c, cudaMalloc(&s->mean3, sizeof(double) * 8), "lag")) return false;
    cudaMemsetAsync(s->mean3, 0, sizeof(double) * 8, c->stream);
  }
  if (!c->tri_coef)
    if (!cuda_ok(c, cudaMalloc(&c->tri_coef, sizeof(double) * 4 * std::max(1, c->maxnf)), "lag")) return false;
  if (!s->bitmap) {
    const size_t n = 108 * (size_t)std::max(1, c->maxnf);
    // runs: at most one per entry and one per key
    const size_t runs = std::min(n, 4 * c->g.cells);
    s->plan_words = (int)(div_up(4 * c->g.cells, 128) * 4);
    bool ok = cuda_ok(c, cudaMalloc(&s->bitmap, sizeof(unsigned) * (size_t)s->plan_words), "plan") &&
              cuda_ok(c, cudaMalloc(&s->wpre, sizeof(int) * (size_t)s->plan_words), "plan") &&
              cuda_ok(c, cudaMalloc(&s->tsum, sizeof(int) * (size_t)div_up(s->plan_words, kPlanTile)), "plan") &&
              cuda_ok(c, cudaMalloc(&s->slot, sizeof(int2) * n), "plan") &&
              cuda_ok(c, cudaMalloc(&s->run_key, sizeof(int) * runs), "plan") &&
              cuda_ok(c, cudaMalloc(&s->run_cnt, sizeof(int) * runs), "plan") &&
              cuda_ok(c, cudaMalloc(&s->run_off, sizeof(int) * runs), "plan") &&
              cuda_ok(c, cudaMalloc(&s->nruns, sizeof(int) * 3), "plan") &&
              cuda_ok(c, cudaMalloc(&s->long_run, sizeof(int) * (n / kLongRun + 1)), "plan") &&
              cuda_ok(c, cudaMalloc(&s->entry, sizeof(int) * n), "plan") &&
              cuda_ok(c, cudaMalloc(&s->src, sizeof(int) * n), "plan") &&
              cuda_ok(c, cudaMalloc(&s->saved, sizeof(int) * 7 * (size_t)std::max(1, c->maxnf)), "plan") &&
              cuda_ok(c, cudaMalloc(&s->dirty, sizeof(int)), "plan") &&
              cuda_ok(c, cudaMalloc(&s->segval, sizeof(double) * runs), "plan");
    if (!ok) return false;
    cudaMemsetAsync(s->bitmap, 0, sizeof(unsigned) * (size_t)s->plan_words, c->stream);
    cudaMemsetAsync(s->saved, 0xff, sizeof(int) * 7 * (size_t)std::max(1, c->maxnf), c->stream);
    cudaMemsetAsync(s->nruns, 0, sizeof(int) * 3, c->stream);
    cudaMemsetAsync(s->dirty, 0, sizeof(int), c->stream);
  }
  return true;
}

// Flags raised by device kernels (singular MLS matrix).  In the fused step
// they are read once at the end of the step.
static bool check_flag(Ctx* c, const char* what) {
  cudaMemcpyAsync(c->hflag, c->dflag, 4, cudaMemcpyDeviceToHost, c->stream);
  if (!cuda_ok(c, cudaStreamSynchronize(c->stream), what)) return false;
  if (c->hflag[0]) {
    fail(c, MIBM_ENUMERIC, std::string(what) + ((c->hflag[0] & 2) ? ": singular inertia tensor (dgetrf info /= 0)"
                                                                  : ": singular MLS moment matrix (dgetrf info /= 0)"));
    cudaMemsetAsync(c->dflag, 0, 4, c->stream);
    return false;
  }
  return true;
}

// Host check of the connectivity every Lagrangian kernel dereferences
// (vertex indices in 1..maxnv); also builds the vertex->face lists.
bool validate_mesh(Ctx* c) {
  LagState* s = lag_of(c);
  s->adj_nf = -1;   // force a rebuild from the current device copy
  return ensure_adjacency(c);
}

// (Re)build the merged scatter plan when the cage centres changed.
// checked: the geometry pass of the substep before compared them already
// (FaceNext; no parameter block carries a request there).
// dp: inside the fused step, the substep's parameter block, whose
// force_plan carries a rebuild request (lagr_take_plan_request); nullptr
// (drop-ins): the pending request is applied now.  A request raised inside
// a step (a remesh, which runs without a step graph) is applied now too.
static void update_plan(Ctx* c, const StepParams* dp, bool checked) {
  LagState* s = lag_of(c);
  const int nf = c->maxnf, words = s->plan_words;
  const unsigned eb = div_up(108 * (size_t)nf, 256), tiles = div_up(words, kPlanTile);
  const int* pind = M<int>(c, MIBM_M_PIND);
  const int* ghost = M<int>(c, MIBM_M_GHOST_FACE);
  if (s->force_rebuild) cudaMemsetAsync(s->dirty, 1, sizeof(int), c->stream);   // non-zero: dirty
  s->force_rebuild = false;
  if (!checked) {
    MIBM_PROF(c, "plan_check");
    plan_check_kernel<<<div_up(nf, 256), 256, 0, c->stream>>>(nf, pind, ghost, s->saved, s->dirty, dp);
    ++c->launches;
  }
  { MIBM_PROF(c, "plan_mark");
    plan_mark_kernel<<<eb, 256, 0, c->stream>>>(c->g, nf, pind, ghost, s->dirty, s->bitmap); }
  { MIBM_PROF(c, "plan_runs");
    plan_count_kernel<<<tiles, 256, 0, c->stream>>>(s->bitmap, words, s->dirty, s->tsum);
    plan_runs_kernel<<<tiles, 256, 0, c->stream>>>(s->bitmap, words, s->dirty, s->tsum, s->wpre, s->run_key,
                                                   s->run_cnt, s->nruns); }
  { MIBM_PROF(c, "plan_slot");
    plan_slot_kernel<<<eb, 256, 0, c->stream>>>(c->g, nf, pind, ghost, s->dirty, s->bitmap, s->wpre, s->run_cnt,
                                                s->slot); }
  { MIBM_PROF(c, "plan_store");
    plan_store_kernel<<<std::min<unsigned>(eb, 304), 256, 0, c->stream>>>(s->dirty, s->run_cnt, s->run_off, s->nruns,
                                                                              s->long_run); }
  { MIBM_PROF(c, "plan_place");
    plan_place_kernel<<<eb, 256, 0, c->stream>>>(nf, pind, ghost, s->dirty, s->slot, s->run_off, s->entry, s->saved); }
  { MIBM_PROF(c, "plan_order");
    plan_order_kernel<<<std::min<unsigned>(eb, kScatterBlocks), 256, 0, c->stream>>>(
        nf, s->dirty, s->nruns, s->run_key, s->run_off, s->run_cnt, s->long_run, s->entry, s->src, s->bitmap); }
  cudaMemsetAsync(s->dirty, 0, sizeof(int), c->stream);
  c->launches += 7;
  MIBM_LAUNCH_CHECK(c, "scatter plan");
}

// m32: base of the FP32 mirrors (u, v, w, T at 0, cells, 2 cells, 3 cells)
// that the scatter keeps equal to the forced fields, or null
static ScatterOut scatter_out(Ctx* c, bool into_fields, float* m32) {
  ScatterOut O;
  for (int q = 0; q < 4; ++q) O.m32[q] = (into_fields && m32) ? m32 + (size_t)q * c->g.cells : nullptr;
  static const int fo[4] = {MIBM_F_FORXC, MIBM_F_FORYC, MIBM_F_FORZC, MIBM_F_FORTEMP};
  static const int fq[4] = {MIBM_F_VX, MIBM_F_VY, MIBM_F_VZ, MIBM_F_TEMP};
  for (int q = 0; q < 4; ++q) O.f[q] = c->df[into_fields ? fq[q] : fo[q]];
  O.phi[0] = M<double>(c, MIBM_M_PTXAB_Q1); O.phi[1] = M<double>(c, MIBM_M_PTXAB_Q2);
  O.phi[2] = M<double>(c, MIBM_M_PTXAB_Q3); O.phi[3] = M<double>(c, MIBM_M_PTXAB_TEMP);
  return O;
}

// An SM divides its memory between L1 and shared memory for the kernel that finds
// it idle, and a kernel that wants more shared memory waits for it to be idle
// again.  The long kernels of the side chain use little shared memory and run beside
// kernels of the FP64 form's main chain that use much (the explicit terms started only
// when the MLS weights ended, up to 25 us after their last input; the line solves
// beside the structural loads), so in that form they, and the scatter and mean force ahead of
// the projection, ask for the others' division:
// moving body at 128^3, two steps, 5270 -> 4982 us, 48^3, four steps, 2769 -> 2739.
// The precision form's main chain lives on L1 and keeps the default
// (128^3 3949 us, with this 4071).
template <typename... P, typename... A>
static void launch_beside(Ctx* c, void (*kern)(P...), unsigned grid, unsigned block, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = c->stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  at.val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
  cfg.attrs = &at;
  cfg.numAttrs = c->precision == 0 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

static void force_coefficients(Ctx* c) {
  ForceArgs F;
  F.q[0] = c->df[MIBM_F_VX]; F.q[1] = c->df[MIBM_F_VY]; F.q[2] = c->df[MIBM_F_VZ]; F.q[3] = c->df[MIBM_F_TEMP];
  F.ptx[0] = M<double>(c, MIBM_M_PTXAB_Q1); F.ptx[1] = M<double>(c, MIBM_M_PTXAB_Q2);
  F.ptx[2] = M<double>(c, MIBM_M_PTXAB_Q3); F.ptx[3] = M<double>(c, MIBM_M_PTXAB_TEMP);
  F.vel_tri = M<double>(c, MIBM_M_VEL_TRI); F.cfac = M<double>(c, MIBM_M_CFAC);
  F.pind = M<int>(c, MIBM_M_PIND); F.ghost = M<int>(c, MIBM_M_GHOST_FACE);
  { MIBM_PROF(c, "force_coef");
    launch_beside(c, force_coef_kernel, div_up(4 * (size_t)c->maxnf, kLagBlock), kLagBlock, c->g, c->maxnf, F, c->S(MIBM_S_TMELT),
                                                                                  c->tri_coef); }
  ++c->launches;
}

static PlanRuns plan_runs(const LagState* s) { return PlanRuns{s->nruns, s->run_key, s->run_off, s->run_cnt, s->src}; }

static void scatter(Ctx* c, bool into_fields, int lo, int hi, bool record, float* m32 = nullptr) {
  LagState* s = lag_of(c);
  { MIBM_PROF(c, "scatter_apply");
    launch_beside(c, scatter_apply_kernel,
                  (unsigned)std::min<size_t>(kScatterBlocks, div_up(108 * (size_t)c->maxnf, 256)), 256, c->maxnf,
                  c->g.cells, plan_runs(s), c->tri_coef, scatter_out(c, into_fields, m32), lo, hi,
                  record ? s->segval : nullptr); }
  ++c->launches;
}

// ---------------------------------------------------------------------
// entry points
// ---------------------------------------------------------------------
void lagr_find_centroid_indices(Ctx* c) {
  if (c->maxnf == 0) return;
  { MIBM_PROF(c, "centroid_idx");
    centroid_idx_kernel<<<div_up(c->maxnf, kLagBlock), kLagBlock, 0, c->stream>>>(
        lag_args(c), M<double>(c, MIBM_M_TRI_BAR), M<int>(c, MIBM_M_GHOST_FACE), M<int>(c, MIBM_M_PIND)); }
  ++c->launches;
  MIBM_LAUNCH_CHECK(c, "findCentroidIndices");
}

static void mls_weight_launch(Ctx* c) {
  if (c->precision == 1) {
    { MIBM_PROF(c, "mls_weight_sep");
      mls_weight_sep_kernel<<<div_up(4 * (size_t)c->maxnf, kLagBlock), kLagBlock, 0, c->stream>>>(
          lag_args(c), M<double>(c, MIBM_M_TRI_BAR), M<int>(c, MIBM_M_GHOST_FACE), M<int>(c, MIBM_M_PIND),
          M<double>(c, MIBM_M_PTXAB_Q1), M<double>(c, MIBM_M_PTXAB_Q2), M<double>(c, MIBM_M_PTXAB_Q3),
          M<double>(c, MIBM_M_PTXAB_TEMP), c->dflag); }
    ++c->launches;
    return;
  }
  { MIBM_PROF(c, "mls_weight");
    launch_beside(c, mls_weight_kernel, div_up(4 * (size_t)c->maxnf, kLagBlock), kLagBlock,
        lag_args(c), M<double>(c, MIBM_M_TRI_BAR), M<int>(c, MIBM_M_GHOST_FACE), M<int>(c, MIBM_M_PIND),
        M<double>(c, MIBM_M_PTXAB_Q1), M<double>(c, MIBM_M_PTXAB_Q2), M<double>(c, MIBM_M_PTXAB_Q3),
        M<double>(c, MIBM_M_PTXAB_TEMP), c->dflag); }
  ++c->launches;
}

void lagr_mls_weight(Ctx* c) {
  if (c->maxnf == 0) return;
  mls_weight_launch(c);
  if (MIBM_LAUNCH_CHECK(c, "mlsWeight")) check_flag(c, "mlsWeight");
}

// mlsforce_ drop-in: spreads into the dense for_* fields
void lagr_mls_force(Ctx* c, const StepParams*, bool) {
  if (c->maxnf == 0) return;
  if (!ensure_lag_buffers(c)) return;
  force_coefficients(c);
  update_plan(c, nullptr, false);
  scatter(c, false, 0, 4, false);
  MIBM_LAUNCH_CHECK(c, "mlsForce");
}

void lagr_velforce(Ctx* c) {
  if (!ensure_lag_buffers(c)) return;
  LagState* s = lag_of(c);
  const double ncell = (double)c->g.n1m * (double)c->g.n2m * (double)c->g.n3m;
  { MIBM_PROF(c, "field_mean");
    field_mean_kernel<<<std::min(kFieldMeanBlocks, c->g.n2m * c->g.n3m), 256, 0, c->stream>>>(c->g, c->df[MIBM_F_FORXC], c->df[MIBM_F_FORYC],
                                                               c->df[MIBM_F_FORZC], c->red + kRedPart, ncell,
                                                               s->mean3); }
  c->launches += 1;
  k_velforce_apply(c, s->mean3);
}

void lagr_tempforce(Ctx* c) { k_tempforce_apply(c); }

void lagr_find_probe_indices(Ctx* c) {
  if (c->maxnf == 0) return;
  { MIBM_PROF(c, "probe_idx");
    probe_idx_kernel<<<div_up(c->maxnf, kLagBlock), kLagBlock, 0, c->stream>>>(
        lag_args(c), M<double>(c, MIBM_M_TRI_BAR), M<double>(c, MIBM_M_TRI_NOR), M<int>(c, MIBM_M_GHOST_FACE),
        c->S(MIBM_S_H_EULERIAN), M<int>(c, MIBM_M_PIND)); }
  ++c->launches;
  MIBM_LAUNCH_CHECK(c, "findProbeIndices");
}

// Which MLS construction evaluates gradients and values at the probes.  The
// reference's (absolute coordinates, condition numbers 1e7-1e8) returns the
// oracle's bits only when its inputs are the oracle's bits: the plain form
// uses it for a body that does not move (fixed, melting or not: the
// geometry follows the Stefan update, which is bit-exact) and for the
// drop-in calls.  Once a body moves, its position carries the fluid solver's
// round-off from the first step on, and the reference's construction turns
// any last-bit difference of the geometry into ~1e-9 noise (its conditioning
// times the rounding unit); there, and in the precision form, the separable
// construction is used, which has none of that noise and agrees with the
// reference's to it, at a quarter of its FP64 operations.
static bool literal_mls(Ctx* c) { return c->precision == 0 && c->I(MIBM_I_IMLSSTR) != 1; }

// fused: without the probe indices in pind, and without the face-to-vertex
// sums (melt_vert_kernel takes them)
static void heat_flux_launch(Ctx* c, bool fused) {
  LagState* s = lag_of(c);
  const int* pind = fused ? nullptr : M<int>(c, MIBM_M_PIND);
  { MIBM_PROF(c, "heat_flux");
    if (literal_mls(c) && c->maxnf <= kHf4Faces)
      launch_beside(c, heat_flux_lit4_kernel, div_up(2 * (size_t)c->maxnf, kHf4Probes), 128,
          lag_args(c), c->df[MIBM_F_TEMP], M<double>(c, MIBM_M_TRI_BAR), M<double>(c, MIBM_M_TRI_NOR),
          M<int>(c, MIBM_M_GHOST_FACE), pind, c->S(MIBM_S_H_EULERIAN), c->S(MIBM_S_PEC),
          M<double>(c, MIBM_M_QW_O), M<double>(c, MIBM_M_QW_I), c->dflag);
    else if (literal_mls(c))
      launch_beside(c, heat_flux_lit_kernel, div_up(2 * (size_t)c->maxnf, kHfProbes), 4 * kHfProbes,
          lag_args(c), c->df[MIBM_F_TEMP], M<double>(c, MIBM_M_TRI_BAR), M<double>(c, MIBM_M_TRI_NOR),
          M<int>(c, MIBM_M_GHOST_FACE), pind, c->S(MIBM_S_H_EULERIAN), c->S(MIBM_S_PEC),
          M<double>(c, MIBM_M_QW_O), M<double>(c, MIBM_M_QW_I), c->dflag);
    else
      launch_beside(c, heat_flux_sep_kernel, div_up(2 * (size_t)c->maxnf, kLagBlock), kLagBlock,
          lag_args(c), c->df[MIBM_F_TEMP], M<double>(c, MIBM_M_TRI_BAR), M<double>(c, MIBM_M_TRI_NOR),
          M<int>(c, MIBM_M_GHOST_FACE), pind, c->S(MIBM_S_H_EULERIAN), c->S(MIBM_S_PEC),
          M<double>(c, MIBM_M_QW_O), M<double>(c, MIBM_M_QW_I), c->dflag); }
  ++c->launches;
  if (fused) return;
  { MIBM_PROF(c, "face_to_vert");
    face_to_vert_kernel<<<div_up(c->maxnv, kLagBlock), kLagBlock, 0, c->stream>>>(
        c->maxnv, s->adj_off, s->adj_face, M<double>(c, MIBM_M_SUR), M<double>(c, MIBM_M_AVERT),
        M<double>(c, MIBM_M_QW_O), M<double>(c, MIBM_M_QW_I), M<double>(c, MIBM_M_QW_OVERT),
        M<double>(c, MIBM_M_QW_IVERT)); }
  ++c->launches;
}

static void melt_vert_launch(Ctx* c, const StepParams* dp) {
  LagState* s = lag_of(c);
  { MIBM_PROF(c, "melt_vert");
    melt_vert_kernel<<<div_up(c->maxnv, kLagBlock), kLagBlock, 0, c->stream>>>(
        c->maxnv, s->adj_off, s->adj_face, M<double>(c, MIBM_M_SUR), M<double>(c, MIBM_M_AVERT),
        M<double>(c, MIBM_M_QW_O), M<double>(c, MIBM_M_QW_I), M<double>(c, MIBM_M_QW_OVERT),
        M<double>(c, MIBM_M_QW_IVERT), M<int>(c, MIBM_M_GHOST_VERT), M<double>(c, MIBM_M_VERT_NOR),
        c->S(MIBM_S_CPLIQUID) / c->S(MIBM_S_LATHEAT), dp, M<double>(c, MIBM_M_VMELT), M<double>(c, MIBM_M_VMELT_M1),
        M<double>(c, MIBM_M_XYZV)); }
  ++c->launches;
  s->weights_valid = false;
}

void lagr_heat_flux(Ctx* c) {
  if (c->maxnf == 0) return;
  if (!ensure_adjacency(c)) return;
  heat_flux_launch(c, false);
  if (MIBM_LAUNCH_CHECK(c, "mls_heatFlux")) check_flag(c, "mls_heatFlux");
}

void lagr_stefan(Ctx* c, const StepParams* dp) {
  if (c->maxnv == 0) return;
  { MIBM_PROF(c, "stefan");
    stefan_kernel<<<div_up(c->maxnv, kLagBlock), kLagBlock, 0, c->stream>>>(
        c->maxnv, M<int>(c, MIBM_M_GHOST_VERT), M<double>(c, MIBM_M_VERT_NOR), M<double>(c, MIBM_M_QW_OVERT),
        M<double>(c, MIBM_M_QW_IVERT), c->S(MIBM_S_CPLIQUID) / c->S(MIBM_S_LATHEAT), dp, M<double>(c, MIBM_M_VMELT),
        M<double>(c, MIBM_M_VMELT_M1), M<double>(c, MIBM_M_XYZV)); }
  ++c->launches;
  MIBM_LAUNCH_CHECK(c, "stefan");
  lag_of(c)->weights_valid = false;
}

// Geometry refresh (particle.f90:165-193): kernels only; the scalars stay
// in the device buffer until geometry_to_host.  body_only: the pass before
// the Newton-Euler update (particle.f90:108-117: centroids, normals,
// volume, centre of mass and inertia tensor of the melted body); it also
// rewrites `sur`, which nothing reads before the full refresh recomputes it.
static FaceNext face_next(Ctx* c) {
  FaceNext N{};
  N.g = c->g;
  N.nv = c->maxnv;
  N.h = c->S(MIBM_S_H_EULERIAN);
  N.celvol = c->S(MIBM_S_CELVOL);
  return N;
}

static void vert_geom_launch(Ctx* c) {
  LagState* s = lag_of(c);
  { MIBM_PROF(c, "vert_geom");
    vert_geom_kernel<<<div_up(c->maxnv, kLagBlock), kLagBlock, 0, c->stream>>>(
        c->maxnv, s->adj_off, s->adj_face, M<int>(c, MIBM_M_GHOST_VERT), M<double>(c, MIBM_M_SUR),
        M<double>(c, MIBM_M_TRI_NOR), M<double>(c, MIBM_M_AVERT), M<double>(c, MIBM_M_VERT_NOR)); }
  ++c->launches;
}

static void edges_launch(Ctx* c) {   // calculate_eLengths, calculate_skewness (particle.f90:173-176)
  if (c->maxne <= 0) return;
  MIBM_PROF(c, "edges");
  elength_kernel<<<div_up(c->maxne, kLagBlock), kLagBlock, 0, c->stream>>>(
      c->maxne, M<int>(c, MIBM_M_VERT_OF_EDGE), M<int>(c, MIBM_M_GHOST_EDGE), M<double>(c, MIBM_M_XYZV), 0.0,
      M<double>(c, MIBM_M_ELENGTHS), nullptr);
  skewness_kernel<<<div_up(c->maxnf, kLagBlock), kLagBlock, 0, c->stream>>>(
      c->maxnf, M<int>(c, MIBM_M_EDGE_OF_FACE), M<int>(c, MIBM_M_GHOST_FACE), M<double>(c, MIBM_M_ELENGTHS),
      M<double>(c, MIBM_M_SUR), M<double>(c, MIBM_M_SKEWNESS));
  c->launches += 2;
}

static void face_geom_launch(Ctx* c, const FaceNext& N, bool sum) {
  LagState* s = lag_of(c);
  { MIBM_PROF(c, "face_geom");
    auto kern = sum ? face_geom_kernel<true> : face_geom_kernel<false>;
    kern<<<div_up(c->maxnf, kGeomBlock), kGeomBlock, 0, c->stream>>>(
        c->maxnf, M<int>(c, MIBM_M_VERT_OF_FACE), M<int>(c, MIBM_M_GHOST_FACE), M<double>(c, MIBM_M_XYZV),
        M<double>(c, MIBM_M_SUR), M<double>(c, MIBM_M_TRI_NOR), M<double>(c, MIBM_M_TRI_BAR), s->face_part,
        s->geom_ticket, c->S(MIBM_S_DENS_RATIO), s->geom_out, N); }
  ++c->launches;
}

static void geom_sum_launch(Ctx* c) {
  LagState* s = lag_of(c);
  { MIBM_PROF(c, "geom_sum");
    geom_sum_kernel<<<1, kGeomBlock, 0, c->stream>>>(s->face_part, (int)div_up(c->maxnf, kGeomBlock),
                                                     c->S(MIBM_S_DENS_RATIO), s->geom_out); }
  ++c->launches;
}

static void geometry_launch(Ctx* c, bool imelt, bool body_only = false) {
  FaceNext N = face_next(c);
  if (imelt && !body_only) N.cfac = M<double>(c, MIBM_M_CFAC);
  face_geom_launch(c, N, true);
  if (body_only) return;
  vert_geom_launch(c);
  edges_launch(c);
}

// Surface, Volume and centre of mass to the registered host scalars
// (calc_rigidBody_params writes Volume last, RigidAuxRoutines.f90:738).
void lagr_geometry_to_host(Ctx* c) {
  if (c->maxnf == 0) return;
  LagState* s = lag_of(c);
  if (!s->geom_out) return;
  cudaMemcpyAsync(c->red_host, s->geom_out, sizeof(double) * 15, cudaMemcpyDeviceToHost, c->stream);
  if (!cuda_ok(c, cudaStreamSynchronize(c->stream), "geometry")) return;
  *c->hs[MIBM_S_SURFACE] = c->red_host[0];
  *c->hs[MIBM_S_VOLUME] = c->red_host[2];
  for (int d = 0; d < 3; ++d) c->hs[MIBM_S_POS_CM][d] = c->red_host[3 + d];
  for (int q = 0; q < 9; ++q) c->hs[MIBM_S_INERT_TENSOR][q] = c->red_host[6 + q];
}

// literal: the reference's MLS construction (the drop-in mls_structloads_
// of the plain form); the fused step of a moving body uses the separable one
// (see literal_mls).
static void struct_loads_launch(Ctx* c, const StepParams* dp, bool literal) {
  LagState* s = lag_of(c);
  const int nb = (int)div_up(std::max(1, c->maxnf), kLoadFaces);   // groups of 32 faces
  if (!s->loads_ev) {
    if (!cuda_ok(c, cudaMalloc(&s->loads_ev, sizeof(double) * (13 * kLoadFaces + 12) * (size_t)nb), "structLoads") ||
        !cuda_ok(c, cudaMalloc(&s->loads_ticket, sizeof(unsigned) * (size_t)(nb + 1)), "structLoads"))
      return;
    cudaMemsetAsync(s->loads_ticket, 0, sizeof(unsigned) * (size_t)(nb + 1), c->stream);
  }
  double h = c->S(MIBM_S_H_EULERIAN);
  { MIBM_PROF(c, "loads_face");
    auto kern = literal ? loads_face_kernel<true> : loads_face_kernel<false>;
    launch_beside(c, kern, 5 * nb, kLoadFaces,
        lag_args(c), c->df[MIBM_F_PR], c->df[MIBM_F_VX], c->df[MIBM_F_VY], c->df[MIBM_F_VZ],
        M<double>(c, MIBM_M_TRI_BAR), M<double>(c, MIBM_M_TRI_NOR), M<double>(c, MIBM_M_SUR),
        M<int>(c, MIBM_M_GHOST_FACE), dp, h, c->S(MIBM_S_REN), s->loads_ev, c->dflag, s->loads_ticket,
        c->drigid); }
  c->launches += 1;
}

// mls_structLoads on the device state; the loads stay in c->drigid.
void lagr_struct_loads(Ctx* c, const StepParams* dp) {
  if (c->maxnf == 0) return;
  if (!ensure_lag_buffers(c) || !rigid_ensure(c)) return;
  struct_loads_launch(c, dp, c->precision == 0);
  if (MIBM_LAUNCH_CHECK(c, "mls_structLoads")) check_flag(c, "mls_structLoads");
}

// particle.f90:108-129: geometry of the melted body, then update_part_pos
// (newton_euler, update_xyz) on the device.
static void motion_launch(Ctx* c, const StepParams* dp) {
  LagState* s = lag_of(c);
  geometry_launch(c, false, true);
  k_newton_euler(c, dp, s->geom_out);
  k_update_xyz(c, false);
}

void lagr_geometry_refresh(Ctx* c, bool imelt) {
  if (c->maxnf == 0) return;
  if (!ensure_adjacency(c) || !ensure_lag_buffers(c)) return;
  geometry_launch(c, imelt);
  lagr_geometry_to_host(c);
}

// the narrow band keeps its minimum distances as integer bit patterns in the
// signed-distance field's own memory (non-negative doubles order as their
// bits) and leaves the signed distances there: no copy pass
static unsigned long long* sdf_bits_of(Ctx* c) { return reinterpret_cast<unsigned long long*>(c->df[MIBM_F_SDF]); }

static bool ensure_band(Ctx* c) {
  LagState* s = lag_of(c);
  if (!s->winner && !cuda_ok(c, cudaMalloc(&s->winner, sizeof(int) * c->g.cells), "band")) return false;
  if (!s->dist_buf) {
    const LagArgs L = lag_args(c);
    bool ok = cuda_ok(c, cudaMalloc(&s->dist_buf, sizeof(double) * 125 * (size_t)c->maxnf), "band") &&
              cuda_ok(c, cudaMalloc(&s->band_ub, sizeof(unsigned) * c->g.cells), "band") &&
              cuda_ok(c, cudaMalloc(&s->band_list, sizeof(int) * 125 * (size_t)c->maxnf), "band") &&
              cuda_ok(c, cudaMalloc(&s->band_count, sizeof(int)), "band") &&
              cuda_ok(c, cudaMalloc(&s->band_face, sizeof(BandFace) * (size_t)c->maxnf), "band") &&
              cuda_ok(c, cudaMalloc(&s->face_cell, sizeof(int4) * (size_t)c->maxnf), "band") &&
              cuda_ok(c, cudaMalloc(&s->cm32, sizeof(float) * 3 * (size_t)L.clen), "band");
    if (!ok) return false;
    cm32_kernel<<<div_up(L.clen, 256), 256, 0, c->stream>>>(L, s->cm32);
    ++c->launches;
  }
  return true;
}

static void band_reset(Ctx* c) {
  LagState* s = lag_of(c);
  { MIBM_PROF(c, "sdf_reset");
    sdf_reset_kernel<<<div_up(c->g.cells, 256), 256, 0, c->stream>>>(c->g, sdf_bits_of(c), nullptr, s->band_ub); }
  cudaMemsetAsync(s->band_count, 0, sizeof(int), c->stream);
  ++c->launches;
}

// later: a tagging of the same step came before, so that vofx, vofy, vofz match
// vofp but around the cells this one writes.
// prepped (fused step): band_reset has run on this stream since the last
// tagging, and the geometry pass has left the faces' bounds (FaceNext)
static void tag_narrow_band(Ctx* c, bool prepped, bool later = false) {
  if (c->maxnf == 0 || !ensure_band(c)) return;
  LagState* s = lag_of(c);
  unsigned long long* const sdf_bits = sdf_bits_of(c);
  TagArgs T;
  T.L = lag_args(c);
  T.x = M<double>(c, MIBM_M_XYZV); T.vof = M<int>(c, MIBM_M_VERT_OF_FACE); T.ghost = M<int>(c, MIBM_M_GHOST_FACE);
  T.bar = M<double>(c, MIBM_M_TRI_BAR); T.nor = M<double>(c, MIBM_M_TRI_NOR);
  if (!prepped) band_reset(c);
  size_t nthr = (size_t)c->maxnf * 125;
  { MIBM_PROF(c, "band_bound");
    if (!prepped) band_prep_kernel<<<div_up(c->maxnf, kLagBlock), kLagBlock, 0, c->stream>>>(T, s->band_face, s->face_cell);
    band_ub_kernel<<<div_up(nthr, 128), 128, 0, c->stream>>>(T, s->band_face, s->face_cell, s->cm32, s->band_ub);
    band_select_kernel<<<div_up(nthr, 128), 128, 0, c->stream>>>(T, s->band_face, s->face_cell, s->cm32, s->band_ub,
                                                                  s->band_list, s->band_count); }
  for (int pass = 0; pass < 3; ++pass) {
    MIBM_PROF(c, "band");
    band_kernel<<<(unsigned)std::min<size_t>(div_up(nthr, kLagBlock), kBandBlocks), kLagBlock, 0, c->stream>>>(T, pass, sdf_bits, s->winner, c->df[MIBM_F_VOFP],
                                                           s->dist_buf, s->face_cell, s->band_list, s->band_count);
  }
  c->launches += prepped ? 5 : 6;
  if (later) {
    MIBM_PROF(c, "band_vof");
    band_vof_kernel<<<(unsigned)std::min<size_t>(div_up(nthr, kLagBlock), kBandBlocks), kLagBlock, 0, c->stream>>>(
        T, s->winner, c->df[MIBM_F_VOFP], c->df[MIBM_F_VOFX], c->df[MIBM_F_VOFY], c->df[MIBM_F_VOFZ],
        s->face_cell, s->band_list, s->band_count);
    ++c->launches;
  } else {
    k_interp_vof(c);
  }
  MIBM_LAUNCH_CHECK(c, "narrowBandTagging");
}

void lagr_tag_narrow_band(Ctx* c) { tag_narrow_band(c, false); }

void lagr_tag_initial(Ctx* c) {
  if (c->maxnf == 0) return;
  // bounding box (tagCells.f90:32-66, dx1 on all axes as in the reference)
  std::vector<double> x(3 * (size_t)c->maxnv);
  std::vector<int> gv(c->maxnv);
  cudaMemcpy(x.data(), c->dm[MIBM_M_XYZV], x.size() * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(gv.data(), c->dm[MIBM_M_GHOST_VERT], gv.size() * 4, cudaMemcpyDeviceToHost);
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int v = 0; v < c->maxnv; ++v) {
    if (gv[v]) continue;
    for (int d = 0; d < 3; ++d) { lo[d] = std::min(lo[d], x[3 * v + d]); hi[d] = std::max(hi[d], x[3 * v + d]); }
  }
  int b0[3], nb[3];
  for (int d = 0; d < 3; ++d) {
    b0[d] = (int)std::floor(lo[d] * c->g.dx1) + 1 - 2;
    int b1 = (int)std::floor(hi[d] * c->g.dx1) + 1 + 2;
    nb[d] = b1 - b0[d] + 1;
  }
  int vids[4] = {MIBM_F_VOFP, MIBM_F_VOFX, MIBM_F_VOFY, MIBM_F_VOFZ};
  for (int q = 0; q < 4; ++q) {
    fill_kernel<<<div_up(c->g.cells, 256), 256, 0, c->stream>>>(c->g, c->df[vids[q]], 1.0);
    ++c->launches;
  }
  TagArgs T;
  T.L = lag_args(c);
  T.x = M<double>(c, MIBM_M_XYZV); T.vof = M<int>(c, MIBM_M_VERT_OF_FACE); T.ghost = M<int>(c, MIBM_M_GHOST_FACE);
  T.bar = M<double>(c, MIBM_M_TRI_BAR); T.nor = M<double>(c, MIBM_M_TRI_NOR);
  size_t ncell = (size_t)nb[0] * nb[1] * nb[2];
  LagState* s = lag_of(c);
  if (!s->winner && !cuda_ok(c, cudaMalloc(&s->winner, sizeof(int) * c->g.cells), "band")) return;
  double* tmp = nullptr;
  if (!cuda_ok(c, cudaMalloc(&tmp, sizeof(double) * std::max<size_t>(1, ncell)), "initial tag")) return;
  sdf_reset_kernel<<<div_up(c->g.cells, 256), 256, 0, c->stream>>>(c->g, sdf_bits_of(c), s->winner, nullptr);
  initial_tag_kernel<<<div_up(ncell, 128), 128, 0, c->stream>>>(T, b0[0], b0[1], b0[2], nb[0], nb[1], nb[2], tmp);
  for (int pass = 0; pass < 2; ++pass)
    initial_claim_kernel<<<div_up(ncell, 256), 256, 0, c->stream>>>(c->g, b0[0], b0[1], b0[2], nb[0], nb[1], nb[2], tmp,
                                                                    s->winner, c->df[MIBM_F_VOFP], pass);
  c->launches += 4;
  bool ok = MIBM_LAUNCH_CHECK(c, "initial tag");
  cudaStreamSynchronize(c->stream);
  cudaFree(tmp);
  if (!ok) return;
  lagr_tag_narrow_band(c);
}

bool lagr_remesh_active(Ctx* c) {
  return c->I(MIBM_I_IREMESH) == 1 && c->I(MIBM_I_IMLSFOR) == 1 && c->maxnf > 0 && c->maxne > 0;
}

// particle.f90:119-160: the trigger (calculate_eLengths of the moved mesh)
// read on the host, and when it fires the hand-off to the host's remesher.
// Returns true if the mesh was remeshed.  Synchronises the stream.
static bool remesh_check(Ctx* c) {
  LagState* s = lag_of(c);
  if (!s->rm_flag && !cuda_ok(c, cudaMalloc(&s->rm_flag, sizeof(int)), "remesh")) return false;
  cudaMemsetAsync(s->rm_flag, 0, sizeof(int), c->stream);
  { MIBM_PROF(c, "edges");
    elength_kernel<<<div_up(c->maxne, kLagBlock), kLagBlock, 0, c->stream>>>(
        c->maxne, M<int>(c, MIBM_M_VERT_OF_EDGE), M<int>(c, MIBM_M_GHOST_EDGE), M<double>(c, MIBM_M_XYZV),
        c->S(MIBM_S_E_THRESH), M<double>(c, MIBM_M_ELENGTHS), s->rm_flag); }
  ++c->launches;
  cudaMemcpyAsync(c->hflag + 1, s->rm_flag, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
  if (!cuda_ok(c, cudaStreamSynchronize(c->stream), "remesh trigger")) return false;
  if (!c->hflag[1]) return false;
  if (!c->remesh_fn) {
    fail(c, MIBM_ESTATE, "remeshing triggered (an edge is shorter than E_thresh) but no remesher is set "
                         "(mibm_set_remesh_callback_)");
    return false;
  }
  // update_tri_normal of the moved mesh and its volume, then every mesh
  // array to the host
  geometry_launch(c, false, true);
  cudaMemcpyAsync(c->red_host, s->geom_out, sizeof(double) * 2, cudaMemcpyDeviceToHost, c->stream);
  for (int i = 0; i < MIBM_NMESH; ++i)
    cudaMemcpyAsync(c->hm[i], c->dm[i], mesh_bytes(c, i), cudaMemcpyDeviceToHost, c->stream);
  if (!cuda_ok(c, cudaStreamSynchronize(c->stream), "remesh download")) return false;
  *c->hs[MIBM_S_VOLUME] = c->red_host[1];          // calculate_volume
  int st = c->remesh_fn(c->remesh_user);
  if (st != 0) {
    fail(c, MIBM_EABORT, "remesher returned " + std::to_string(st));
    return false;
  }
  for (int i = 0; i < MIBM_NMESH; ++i)
    cudaMemcpyAsync(c->dm[i], c->hm[i], mesh_bytes(c, i), cudaMemcpyHostToDevice, c->stream);
  if (!cuda_ok(c, cudaStreamSynchronize(c->stream), "remesh upload")) return false;
  lagr_topology_changed(c);
  ++c->remesh_count;
  return ensure_adjacency(c);
}

static void tri_velocity_launch(Ctx* c, const double* vel, const double* om) {
  MIBM_PROF(c, "tri_velocity");
  tri_velocity_kernel<<<div_up(c->maxnf, 128), 128, 0, c->stream>>>(
      c->maxnf, M<int>(c, MIBM_M_GHOST_FACE), M<double>(c, MIBM_M_TRI_BAR), lag_of(c)->geom_out, vel, om,
      M<double>(c, MIBM_M_VEL_TRI));
  ++c->launches;
}

// device addresses of vel_CM and omega_c for update_tri_velocity: the moving
// body's state, else the values the substep was given
static void body_velocity(Ctx* c, const StepParams* dp, const double** vel, const double** om) {
  if (c->I(MIBM_I_IMLSSTR) == 1 && c->drigid) {
    *vel = (const double*)((const char*)c->drigid + offsetof(RigidDev, vel));
    *om = (const double*)((const char*)c->drigid + offsetof(RigidDev, om));
  } else {
    *vel = (const double*)((const char*)dp + offsetof(StepParams, vel));
    *om = (const double*)((const char*)dp + offsetof(StepParams, om));
  }
}

// particle.f90:38-193 (drop-in particle_): dense force fields, host checks
void lagr_particle(Ctx* c, const StepParams* dp) {
  if (c->I(MIBM_I_IMLSFOR) != 1 || c->maxnf == 0) return;
  lagr_find_centroid_indices(c);
  lagr_mls_weight(c);
  if (c->status != MIBM_OK) return;
  static const int fo[4] = {MIBM_F_FORXC, MIBM_F_FORYC, MIBM_F_FORZC, MIBM_F_FORTEMP};
  for (int q = 0; q < 4; ++q) cudaMemsetAsync(c->df[fo[q]], 0, c->g.cells * sizeof(double), c->stream);
  lagr_mls_force(c, dp, true);
  bool imelt = c->I(MIBM_I_IMELT) == 1;
  if (imelt) {
    lagr_find_probe_indices(c);
    lagr_heat_flux(c);
    if (c->status != MIBM_OK) return;
  }
  bool str = c->I(MIBM_I_IMLSSTR) == 1;
  if (str) {
    if (!ensure_lag_buffers(c) || !rigid_ensure(c)) return;
    rigid_pack(c, c->hrigid_in, false);
    rigid_upload(c);
    lagr_struct_loads(c, dp);
    if (c->status != MIBM_OK) return;
  }
  lagr_velforce(c);
  lagr_tempforce(c);
  if (imelt) lagr_stefan(c, dp);
  if (!ensure_adjacency(c) || !ensure_lag_buffers(c)) return;
  if (str) motion_launch(c, dp);
  bool remeshed = lagr_remesh_active(c) && remesh_check(c);
  if (c->status != MIBM_OK) return;
  geometry_launch(c, imelt);
  if (remeshed) {
    const double *vel, *om;
    body_velocity(c, dp, &vel, &om);
    tri_velocity_launch(c, vel, om);
  }
  if (str) {
    k_rigid_publish(c, lag_of(c)->geom_out, nullptr);
    rigid_download(c);
  }
  lagr_geometry_to_host(c);
  if (str) {
    if (!check_flag(c, "update_part_pos")) return;
    rigid_unpack(c, c->hrigid_out, false);
  }
  if (c->S(MIBM_S_VOLUME) < c->S(MIBM_S_V_THRESH)) fail(c, MIBM_EABORT, "Geometry V/VE smaller than threshold");
}

// particle.f90:38-193 inside the fused step: no host synchronisation.  The
// forces are added straight into u, v, w (the mean force is left in
// `mean3` for the projection update to subtract) and, after the heat flux
// has read the unforced temperature, into T.  MLS weights of a stationary
// cage are reused.  Flags and geometry scalars are read by the caller at the
// end of the step.
// The work of a substep that depends on the geometry alone: narrow-band
// tagging (tagCells at the start of the substep, tsch.f90:45-47) and, from
// particle, the cage indices, the MLS weights and the scatter plan.  The fused
// step runs it on the side stream of the substep before (the geometry is
// final once that substep's particle is done): for substeps 1 and 2, and for
// substep 0 of the next step (slot 3: no parameter block, the host's plan
// rebuild requests invalidate it instead).
// prepped: the geometry pass has left the cage indices and the band's bounds,
// and band_reset has run on the tagging's stream (lagr_particle_fused, whose
// geometry refresh is finished here)
static void substep_prologue(Ctx* c, int slot, bool prepped) {
  if (c->I(MIBM_I_IMLSFOR) != 1 || c->maxnf == 0) return;
  // the tagging (VOF fields) and the cage indices, weights and plan read the
  // same geometry and write disjoint buffers: the tagging goes to a stream of
  // its own and is joined back before the prologue ends
  const bool split = !c->I(MIBM_I_STATIONARY) && c->side2 && lagr_fork_enabled(c);
  c->geom_join_tag = split;
  if (split) {
    cudaEventRecord(c->ev_tfork, c->stream);
    wait_event(c, c->side2, c->ev_tfork);
    std::swap(c->stream, c->side2);
    tag_narrow_band(c, prepped, prepped && (slot == 1 || slot == 2));
    cudaEventRecord(c->ev_tjoin, c->stream);
    std::swap(c->stream, c->side2);
  } else if (!c->I(MIBM_I_STATIONARY)) {
    lagr_tag_narrow_band(c);
  }
  if (!ensure_adjacency(c) || !ensure_lag_buffers(c)) {
    if (split) wait_event(c, c->stream, c->ev_tjoin);
    return;
  }
  LagState* s = lag_of(c);
  bool stationary = c->I(MIBM_I_STATIONARY) != 0;
  if (!prepped) lagr_find_centroid_indices(c);
  // the MLS weights and the scatter plan both read the cage indices and
  // nothing the other writes: the weights go to a third stream
  const bool wsplit = split && c->side3;
  if (wsplit) {
    cudaEventRecord(c->ev_wfork, c->stream);
    wait_event(c, c->side3, c->ev_wfork);
    std::swap(c->stream, c->side3);
  }
  if (!(stationary && s->weights_valid)) {
    mls_weight_launch(c);
    s->weights_valid = stationary;
    if (stationary) ++c->lag_gen;     // later steps skip the weights: another launch sequence
  }
  if (wsplit) {
    cudaEventRecord(c->ev_wjoin, c->stream);
    std::swap(c->stream, c->side3);
  }
  update_plan(c, slot < 3 ? c->dparams + slot : nullptr, prepped);
  if (prepped) {                 // the rest of the geometry refresh: nothing of the next substep's chain needs it
    vert_geom_launch(c);
    edges_launch(c);
  }
  if (wsplit) wait_event(c, c->stream, c->ev_wjoin);
  if (split) wait_event(c, c->stream, c->ev_tjoin);
}

void lagr_substep_prologue(Ctx* c, int slot) { substep_prologue(c, slot, false); }

// The side stream takes the second half of particle (and the work that
// follows it) unless the host's remesher may be needed mid-way or kernels
// are timed one by one (mibm_profile_: serial, so each time is its own).
bool lagr_fork_enabled(Ctx* c) {
  return c->side && !lagr_remesh_active(c) && !c->profiling && c->I(MIBM_I_IMLSFOR) == 1 && c->maxnf > 0;
}

// The structural loads read u, v, w after their line solves, p, and the
// geometry, nothing that the temperature's line solves write: the fused step
// starts them on the side stream once w is solved, so that they run beside
// the temperature solves; the velocity scatter, which changes u, v, w, waits
// for them (lagr_particle_fused).  Same conditions as the particle fork.
void lagr_loads_early(Ctx* c, const StepParams* dp) {
  c->loads_pending = false;
  if (c->I(MIBM_I_IMLSFOR) != 1 || c->maxnf == 0 || c->I(MIBM_I_IMLSSTR) != 1) return;
  if (!lagr_fork_enabled(c)) return;
  if (!ensure_adjacency(c) || !ensure_lag_buffers(c)) return;
  cudaEventRecord(c->ev_lfork, c->stream);
  wait_event(c, c->side, c->ev_lfork);
  std::swap(c->stream, c->side);
  struct_loads_launch(c, dp, false);
  cudaEventRecord(c->ev_ldone, c->stream);
  std::swap(c->stream, c->side);
  c->loads_pending = true;
}

// The heat flux reads the solved temperature (before the temperature forcing)
// and the geometry, nothing of the velocity forcing: the fused step starts it
// on the tagging's stream, idle at this point, once T is solved (called with
// the context's stream the one that solves T).  Same conditions as above, and
// not on large grids: there the chain hides beside the projection anyway, and
// the flux would take the FP64 pipe from kernels the main stream waits for
// (128^3 free body 7.44 -> 7.35 ms, 48^3 5.19 -> 3.78 ms for two and four
// steps; 256^3 FP64 81.9 -> 82.5 ms for three).
constexpr size_t kHeatEarlyCells = 4u << 20;
void lagr_heat_early(Ctx* c) {
  c->heat_pending = false;
  if (c->I(MIBM_I_IMLSFOR) != 1 || c->maxnf == 0 || c->I(MIBM_I_IMELT) != 1) return;
  if (!lagr_fork_enabled(c) || !c->side2 || c->g.cells > kHeatEarlyCells) return;
  if (!ensure_adjacency(c) || !ensure_lag_buffers(c)) return;
  cudaEventRecord(c->ev_hfork, c->stream);
  wait_event(c, c->side2, c->ev_hfork);
  std::swap(c->stream, c->side2);
  heat_flux_launch(c, true);
  cudaEventRecord(c->ev_hflux, c->stream);
  std::swap(c->stream, c->side2);
  c->heat_pending = true;
}

const double* lagr_particle_fused(Ctx* c, const StepParams* dp, float* m32, StepParams* next,
                                  int next_prologue) {
  if (c->I(MIBM_I_IMLSFOR) != 1 || c->maxnf == 0) return nullptr;
  if (!ensure_adjacency(c) || !ensure_lag_buffers(c)) return nullptr;
  LagState* s = lag_of(c);
  lagr_join(c);                   // cage indices, MLS weights, scatter plan of this substep
  force_coefficients(c);
  bool str = c->I(MIBM_I_IMLSSTR) == 1;
  if (str) {                                 // reads the unforced u, v, w and p
    if (c->loads_pending) {
      wait_event(c, c->stream, c->ev_ldone);
      c->loads_pending = false;
    } else {
      struct_loads_launch(c, dp, false);
    }
  }
  scatter(c, true, 0, 3, true);
  double ncell = (double)c->g.n1m * (double)c->g.n2m * (double)c->g.n3m;
  { MIBM_PROF(c, "seg_mean");
    launch_beside(c, seg_mean_kernel, kMeanBlocks, 256, plan_runs(s), c->g.cells, s->segval, c->red + kRedPart, ncell,
                  s->mean3); }
  c->launches += 1;
  // Fork: the rest of particle (heat flux, temperature forcing, Stefan
  // front, motion, geometry) reads and writes none of the buffers of the
  // pressure projection that the caller enqueues next, so it runs on the
  // side stream; lagr_join makes the main stream wait for it before the next
  // substep.
  const bool fork = lagr_fork_enabled(c);
  if (fork) {
    cudaEventRecord(c->ev_fork, c->stream);
    wait_event(c, c->side, c->ev_fork);
    std::swap(c->stream, c->side);
  }
  const bool next_here = fork && next_prologue >= 0 && c->side3;     // the next substep's geometry work follows
  const bool tag_next = next_here && c->side2 && !c->I(MIBM_I_STATIONARY) && ensure_band(c);
  bool imelt = c->I(MIBM_I_IMELT) == 1;
  if (imelt && !c->heat_pending) {
    if (!fork) lagr_find_probe_indices(c);   // no next substep's cage indices follow: the host finds the probes in pind
    heat_flux_launch(c, true);
  }
  // the temperature forcing (after the heat flux, which reads the unforced
  // temperature) and the reset of the narrow band need nothing of what
  // follows here: they go to the tagging's stream, off the chain to the next
  // substep
  const bool tside = fork && c->side2;
  if (tside) {
    if (!c->heat_pending) cudaEventRecord(c->ev_hfork, c->stream);
    wait_event(c, c->side2, c->heat_pending ? c->ev_fork : c->ev_hfork);
    std::swap(c->stream, c->side2);
  }
  scatter(c, true, 3, 4, false, m32);
  if (tside) {
    if (tag_next) band_reset(c);
    cudaEventRecord(c->ev_tscat, c->stream);
    std::swap(c->stream, c->side2);
    c->tscat_pending = true;
  }
  if (c->heat_pending) {
    wait_event(c, c->stream, c->ev_hflux);
    c->heat_pending = false;
  }
  if (imelt) melt_vert_launch(c, dp);
  if (str) motion_launch(c, dp);
  bool remeshed = !fork && lagr_remesh_active(c) && remesh_check(c);
  if (c->status == MIBM_OK && next_here) {
    // the next substep's geometry-only work needs the new face centroids and
    // normals alone: it starts after the per-face pass, while a third stream
    // finishes the body's sums and publishes the moved body (ev_pub)
    FaceNext N = face_next(c);
    N.pind = M<int>(c, MIBM_M_PIND);
    N.saved = s->saved;
    N.dirty = s->dirty;
    if (tag_next) { N.band_face = s->band_face; N.face_cell = s->face_cell; }
    if (imelt) N.cfac = M<double>(c, MIBM_M_CFAC);
    face_geom_launch(c, N, false);
    cudaEventRecord(c->ev_gfork, c->stream);
    wait_event(c, c->side3, c->ev_gfork);
    std::swap(c->stream, c->side3);
    geom_sum_launch(c);
    if (str) k_rigid_publish(c, s->geom_out, next);
    cudaEventRecord(c->ev_pub, c->stream);
    std::swap(c->stream, c->side3);
    c->geom_join_tag = false;
    // the temperature forcing reads the plan and the weights of this substep
    if (tside) wait_event(c, c->stream, c->ev_tscat);
    substep_prologue(c, next_prologue, true);
    c->prologue_done = true;
    wait_event(c, c->stream, c->ev_pub);     // the full join covers the body's sums
    MIBM_LAUNCH_CHECK(c, "particle");
  } else if (c->status == MIBM_OK) {
    geometry_launch(c, imelt);
    if (remeshed) {
      const double *vel, *om;
      body_velocity(c, dp, &vel, &om);
      tri_velocity_launch(c, vel, om);
    }
    if (str) k_rigid_publish(c, s->geom_out, next);
    if (fork) cudaEventRecord(c->ev_pub, c->stream);
    c->geom_join_tag = false;
    if (tside) wait_event(c, c->stream, c->ev_tscat);
    if (fork && next_prologue >= 0) {
      lagr_substep_prologue(c, next_prologue);
      c->prologue_done = true;
    }
    MIBM_LAUNCH_CHECK(c, "particle");
  }
  if (fork) {
    cudaEventRecord(c->ev_join, c->stream);
    std::swap(c->stream, c->side);
    c->join_pending = true;
    c->geom_join_pending = true;
  }
  return c->status == MIBM_OK ? s->mean3 : nullptr;
}

// the main stream waits for the side-stream half of the last particle
void lagr_join(Ctx* c) {
  if (c->tscat_pending) {
    wait_event(c, c->stream, c->ev_tscat);
    c->tscat_pending = false;
  }
  if (!c->join_pending) return;
  wait_event(c, c->stream, c->ev_join);
  c->join_pending = false;
  c->geom_join_pending = false;
}

// the main stream waits for what the next substep's explicit terms read
// from the side branch: the moved body (published state, geometry) and,
// when the tagging ran on its own stream, the VOF fields
void lagr_join_geom(Ctx* c) {
  if (c->tscat_pending) {          // the forced temperature
    wait_event(c, c->stream, c->ev_tscat);
    c->tscat_pending = false;
  }
  if (!c->geom_join_pending) return;
  wait_event(c, c->stream, c->ev_pub);
  if (c->geom_join_tag) wait_event(c, c->stream, c->ev_tjoin);
  c->geom_join_pending = false;
}

// End of the fused step, in two halves so that the device half can sit in
// a captured step graph: lagr_step_readback enqueues the copies of the MLS
// flag and the geometry scalars into pinned host memory; after the stream
// has completed, lagr_step_host_finish reads them (MLS failure status,
// Surface, Volume, centre of mass, V_thresh abort of particle.f90:218-224).
void lagr_step_readback(Ctx* c) {
  if (c->I(MIBM_I_IMLSFOR) != 1 || c->maxnf == 0) return;
  LagState* s = lag_of(c);
  cudaMemcpyAsync(c->hflag, c->dflag, 4, cudaMemcpyDeviceToHost, c->stream);
  if (s->geom_out) cudaMemcpyAsync(c->step_host, s->geom_out, sizeof(double) * 15, cudaMemcpyDeviceToHost, c->stream);
  if (c->I(MIBM_I_IMLSSTR) == 1 && c->drigid) rigid_download(c);
}

void lagr_step_host_finish(Ctx* c) {
  if (c->I(MIBM_I_IMLSFOR) != 1 || c->maxnf == 0) return;
  if (c->hflag[0]) {
    fail(c, MIBM_ENUMERIC, (c->hflag[0] & 2) ? "particle: singular inertia tensor (dgetrf info /= 0)"
                                             : "particle: singular MLS moment matrix (dgetrf info /= 0)");
    c->hflag[0] = 0;
    cudaMemsetAsync(c->dflag, 0, 4, c->stream);
    return;
  }
  if (!lag_of(c)->geom_out) return;
  if (c->I(MIBM_I_IMLSSTR) == 1 && c->drigid) rigid_unpack(c, c->hrigid_out, false);
  *c->hs[MIBM_S_SURFACE] = c->step_host[0];
  *c->hs[MIBM_S_VOLUME] = c->step_host[2];
  for (int d = 0; d < 3; ++d) c->hs[MIBM_S_POS_CM][d] = c->step_host[3 + d];
  for (int q = 0; q < 9; ++q) c->hs[MIBM_S_INERT_TENSOR][q] = c->step_host[6 + q];
  if (c->S(MIBM_S_VOLUME) < c->S(MIBM_S_V_THRESH)) fail(c, MIBM_EABORT, "Geometry V/VE smaller than threshold");
}

void lagr_free(Ctx* c) {
  for (size_t q = 0; q < g_lag.size(); ++q)
    if (g_lag[q]->c == c) {
      LagState* s = g_lag[q];
      cudaFree(s->adj_off); cudaFree(s->adj_face); cudaFree(s->face_part); cudaFree(s->geom_out); cudaFree(s->geom_ticket);
      cudaFree(s->loads_ev); cudaFree(s->loads_ticket); cudaFree(s->rm_flag);
      cudaFree(s->mean3); cudaFree(s->winner); cudaFree(s->dist_buf);
      cudaFree(s->band_ub); cudaFree(s->band_face); cudaFree(s->face_cell); cudaFree(s->cm32);
      cudaFree(s->band_list); cudaFree(s->band_count);
      cudaFree(s->bitmap); cudaFree(s->wpre); cudaFree(s->tsum); cudaFree(s->slot);
      cudaFree(s->run_key); cudaFree(s->run_cnt); cudaFree(s->run_off); cudaFree(s->nruns); cudaFree(s->long_run);
      cudaFree(s->entry); cudaFree(s->src);
      cudaFree(s->saved); cudaFree(s->dirty); cudaFree(s->segval);
      delete s;
      g_lag.erase(g_lag.begin() + q);
      break;
    }
}

}  // namespace mibm
