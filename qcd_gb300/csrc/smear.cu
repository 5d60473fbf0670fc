// smear.cu -- source construction on the GPU: 3D APE smearing of the links,
// 3D Gaussian smearing of a spinor on one time-slice, and the smeared point
// source built from both (the setup of the 24^3 x 48 single-RHS workload).
//
// APE step (qcd_apeSmear3d, lib/src/qcd_smearing.c:209-276): for spatial
// mu, U'_mu(x) = Proj_SU3( U_mu(x) + alpha * sum over spatial nu != mu of
//   U_nu(x) U_mu(x+nu) U_nu(x+mu)^+  +  U_nu(x-nu)^+ U_mu(x-nu) U_nu(x-nu+mu) );
// temporal links are copied. Proj_SU3 (qcd_projectSU33d, lib/src/qcd_blas.c:
// 950) is the unitary polar factor of M times exp(-i arg(det M) / 3) with
// the columns re-orthonormalised (project_su3 below).
//
// Gaussian step (qcd_gaussIteration3d, lib/src/qcd_smearing.c:25-113): on
// time-slice t, v <- (v + alpha H v) / (1 + 6 alpha) with
//   H v(x) = sum_{nu=1..3} U_nu(x) v(x+nu) + U_nu(x-nu)^+ v(x-nu);
// other time-slices are unchanged. FP64 throughout, which runs at two
// multiply-adds per clock and SM: both steps are bound by their FP64
// operations, so products are multiply-add chains into their sums.
//
// Both steps stay inside a time-slice. The Gaussian steps, and the APE steps
// of a smeared source (whose other slices nobody reads), run on copies of the
// slice's links and spinor that are dense in the spatial index: the fields
// keep t fastest, so a slice read in place uses half of every 32-byte sector.
#include <math.h>

#include "su3.cuh"

namespace qg {

__device__ __forceinline__ C<double> m3det(const C<double> m[9])
{
  C<double> d = m[0] * (m[4] * m[8] - m[5] * m[7]);
  d = d - m[1] * (m[3] * m[8] - m[5] * m[6]);
  return d + m[2] * (m[3] * m[7] - m[4] * m[6]);
}

// r = (m^{-1})^+ by cofactors
__device__ __forceinline__ void m3inv_dag(const C<double> m[9], C<double> r[9])
{
  const C<double> d = m3det(m);
  const double dd = d.re * d.re + d.im * d.im;
  const C<double> id{d.re / dd, -d.im / dd};
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int i1 = (j + 1) % 3, i2 = (j + 2) % 3, j1 = (i + 1) % 3, j2 = (i + 2) % 3;
      const C<double> cof = m[3 * i1 + j1] * m[3 * i2 + j2] - m[3 * i1 + j2] * m[3 * i2 + j1];
      r[3 * j + i] = conj(cof * id);  // (m^{-1})_{ij} = cof_ij / det, stored transposed and conjugated
    }
}

// the polar factor by Newton's iteration W <- (W + W^{-+}) / 2 (N. J. Higham,
// SIAM J. Sci. Stat. Comput. 7 (1986) 1160) to a relative step of 1e-15, any
// condition: about 1,000-2,000 FP64 operations a link
__device__ __noinline__ void project_su3_newton(C<double> W[9])
{
  const C<double> d = m3det(W);
  const double phase = atan2(d.im, d.re) / 3.0;
  for (int it = 0; it < 100; it++) {
    C<double> Wi[9];
    m3inv_dag(W, Wi);
    double diff = 0, nrm = 0;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const C<double> nw{0.5 * (W[k].re + Wi[k].re), 0.5 * (W[k].im + Wi[k].im)};
      diff += fabs(nw.re - W[k].re) + fabs(nw.im - W[k].im);
      nrm += fabs(nw.re) + fabs(nw.im);
      W[k] = nw;
    }
    if (diff <= 1e-15 * nrm) break;
  }
  double s, c;
  sincos(phase, &s, &c);
  const C<double> ph{c, -s};
#pragma unroll
  for (int k = 0; k < 9; k++) W[k] = W[k] * ph;
  reunit_cols(W);
}

// re += |a|^2
__device__ __forceinline__ double sq_acc(C<double> a, double r) { return fma(a.im, a.im, fma(a.re, a.re, r)); }

// M <- (s M + (s M)^{-+}) / 2 with s about 1 / |det M|^{1/3}, d = det M, i3 =
// |d| (N. J. Higham, SIAM J. Sci. Stat. Comput. 7 (1986) 1160): the same polar
// factor and phase of the determinant, singular values closer together
__device__ __forceinline__ void polar_step(C<double> M[9], C<double> d, double i3)
{
  const float sf = rcbrtf((float)i3);
  const double s = 0.5 * (double)sf, r = (double)(0.5f / sf) / (i3 * i3);
  const C<double> id{r * d.re, -r * d.im};
  C<double> N[9];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
      const C<double> cof = cmsub(M[3 * i1 + j2], M[3 * i2 + j1], M[3 * i1 + j1] * M[3 * i2 + j2]);
      const C<double> t = cof * id, m = M[3 * i + j];  // (M^{-1})_ji / (2 s)
      N[3 * i + j] = C<double>{fma(s, m.re, t.re), fma(s, m.im, -t.im)};
    }
#pragma unroll
  for (int k = 0; k < 9; k++) M[k] = N[k];
}

// M <- its SU(3) projection, the polar factor in closed form:
// M (M^+ M)^{-1/2} with the inverse square root as a polynomial in
// G = M^+ M (Cayley-Hamilton; A. Hoger and D. E. Carlson, Quart. Appl. Math.
// 42 (1984) 113). With i1, i2, i3 the invariants of sqrt(G),
//   G^{-1/2} = [ i1 G^2 - (i3 + i1 (i1^2 - 2 i2)) G + (i1 i2^2 - i3 (i1^2 + i2)) ] / (i3 (i1 i2 - i3)),
// i3 = |det M|, i2 = (i1^2 - tr G) / 2 and i1 the largest root of
//   x^4 - 2 (tr G) x^2 - 8 i3 x + (tr G)^2 - 4 I2(G)
// (simple unless two singular values vanish): Newton from above in FP32, two
// steps in FP64. The factor e^{-i arg(det) / 3} starts in FP32 as well and
// takes two FP64 Newton steps of w <- w (4 - z w^3) / 3. Only two columns are
// formed, the third is their cross product: about 400 FP64 operations a link.
// Working on M^+ M loses the square of M's condition number kappa, where
// Newton's iteration stays at its error for kappa = 1: 1.35 times that at
// kappa = 1.5, 3.8 times at 3, 26 times at 10 (root mean square of 20,000 links
// each, against 113 bits). i1^3 / (27 i3) is 1 for equal singular values and
// 1.02 at kappa = 1.3; links beyond that take one or two steps of polar_step
// first (kappa 3 -> 1.2, 10 -> at most 1.9), about 350 operations each where any
// of a warp's 32 links needs it (a smeared source at 24^3 x 48, whose links are
// beyond in the first APE steps only: 2.99 -> 3.04 ms). Then the error is 0.90 to
// 1.02 times the iteration's for smooth, rough and random links and for kappa =
// 1.2 to 20.
// Links with i1^3 > 135 i3 (from kappa = 8.4 to 15.6 on, by the middle singular
// value), those still beyond after two steps and those whose root has not
// settled (out of FP32's range, singular, not finite) take the iteration.
__device__ __forceinline__ void project_su3(C<double> M[9])
{
  C<double> d, g01, g02, g12;
  double g0, g1, g2, n01, n02, n12, I1, i1, i3;
#pragma unroll 1
  for (int pass = 0;; pass++) {
    d = cmadd(M[0], cmsub(M[5], M[7], M[4] * M[8]),
              cmadd(M[1], cmsub(M[3], M[8], M[5] * M[6]), M[2] * cmsub(M[4], M[6], M[3] * M[7])));
    // G = M^+ M
    g0 = sq_acc(M[6], sq_acc(M[3], sq_acc(M[0], 0.0)));
    g1 = sq_acc(M[7], sq_acc(M[4], sq_acc(M[1], 0.0)));
    g2 = sq_acc(M[8], sq_acc(M[5], sq_acc(M[2], 0.0)));
    g01 = cmadd_conj(M[6], M[7], cmadd_conj(M[3], M[4], cdot(M[0], M[1])));
    g02 = cmadd_conj(M[6], M[8], cmadd_conj(M[3], M[5], cdot(M[0], M[2])));
    g12 = cmadd_conj(M[7], M[8], cmadd_conj(M[4], M[5], cdot(M[1], M[2])));
    n01 = sq_acc(g01, 0.0);
    n02 = sq_acc(g02, 0.0);
    n12 = sq_acc(g12, 0.0);
    I1 = g0 + g1 + g2;
    const double I2 = fma(g0, g1, fma(g1, g2, g0 * g2)) - (n01 + n02 + n12), c0 = fma(I1, I1, -4.0 * I2);
    i3 = sqrt(sq_acc(d, 0.0));
    float xf = sqrtf(3.0f * (float)I1);
    {
      const float a = 2.0f * (float)I1, b = 8.0f * (float)i3, c = (float)c0;
#pragma unroll
      for (int k = 0; k < 6; k++) {
        const float x2 = xf * xf;
        xf -= (((x2 - a) * xf - b) * xf + c) / ((4.0f * x2 - 2.0f * a) * xf - b);
      }
    }
    i1 = (double)xf;
    double dx = 0.0;
    const double slope = (double)(1.0f / ((4.0f * xf * xf - 4.0f * (float)I1) * xf - 8.0f * (float)i3));
#pragma unroll
    for (int k = 0; k < 2; k++) {
      dx = slope * fma(fma(fma(i1, i1, -2.0 * I1), i1, -8.0 * i3), i1, c0);
      i1 -= dx;
    }
    const double cube = i1 * i1 * i1;
    const bool settled = 135.0 * i3 >= cube && fabs(dx) <= 1e-9 * i1;
    if (settled && 27.54 * i3 >= cube) break;
    if (!settled || pass == 2) {
      C<double> W[9];
#pragma unroll
      for (int k = 0; k < 9; k++) W[k] = M[k];
      project_su3_newton(W);
#pragma unroll
      for (int k = 0; k < 9; k++) M[k] = W[k];
      return;
    }
    polar_step(M, d, i3);
  }
  const double i2 = 0.5 * fma(i1, i1, -I1), e = fma(i1, i2, -i3);
  const double r = 1.0 / (i3 * e);
  const double a2 = i1 * r, a1 = -fma(i1, fma(i1, i1, -2.0 * i2), i3) * r,
               a0 = fma(i1 * i2, i2, -i3 * fma(i1, i1, i2)) * r;
  // columns 0 and 1 of X = a2 G^2 + a1 G + a0 (Hermitian)
  const double x0 = fma(a2, fma(g0, g0, n01 + n02), fma(a1, g0, a0));
  const double x1 = fma(a2, fma(g1, g1, n01 + n12), fma(a1, g1, a0));
  const double s01 = g0 + g1, s02 = g0 + g2, s12 = g1 + g2;
  const C<double> q01{fma(s01, g01.re, fma(g02.re, g12.re, g02.im * g12.im)),
                      fma(s01, g01.im, fma(g02.im, g12.re, -g02.re * g12.im))};  // + g02 conj(g12)
  const C<double> q02 = cmadd(g01, g12, C<double>{s02 * g02.re, s02 * g02.im});
  const C<double> q12 = cmadd_conj(g01, g02, C<double>{s12 * g12.re, s12 * g12.im});
  const C<double> x01{fma(a2, q01.re, a1 * g01.re), fma(a2, q01.im, a1 * g01.im)};
  const C<double> x02{fma(a2, q02.re, a1 * g02.re), fma(a2, q02.im, a1 * g02.im)};
  const C<double> x12{fma(a2, q12.re, a1 * g12.re), fma(a2, q12.im, a1 * g12.im)};
  // w = z^{-1/3}, z = det / |det|
  const double r3 = r * e;
  const C<double> z{d.re * r3, d.im * r3};
  float sf, cf;
  sincosf(atan2f((float)z.im, (float)z.re) / 3.0f, &sf, &cf);
  C<double> w{(double)cf, -(double)sf};
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const C<double> t = z * (w * (w * w));
    w = w * C<double>{fma(t.re, -1.0 / 3.0, 4.0 / 3.0), t.im * (-1.0 / 3.0)};
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const C<double> m0 = M[3 * i], m1 = M[3 * i + 1], m2 = M[3 * i + 2];
    // (M X)_i0 = m0 x0 + m1 conj(x01) + m2 conj(x02); (M X)_i1 = m0 x01 + m1 x1 + m2 conj(x12)
    const C<double> u = cmadd_conj(x02, m2, cmadd_conj(x01, m1, C<double>{m0.re * x0, m0.im * x0}));
    const C<double> v = cmadd_conj(x12, m2, cmadd(x01, m0, C<double>{m1.re * x1, m1.im * x1}));
    M[3 * i] = u * w;
    M[3 * i + 1] = v * w;
  }
  reunit_cols(M);
}

__device__ __forceinline__ C<double> load_entry(const double2 *u, int64_t stride, int x, int mu, int k)
{
  const double2 v = __ldg(u + ((int64_t)mu * 9 + k) * stride + x);
  return C<double>{v.x, v.y};
}

// S += A (B C^+) (DAG: A^+ (B C)) for the links A = (xa, ma), B = (xb, mb),
// C = (xc, mc), one row of the inner product at a time
template <bool DAG>
__device__ __forceinline__ void staple_acc(C<double> S[9], const double2 *u, int64_t stride, int xa, int ma, int xb,
                                           int mb, int xc, int mc)
{
  C<double> c[9];
#pragma unroll
  for (int k = 0; k < 9; k++) c[k] = load_entry(u, stride, xc, mc, k);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    C<double> b[3], t[3];
#pragma unroll
    for (int j = 0; j < 3; j++) b[j] = load_entry(u, stride, xb, mb, 3 * k + j);
#pragma unroll
    for (int j = 0; j < 3; j++)
      t[j] = DAG ? cmadd(c[6 + j], b[2], cmadd(c[3 + j], b[1], c[j] * b[0]))
                 : cmadd_conj(c[3 * j + 2], b[2], cmadd_conj(c[3 * j + 1], b[1], cdot(c[3 * j], b[0])));
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const C<double> a = load_entry(u, stride, xa, ma, DAG ? 3 * k + i : 3 * i + k);
#pragma unroll
      for (int j = 0; j < 3; j++) S[3 * i + j] = DAG ? cmadd_conj(a, t[j], S[3 * i + j]) : cmadd(a, t[j], S[3 * i + j]);
    }
  }
}

// One APE step, one thread per site and spatial direction mu = 1 + blockIdx.y.
// mu0: direction of the arrays' first nine blocks (0: whole fields, whose
// temporal links are copied; 1: a time-slice's spatial links).
constexpr int kApeThreads = 32;
__global__ void __launch_bounds__(kApeThreads, 12) k_ape3d(double2 *out, const double2 *in, int64_t stride, Geom geo,
                                                          int V, double alpha, int mu0)
{
  const int x = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (x >= V) return;
  int c[4];
  coords(geo, x, c);
  const int mu = 1 + (int)blockIdx.y;
  if (mu0 == 0)
    for (int k = 3 * (mu - 1); k < 3 * mu; k++) out[(int64_t)k * stride + x] = in[(int64_t)k * stride + x];
  C<double> S[9];
#pragma unroll
  for (int k = 0; k < 9; k++) S[k] = C<double>{0.0, 0.0};
  const int xm = fwd(geo, x, c, mu);
#pragma unroll 1
  for (int i = 1; i < 3; i++) {
    const int nu = 1 + (mu - 1 + i) % 3, b = bwd(geo, x, c, nu);
    // b's neighbour in direction mu (b has x's mu coordinate)
    const int bm = b + (xm - x);
    staple_acc<false>(S, in, stride, x, nu - mu0, fwd(geo, x, c, nu), mu - mu0, xm, nu - mu0);
    staple_acc<true>(S, in, stride, b, nu - mu0, b, mu - mu0, bm, nu - mu0);
  }
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const C<double> u = load_entry(in, stride, x, mu - mu0, k);
    S[k] = C<double>{fma(alpha, S[k].re, u.re), fma(alpha, S[k].im, u.im)};
  }
  project_su3(S);
#pragma unroll
  for (int k = 0; k < 9; k++) out[((int64_t)(mu - mu0) * 9 + k) * stride + x] = make_double2(S[k].re, S[k].im);
}

// --------------------------------------------------- a time-slice, dense
// blocks blockIdx.y = 0 .. n-1 of V3 sites at a distance of step sites,
// from / to a dense array of stride sstride
__global__ void k_slice_get(double2 *d, int64_t sstride, const double2 *f, int64_t stride, int V3, int t, int step)
{
  const int s = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (s < V3) d[(int64_t)blockIdx.y * sstride + s] = f[(int64_t)blockIdx.y * stride + t + (int64_t)step * s];
}
__global__ void k_slice_put(double2 *f, int64_t stride, const double2 *d, int64_t sstride, int V3, int t, int step)
{
  const int s = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (s < V3) f[(int64_t)blockIdx.y * stride + t + (int64_t)step * s] = d[(int64_t)blockIdx.y * sstride + s];
}

// what a dense time-slice holds: flag[0] = 1 when a link is infinite or not a
// number, flag[1 + spin] = 1 when a value of that spin is not +0
__global__ void k_slice_flags(const double2 *u, const double2 *v, int64_t sstride, int V3, int *flag)
{
  const int s = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (s >= V3) return;
  const int k = (int)blockIdx.y;  // 27 blocks of links, then 12 of the spinor
  const double2 w = k < 27 ? u[k * sstride + s] : v[(k - 27) * sstride + s];
  if (k < 27) {
    if (!isfinite(w.x) || !isfinite(w.y)) flag[0] = 1;
  } else if ((__double2hiint(w.x) | __double2loint(w.x) | __double2hiint(w.y) | __double2loint(w.y)) != 0) {
    flag[1 + (k - 27) / 3] = 1;
  }
}

// one of the three values is not zero (integer test: the FP64 pipe is the bottleneck)
__device__ __forceinline__ bool nonzero(const double2 v[3])
{
  int m = 0;
#pragma unroll
  for (int b = 0; b < 3; b++)
    m |= ((__double2hiint(v[b].x) | __double2hiint(v[b].y)) & 0x7fffffff) | __double2loint(v[b].x) |
         __double2loint(v[b].y);
  return m != 0;
}

// out = (in + alpha H in) / (1 + 6 alpha) on a dense time-slice: a block takes
// one spin (blockIdx.y) of 32 sites, one warp per direction, whose sums meet in
// shared memory; the step does not mix spins. Zeros are left out while the
// links are finite: an empty spin stays empty (the host clears it in both
// arrays), and a neighbour whose three colours are zero at all 32 sites adds
// nothing, so its product is skipped. A point source fills one spin of four,
// and the sites within k of it after k steps; dense spinors take the same path
// and skip nothing. Twelve point sources on a 32^3 slice, 50 steps: 72.9 ms with
// one thread per site, in place; 15.0 with one warp per spin and 32 sites (its
// six neighbours one latency chain after the other); 13.7 now (a step is 23 us,
// 12 of them the FP64 operations of one full spin, 234 a site). The sum by
// direction, chains of 12 multiply-adds, also rounds less than one chain of 36:
// 2.1e-16 off the 64-bit result after 50 steps, 3.8e-16, and 2.5e-16 for
// separately summed products.
constexpr int kGaussSites = 32;
__global__ void __launch_bounds__(3 * kGaussSites) k_gauss3d(double2 *out, const double2 *in, const double2 *u,
                                                             int64_t stride, Geom geo, int V3, double alpha,
                                                             double nrm, const int *flag)
{
  __shared__ double2 part[3][3][kGaussSites];  // [direction][colour][site]
  const int lane = threadIdx.x, mu = threadIdx.y, id = (int)blockIdx.x * kGaussSites + lane, sp = (int)blockIdx.y;
  const bool all = flag[0] != 0 || !isfinite(alpha) || !isfinite(nrm);
  if (!all && flag[1 + sp] == 0) return;  // the whole block
  const int x = id < V3 ? id : V3 - 1;    // idle lanes repeat the last site
  int c[4];
  coords(geo, x, c);
  const double2 *v = in + (int64_t)(3 * sp) * stride;
  const int xf = fwd(geo, x, c, 1 + mu), xb = bwd(geo, x, c, 1 + mu);
  double2 p[2][3];
#pragma unroll
  for (int b = 0; b < 3; b++) {
    p[0][b] = v[b * stride + xf];
    p[1][b] = v[b * stride + xb];
  }
  const double2 w0 = v[mu * stride + x];
  C<double> t[3];
#pragma unroll
  for (int k = 0; k < 3; k++) t[k] = C<double>{0.0, 0.0};
#pragma unroll
  for (int d = 0; d < 2; d++) {
    if (!__any_sync(0xffffffffu, all || nonzero(p[d]))) continue;
#pragma unroll
    for (int b = 0; b < 3; b++) {
      const C<double> w{p[d][b].x, p[d][b].y};
#pragma unroll
      for (int a = 0; a < 3; a++)
        t[a] = d ? cmadd_conj(load_entry(u, stride, xb, mu, 3 * b + a), w, t[a])
                 : cmadd(load_entry(u, stride, x, mu, 3 * a + b), w, t[a]);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++) part[mu][k][lane] = make_double2(t[k].re, t[k].im);
  __syncthreads();
  if (id >= V3) return;
  const double2 a = part[0][mu][lane], b = part[1][mu][lane], d = part[2][mu][lane];
  out[(int64_t)(3 * sp + mu) * stride + x] =
      make_double2((w0.x + alpha * (a.x + b.x + d.x)) * nrm, (w0.y + alpha * (a.y + b.y + d.y)) * nrm);
}

static Geom make_geom(const int L[4])
{
  Geom g;
  for (int i = 0; i < 4; i++) g.L[i] = L[i];
  g.st[0] = 1;
  g.st[1] = L[0];
  g.st[2] = L[0] * L[1];
  g.st[3] = L[0] * L[1] * L[2];
  return g;
}

static bool same_lattice(qcdgpu_gauge a, qcdgpu_gauge b)
{
  return a->L[0] == b->L[0] && a->L[1] == b->L[1] && a->L[2] == b->L[2] && a->L[3] == b->L[3];
}

// one APE step out <- in (FP64 fields, out != in)
bool ape3d(qcdgpu_gauge out, qcdgpu_gauge in, double alpha)
{
  if (!out || !in || out == in || out->prec != QCDGPU_F64 || in->prec != QCDGPU_F64 || !same_lattice(out, in)) {
    set_error("APE smearing: two distinct FP64 gauge fields on the same lattice");
    return false;
  }
  const dim3 nb((unsigned)((in->V + kApeThreads - 1) / kApeThreads), 3);
  k_ape3d<<<nb, kApeThreads, 0, stream()>>>((double2 *)out->data, (const double2 *)in->data, in->stride,
                                            make_geom(in->L), (int)in->V, alpha, 0);
  if (!QG_LAUNCHED("ape3d")) return false;
  out->recon = 12;  // SU(3) by construction
  gauge_forget(out);
  return true;
}

// n Gaussian steps of v on time-slice t, with the links of g after ape_n APE
// steps (g itself stays)
static bool smear_slice(qcdgpu_field v, qcdgpu_gauge g, double ape_alpha, int ape_n, double alpha, int t, int n)
{
  if (!v || !g || v->prec != QCDGPU_F64 || g->prec != QCDGPU_F64 || v->V != g->V ||
      memcmp(v->L, g->L, sizeof(v->L)) != 0 || t < 0 || t >= v->L[0] || n < 0) {
    set_error("Gaussian smearing: FP64 field and gauge on one lattice, 0 <= t < L_t, n >= 0");
    return false;
  }
  if (n == 0) return true;
  const int V3 = (int)(v->V / v->L[0]);
  const int64_t S = pad_stride(V3);
  // dense copies: two of the spinor's 12 blocks, one or two of the 27 link
  // blocks, and the flags
  const int64_t blocks = 24 + (ape_n > 0 ? 54 : 27);
  Scratch w(sizeof(double2) * (size_t)(blocks * S) + 5 * sizeof(int));
  if (!w.data) return false;
  double2 *a = (double2 *)w.data, *b = a + 12 * S, *u = b + 12 * S, *u2 = u + 27 * S;
  int *flag = (int *)(a + blocks * S);
  cudaStream_t st = stream();
  Geom geo = make_geom(v->L);
  geo.L[0] = 1;
  for (int i = 1; i < 4; i++) geo.st[i] /= v->L[0];
  const unsigned nb = (unsigned)((V3 + 127) / 128);
  const double2 *links = (const double2 *)g->data + 9 * g->stride;  // the spatial directions
  k_slice_get<<<dim3(nb, 12), 128, 0, st>>>(a, S, (const double2 *)v->data, v->stride, V3, t, v->L[0]);
  bool ok = QG_LAUNCHED("slice_get");
  k_slice_get<<<dim3(nb, 27), 128, 0, st>>>(u, S, links, g->stride, V3, t, v->L[0]);
  ok = QG_LAUNCHED("slice_get") && ok;
  for (int i = 0; ok && i < ape_n; i++) {
    const dim3 na((unsigned)((V3 + kApeThreads - 1) / kApeThreads), 3);
    k_ape3d<<<na, kApeThreads, 0, st>>>(u2, u, S, geo, V3, ape_alpha, 1);
    ok = QG_LAUNCHED("ape3d");
    double2 *tmp = u;
    u = u2;
    u2 = tmp;
  }
  ok = ok && QG_CUDA(cudaMemsetAsync(flag, 0, 5 * sizeof(int), st)) &&
       QG_CUDA(cudaMemsetAsync(b, 0, sizeof(double2) * 12 * S, st));
  if (ok) {
    k_slice_flags<<<dim3(nb, 39), 128, 0, st>>>(u, a, S, V3, flag);
    ok = QG_LAUNCHED("slice_flags");
  }
  const double nrm = 1.0 / (1.0 + 6.0 * alpha);
  const dim3 ng((unsigned)((V3 + kGaussSites - 1) / kGaussSites), 4);
  for (int i = 0; ok && i < n; i++) {
    k_gauss3d<<<ng, dim3(kGaussSites, 3), 0, st>>>(b, a, u, S, geo, V3, alpha, nrm, flag);
    ok = QG_LAUNCHED("gauss3d");
    double2 *tmp = a;
    a = b;
    b = tmp;
  }
  if (ok) {
    k_slice_put<<<dim3(nb, 12), 128, 0, st>>>((double2 *)v->data, v->stride, a, S, V3, t, v->L[0]);
    ok = QG_LAUNCHED("slice_put");
  }
  return ok;
}

// n Gaussian steps of v on time-slice t with links g
bool gauss3d(qcdgpu_field v, qcdgpu_gauge g, double alpha, int t, int n)
{
  return smear_slice(v, g, 0.0, 0, alpha, t, n);
}

bool ape3d_steps(qcdgpu_gauge out, qcdgpu_gauge in, double alpha, int n)
{
  if (!out || !in || out == in || n < 1) {
    set_error("APE smearing: distinct fields and n >= 1");
    return false;
  }
  if (n == 1) return ape3d(out, in, alpha);
  qcdgpu_gauge w = gauge_new(in->L, in->theta, QCDGPU_F64, 18);
  if (!w) return false;
  // ping-pong so that the last step writes `out`
  qcdgpu_gauge src = in;
  bool ok = true;
  for (int i = 0; ok && i < n; i++) {
    qcdgpu_gauge dst = ((n - 1 - i) % 2 == 0) ? out : w;
    ok = ape3d(dst, src, alpha);
    src = dst;
  }
  if (!QG_CUDA(cudaStreamSynchronize(stream()))) ok = false;
  gauge_forget(w);
  gauge_free(w);
  return ok;
}

}  // namespace qg

extern "C" {

int qcdgpu_gauge_ape3d(qcdgpu_gauge out, qcdgpu_gauge in, double alpha, int n)
{
  return qg::ape3d_steps(out, in, alpha, n) ? 0 : 1;
}

int qcdgpu_field_gauss3d(qcdgpu_field v, qcdgpu_gauge g, double alpha, int t, int n)
{
  return qg::gauss3d(v, g, alpha, t, n) ? 0 : 1;
}

int qcdgpu_smeared_source(qcdgpu_field f, qcdgpu_gauge g, const int x[4], int spin, int colour, double ape_alpha,
                          int ape_n, double gauss_alpha, int gauss_n)
{
  if (!f || !g || f->prec != QCDGPU_F64) {
    qg::set_error("smeared source: FP64 field and gauge field");
    return 1;
  }
  if (!qg::field_point(f, x, spin, colour)) return 1;
  if (gauss_n == 0) return 0;
  // the Gaussian steps read the links of the source's time-slice only, and
  // the APE steps do not couple time-slices: only that slice is smeared
  const bool ok = qg::smear_slice(f, g, ape_alpha, ape_n, gauss_alpha, x[0], gauss_n);
  // with APE steps the call ends when the source is there, for callers that
  // go on on another stream (15 to 22 us a call where calls follow each other)
  return (ape_n <= 0 || QG_CUDA(cudaStreamSynchronize(qg::stream()))) && ok ? 0 : 1;
}

}  // extern "C"
