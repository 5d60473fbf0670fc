// contract.cu -- proton two-point function on GPU-resident propagators, the
// contraction of twop.c (twop.c:219-226 boundary phases, :264-282 C g5 x
// bar C g5 entries, :324-399 block and Fourier sum).
//
// Propagators are 12 FP64 fields per flavour: column nu * 3 + c2 (source spin
// nu, source colour c2) holds the spinor (sink spin mu, sink colour c1), i.e.
// qcd_lib's D[v][mu][nu][c1][c2]. For every requested time-slice t (relative
// to the source) and spatial site x of slice (t + x_src,t) mod L_t:
//
//   block(x) = - f(t)^3 sum_{al,be} P13[al][be] sum_{mu nu ku lu} Cg5[mu][nu] barCg5[ku][lu]
//              sum_{eps, eps'} sgn sgn' [ u(mu,ku;c1,c1') d(nu,lu;c2,c2') u(be,al;c3,c3')
//                                        + u(mu,al;c1,c1') d(nu,lu;c2,c2') u(be,ku;c3,c3') ]
//
// with f(t) = exp(i pi t / L_t) (the antiperiodic-to-periodic phase twop.c
// multiplies into both propagators), and corr(t, p) = 1/2 sum_x block(x)
// exp(-2 pi i p.(x - x_src) / L).
//
// FP64 arithmetic bounds it (two multiply-adds per clock and SM), so the sum
// is factorised. Every term is D3(A, B, C) = sum eps eps' A[c1][d1] B[c2][d2]
// C[c3][d3], which is linear in each matrix and symmetric, and the projector
// has rank two: P13 = i/2 sum_g w_g w_g^T, g = 0, 1, w_g = e_g + i e_{g+2}. With
//   X = sum_g u(w_g, w_g), R_g(mu) = u(mu, w_g), S_g(ku) = u(w_g, ku)
// and (A x B)[c3][d3] = sum eps eps' A[c1][d1] B[c2][d2],
//   block(x) = -(i/2) f(t)^3 sum_{mu ku} +-d(nu, lu) . [ u(mu,ku) x X + sum_g R_g(mu) x S_g(ku) ]
// where nu, lu and the sign follow from mu, ku (one entry per row of C g5 and
// bar C g5): 48 matrix pairs of 36 complex products a site, about 7,900
// multiply-adds, against 18,432 products of three factors in the written-out
// sum (115 ms at 24^3 x 48 in that form; the FP64 floor of this one is 8 ms).
#include <math.h>

#include "dslash_args.h"

namespace qg {

using namespace qgd;

namespace {

struct Props {
  const double2 *u[12], *d[12];  // column nu * 3 + c2
  int64_t stride;
};

// u(mu, nu; c1, c2) at site v
__device__ __forceinline__ C<double> pr(const double2 *const *col, int64_t stride, int v, int mu, int nu, int c1,
                                         int c2)
{
  const double2 w = __ldg(col[nu * 3 + c2] + (int64_t)(mu * 3 + c1) * stride + v);
  return C<double>{w.x, w.y};
}

// e += a x b: (a x b)[c3][d3] = sum eps(c1 c2 c3) eps(d1 d2 d3) a[c1][d1] b[c2][d2],
// b's nine entries read once each at a distance of `step`
__device__ __forceinline__ void cross_acc(C<double> e[9], const C<double> a[9], const double2 *b, int step)
{
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double2 w = b[k * step];
    const C<double> v{w.x, w.y};
    const int c2 = k / 3, d2 = k % 3;
#pragma unroll
    for (int i = 1; i < 3; i++)
#pragma unroll
      for (int j = 1; j < 3; j++) {
        // c1 = c2 + i: eps(c2 + 1, c2, c2 + 2) = -1, eps(c2 + 2, c2, c2 + 1) = +1
        const int c1 = (c2 + i) % 3, c3 = (c2 + 3 - i) % 3, d1 = (d2 + j) % 3, d3 = (d2 + 3 - j) % 3;
        C<double> &r = e[3 * c3 + d3];
        r = i == j ? cmadd(a[3 * c1 + d1], v, r) : cmsub(a[3 * c1 + d1], v, r);
      }
  }
}

// a block's 32 sites times four warps, one per sink spin mu: the warps build
// S_g(ku = mu) and a share of X in shared memory, then each takes its mu's
// four ku. One site per thread would need all eight S_g in registers.
constexpr int kTwSites = 32;
constexpr size_t kTwShared = sizeof(double2) * kTwSites * 9 * (8 + 4);

__global__ void __launch_bounds__(4 * kTwSites, 3) k_twop_block(Props p, Geom geo, int t0, int nt, int xsrc_t,
                                                                double2 *block)
{
  extern __shared__ double2 tw_sh[];
  double2 *S = tw_sh;                    // [ku][g][entry][site]
  double2 *X = tw_sh + 8 * 9 * kTwSites;  // [share][entry][site]; the sum in share 0
  const int lane = threadIdx.x & 31, mu = threadIdx.x >> 5;
  const unsigned V3 = (unsigned)geo.L[1] * geo.L[2] * geo.L[3], n = V3 * (unsigned)nt;
  const unsigned id = blockIdx.x * kTwSites + lane;
  const bool act = id < n;
  const unsigned i = act ? id : n - 1;  // idle lanes repeat the last site
  // the time runs fastest, as in the fields
  const int ti = (int)(i % (unsigned)nt), s = (int)(i / (unsigned)nt);
  const int t = t0 + ti, v = (t + xsrc_t) % geo.L[0] + geo.L[0] * s;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const int c1 = k / 3, d1 = k % 3;
#pragma unroll
    for (int g = 0; g < 2; g++) {
      const C<double> a = pr(p.u, p.stride, v, g, mu, c1, d1), b = pr(p.u, p.stride, v, g + 2, mu, c1, d1);
      S[((mu * 2 + g) * 9 + k) * kTwSites + lane] = make_double2(a.re - b.im, a.im + b.re);
    }
    const C<double> a = pr(p.u, p.stride, v, mu, mu, c1, d1), b = pr(p.u, p.stride, v, mu, mu ^ 2, c1, d1);
    const double sg = mu < 2 ? 1.0 : -1.0;
    X[(mu * 9 + k) * kTwSites + lane] = make_double2(fma(sg, a.re, -b.im), fma(sg, a.im, b.re));
  }
  __syncthreads();
  for (int k = mu; k < 9; k += 4) {
    double2 x = X[k * kTwSites + lane];
    for (int j = 1; j < 4; j++) {
      const double2 y = X[(j * 9 + k) * kTwSites + lane];
      x = make_double2(x.x + y.x, x.y + y.y);
    }
    X[k * kTwSites + lane] = x;
  }
  C<double> R[2][9];
#pragma unroll
  for (int g = 0; g < 2; g++)
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const C<double> a = pr(p.u, p.stride, v, mu, g, k / 3, k % 3), b = pr(p.u, p.stride, v, mu, g + 2, k / 3, k % 3);
      R[g][k] = C<double>{a.re - b.im, a.im + b.re};
    }
  __syncthreads();
  C<double> acc{0.0, 0.0};
#pragma unroll 1
  for (int ku = 0; ku < 4; ku++) {
    C<double> E[9], A[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
      E[k] = C<double>{0.0, 0.0};
      A[k] = pr(p.u, p.stride, v, mu, ku, k / 3, k % 3);
    }
    cross_acc(E, A, X + lane, kTwSites);
    cross_acc(E, R[0], S + (ku * 2) * 9 * kTwSites + lane, kTwSites);
    cross_acc(E, R[1], S + (ku * 2 + 1) * 9 * kTwSites + lane, kTwSites);
    // C g5 and bar C g5: entry (mu, mu ^ 1) = +1 for even mu, -1 for odd; the
    // other sign for ku
    const bool neg = ((mu ^ ku) & 1) == 0;
    // a sum for each ku, then their sum: one chain of all four rounds more
    // (3.4e-16 off 113 bits in the root mean square, against 2.6e-16 and 2.9e-16
    // for the written-out sum) and takes 0.6 % less time
    C<double> sum{0.0, 0.0};
#pragma unroll
    for (int k = 0; k < 9; k++) {
      C<double> d = pr(p.d, p.stride, v, mu ^ 1, ku ^ 1, k / 3, k % 3);
      if (neg) d = -d;
      sum = cmadd(E[k], d, sum);
    }
    acc = acc + sum;
  }
  __syncthreads();  // X is read no more
  X[mu * kTwSites + lane] = make_double2(acc.re, acc.im);
  __syncthreads();
  if (mu != 0 || !act) return;
  for (int j = 1; j < 4; j++) {
    const double2 y = X[j * kTwSites + lane];
    acc = acc + C<double>{y.x, y.y};
  }
  // -(i/2) and the boundary phase of the three propagator factors, exp(3 i pi t / L_t)
  double sn, cs;
  sincospi(3.0 * (double)t / (double)geo.L[0], &sn, &cs);
  acc = C<double>{0.5 * acc.im, -0.5 * acc.re} * C<double>{cs, sn};
  block[(int64_t)ti * V3 + s] = make_double2(acc.re, acc.im);
}

// the Fourier phases of momentum j, exp(-2 pi i p.(x - x_src) / L), as an x
// factor (Lx entries) and a (y, z) factor (Ly Lz entries) after it
__global__ void k_twop_phase(Geom geo, const int *mom, int nmom, int sx, int sy, int sz, double2 *ph)
{
  const int Lx = geo.L[1], Ly = geo.L[2], Lz = geo.L[3], m = Lx + Ly * Lz;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)m * nmom) return;
  const int j = (int)(i / m), k = (int)(i % m);
  double a;
  if (k < Lx) {
    a = (double)mom[3 * j] / Lx * (k - sx);
  } else {
    const int r = k - Lx;
    a = (double)mom[3 * j + 1] / Ly * (r % Ly - sy) + (double)mom[3 * j + 2] / Lz * (r / Ly - sz);
  }
  double sn, cs;
  sincospi(2.0 * a, &sn, &cs);
  ph[i] = make_double2(cs, -sn);
}

// corr[t][j] = 1/2 sum_x block(x) phase_j(x); one CTA per (t, j), sites
// summed in a fixed order: a thread sums one x over its (y, z) rows, then
// multiplies by the x factor. (One FP64 sincospi per site and momentum
// instead of the tables: 464 us at 24^3 x 48 and 7 momenta.)
constexpr int kFtThreads = 256;
__global__ void __launch_bounds__(kFtThreads) k_twop_ft(const double2 *block, Geom geo, const double2 *ph, int nmom,
                                                        double2 *corr)
{
  const int t = blockIdx.x / nmom, j = blockIdx.x % nmom;
  const int Lx = geo.L[1], rows = geo.L[2] * geo.L[3];
  const double2 *ex = ph + (int64_t)j * (Lx + rows), *eyz = ex + Lx, *b0 = block + (int64_t)t * Lx * rows;
  const int nx = Lx < kFtThreads ? Lx : kFtThreads, ny = kFtThreads / nx;
  const int tx = threadIdx.x % nx, ty = threadIdx.x / nx;
  C<double> sum{0.0, 0.0};
  if (ty < ny)
    for (int x = tx; x < Lx; x += nx) {
      // four partial sums: 58 rows in one chain round to 5.4e-16 at 24^3 sites
      // (root mean square against 113 bits), so split to 4.3e-16
      C<double> a[4];
#pragma unroll
      for (int k = 0; k < 4; k++) a[k] = C<double>{0.0, 0.0};
      for (int r0 = ty; r0 < rows; r0 += 4 * ny) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int r = r0 + k * ny;
          if (r >= rows) continue;
          const double2 b = b0[(int64_t)r * Lx + x], e = eyz[r];
          a[k] = cmadd(C<double>{b.x, b.y}, C<double>{e.x, e.y}, a[k]);
        }
      }
      sum = cmadd((a[0] + a[1]) + (a[2] + a[3]), C<double>{ex[x].x, ex[x].y}, sum);
    }
  __shared__ double sr[kFtThreads], si[kFtThreads];
  sr[threadIdx.x] = sum.re;
  si[threadIdx.x] = sum.im;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      sr[threadIdx.x] += sr[threadIdx.x + w];
      si[threadIdx.x] += si[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) corr[blockIdx.x] = make_double2(0.5 * sr[0], 0.5 * si[0]);
}

}  // namespace

bool twop_proton(const qcdgpu_field *up, const qcdgpu_field *dn, const int xsrc[4], int t0, int t1, const int *mom,
                 int nmom, double *corr)
{
  if (!up || !dn || !xsrc || !mom || !corr || nmom < 1 || t0 < 0 || t1 < t0) {
    set_error("two-point function: 12 + 12 propagator columns, 0 <= t0 <= t1, at least one momentum");
    return false;
  }
  const qcdgpu_field f0 = up[0];
  if (!f0 || t1 >= f0->L[0]) {
    set_error("two-point function: time-slices beyond the lattice");
    return false;
  }
  Props p;
  for (int k = 0; k < 12; k++) {
    if (!up[k] || !dn[k] || up[k]->prec != QCDGPU_F64 || dn[k]->prec != QCDGPU_F64 || !same_shape(up[k], f0) ||
        !same_shape(dn[k], f0)) {
      set_error("two-point function: FP64 propagator columns of one lattice");
      return false;
    }
    p.u[k] = (const double2 *)up[k]->data;
    p.d[k] = (const double2 *)dn[k]->data;
  }
  for (int i = 0; i < 4; i++)
    if (xsrc[i] < 0 || xsrc[i] >= f0->L[i]) {
      set_error("two-point function: source outside the lattice");
      return false;
    }
  p.stride = f0->stride;
  Geom geo;
  for (int i = 0; i < 4; i++) geo.L[i] = f0->L[i];
  geo.st[0] = 1;
  geo.st[1] = f0->L[0];
  geo.st[2] = f0->L[0] * f0->L[1];
  geo.st[3] = f0->L[0] * f0->L[1] * f0->L[2];
  const int nt = t1 - t0 + 1, V3 = f0->L[1] * f0->L[2] * f0->L[3];
  // block, corr, the phase tables and the momenta
  const size_t nb = (size_t)nt * V3, nc = (size_t)nt * nmom;
  const size_t np = (size_t)nmom * (f0->L[1] + (size_t)f0->L[2] * f0->L[3]);
  const size_t need = sizeof(double2) * (nb + nc + np) + sizeof(int) * 3 * (size_t)nmom;
  cudaStream_t st = stream();
  Scratch w(need);
  if (!w.data) return false;
  double2 *block = (double2 *)w.data, *dcorr = block + nb, *ph = dcorr + nc;
  int *dmom = (int *)(ph + np);
  bool ok = QG_CUDA(cudaMemcpyAsync(dmom, mom, sizeof(int) * 3 * (size_t)nmom, cudaMemcpyHostToDevice, st)) &&
            QG_CUDA(cudaFuncSetAttribute(k_twop_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTwShared));
  if (ok) {
    k_twop_phase<<<(unsigned)((np + 127) / 128), 128, 0, st>>>(geo, dmom, nmom, xsrc[1], xsrc[2], xsrc[3], ph);
    ok = QG_LAUNCHED("twop_phase");
  }
  if (ok) {
    k_twop_block<<<(unsigned)((nb + kTwSites - 1) / kTwSites), 4 * kTwSites, kTwShared, st>>>(p, geo, t0, nt, xsrc[0],
                                                                                              block);
    ok = QG_LAUNCHED("twop_block");
  }
  if (ok) {
    k_twop_ft<<<(unsigned)(nt * nmom), kFtThreads, 0, st>>>(block, geo, ph, nmom, dcorr);
    ok = QG_LAUNCHED("twop_ft") &&
         QG_CUDA(cudaMemcpyAsync(corr, dcorr, sizeof(double2) * nc, cudaMemcpyDeviceToHost, st));
  }
  return QG_CUDA(cudaStreamSynchronize(st)) && ok;
}

}  // namespace qg

extern "C" {

int qcdgpu_twop_proton(const qcdgpu_field *up, const qcdgpu_field *dn, const int xsrc[4], int t0, int t1,
                       const int *mom, int nmom, double *corr)
{
  return qg::twop_proton(up, dn, xsrc, t0, t1, mom, nmom, corr) ? 0 : 1;
}

}  // extern "C"
