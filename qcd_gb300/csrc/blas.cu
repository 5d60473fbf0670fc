// blas.cu -- BLAS-1 and reductions on device spinor fields
// (qcd_blas.c:137-492: zero, set, copy, scale, mulC, add, sub, axpy, the
// complex dot <a,b> = sum conj(a) b and the 2-norm).
//
// Kernels work one site per thread through the precision accessors, so the
// same code serves FP64, FP32 and FP16(+norm) storage. Reductions accumulate
// in double: each block reduces with warp shuffles into one partial, and a
// single block sums the partials in a fixed order, so results do not depend
// on scheduling (the reference's MPI_Allreduce becomes this second pass).
#include <string.h>

#include <complex>

#include "internal.h"

namespace qg {

using namespace qgd;

static inline unsigned grid_sites(int64_t V) { return (unsigned)((V + 127) / 128); }

// -------------------------------------------------------------- elementwise
template <int P, typename R>
__global__ void k_axpby(void *out, float *onorm, R ar, R ai, const void *x, const float *xn, R br,
                        R bi, const void *y, const float *yn, int64_t stride, int64_t V)
{
  int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  C<R> a{ar, ai}, b{br, bi}, vx[12], vy[12];
  Spinor<P, R>::load(x, xn, stride, s, vx);
  Spinor<P, R>::load(y, yn, stride, s, vy);
#pragma unroll
  for (int k = 0; k < 12; k++) vx[k] = a * vx[k] + b * vy[k];
  Spinor<P, R>::store(out, onorm, stride, s, vx);
}

// out = a x + b y with real a, b: b y + x (a = 1: exact for b = +-1) or
// b y + (a x); one or two FP64 operations per real instead of the complex
// form's six (GB300's FP64 pipe, not HBM, bounds the complex form)
template <int P, typename R>
__global__ void k_axpby_real(void *out, float *onorm, R a, const void *x, const float *xn, R b, const void *y,
                             const float *yn, int64_t stride, int64_t V)
{
  int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  C<R> vx[12], vy[12];
  Spinor<P, R>::load(x, xn, stride, s, vx);
  Spinor<P, R>::load(y, yn, stride, s, vy);
  const bool unit = a == (R)1;
#pragma unroll
  for (int k = 0; k < 12; k++) {
    const R xr = unit ? vx[k].re : a * vx[k].re, xi = unit ? vx[k].im : a * vx[k].im;
    vx[k].re = qfma(b, vy[k].re, xr);
    vx[k].im = qfma(b, vy[k].im, xi);
  }
  Spinor<P, R>::store(out, onorm, stride, s, vx);
}

// y = a x + y with real a: one fused multiply-add per real
template <int P, typename R>
__global__ void k_axpy_real(void *y, float *yn, R a, const void *x, const float *xn, int64_t stride,
                            int64_t V)
{
  int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  C<R> vx[12], vy[12];
  Spinor<P, R>::load(x, xn, stride, s, vx);
  Spinor<P, R>::load(y, yn, stride, s, vy);
#pragma unroll
  for (int k = 0; k < 12; k++) {
    vy[k].re = qfma(a, vx[k].re, vy[k].re);
    vy[k].im = qfma(a, vx[k].im, vy[k].im);
  }
  Spinor<P, R>::store(y, yn, stride, s, vy);
}

template <int P, typename R>
__global__ void k_set(void *out, float *onorm, R cr, R ci, int64_t stride, int64_t V)
{
  int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  C<R> v[12];
#pragma unroll
  for (int k = 0; k < 12; k++) v[k] = C<R>{cr, ci};
  Spinor<P, R>::store(out, onorm, stride, s, v);
}

// mode 0: g5 in ; mode 1: i g5 in
template <int P, typename R>
__global__ void k_g5(void *out, float *onorm, const void *in, const float *inorm, int mode,
                     int64_t stride, int64_t V)
{
  int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  C<R> v[12];
  Spinor<P, R>::load(in, inorm, stride, s, v);
#pragma unroll
  for (int k = 0; k < 12; k++) {
    C<R> w = mode ? mul_i(v[k]) : v[k];
    v[k] = k < 6 ? w : -w;
  }
  Spinor<P, R>::store(out, onorm, stride, s, v);
}

// --------------------------------------------------------------- reductions
__device__ __forceinline__ double warp_sum(double v)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block-level sum of (v0, v1) into partials[2*blockIdx.x + {0,1}]
__device__ __forceinline__ void block_sum2(double v0, double v1, double *partials)
{
  __shared__ double sh[2][32];
  v0 = warp_sum(v0);
  v1 = warp_sum(v1);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sh[0][w] = v0;
    sh[1][w] = v1;
  }
  __syncthreads();
  if (w == 0) {
    int nw = blockDim.x >> 5;
    v0 = l < nw ? sh[0][l] : 0.0;
    v1 = l < nw ? sh[1][l] : 0.0;
    v0 = warp_sum(v0);
    v1 = warp_sum(v1);
    if (l == 0) {
      partials[2 * blockIdx.x] = v0;
      partials[2 * blockIdx.x + 1] = v1;
    }
  }
}

// kind 0: |a|^2 ; kind 1: <a,b> ; kind 2: b = b + (ar,ai) a, then |b|^2
template <int P, typename R, int KIND>
__global__ void __launch_bounds__(256) k_reduce(const void *a, const float *an, void *b, float *bn,
                                                R ar, R ai, int64_t stride, int64_t V, double *partials)
{
  double s0 = 0, s1 = 0;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < V;
       s += (int64_t)gridDim.x * blockDim.x) {
    C<R> va[12];
    Spinor<P, R>::load(a, an, stride, s, va);
    // FP64 fields: FP64 products and sums; FP32 / FP16 fields: the site's
    // twelve terms in FP32 (their own precision), the sum over sites in FP64
    // (FP64 arithmetic per component would make these kernels FP64-pipe bound)
    constexpr bool F = sizeof(R) == 4;
    if (KIND == 0) {
      if (F) {
        R t = (R)0;
#pragma unroll
        for (int k = 0; k < 12; k++) t += va[k].re * va[k].re + va[k].im * va[k].im;
        s0 += (double)t;
      } else {
#pragma unroll
        for (int k = 0; k < 12; k++) s0 += (double)va[k].re * va[k].re + (double)va[k].im * va[k].im;
      }
    } else if (KIND == 1) {
      C<R> vb[12];
      Spinor<P, R>::load(b, bn, stride, s, vb);
      if (F) {
        R t0 = (R)0, t1 = (R)0;
#pragma unroll
        for (int k = 0; k < 12; k++) {
          t0 += va[k].re * vb[k].re + va[k].im * vb[k].im;
          t1 += va[k].re * vb[k].im - va[k].im * vb[k].re;
        }
        s0 += (double)t0;
        s1 += (double)t1;
      } else {
#pragma unroll
        for (int k = 0; k < 12; k++) {
          s0 += (double)va[k].re * vb[k].re + (double)va[k].im * vb[k].im;
          s1 += (double)va[k].re * vb[k].im - (double)va[k].im * vb[k].re;
        }
      }
    } else {
      C<R> vb[12], c{ar, ai};
      Spinor<P, R>::load(b, bn, stride, s, vb);
      R t = (R)0;
#pragma unroll
      for (int k = 0; k < 12; k++) {
        vb[k] = vb[k] + c * va[k];
        if (F) t += vb[k].re * vb[k].re + vb[k].im * vb[k].im;
        else s0 += (double)vb[k].re * vb[k].re + (double)vb[k].im * vb[k].im;
      }
      if (F) s0 += (double)t;
      Spinor<P, R>::store(b, bn, stride, s, vb);
    }
  }
  block_sum2(s0, s1, partials);
}

// one block: res[0..1] = sum of n partial pairs, in index order per lane
__global__ void k_finalize(const double *partials, int n, double *res)
{
  double v0 = 0, v1 = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    v0 += partials[2 * i];
    v1 += partials[2 * i + 1];
  }
  __shared__ double sh[2][32];
  v0 = warp_sum(v0);
  v1 = warp_sum(v1);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sh[0][w] = v0;
    sh[1][w] = v1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0, b = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
      a += sh[0][i];
      b += sh[1][i];
    }
    res[0] = a;
    res[1] = b;
  }
}

static int reduce_blocks(int64_t V)
{
  int64_t n = (V + 255) / 256;
  return (int)(n < kMaxPartials ? n : kMaxPartials);
}

// --------------------------------------------------------------- dispatch
#define QG_DISPATCH(prec, F64CALL, F32CALL, F16CALL) \
  do {                                               \
    if ((prec) == QCDGPU_F64) { F64CALL; }           \
    else if ((prec) == QCDGPU_F32) { F32CALL; }      \
    else { F16CALL; }                                \
  } while (0)

bool blas_zero(qcdgpu_field x) { return QG_CUDA(cudaMemsetAsync(x->data, 0, x->bytes, stream())); }

bool blas_copy(qcdgpu_field d, qcdgpu_field s)
{
  if (!same_shape(d, s) || d->prec != s->prec) {
    set_error("copy: fields differ in shape or precision");
    return false;
  }
  if (d == s) return true;
  return QG_CUDA(cudaMemcpyAsync(d->data, s->data, d->bytes, cudaMemcpyDeviceToDevice, stream()));
}

bool blas_axpby(qcdgpu_field out, double ar, double ai, qcdgpu_field x, double br, double bi, qcdgpu_field y)
{
  if (!same_shape(out, x) || !same_shape(out, y) || out->prec != x->prec || out->prec != y->prec) {
    set_error("axpby: fields differ in shape or precision");
    return false;
  }
  unsigned g = grid_sites(out->V);
  cudaStream_t st = stream();
  if (ai == 0.0 && br == 1.0 && bi == 0.0 && out == y) {
    QG_DISPATCH(out->prec,
                (k_axpy_real<QCDGPU_F64, double><<<g, 128, 0, st>>>(y->data, y->norm, ar, x->data, x->norm, out->stride, out->V)),
                (k_axpy_real<QCDGPU_F32, float><<<g, 128, 0, st>>>(y->data, y->norm, (float)ar, x->data, x->norm, out->stride, out->V)),
                (k_axpy_real<QCDGPU_F16, float><<<g, 128, 0, st>>>(y->data, y->norm, (float)ar, x->data, x->norm, out->stride, out->V)));
    return QG_LAUNCHED("axpy_real");
  }
  if (ai == 0.0 && bi == 0.0) {
    QG_DISPATCH(out->prec,
                (k_axpby_real<QCDGPU_F64, double><<<g, 128, 0, st>>>(out->data, out->norm, ar, x->data, x->norm, br, y->data, y->norm, out->stride, out->V)),
                (k_axpby_real<QCDGPU_F32, float><<<g, 128, 0, st>>>(out->data, out->norm, (float)ar, x->data, x->norm, (float)br, y->data, y->norm, out->stride, out->V)),
                (k_axpby_real<QCDGPU_F16, float><<<g, 128, 0, st>>>(out->data, out->norm, (float)ar, x->data, x->norm, (float)br, y->data, y->norm, out->stride, out->V)));
    return QG_LAUNCHED("axpby_real");
  }
  QG_DISPATCH(out->prec,
              (k_axpby<QCDGPU_F64, double><<<g, 128, 0, st>>>(out->data, out->norm, ar, ai, x->data, x->norm, br, bi, y->data, y->norm, out->stride, out->V)),
              (k_axpby<QCDGPU_F32, float><<<g, 128, 0, st>>>(out->data, out->norm, (float)ar, (float)ai, x->data, x->norm, (float)br, (float)bi, y->data, y->norm, out->stride, out->V)),
              (k_axpby<QCDGPU_F16, float><<<g, 128, 0, st>>>(out->data, out->norm, (float)ar, (float)ai, x->data, x->norm, (float)br, (float)bi, y->data, y->norm, out->stride, out->V)));
  return QG_LAUNCHED("axpby");
}

bool blas_set(qcdgpu_field x, double cr, double ci)
{
  unsigned g = grid_sites(x->V);
  cudaStream_t st = stream();
  QG_DISPATCH(x->prec,
              (k_set<QCDGPU_F64, double><<<g, 128, 0, st>>>(x->data, x->norm, cr, ci, x->stride, x->V)),
              (k_set<QCDGPU_F32, float><<<g, 128, 0, st>>>(x->data, x->norm, (float)cr, (float)ci, x->stride, x->V)),
              (k_set<QCDGPU_F16, float><<<g, 128, 0, st>>>(x->data, x->norm, (float)cr, (float)ci, x->stride, x->V)));
  return QG_LAUNCHED("set");
}

static bool g5_common(qcdgpu_field out, qcdgpu_field in, int mode)
{
  if (!same_shape(out, in) || out->prec != in->prec) {
    set_error("gamma5: fields differ in shape or precision");
    return false;
  }
  unsigned g = grid_sites(out->V);
  cudaStream_t st = stream();
  QG_DISPATCH(out->prec,
              (k_g5<QCDGPU_F64, double><<<g, 128, 0, st>>>(out->data, out->norm, in->data, in->norm, mode, out->stride, out->V)),
              (k_g5<QCDGPU_F32, float><<<g, 128, 0, st>>>(out->data, out->norm, in->data, in->norm, mode, out->stride, out->V)),
              (k_g5<QCDGPU_F16, float><<<g, 128, 0, st>>>(out->data, out->norm, in->data, in->norm, mode, out->stride, out->V)));
  return QG_LAUNCHED("gamma5");
}
bool blas_gamma5(qcdgpu_field out, qcdgpu_field in) { return g5_common(out, in, 0); }
bool blas_ig5(qcdgpu_field out, qcdgpu_field in) { return g5_common(out, in, 1); }

template <int KIND>
static bool reduce_common(qcdgpu_field a, qcdgpu_field b, double ar, double ai, double *res)
{
  double *part = reduce_scratch();
  if (!part) return false;
  int nb = reduce_blocks(a->V);
  cudaStream_t st = stream();
  const void *bd = b ? b->data : nullptr;
  float *bn = b ? b->norm : nullptr;
  QG_DISPATCH(a->prec,
              (k_reduce<QCDGPU_F64, double, KIND><<<nb, 256, 0, st>>>(a->data, a->norm, (void *)bd, bn, ar, ai, a->stride, a->V, part)),
              (k_reduce<QCDGPU_F32, float, KIND><<<nb, 256, 0, st>>>(a->data, a->norm, (void *)bd, bn, (float)ar, (float)ai, a->stride, a->V, part)),
              (k_reduce<QCDGPU_F16, float, KIND><<<nb, 256, 0, st>>>(a->data, a->norm, (void *)bd, bn, (float)ar, (float)ai, a->stride, a->V, part)));
  if (!QG_LAUNCHED("reduce")) return false;
  k_finalize<<<1, 256, 0, st>>>(part, nb, res);
  return QG_LAUNCHED("reduce_finalize");
}

bool blas_norm2_dev(qcdgpu_field x, double *res) { return reduce_common<0>(x, nullptr, 0, 0, res); }

bool blas_dot_dev(qcdgpu_field a, qcdgpu_field b, double *res)
{
  if (!same_shape(a, b) || a->prec != b->prec) {
    set_error("dot: fields differ in shape or precision");
    return false;
  }
  return reduce_common<1>(a, b, 0, 0, res);
}

bool blas_axpy_norm2_dev(qcdgpu_field y, double ar, double ai, qcdgpu_field x, double *res)
{
  if (!same_shape(x, y) || x->prec != y->prec) {
    set_error("axpy_norm: fields differ in shape or precision");
    return false;
  }
  return reduce_common<2>(x, y, ar, ai, res);
}

static bool fetch(double *dev_res, double *out, int n)
{
  double *h = host_result();
  if (!h) return false;
  if (!QG_CUDA(cudaMemcpyAsync(h, dev_res, sizeof(double) * n, cudaMemcpyDeviceToHost, stream()))) return false;
  if (!QG_CUDA(cudaStreamSynchronize(stream()))) return false;
  memcpy(out, h, sizeof(double) * n);
  return true;
}

bool blas_norm2(qcdgpu_field x, double *out)
{
  double *r = reduce_scratch();
  if (!r) return false;
  r += 2 * kMaxPartials;
  return blas_norm2_dev(x, r) && fetch(r, out, 1);
}

bool blas_dot(qcdgpu_field a, qcdgpu_field b, double out[2])
{
  double *r = reduce_scratch();
  if (!r) return false;
  r += 2 * kMaxPartials;
  return blas_dot_dev(a, b, r) && fetch(r, out, 2);
}


// ------------------------------------------------ Gram-Schmidt steps
// The Gram-Schmidt step of GCR: k dot products against one field and one
// field plus k scaled fields, in passes of up to kMulti fields (FP64 fields
// of one shape, taken as flat arrays of 12 x stride complex numbers whose
// padding sites are passed over: a coefficient that is not a number would make
// NaNs of their zeros). The scalars stay on the device: a pass of dots leaves
// the coefficients that the update pass reads, and the last update pass sums
// the norm and the dot with the source of the field it writes, so no step
// waits for the host. Block partial sums are added in a fixed order by the
// block that finishes last, so the results are deterministic.
//
// FP64 arithmetic bounds both passes (four multiply-adds per complex element
// and field: 80 us for 8 fields at 16^3 x 32, against 34 us for their bytes).
// Two resident blocks per SM share the elements evenly, and the warps' sums
// are reduced by halves (16 adds for 16 values instead of 80): with 1,024
// blocks and a shuffle tree per value a pass of dots took 132 us there, now
// 96; an update pass 104 us, now 87.
constexpr int kMulti = 8, kMultiThreads = 256, kMultiBlocks = 304;

struct MultiPtr {
  const double2 *p[kMulti];
};

// A thread's elements i of the 12 blocks of `stride` sites, gridDim.x *
// kMultiThreads apart, with the site x within the block beside them (no
// division in the loop)
struct MultiIter {
  int64_t i, n;
  unsigned x, stride, V, step;
  __device__ __forceinline__ MultiIter(int64_t V_, int64_t stride_)
      : i((int64_t)blockIdx.x * kMultiThreads + threadIdx.x), n(12 * stride_), stride((unsigned)stride_), V((unsigned)V_)
  {
    x = (unsigned)i % stride;
    step = gridDim.x * kMultiThreads % stride;
  }
  __device__ __forceinline__ bool site() const { return x < V; }
  __device__ __forceinline__ void next()
  {
    i += (int64_t)gridDim.x * kMultiThreads;
    x += step;
    if (x >= stride) x -= stride;
  }
};

// v[0 .. W-1] summed over the warp: lane l returns the sum of entry l >> (5 - log2 W)
template <int W>
__device__ __forceinline__ double warp_sums(double *v)
{
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int w = W / 2; w >= 1; w /= 2, o /= 2) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < w; i++) {
      const double keep = up ? v[i + w] : v[i], send = up ? v[i] : v[i + w];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  for (; o >= 1; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// the block's sums of W values per thread to part[blockIdx.x * 16 + entry]; in
// the block that finishes last, total[0 .. W-1] (shared) of all blocks and
// true. done is zero between launches.
template <int W>
__device__ __forceinline__ bool multi_total(double *v, double *part, unsigned *done, double *total)
{
  constexpr int S = W == 16 ? 1 : W == 8 ? 2 : W == 4 ? 3 : 4;  // 5 - log2 W
  __shared__ double sh[kMultiThreads / 16][16];
  __shared__ unsigned last;
  const int tid = threadIdx.x, lane = tid & 31;
  const double t = warp_sums<W>(v);
  if ((lane & ((1 << S) - 1)) == 0) sh[tid >> 5][lane >> S] = t;
  __syncthreads();
  if (tid < W) {
    double s = 0.0;
    for (int k = 0; k < kMultiThreads / 32; k++) s += sh[k][tid];
    part[(int64_t)blockIdx.x * 16 + tid] = s;
  }
  __threadfence();  // the block's partials before its count
  __syncthreads();
  if (tid == 0) last = atomicAdd(done, 1u) == gridDim.x - 1 ? 1u : 0u;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  const int col = tid & 15, row = tid >> 4;
  double s = 0.0;
  if (col < W)
    for (int b = row; b < (int)gridDim.x; b += kMultiThreads / 16) s += __ldcg(part + (int64_t)b * 16 + col);
  sh[row][col] = s;
  __syncthreads();
  if (tid < W) {
    double r = 0.0;
    for (int k = 0; k < kMultiThreads / 16; k++) r += sh[k][tid];
    total[tid] = r;
  }
  if (tid == 0) *done = 0u;
  __syncthreads();
  return true;
}

// dots[j] = <x_j, y> and coef[j] = -dots[j] inv2[j]
template <int J>
__global__ void __launch_bounds__(kMultiThreads, 2) k_multi_dot(MultiPtr x, const double2 *y, int64_t V, int64_t stride,
                                                                double *part, unsigned *done, double2 *dots,
                                                                const double *inv2, double2 *coef)
{
  constexpr int W = J > 4 ? 16 : J > 2 ? 8 : J > 1 ? 4 : 2;
  double v[W];
#pragma unroll
  for (int j = 0; j < W; j++) v[j] = 0.0;
  for (MultiIter it(V, stride); it.i < it.n; it.next()) {
    const bool in = it.site();  // selected loads, no branch: a jump over the body costs 0.6 % of a GCR(32)
    const double2 zero = make_double2(0.0, 0.0), b = in ? y[it.i] : zero;
#pragma unroll
    for (int j = 0; j < J; j++) {
      const double2 a = in ? x.p[j][it.i] : zero;  // conj(a) b
      v[2 * j] = fma(a.x, b.x, fma(a.y, b.y, v[2 * j]));
      v[2 * j + 1] = fma(a.x, b.y, fma(-a.y, b.x, v[2 * j + 1]));
    }
  }
  __shared__ double total[16];
  if (!multi_total<W>(v, part, done, total)) return;
  if (threadIdx.x < J) {
    const int j = threadIdx.x;
    dots[j] = make_double2(total[2 * j], total[2 * j + 1]);
    coef[j] = make_double2(-total[2 * j] * inv2[j], -total[2 * j + 1] * inv2[j]);
  }
}

// y += sum_j coef[j] x_j; SUMS: also the sums of the updated y
template <int J, bool SUMS>
__global__ void __launch_bounds__(kMultiThreads, 2) k_multi_axpy(MultiPtr x, const double2 *coef, double2 *y, int64_t V,
                                                                 int64_t stride, const double2 *src, double *part,
                                                                 unsigned *done, double *inv2, GsSums *sums)
{
  double2 c[J > 0 ? J : 1];
#pragma unroll
  for (int j = 0; j < J; j++) c[j] = coef[j];
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (MultiIter it(V, stride); it.i < it.n; it.next()) {
    if (!it.site()) continue;
    double2 v = y[it.i];
#pragma unroll
    for (int j = 0; j < J; j++) {
      const double2 b = x.p[j][it.i];
      v.x = fma(c[j].x, b.x, fma(-c[j].y, b.y, v.x));
      v.y = fma(c[j].x, b.y, fma(c[j].y, b.x, v.y));
    }
    if (J > 0) y[it.i] = v;
    if (SUMS) {
      const double2 b = src[it.i];
      s[0] = fma(v.x, v.x, fma(v.y, v.y, s[0]));
      s[1] = fma(v.x, b.x, fma(v.y, b.y, s[1]));
      s[2] = fma(v.x, b.y, fma(-v.y, b.x, s[2]));
    }
  }
  if (!SUMS) return;
  __shared__ double total[16];
  if (!multi_total<4>(s, part, done, total)) return;
  if (threadIdx.x == 0) {
    const double r = 1.0 / total[0];
    *inv2 = r;
    sums->n2 = total[0];
    sums->inv2 = r;
    sums->dot = make_double2(total[1], total[2]);
    sums->step = make_double2(-total[1] * r, -total[2] * r);
  }
}

// out = y + *c x, component blockIdx.y
__global__ void __launch_bounds__(kMultiThreads) k_axpy_dev(double2 *out, const double2 *c, const double2 *x,
                                                            const double2 *y, int64_t V, int64_t stride)
{
  const int64_t s = (int64_t)blockIdx.x * kMultiThreads + threadIdx.x;
  if (s >= V) return;
  const int64_t i = blockIdx.y * stride + s;
  const double2 a = *c, b = x[i], v = y[i];
  out[i] = make_double2(fma(a.x, b.x, fma(-a.y, b.y, v.x)), fma(a.x, b.y, fma(a.y, b.x, v.y)));
}

static unsigned multi_blocks(int64_t n)
{
  const int64_t b = (n + kMultiThreads - 1) / kMultiThreads;
  return (unsigned)(b < kMultiBlocks ? b : kMultiBlocks);
}

static bool multi_shapes(const char *what, const qcdgpu_field *x, int k, qcdgpu_field y)
{
  bool ok = y->prec == QCDGPU_F64;
  for (int j = 0; j < k; j++) ok = ok && same_shape(x[j], y) && x[j]->prec == QCDGPU_F64;
  if (!ok) set_error("%s: FP64 fields of one shape", what);
  return ok;
}

// scratch of the passes: block partials, then the counter
constexpr int64_t kGsPart = 16 * kMultiBlocks;
int64_t gs_scratch_doubles() { return kGsPart + 2; }
bool gs_init(double *scratch) { return QG_CUDA(cudaMemsetAsync(scratch + kGsPart, 0, 2 * sizeof(double), stream())); }

bool gs_dots(const qcdgpu_field *x, int k, qcdgpu_field y, double *scratch, double2 *dots, const double *inv2,
             double2 *coef)
{
  if (!multi_shapes("multi-dot", x, k, y)) return false;
  const unsigned nb = multi_blocks(12 * y->stride);
  const double2 *yy = (const double2 *)y->data;
  unsigned *done = (unsigned *)(scratch + kGsPart);
  cudaStream_t st = stream();
  for (int j0 = 0; j0 < k; j0 += kMulti) {
    MultiPtr mp{};
    const int J = k - j0 < kMulti ? k - j0 : kMulti;
    for (int j = 0; j < J; j++) mp.p[j] = (const double2 *)x[j0 + j]->data;
#define QG_DOTS(J)                                                                                                   \
  case J:                                                                                                            \
    k_multi_dot<J><<<nb, kMultiThreads, 0, st>>>(mp, yy, y->V, y->stride, scratch, done, dots + j0, inv2 + j0, coef + j0); \
    break;
    switch (J) {
      QG_DOTS(1) QG_DOTS(2) QG_DOTS(3) QG_DOTS(4) QG_DOTS(5) QG_DOTS(6) QG_DOTS(7) QG_DOTS(8)
    }
#undef QG_DOTS
    if (!QG_LAUNCHED("multi_dot")) return false;
  }
  return true;
}

bool gs_update(qcdgpu_field y, const qcdgpu_field *x, const double2 *coef, int k, qcdgpu_field src, double *scratch,
               double *inv2, GsSums *sums)
{
  if (!multi_shapes("multi-axpy", x, k, y) || (src && !multi_shapes("multi-axpy", &src, 1, y))) return false;
  const unsigned nb = multi_blocks(12 * y->stride);
  double2 *yy = (double2 *)y->data;
  const double2 *ss = src ? (const double2 *)src->data : nullptr;
  unsigned *done = (unsigned *)(scratch + kGsPart);
  cudaStream_t st = stream();
  for (int j0 = 0; j0 < k || (j0 == 0 && src); j0 += kMulti) {
    MultiPtr mp{};
    const int J = k - j0 < kMulti ? k - j0 : kMulti;
    const bool last = src && j0 + J == k;
    for (int j = 0; j < J; j++) mp.p[j] = (const double2 *)x[j0 + j]->data;
#define QG_AXPY(J)                                                                                               \
  case J:                                                                                                        \
    if (last)                                                                                                    \
      k_multi_axpy<J, true><<<nb, kMultiThreads, 0, st>>>(mp, coef + j0, yy, y->V, y->stride, ss, scratch, done, \
                                                          inv2, sums);                                           \
    else                                                                                                         \
      k_multi_axpy<J, false><<<nb, kMultiThreads, 0, st>>>(mp, coef + j0, yy, y->V, y->stride, ss, scratch, done, \
                                                           inv2, sums);                                          \
    break;
    switch (J) {
      QG_AXPY(0) QG_AXPY(1) QG_AXPY(2) QG_AXPY(3) QG_AXPY(4) QG_AXPY(5) QG_AXPY(6) QG_AXPY(7) QG_AXPY(8)
    }
#undef QG_AXPY
    if (!QG_LAUNCHED("multi_axpy")) return false;
  }
  return true;
}

bool blas_axpy_dev(qcdgpu_field out, const double2 *c, qcdgpu_field x, qcdgpu_field y)
{
  if (!multi_shapes("axpy", &x, 1, y) || !same_shape(out, y) || out->prec != QCDGPU_F64) return false;
  const dim3 nb((unsigned)((y->V + kMultiThreads - 1) / kMultiThreads), 12);
  k_axpy_dev<<<nb, kMultiThreads, 0, stream()>>>((double2 *)out->data, c, (const double2 *)x->data,
                                                 (const double2 *)y->data, y->V, y->stride);
  return QG_LAUNCHED("axpy_dev");
}

}  // namespace qg

extern "C" {

int qcdgpu_axpy(qcdgpu_field out, double are, double aim, qcdgpu_field x, qcdgpu_field y)
{
  return qg::blas_axpby(out, are, aim, x, 1.0, 0.0, y) ? 0 : 1;
}

int qcdgpu_norm2(qcdgpu_field x, double *result) { return qg::blas_norm2(x, result) ? 0 : 1; }

int qcdgpu_dot(qcdgpu_field a, qcdgpu_field b, double result[2]) { return qg::blas_dot(a, b, result) ? 0 : 1; }

}  // extern "C"
